// rs_step_f32.cu — the FP32 step on tiles: the column table, the exact kernels of
// fields with 16-byte aligned rows and the launch (rs_tile_f32.cuh).
#include "rs_tile_f32.cuh"

namespace rs {
namespace {

__global__ void __launch_bounds__(kTabBlock) column_table_kernel(const StepCoef K, const double d0, const double d1,
                                                                 const int len, float *__restrict__ tab) {
  // the tile kernel may start now; it waits for this grid before reading tab
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ double kc[kTabBlock];
  table_block(K, d0, d1, len, tab, blockIdx.x, kc);
}

}  // namespace

// Output rows of the tiles of an nx x ny FP32 step, as tile_rows_f64, in waves
// of five CTAs per SM of 16 x 128 tiles (us a step with a planar front, 4 / 8 /
// 16 rows): 256^2, 0.04 waves, 6.2 / 8.3 / 12.2; 1024^2, 0.7 waves, 8.7 / 10.7 /
// 16.0; 1280^2, 1.1 waves, 12.6 / 11.4 / 15.2; 2048 x 1536, 2.1 waves, 20.9 /
// 18.1 / 19.3 (all melt 19.1 / 16.5 / 14.6); 2048^2, 2.8 waves, 26.6 / 22.9 /
// 21.1.  The network's tiles at the front take two to three times as long:
// 1024^2 19.1 / 26.0 / 45.6; 1536^2, 1.6 waves, 29.8 / 28.0 / 41.1; 2048 x 3072,
// 4.2 waves, 67 / 47.9 / 49.5; 4096^2, 11 waves, 146 / 98 / 80.
// Tall grids, whose front tiles fill every SM by themselves, as in FP64 (planar,
// cellular front): 64 x 8000, 0.7 waves, 18.9, 18.3 / 20, 19 / 18.1, 17.0; with
// the network 67 / 53 / 50; 600 x 2300, 1 wave, network, in units of 16 rows 0.86
// / 0.78 / 1.
// And where the front's column, which i_tip_target gives, lies so near the border of
// two tile columns that both hold it: twice the front tiles, for which 16 rows with the
// late trigger are best (before the tile heights / rule without the border / now):
// 448 x 3000, front at 134, 15.0, 15.4 / 16.7, 17.2 / 14.8, 15.4, network 35.1, 48.9 /
// 41.7, 51.9 / 35.5, 49.7; 512 x 4000, front at 272, 1 / 1.07, 1.14 / 0.99, 1.00; the
// front in the middle of a column 448 x 3000, 44, 14.8 / 12.8 / 14.6, network 40.9 /
// 29.1 / 40.8: it keeps 8 rows, and so does a front near column 0, where there is no
// second tile column (448 x 3000, 16, 14.9 / 13.0 / 14.6, network 36.3 / 27.1 / 36.4).
// The network's tiles of one column fit on the device at once at 4 rows up to 16 rows
// per SM (at 8 up to 32): 192 x 3968, front at 104, 1 / 1.17 with 4 rows / 0.98 with
// 8; 384 x 3968, 40, 1 / 0.84 / 0.70.  At a border below these lines 8 rows beat 4:
// 512 x 2300, 121, 1 / 1.07 / 1.00; 192 x 2300, 134, network, 1 / 1.05 / 0.79.
// Beyond 24 rows per SM the exact step takes 16 rows wherever the front is: 448 x
// 3600, cellular front at 153, 1 / 1.14 / 1.01.  (i_front < 0: unaligned rows,
// without these lines)
int tile_rows_f32(int nx, int ny, bool tfc, bool network, int i_front) {
  if (tfc) return kTfcTR;
  const int64_t sms = sm_count(), rows = ny - 2;
  const int64_t tiles = (int64_t)((nx + kW - 1) / kW) * ((rows + 15) / 16), wave = 5 * sms;
  if (rows > (network || i_front < 0 ? 28 : 24) * sms && (network || tiles < 2 * wave)) return 16;
  const bool border = i_front >= kW - 14 && i_front < nx && (i_front + 14) % kW < 34;
  if (border && rows > (network ? 16 : 18) * sms && 2 * tiles < 5 * wave) return 16;
  if (network) {
    if (2 * tiles >= 9 * wave) return 16;
    return 2 * tiles >= 3 * wave || rows > 16 * sms || (rows > 14 * sms && (border || 20 * tiles >= 19 * wave)) ? 8 : 4;
  }
  return tiles >= 2 * wave ? 16 : tiles >= wave || (border && rows > 14 * sms) ? 8 : 4;
}
// Rows that are not 16-byte aligned: the tiles, which copy their boxes cell by
// cell, but for grids of more than a wave and a half of them (at 4 rows a tile)
// where the register kernel is the faster one with a cellular front and no noise
// (us a step, register kernel / tiles): narrow ones, 319 x 2300 13.0 / 15.2, 417 x
// 1568 12.6 / 13.5, 63 x 8000 14.2 / 20.2 (639 x 1600 16.9 / 12.8), and steps with
// a shift, whose tiles load from two places: 1279 x 700 13.1 / 15.3, 4095 x 2048
// 88 / 108 (639 x 640 11.5 / 10.5).  With the coarse-grid temperature narrow grids
// of little more than one wave: 199 x 4002 1 / 1.14, 63 x 8002 31.4 / 43.9 (255 x
// 6002, two waves, 1 / 0.95).
bool raw_on_tiles_f32(int nx, int ny, bool tfc, bool pull_back) {
  const int rows = tfc ? kTfcTR : 4;
  const int64_t tiles = (int64_t)((nx - 1 + kW - 1) / kW) * ((ny - 2 + rows - 1) / rows), wave = 5 * (int64_t)sm_count();
  const bool few = 2 * tiles <= 3 * wave;
  if (!register_grid_fits(nx)) return true;
  if (tfc) return nx > 448 || tiles <= wave || !few;
  return few || (!pull_back && nx > 432);
}

int launch_step_f32_tma(const StepCoef &K, const Coef<float> &F, const StepScalars &P, const TmaMaps &tm,
                        float *psi_n, float *c_n, float *phi_n, BlockPartial *partials, int max_partials,
                        int *nparts_out, int *err, cudaStream_t st) {
  const bool raw = P.raw != 0;
  if ((K.nx % 4 && !raw) || K.pitch != K.nx) return -1;  // rows are copied in 16-byte units
  const bool surr = tm.surr != nullptr, tfc = K.tfc != 0;
  // the coarse-grid temperature has no table kernel, surrogate or pipeline
  if (tfc && (!P.T_coarse || surr)) return -1;
  if (raw && surr) return -1;
  const bool pipe = tm.pipeline != 0 && !surr && !tfc && !P.pull_back && !raw;  // the persistent warp-role kernel (exact path)
  const int TR = tm.rows;  // the tensor maps' box is TR + 2 rows high
  if (tfc ? TR != kTfcTR : (TR != 4 && TR != 8 && TR != 16)) return -1;
  // column-major: consecutive CTAs share a column strip and its halo rows in L2
  // (raw: the tile that holds the last interior column writes the ghost column)
  const int nrt = (K.ny - 2 + TR - 1) / TR, ncb = (K.nx - raw + kW - 1) / kW;
  if (ncb > 65535 || (int64_t)nrt * ncb > (1 << 30)) return -1;
  const int nparts = nrt * ncb;
  if (partials && nparts > max_partials) return -1;
  if (tm.col_tab_len < ncb * kW + kWin) return -1;
  const int sh = TR == 4 ? 0 : TR == 8 ? 1 : 2;
  const int which = tfc ? 12 + raw : pipe ? 9 + sh : 3 * (raw ? 2 : surr) + sh;
  StepKernel32 k = {};
  ExactKernel32 x = {};  // (the forms without a surrogate argument)
  if (tfc) x = tfc_kernel_f32(raw);
  else if (pipe) x = pipe_kernel_of_f32(TR);
  else if (raw) k = raw_kernel_f32(TR);
  else if (surr) k = net_kernel_f32(TR);
  else if (TR == 4) k = {tile_kernel<false, 4, false>, sizeof(TileSmemT<4>)};
  else if (TR == 8) k = {tile_kernel<false, 8, false>, sizeof(TileSmemT<8>)};
  else k = {tile_kernel<false, 16, false>, sizeof(TileSmemT<16>)};
  const void *kfn = x.fn ? (const void *)x.fn : (const void *)k.fn;
  const size_t smem = x.fn ? x.smem : k.smem;
  const dim3 block(pipe ? kPipeThreads32 : kTileThreads32);
  static std::atomic<unsigned long long> attr_done[14];
  if (!smem_limit_once(kfn, (int)smem, attr_done[which])) return -3;
  static std::atomic<int> resident_of[14][64];
  const int resident = resident_ctas(kfn, (int)block.x, smem, resident_of[which]);
  if (resident <= 0) return -3;
  // the late trigger (rs_step_f64t.cu) where it pays: tiles of the coarse-grid
  // temperature in few waves (96 x 3002, cellular: 0.95 -> 0.80 of the 16-row
  // form), unaligned rows (1279 x 700, cellular: 13.6 -> 12.8 us; from 2.5 waves on
  // it costs: 1023 x 1024 12.6 / 13.4), the network's higher tiles (320 x 2300 at 8
  // rows: 41.9 -> 39.2), tall grids (64 x 8000 at 16 rows: 1.15 -> 1.01)
  StepScalars Q = P;
  const int64_t sms = sm_count();
  Q.late = tfc    ? nparts < 3 * (int64_t)resident
           : raw  ? 2 * (int64_t)nparts < 25 * sms
           : surr ? TR > 4 && nparts < 3 * (int64_t)resident
                  : !pipe && TR == 16 && K.ny - 2 > 18 * sms && nparts < 10 * sms;
  // every kernel of the step is a programmatic dependent of the one before it
  // in the stream (rs_step_f64t.cu)
  const float *tab = tm.col_tab;
  cudaError_t e = cudaSuccess;
  if (!tfc)
    e = launch_dep(column_table_kernel, dim3((tm.col_tab_len + kTabBlock - 2) / (kTabBlock - 1)), dim3(kTabBlock), st,
                   K, P.d0, P.d1, tm.col_tab_len, tm.col_tab);
  if (e != cudaSuccess) return -3;
  const dim3 grid(nrt, ncb);
  const int wx = resident % nrt, wy = resident / nrt;
  if (tfc) {
    e = launch_dep_smem(x.fn, grid, block, smem, st, K, F, Q, tm.psi, tm.c, tab, tm.col_tab_len, psi_n, c_n,
                        phi_n, partials, err, wx, wy);
  } else if (pipe) {
    e = launch_dep_smem(x.fn, dim3((unsigned)std::min(resident, nparts)), block, smem, st, K, F, Q, tm.psi, tm.c,
                        tab, tm.col_tab_len, psi_n, c_n, phi_n, partials, err, nrt, ncb);
  } else {
    SurrArgs sa = {};
    if (surr) sa = *tm.surr;
    e = launch_dep_smem(k.fn, grid, block, smem, st, K, F, Q, tm.psi, tm.c, tab, tm.col_tab_len, psi_n,
                        c_n, phi_n, partials, err, sa, wx, wy);
  }
  if (e != cudaSuccess) return -3;
  // the final reduction is a programmatic dependent launch after the step
  FinalRed fr = tm.red;
  fr.partials = partials;
  fr.nparts = nparts;
  if (partials && (fr.mass_out || fr.itip_out) && launch_reduce_partials_dep(fr, st)) return -3;
  if (nparts_out) *nparts_out = nparts;
  return 0;
}

}  // namespace rs
