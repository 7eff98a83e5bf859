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
int tile_rows_f32(int nx, int ny, bool tfc, bool network) {
  if (tfc) return kTfcTR;
  const int64_t tiles = (int64_t)((nx + kW - 1) / kW) * ((ny - 2 + 15) / 16), wave = 5 * (int64_t)sm_count();
  if (network) return 2 * tiles >= 9 * wave ? 16 : 2 * tiles >= 3 * wave ? 8 : 4;
  return tiles >= 2 * wave ? 16 : tiles >= wave ? 8 : 4;
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
    e = launch_dep_smem(x.fn, grid, block, smem, st, K, F, P, tm.psi, tm.c, tab, tm.col_tab_len, psi_n, c_n,
                        phi_n, partials, err, wx, wy);
  } else if (pipe) {
    e = launch_dep_smem(x.fn, dim3((unsigned)std::min(resident, nparts)), block, smem, st, K, F, P, tm.psi, tm.c,
                        tab, tm.col_tab_len, psi_n, c_n, phi_n, partials, err, nrt, ncb);
  } else {
    SurrArgs sa = {};
    if (surr) sa = *tm.surr;
    e = launch_dep_smem(k.fn, grid, block, smem, st, K, F, P, tm.psi, tm.c, tab, tm.col_tab_len, psi_n,
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
