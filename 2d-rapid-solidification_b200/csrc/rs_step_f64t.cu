// rs_step_f64t.cu — the FP64 step on tiles: the column table, the kernels of
// fields with 16-byte aligned rows and the launch (rs_tile_f64.cuh).
#include "rs_tile_f64.cuh"

namespace rs {
namespace {

// One thread per column, one exact FP64 col_terms each; K + C0 of the next
// column comes from the neighbouring thread, so blocks overlap by one column
// and write 127 entries.
constexpr int kTabBlock = 128;
__global__ void __launch_bounds__(kTabBlock) column_table_kernel_f64(const StepCoef K, const double d0,
                                                                     const double d1, const int len,
                                                                     double *__restrict__ tab) {
  // the tile kernel may start now; it waits for this grid before reading tab
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __shared__ double kc[kTabBlock];
  const int k = blockIdx.x * (kTabBlock - 1) + threadIdx.x;  // table entry; column k - 4
  const int gi = min(max(k - 4, 0), K.nx - 1);
  const double T = (d0 + d1 * gi) * K.deltaT0 + K.Tmelt;  // get_delta, fun.cu:1610-1619
  const ColEntry ct = col_entry(T, K.RR, K.cinf, K.Lref);
  kc[threadIdx.x] = ct.KC;
  __syncthreads();
  // the previous step's tiles have read the table
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (threadIdx.x == kTabBlock - 1 || k >= len) return;
  tab[kTabRT * len + k] = ct.RT;
  tab[kTabC0 * len + k] = ct.C0;
  tab[kTabDK * len + k] = kc[threadIdx.x + 1] - kc[threadIdx.x];  // (K + C0)(i+1) - (K + C0)(i)
  tab[kTabAnb * len + k] = ct.Anb;
  tab[kTabAti * len + k] = ct.Ati;
}

}  // namespace

// Output rows of the tiles of an nx x ny step.  Low tiles share the latency of
// a front tile (load, phases, stores in series, 12 to 21 us at 16 rows) among
// more CTAs; high ones load and compute fewer halo rows.  The lines are where
// they break even, in waves of five CTAs per SM of 16-row tiles (us a step with
// a planar front, 4 / 8 / 16 rows): 512^2, 0.3 waves, 13.7 / 14.1 / 18.4; 768 x
// 832, 0.8 waves, 13.8 / 12.4 / 17.5; 1024^2, 1.4 waves, 18.5 / 16.5 / 17.9;
// 1536^2, 3.1 waves, 33.7 / 23.7 / 20.3; 2048^2, 5.5 waves, 57 / 41.3 / 38.9.
// A tall grid has front tiles enough for every SM at 8 or 16 rows, and then the
// rows that a tile reads beside its own decide, and whether all tiles are resident
// at once (planar, cellular front, 4 / 8 / 16 rows): 128 x 1800, 0.3 waves, 14.2,
// 13.4 / 11.3, 10.9 / 15.8, 14.7; 352 x 1568, 0.8 waves, 15.8, 18.7 / 13.5, 18.4 /
// 16.6, 16.2; 96 x 4000, 0.7 waves, 16.1, 22.0 / 14.8, 20.1 / 18.9, 17.5; 160 x
// 3776, 0.96 waves, 24.2, 24.6 / 21.4, 21.7 / 19.3, 19.5; with a shift 28.3, 28.3 /
// 24.1, 24.4 / 21.8, 21.4.  A step with a shift gathers its tiles cell by cell, so
// their halo rows cost more: 640 x 1100, 0.9 waves, cellular, in units of the
// 16-row tile without its whole-tile forms 1.12 / 1.04 / 0.99.
// With the coarse-grid temperature a tile also sets up its temperature tables:
// 768 x 832, 28.8 / 22.5 / 30.2 us a step, so 4 rows are left out, and 16 pay from
// 1.45 waves on (in units of the 16-row tile without its polynomials, planar front
// at column 16, 8 / 16 rows): 1024^2, 1.4 waves, 0.65 / 0.74 (in a tile column's
// middle 0.80 / 0.76); 1200^2, 1.9 waves, 0.87 / 0.71; 1400 x 1600, 3 waves less a
// tile row, 1.13 / 0.86; 512 x 4002, 2.7 waves, 1.11 / 0.87.
int tile_rows_f64(int nx, int ny, bool tfc, bool pull_back) {
  const int64_t sms = sm_count(), rows = ny - 2;
  const int64_t tiles = (int64_t)((nx + kW - 1) / kW) * ((rows + 15) / 16), wave = 5 * sms;
  if (tfc) return 20 * tiles >= 29 * wave ? 16 : 8;
  if (tiles >= 3 * wave) return 16;
  if (rows > 21 * sms && tiles >= 2 * wave) return 16;
  if (2 * rows > 21 * sms && tiles < wave) return 20 * tiles >= 9 * wave ? 16 : 8;
  if (pull_back && rows > 7 * sms && 4 * tiles >= 3 * wave && tiles < wave) return 16;
  return 5 * tiles >= 4 * wave || rows > 10 * sms ? 8 : 4;
}
// Rows that are not 16-byte aligned: the tiles but for tall grids of two tile
// columns, where the second is mostly empty, or whose tiles a shift makes dear
// (95 x 4000: the register kernel 26.7 us a step with a planar front and noise,
// 17.9 with a cellular one without, 16-row tiles 20.7, 20.0; 127 x 3000 with a
// shift, cellular: 1.06 of the register kernel's time, without one 1.02, 0.71).
bool raw_on_tiles_f64(int nx, int ny, bool tfc, bool pull_back) {
  const int64_t columns = (nx - 1 + kW - 1) / kW, tiles = columns * ((ny - 2 + 15) / 16), wave = 5 * (int64_t)sm_count();
  if (!register_grid_fits(nx)) return true;
  if (columns > 65535) return false;  // (the tiles' grid: 4194240 columns)
  return tfc || columns != 2 || 20 * tiles < 9 * wave || (nx >= 104 && !pull_back);
}

int launch_step_f64_tma(const StepCoef &K, const Coef<double> &F, const StepScalars &P, const TmaMaps &tm,
                        double *psi_n, double *c_n, double *phi_n, BlockPartial *partials, int max_partials,
                        int *nparts_out, int *err, cudaStream_t st) {
  const int nj = K.ny - 2;
  const bool raw = P.raw != 0;
  if ((K.nx % 2 && !raw) || K.pitch != K.nx) return -1;  // rows are copied in 16-byte units
  // the coarse-grid temperature: per-cell groups, no column table (the
  // persistent pipeline has no TFC form and is not taken then)
  const bool tfc = K.tfc != 0;
  if (tfc && !P.T_coarse) return -1;
  const bool pipe = tm.pipeline != 0 && !tfc && !P.pull_back && !raw;
  const int TR = tm.rows;  // the tensor maps' box is TR + 2 rows high
  if (!((TR == 4 && !tfc) || TR == 8 || TR == 16)) return -1;
  // (raw: the tile that holds the last interior column writes the ghost column)
  const int nrt = (nj + TR - 1) / TR, ncb = (K.nx - raw + kW - 1) / kW;
  if (ncb > 65535 || (int64_t)nrt * ncb > (1 << 30)) return -1;
  const int nparts = nrt * ncb;
  if (partials && nparts > max_partials) return -1;
  if (!tm.col_tab64 || tm.col_tab64_len < ncb * kW + kWin) return -1;
  const int sh = TR == 4 ? 0 : TR == 8 ? 1 : 2;
  auto frozen = [&](bool own) {
    return raw       ? raw_kernel_f64(TR, own)
           : TR == 4 ? frozen_kernel<4, false>(own)
           : TR == 8 ? frozen_kernel<8, false>(own)
                     : frozen_kernel<16, false>(own);
  };
  static std::atomic<unsigned long long> attr_done[21];
  static std::atomic<int> resident_of[21][64];
  StepKernel64 k = {};
  auto resident_at = [&](int which) {
    return smem_limit_once((const void *)k.fn, (int)k.smem, attr_done[which])
               ? resident_ctas((const void *)k.fn, pipe ? kPipeThreads64 : kTileThreads64, k.smem, resident_of[which])
               : -1;
  };
  // a grid of one wave: the tiles compute their columns' entries themselves
  bool own = !tfc && !pipe;
  int resident = 0;
  if (own) {
    k = frozen(true);
    resident = resident_at(15 + 3 * raw + sh);
    own = nparts <= resident;
  }
  if (!own) {
    k = pipe  ? pipe_kernel_of_f64(TR)
        : tfc ? (raw ? tfc_raw_kernel_f64(TR) : tfc_kernel_f64(TR))
              : frozen(false);
    resident = resident_at(pipe ? 12 + sh : 6 * raw + 3 * tfc + sh);
  }
  if (resident <= 0) return -3;
  // CTAs of the next step that are scheduled while this one's last tiles are at
  // work fill the slots of SMs that have finished first, its front tiles, which
  // are launched first, several to an SM.  Where a grid has few waves that costs
  // more than the launch latency it hides: 96 x 4000 with a cellular front on
  // 16-row tiles, 22.5 us a step with the early trigger, 18.5 with the late one;
  // 768 x 832 on 8-row tiles 15.9 / 14.9; 1536^2, 3.1 waves of 16-row tiles, with
  // a planar front 20.3 / 21.0.  (4-row tiles: no difference, and the early
  // trigger lets those that compute their own columns start on them.)
  StepScalars Q = P;
  Q.late = TR > 4 && !tfc && !pipe && nparts < 15 * (int64_t)sm_count();
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  // every kernel of the step is a programmatic dependent of the one before it
  // in the stream: it is scheduled while that one drains and waits
  // (griddepcontrol.wait) before it reads or writes what the other may touch
  cudaLaunchConfig_t cfg = {};
  cfg.stream = st;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const double *tab = tm.col_tab64;
  cudaError_t e = cudaSuccess;
  if (!tfc && !own) {
    cfg.gridDim = dim3((tm.col_tab64_len + kTabBlock - 2) / (kTabBlock - 1));
    cfg.blockDim = dim3(kTabBlock);
    e = cudaLaunchKernelEx(&cfg, column_table_kernel_f64, K, P.d0, P.d1, tm.col_tab64_len, tm.col_tab64);
    if (e != cudaSuccess) return -3;
  }
  cfg.dynamicSmemBytes = k.smem;
  if (pipe) {
    // persistent: every CTA resident at once, each walking tiles b, b + G, ...
    cfg.gridDim = dim3((unsigned)std::min(resident, nparts));
    cfg.blockDim = dim3(kPipeThreads64);
    e = cudaLaunchKernelEx(&cfg, k.fn, K, F, P, tm.psi, tm.c, tab, tm.col_tab64_len, psi_n, c_n, phi_n,
                           partials, err, nrt, ncb);
  } else {
    // column-major: consecutive CTAs share a column strip and its halo rows in L2
    cfg.gridDim = dim3(nrt, ncb);
    cfg.blockDim = dim3(kTileThreads64);
    e = cudaLaunchKernelEx(&cfg, k.fn, K, F, Q, tm.psi, tm.c, tab, tm.col_tab64_len, psi_n, c_n, phi_n, partials,
                           err, resident % nrt, resident / nrt);
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
