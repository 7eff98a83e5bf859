// rs_ensemble_walk.cu — the persistent walk: many steps of a batch of FP32 runs in
// one cooperative launch (rs_ensemble.cuh).
#include "rs_ens_tile.cuh"

namespace rs {
namespace {

// The persistent walk: one cooperative launch for nsteps steps of every run.
// Per step the CTAs compute the runs' column tables (table blocks b, b + G,
// ...), meet at a grid barrier, step the tiles b, b + G, ... of the order
// with tile_body, wait for their bulk stores to complete, and meet again.  A
// run's state at step s of the launch is step + s and l = lv[s * nruns + r],
// which the host fills by the additions of inc_l that ens_advance_kernel
// makes, so every tile computes what the per-step launches compute, bit for
// bit.  The barriers are bounded: one that gives up sets *err; a CTA that
// sees *err set stops working but keeps arriving at the barriers, so the
// others do not wait out their limits.  advance: at the end (block 0, after
// the last barrier) the runs move on to step + nsteps and l = lv[nsteps *
// nruns + r].
constexpr uint32_t kWalkBarrierLimit = 1u << 22;

template <bool SURR, int SHAPE>
__global__ void __launch_bounds__(kThreads, min_ctas(SURR, shape_rows(SHAPE)))
    ens_walk_kernel(EnsRun *__restrict__ runs, const int nruns, const int32_t *__restrict__ tblk, const int ntblk,
                    const int32_t *__restrict__ order, const int ntiles, const int nsteps,
                    const double *__restrict__ lv, const int advance, unsigned *bar, int *err,
                    const uint32_t barrier_limit) {
  constexpr int TR = shape_rows(SHAPE);
  extern __shared__ __align__(128) unsigned char smem_raw[];
  TileSmemT<TR> &sm = *reinterpret_cast<TileSmemT<TR> *>(smem_raw);
  const unsigned G = gridDim.x;
  unsigned target = 0;
  bool dead = false;
  const SurrArgs none = {};
  auto l_at = [&](int r, int s) { return lv[(int64_t)s * nruns + r]; };
  for (int s = 0; s < nsteps; ++s) {
    if (!dead)
      for (int i = blockIdx.x; i < ntblk; i += G) {
        const int32_t e = tblk[i];
        const EnsRun &R = runs[e >> 16];
        if (R.active) table_block(R.K, ens_d0(R, l_at(e >> 16, s)), R.d1, R.tab_len, R.tab, e & 0xFFFF,
                                  reinterpret_cast<double *>(smem_raw));
        __syncthreads();  // the scratch is reused by the next block
      }
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // the scratch lies where tiles' loads land
    target += G;
    if (!grid_barrier(bar, target, err, barrier_limit)) dead = true;
    // tiles are handed out by a ticket counter (bar[1]): a CTA takes the next
    // tile of the order when it finishes one, so the step ends when the
    // work does, whatever the tiles cost; each CTA takes one ticket past the
    // last tile per step, so step s's tickets start at s (ntiles + G)
    const unsigned t0 = (unsigned)s * ((unsigned)ntiles + G);
    while (!dead) {
      __shared__ int tk;
      if (threadIdx.x == 0) tk = (int)(atomicAdd(bar + 1, 1u) - t0);
      __syncthreads();
      const int i = tk;
      __syncthreads();  // every thread has read the ticket
      if (i < 0 || i >= ntiles) break;  // (i < 0 only after an error left tickets untaken)
      {
        const int32_t e = order[i];
        const EnsRun &R = runs[e >> 16];
        if (!R.active) continue;  // (every thread: the run is the same)
        const int t = e & 0xFFFF;
        const int64_t step = R.step + s;
        const int par = (int)(step & 1);
        StepScalars PS;
        memset(&PS, 0, sizeof(PS));
        PS.step = step;
        PS.d0 = ens_d0(R, l_at(e >> 16, s));
        PS.d1 = R.d1;
        // L2 prefetch of this CTA's next tile of the step (as the per-step
        // launch prefetches the tile one resident wave later)
        auto prefetch = [&]() {
          const int i2 = i + (int)G;
          if (i2 >= ntiles) return;
          const int32_t e2 = order[i2];
          const EnsRun &R2 = runs[e2 >> 16];
          if (!R2.active) return;
          const int t2 = e2 & 0xFFFF, p2 = (int)((R2.step + s) & 1), n2 = R2.nrt[SHAPE];
          tma_prefetch_2d(&R2.map_psi[SHAPE][p2], kW * (t2 / n2) - 4, TR * (t2 % n2));
          tma_prefetch_2d(&R2.map_c[SHAPE][p2], kW * (t2 / n2) - 4, TR * (t2 % n2));
        };
        const int nrt = R.nrt[SHAPE];
        tile_body<SURR, TR>(R.K, R.F, PS, &R.map_psi[SHAPE][par], &R.map_c[SHAPE][par], R.tab, R.tab_len,
                            R.psi[par ^ 1], R.c[par ^ 1], nullptr, nullptr, err, SURR ? R.surr : none, t % nrt,
                            t / nrt, prefetch);
        // what this thread wrote into the input tile (the columns beyond the
        // array; a far-melt or solid tile ends without the fence of the bulk
        // stores) comes before the next tile's load into the same memory
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        __syncthreads();  // every thread is done with the tile's barrier and shared memory
        if (threadIdx.x == 0) mbar_inval(&sm.full);
        if (__syncthreads_or(*(volatile int *)err != 0)) dead = true;
      }
    }
    // the bulk stores of this step complete before the barrier releases them
    asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
    target += G;
    if (!grid_barrier(bar, target, err, barrier_limit)) dead = true;
  }
  if (advance && blockIdx.x == 0 && !dead)
    for (int r = threadIdx.x; r < nruns; r += blockDim.x)
      if (runs[r].active) {
        runs[r].l = l_at(r, nsteps);
        runs[r].step += nsteps;
      }
}

using EnsWalkFn = void (*)(EnsRun *, int, const int32_t *, int, const int32_t *, int, int, const double *, int,
                           unsigned *, int *, uint32_t);
template <bool SURR>
EnsWalkFn ens_walk_of(int shape) {
  return shape == 0   ? ens_walk_kernel<SURR, 0>
         : shape == 1 ? ens_walk_kernel<SURR, 1>
                      : ens_walk_kernel<SURR, 2>;
}

}  // namespace

int launch_ensemble_walk(EnsRun *runs, int nruns, const int32_t *tblk, int ntblk, const int32_t *order, int ntiles,
                         int shape, int nsteps, const double *lv, bool advance, bool surr, unsigned *bar, int *err,
                         uint32_t barrier_limit, cudaStream_t st) {
  if (nsteps <= 0) return 0;
  if (shape < 0 || shape >= kTileShapes) return -1;
  const EnsWalkFn kfn = surr ? ens_walk_of<true>(shape) : ens_walk_of<false>(shape);
  const size_t smem = shape == 0   ? sizeof(TileSmemT<shape_rows(0)>)
                      : shape == 1 ? sizeof(TileSmemT<shape_rows(1)>)
                                   : sizeof(TileSmemT<shape_rows(2)>);
  static_assert(sizeof(TileSmemT<8>) >= kTabBlock * sizeof(double), "table scratch fits the tile's shared memory");
  static std::atomic<unsigned long long> attr_done[2][kTileShapes];
  if (!smem_limit_once((const void *)kfn, (int)smem, attr_done[surr][shape])) return -3;
  static std::atomic<int> res_of[2][kTileShapes][64];
  const int res = resident_ctas((const void *)kfn, kThreads, smem, res_of[surr][shape]);
  if (res <= 0) return -3;
  const int grid = std::max(1, std::min(res, std::max(ntiles, ntblk)));
  if (cudaMemsetAsync(bar, 0, 2 * sizeof(unsigned), st) != cudaSuccess) return -2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)grid);
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeCooperative;
  at[0].val.cooperative = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  const int adv = advance ? 1 : 0;
  const uint32_t lim = barrier_limit ? barrier_limit : kWalkBarrierLimit;
  if (cudaLaunchKernelEx(&cfg, kfn, runs, nruns, tblk, ntblk, order, ntiles, nsteps, lv, adv, bar, err, lim) !=
      cudaSuccess)
    return -2;
  return 0;
}

}  // namespace rs
