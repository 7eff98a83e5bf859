// rs_ens_tile.cuh — the ensemble's tile kernel and what its translation units
// share (rs_ensemble.cu, rs_ensemble_net.cu, rs_ensemble_walk.cu).
#pragma once

#include "rs_ensemble.cuh"
#include "rs_tile_f32.cuh"

namespace rs {
namespace {

// d0 of the frozen temperature line, evaluated in the order rs_step uses on
// the host (no contraction), so an ensemble run matches the same run stepped
// alone bit for bit
__device__ __forceinline__ double ens_d0(const EnsRun &R, const double l) {
  double t = __dmul_rn(R.GG, __dsub_rn(l, R.l_init));
  t = __dmul_rn(t, R.S);
  t = __dmul_rn(t, R.W0);
  t = __ddiv_rn(t, R.deltaT0);
  const double k = (double)(-R.i_tip_target + R.hist - R.hist_init);
  return __dsub_rn(__dadd_rn(R.delta_initial, __dmul_rn(R.d1, k)), t);
}

// CTAs per SM the tile kernels are built for, by tile height (32-row tiles
// take 83 KB of shared memory: two per SM)
constexpr int min_ctas(bool surr, int TR) { return TR > 16 ? 2 : surr ? 4 : 5; }

template <bool SURR, int SHAPE>
__global__ void __launch_bounds__(kThreads, min_ctas(SURR, shape_rows(SHAPE)))
    ens_tile_kernel(const EnsRun *__restrict__ runs, const int32_t *__restrict__ order, int *err, const int wave) {
  constexpr int TR = shape_rows(SHAPE);
  pdl_wait();  // the runs' state
  const int32_t e = order[blockIdx.x];
  const EnsRun &R = runs[e >> 16];
  if (!R.active) return;
  const int t = e & 0xFFFF, par = (int)(R.step & 1);
  StepScalars PS;
  memset(&PS, 0, sizeof(PS));
  PS.step = R.step;
  PS.d0 = ens_d0(R, R.l);
  PS.d1 = R.d1;
  const SurrArgs none = {};
  // the tile of the block launched `wave` (CTAs resident at once) positions
  // later, looked up by the issuing thread only: it may belong to another run
  auto prefetch = [&]() {
    const int nb = (int)blockIdx.x + wave;
    if (wave <= 0 || nb >= (int)gridDim.x) return;
    const int32_t e2 = order[nb];
    const EnsRun &R2 = runs[e2 >> 16];
    if (!R2.active) return;
    const int t2 = e2 & 0xFFFF, p2 = (int)(R2.step & 1), n2 = R2.nrt[SHAPE];
    tma_prefetch_2d(&R2.map_psi[SHAPE][p2], kW * (t2 / n2) - 4, TR * (t2 % n2));
    tma_prefetch_2d(&R2.map_c[SHAPE][p2], kW * (t2 / n2) - 4, TR * (t2 % n2));
  };
  const int nrt = R.nrt[SHAPE];
  tile_body<SURR, TR>(R.K, R.F, PS, &R.map_psi[SHAPE][par], &R.map_c[SHAPE][par], R.tab, R.tab_len, R.psi[par ^ 1],
                      R.c[par ^ 1], nullptr, nullptr, err, SURR ? R.surr : none, t % nrt, t / nrt, prefetch);
}

}  // namespace

// the per-step kernel of a tile shape and the shared memory it takes
using EnsTileFn = void (*)(const EnsRun *, const int32_t *, int *, int);
struct EnsTileKernel {
  EnsTileFn fn;
  size_t smem;
};
template <bool SURR>
EnsTileKernel ens_tile_of(int shape) {
  static_assert(kTileShapes == 3, "every tile shape");
  if (shape == 0) return {ens_tile_kernel<SURR, 0>, sizeof(TileSmemT<shape_rows(0)>)};
  if (shape == 1) return {ens_tile_kernel<SURR, 1>, sizeof(TileSmemT<shape_rows(1)>)};
  return {ens_tile_kernel<SURR, 2>, sizeof(TileSmemT<shape_rows(2)>)};
}
EnsTileKernel ens_net_kernel(int shape);  // rs_ensemble_net.cu

}  // namespace rs
