// rs_step_f64t_pipe.cu — the persistent FP64 step kernel of three warp roles on
// the phases of rs_tile_f64.cuh.
#include "rs_tile_f64.cuh"

namespace rs {
namespace {

// the persistent pipeline's rings
constexpr int kRing = 3, kStage = 2;
template <int TR>
struct alignas(128) StSlot {
  typename TileOps<TR>::StArr a;
  typename TileOps<TR>::StFlags f;
};
template <int TR>
struct alignas(128) PipeSmem64 {
  typename TileOps<TR>::InSlot in[kRing];
  StSlot<TR> st[kStage];
  typename TileOps<TR>::P2Smem p2;
  uint64_t in_full[kRing], in_empty[kRing], st_full[kStage], st_empty[kStage];
  int abort;  // a wait gave up: every role stops
};
// ---------------------------------------------------------------- persistent, warp roles
constexpr int kPipeThreads = kPipeThreads64;
enum { kBarP1 = 1, kBarP2 = 2 };                 // named barriers of the two groups

// AND of a predicate over the 128 threads of a phase group (named barrier)
__device__ __forceinline__ bool group_and(bool v, int id) {
  uint32_t r;
  asm volatile(
      "{\n .reg .pred p, q;\n setp.ne.u32 p, %1, 0;\n barrier.red.and.pred q, %2, 128, p;\n"
      " selp.u32 %0, 1, 0, q;\n}\n"
      : "=r"(r)
      : "r"((uint32_t)v), "r"(id)
      : "memory");
  return r != 0;
}

// bounded wait on an mbarrier phase; gives up (error flag, abort flag) after
// the limit or when another role has given up
__device__ __forceinline__ bool pipe_wait(uint64_t *bar, uint32_t parity, volatile int *abort, uint32_t limit,
                                          int *err, bool poll) {
  uint32_t tries = 0;
  while (!mbar_try(bar, parity, poll)) {
    if (*abort) return false;
    if (++tries >= limit) {
      atomicExch(err, 1);
      *abort = 1;
      return false;
    }
  }
  return true;
}

template <int TR>
__global__ void __launch_bounds__(kPipeThreads, 2)
    pipe_kernel_f64(const __grid_constant__ StepCoef K, const __grid_constant__ Coef<double> F,
                    const __grid_constant__ StepScalars PS, const __grid_constant__ CUtensorMap tm_psi,
                    const __grid_constant__ CUtensorMap tm_c, const double *__restrict__ tab, const int tab_len,
                    double *__restrict__ psi_n, double *__restrict__ c_n, double *__restrict__ phi_n,
                    BlockPartial *partials, int *err, const int nrt, const int ncb) {
  extern __shared__ __align__(128) unsigned char smem_raw[];
  using Ops = TileOps<TR>;
  PipeSmem64<TR> &sm = *reinterpret_cast<PipeSmem64<TR> *>(smem_raw);
  const int warp = threadIdx.x >> 5;
  const int ntiles = nrt * ncb;
  const int f = max(PS.i_front, 0) / kW;
  const uint32_t limit = PS.wait_limit ? PS.wait_limit : kWaitLimit;
  const bool poll = PS.wait_limit != 0;
  volatile int *abort = &sm.abort;
  if (smem_u32(smem_raw) & 127u) {  // TMA destinations must be 128-byte aligned
    if (threadIdx.x == 0) atomicExch(err, 2);
    return;
  }
  if (threadIdx.x == 0) {
    for (int s = 0; s < kRing; ++s) {
      mbar_init(&sm.in_full[s], 1);
      mbar_init(&sm.in_empty[s], 1);
    }
    for (int s = 0; s < kStage; ++s) {
      mbar_init(&sm.st_full[s], 1);
      mbar_init(&sm.st_empty[s], 1);
    }
    sm.abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  // the column table of this step (programmatic dependency on its kernel)
  asm volatile("griddepcontrol.wait;" ::: "memory");
  // the step's final reduction (a programmatic dependent) may be scheduled now
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  __syncthreads();

  if (warp == 0) {
    // ---- producer: the input boxes of this CTA's tiles, kRing - 1 ahead of
    // phases 2-4 (a slot is refilled once its tile's bulk stores have read it)
    if ((threadIdx.x & 31) == 0) {
      int k = 0;
      for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++k) {
        const int s = k % kRing;
        if (k >= kRing && !pipe_wait(&sm.in_empty[s], ((k / kRing) - 1) & 1, abort, limit, err, poll)) break;
        int tr, tc;
        tile_of(t, nrt, ncb, f, tr, tc);
        mbar_expect_tx(&sm.in_full[s], Ops::kTileBytes);
        tma_load_2d(&sm.in[s].psi[0][0], &tm_psi, &sm.in_full[s], kW * tc - 4, TR * tr);
        tma_load_2d(&sm.in[s].c[0][0], &tm_c, &sm.in_full[s], kW * tc - 4, TR * tr);
      }
      // loads still in flight into this CTA's shared memory complete before
      // it exits (bounded)
      // (a load's slot is only refilled after its tile is done, so only the
      // last kRing loads can still be in flight)
      for (int q = max(k - kRing, 0); q < k; ++q)
        for (uint32_t tt = 0; tt < kWaitLimit && !mbar_try_wait(&sm.in_full[q % kRing], (q / kRing) & 1); ++tt) {
        }
    }
    return;
  }
  if (warp <= kWarps) {
    // ---- phase 1 of tile k into staging slot k % kStage
    const int gtid = (int)threadIdx.x - 32;
    int k = 0;
    for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++k) {
      const int s = k % kRing, q = k % kStage;
      // every thread waits (bounded); the group goes on only if all of them saw the phases
      bool ok = pipe_wait(&sm.in_full[s], (k / kRing) & 1, abort, limit, err, poll);
      if (ok && k >= kStage) ok = pipe_wait(&sm.st_empty[q], ((k / kStage) - 1) & 1, abort, limit, err, poll);
      if (!group_and(ok, kBarP1)) break;
      int tr, tc;
      tile_of(t, nrt, ncb, f, tr, tc);
      const typename Ops::TileView V(K, F, PS, tab, tab_len, kW * tc, 1 + TR * tr, gtid);
      if (gtid == 0) {
        sm.st[q].f.liq = 0u;
        sm.st[q].f.sol = 0u;
      }
      Ops::fix_beyond(V, sm.in[s]);
      gsync(kBarP1);
      Ops::template phase1<false>(V, Ops::template lane_cols<false>(V), sm.in[s], sm.st[q].a, sm.st[q].f, nullptr);
      gsync(kBarP1);
      if (gtid == 0) mbar_arrive(&sm.st_full[q]);
    }
    return;
  }
  // ---- phases 2-4 of tile k: fluxes, interface cells, stores
  const int gtid = (int)threadIdx.x - 32 - kThreads;
  int k = 0;
  for (int t = blockIdx.x; t < ntiles; t += gridDim.x, ++k) {
    const int s = k % kRing, q = k % kStage;
    if (!group_and(pipe_wait(&sm.st_full[q], (k / kStage) & 1, abort, limit, err, poll), kBarP2)) break;
    int tr, tc;
    tile_of(t, nrt, ncb, f, tr, tc);
    const typename Ops::TileView V(K, F, PS, tab, tab_len, kW * tc, 1 + TR * tr, gtid);
    BlockPartial *part = partials ? partials + ((int64_t)tc * nrt + tr) : nullptr;
    const bool red = part != nullptr;
    if (gtid == 0) sm.p2.nlist = 0u;
    gsync(kBarP2);
    double mass = 0.0;
    int itip = 0;
    double dn[Ops::kRowsPerWarp][2];
    const uint32_t needs_all = Ops::phase2(V, Ops::template lane_cols<false>(V), sm.in[s], sm.st[q].a, sm.st[q].f, sm.p2, dn, mass, red);
    gsync(kBarP2);
    Ops::template phase3<false>(V, sm.in[s], sm.p2, nullptr, sm.st[q].a.S, red, itip);  // S of the slot is free after phase 2
    gsync(kBarP2);
    Ops::phase4_rows(V, sm.in[s], sm.st[q].a.S, needs_all, dn, red, itip);
    const bool issued = Ops::store_tile(V, sm.in[s], psi_n, c_n, phi_n, kBarP2);
    Ops::finish_tile(V, sm.p2, mass, itip, part, kBarP2);
    // the slots are free once the bulk copies have read the input tile
    if (issued) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
    gsync(kBarP2);
    if (gtid == 0) {
      mbar_arrive(&sm.st_empty[q]);
      mbar_arrive(&sm.in_empty[s]);
    }
  }
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

}  // namespace

StepKernel64 pipe_kernel_of_f64(int rows) {
  if (rows == 4) return {pipe_kernel_f64<4>, sizeof(PipeSmem64<4>)};
  if (rows == 8) return {pipe_kernel_f64<8>, sizeof(PipeSmem64<8>)};
  return {pipe_kernel_f64<16>, sizeof(PipeSmem64<16>)};
}

}  // namespace rs
