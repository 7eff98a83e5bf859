// rs_kernels.cuh — launcher declarations and block-reduction helpers.
#pragma once

#include <cuda.h>

#include "rs_common.cuh"

namespace rs {

// Programmatic dependent launch: the kernel is scheduled while the one before
// it in the stream drains, and must execute pdl_wait() before it touches
// memory (its launch latency hides; the order of the stream stays).
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
// the next kernel of the stream may be scheduled (if it is such a launch)
__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
template <typename T>
struct Same {  // (the kernel's own parameter types: no deduction from the arguments)
  using type = T;
};
template <typename... Args>
cudaError_t launch_dep_smem(void (*kernel)(Args...), dim3 grid, dim3 block, size_t smem, cudaStream_t st,
                            const typename Same<Args>::type &...args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = block;
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[0].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, kernel, args...);
}
template <typename... Args>
cudaError_t launch_dep(void (*kernel)(Args...), dim3 grid, dim3 block, cudaStream_t st,
                       const typename Same<Args>::type &...args) {
  return launch_dep_smem(kernel, grid, block, 0, st, args...);
}

// Per-block partial results of a grid pass: sum of interior c (FP64) and the
// largest column with psi > 0 (the coarse tip, get_itip_all_grain fun.cu:1745).
struct BlockPartial {
  double mass;
  int32_t itip;
  int32_t pad;
};

template <int NT>
__device__ __forceinline__ void block_partial(double mass, int itip, BlockPartial *out) {
  __shared__ double s_m[NT / 32];
  __shared__ int s_i[NT / 32];
  const int tid = threadIdx.y * blockDim.x + threadIdx.x;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mass += __shfl_down_sync(0xffffffffu, mass, o);
  itip = __reduce_max_sync(0xffffffffu, itip);
  if ((tid & 31) == 0) {
    s_m[tid >> 5] = mass;
    s_i[tid >> 5] = itip;
  }
  __syncthreads();
  if (tid == 0) {
    double m = 0.0;
    int it = 0;
#pragma unroll
    for (int w = 0; w < NT / 32; ++w) {
      m += s_m[w];
      it = max(it, s_i[w]);
    }
    BlockPartial b;
    b.mass = m;
    b.itip = it;
    b.pad = 0;
    out[blockIdx.y * gridDim.x + blockIdx.x] = b;
  }
}

// Inputs of the TMA-staged FP32 kernel: descriptors of the current psi and c
// fields (built on the host) and the context's per-column table workspace.
struct SurrArgs;
// The final reduction of a launch's partials (a dependent launch).
struct FinalRed {
  const BlockPartial *partials;
  int nparts;
  double mass_offset;
  double *mass_out;
  int32_t *itip_out;
};
// It runs on one CTA of kRedThreads: slot v = 0 .. kRedThreads-1 adds partials v,
// v + kRedThreads, ... in turn (four 16-byte loads in flight), then a tree over
// each warp's slots and over the warps.  The next step waits for it, so its
// latency counts: 128 threads with a tree in shared memory took 3.5 us for
// 2048 partials.
constexpr int kRedThreads = 1024;
__device__ __forceinline__ void final_reduce(const FinalRed &FR) {
  constexpr int kB = 4;
  static_assert(sizeof(BlockPartial) == 16, "a partial is one 16-byte load");
  __shared__ double s_m[kRedThreads / 32];
  __shared__ int s_i[kRedThreads / 32];
  const int tid = threadIdx.x, n = FR.nparts;
  const double2 *P = reinterpret_cast<const double2 *>(FR.partials);
  auto itip_of = [](double2 x) { return (int)(uint32_t)(unsigned long long)__double_as_longlong(x.y); };
  double m = 0.0;
  int it = 0;
  for (int k = tid; k < n; k += kB * kRedThreads) {
    double2 x[kB];
#pragma unroll
    for (int u = 0; u < kB; ++u)
      x[u] = k + u * kRedThreads < n ? __ldcg(P + k + u * kRedThreads) : make_double2(0.0, 0.0);
#pragma unroll
    for (int u = 0; u < kB; ++u) {
      m += x[u].x;
      it = max(it, itip_of(x[u]));
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m += __shfl_down_sync(0xffffffffu, m, o);
  it = __reduce_max_sync(0xffffffffu, it);
  if ((tid & 31) == 0) {
    s_m[tid >> 5] = m;
    s_i[tid >> 5] = it;
  }
  __syncthreads();
  if (tid >= 32) return;
  m = s_m[tid];
  it = __reduce_max_sync(0xffffffffu, s_i[tid]);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) m += __shfl_down_sync(0xffffffffu, m, o);
  if (tid == 0) {
    if (FR.mass_out) *FR.mass_out = m + FR.mass_offset;
    if (FR.itip_out) *FR.itip_out = max(1, it);  // get_itip_all_grain starts at 1
  }
}

struct TmaMaps {
  CUtensorMap psi;
  CUtensorMap c;
  float *col_tab;   // kColTabFields arrays of col_tab_len floats (FP32 step)
  int col_tab_len;
  double *col_tab64;  // kColTabFields arrays of col_tab64_len doubles (FP64 step)
  int col_tab64_len;
  const SurrArgs *surr;  // learned CALPHAD surrogate, or nullptr (exact)
  FinalRed red;          // offset and outputs (partials, nparts set by the launcher)
  int pipeline;          // the persistent warp-role kernel instead of one tile per CTA
  int rows;              // output rows of a tile (the maps' boxes are two rows higher)
};
constexpr int kTileOutW = 128;                  // output columns of an FP32 tile
constexpr int kTmaBoxW32 = kTileOutW + 8;        // input columns (4 each side keep x 16-byte aligned)
constexpr int kTileOutW64 = 64;                  // output columns of an FP64 tile
constexpr int kTmaBoxW64 = kTileOutW64 + 8;      // its input columns
constexpr int kTileRows = 16;    // output rows of a tile
constexpr int kTmaBoxH = kTileRows + 2;  // input rows of a tile
int tile_rows_f64(int nx, int ny, bool tfc, bool pull_back);  // output rows of an FP64 tile: 4, 8 or 16
// and of an FP32 tile (i_front: the column of the front, < 0 on unaligned rows)
int tile_rows_f32(int nx, int ny, bool tfc, bool network, int i_front);
// whether the tile kernels take a step on rows that are not 16-byte aligned (else
// the register kernel, whose grid is 4 strips of 30 columns wide)
constexpr bool register_grid_fits(int nx) { return ((nx - 2 + 29) / 30 + 3) / 4 <= 65535; }
bool raw_on_tiles_f64(int nx, int ny, bool tfc, bool pull_back);
bool raw_on_tiles_f32(int nx, int ny, bool tfc, bool pull_back);
constexpr int kTfcTileRows32 = 8;        // output rows of an FP32 coarse-grid-temperature tile
constexpr int kColTabFields = 5;
// length of the per-column table (entry k is column k - 4) for nx_all columns
inline int col_tab_len(int nx_all) { return ((nx_all + kTileOutW - 1) / kTileOutW) * kTileOutW + kTmaBoxW32; }
inline int col_tab64_len(int nx_all) {
  return ((nx_all + kTileOutW64 - 1) / kTileOutW64) * kTileOutW64 + kTmaBoxW64;
}

// ---- launchers (return 0, or -1 when a size limit is exceeded)
int launch_step_f64(const StepCoef &K, const StepScalars &P, const double *psi, const double *c,
                    double *psi_n, double *c_n, double *phi_n, BlockPartial *partials,
                    int max_partials, int *nblocks_out, const TmaMaps *tm, int *err, cudaStream_t st);
int launch_step_f32(const StepCoef &K, const StepScalars &P, const float *psi, const float *c,
                    float *psi_n, float *c_n, float *phi_n, BlockPartial *partials, int max_partials,
                    int *nblocks_out, const TmaMaps *tm, int *err, cudaStream_t st);
template <typename R>
struct Coef;
// FP32 TMA-staged kernels (rs_tile_f32.cuh): the frozen and the coarse-grid
// temperature, with or without a fused pull-back, the fields by TMA or, of rows
// that TMA cannot address, element by element.  Launches the per-column table
// kernel (frozen temperature) and the tile kernel; nparts_out gets the number of
// partials written.
int launch_step_f32_tma(const StepCoef &K, const Coef<float> &F, const StepScalars &P, const TmaMaps &tm,
                        float *psi_n, float *c_n, float *phi_n, BlockPartial *partials, int max_partials,
                        int *nparts_out, int *err, cudaStream_t st);
// FP64 TMA-staged kernels (rs_tile_f64.cuh), the same calls.  (Frozen
// temperature, a grid of one wave of CTAs: no table kernel.)
int launch_step_f64_tma(const StepCoef &K, const Coef<double> &F, const StepScalars &P, const TmaMaps &tm,
                        double *psi_n, double *c_n, double *phi_n, BlockPartial *partials, int max_partials,
                        int *nparts_out, int *err, cudaStream_t st);
// The final reduction of FR as a programmatic dependent of
// the kernel just launched on st, which wrote the partials: it is scheduled
// while that kernel runs and waits for its completion on the device
// (griddepcontrol.wait), so no host-side launch gap follows the step.  (A
// kernel that does not execute griddepcontrol.launch_dependents lets it start
// when it ends.)
int launch_reduce_partials_dep(const FinalRed &FR, cudaStream_t st);

// frame / reductions / tip (rs_frame.cu); precision 0 = double, 1 = float
void launch_pull_back(int precision, const StepCoef &K, const void *c, const void *psi,
                      const void *phi, void *c_n, void *psi_n, void *phi_n, int i_offset,
                      cudaStream_t st);
int launch_itip_partials(int precision, const StepCoef &K, const void *psi, BlockPartial *partials, int max_partials,
                         int *nblocks_out, cudaStream_t st);
int launch_mass_partials(int precision, const StepCoef &K, const void *c, double c_offset, BlockPartial *partials,
                         int max_partials, int *nblocks_out, cudaStream_t st);
int launch_precise_tip(int precision, const StepCoef &K, const void *psi, int *row_last, double *row_f, double *row_g,
                       rs_tip *out, cudaStream_t st);

// initial conditions and coarse temperature (rs_init.cu)
void launch_initial_reference(int precision, const StepCoef &K, int i_tip_target, void *c,
                              void *psi, void *phi, cudaStream_t st);
void launch_initial_planar(int precision, const StepCoef &K, int i_tip_target, double c_liquid,
                           double c_solid, uint64_t seed, void *c, void *psi, void *phi,
                           cudaStream_t st);

struct TfcCoef {
  int32_t nx, ny, pitch, ratio;
  int32_t NxT, NyT, NxT_all, NyT_all;
  int32_t jTmin, jTmax;
  int32_t ratio_dt_dtT, Sint;
  double Tcold, Thot, dx, dxT, dtT, W0, GG, S;
  double diff;    // DT / (Gamma muk0 dxT^2)
  double source;  // Lcp / (ratio_dt_dtT ratio^2)
};
void launch_temperature_init(const TfcCoef &T, double *d_T, cudaStream_t st);
// adv = Vp_ramp(step tau0 dt) tau0 / (S W0), per step (fun.cu:1563)
int launch_temperature_substep(const TfcCoef &T, const double *Tin, double *Tout, const double *dphidt, double adv,
                               cudaStream_t st);
int launch_temperature_copy(const TfcCoef &T, const double *src, double *dst, cudaStream_t st);
void launch_interpolate_temperature(const TfcCoef &T, const StepCoef &K, const double *d_T,
                                    double *d_T_fine, int i_left_end, cudaStream_t st);
int launch_integrate_phi(int precision, const TfcCoef &T, const void *psi, const void *psi_n, double *dphidt,
                         int i_left_end, int i_offset, cudaStream_t st);

// records a message for rs_last_error() and returns code (rs_capi.cu)
int set_error(int code, const char *msg);

}  // namespace rs
