// rs_mlp.cu — the learned stand-in for the per-cell CALPHAD evaluation:
// training data from the exact evaluator, forward/backward and Adam kernels.
//
// Network: (T, c, phi) -> (mu'', dG), 3 -> 32 -> 32 -> 2, SiLU, inputs scaled
// to [-1, 1] over the training box, outputs scaled by the box's
// mean/scale.  mu'' is the chemical potential relative to the melt's column
// value used by the FP32 tile kernel (rs_tile_f32.cuh),
//   mu'' = -(g+1) C0(T) - delta (L0_BCC + L0_Liq + g (L0_BCC - L0_Liq)) + RT lam(c),
// and dG = Gl - Gs = (1-c) A_Nb + c A_Ti + c (1-c) (L0_Liq - L0_BCC)
// (fun.cu:1671-1720 regrouped, rs_common.cuh).  Targets are evaluated in FP64
// with the same device functions as the exact kernels.
//
// Parameters are one flat FP32 vector (RS_MLP_NPARAMS):
//   W1[32][3], b1[32], W2[32][32], b2[32], W3[2][32], b3[2]   (row = output unit)
#include <cooperative_groups.h>

#include "rs_mlp.cuh"

namespace cg = cooperative_groups;

namespace rs {
namespace {

constexpr int kGradThreads = 256;

// g: the interpolation weight, gg(phi) for the 2D model, 2 gS - 1 for the 3D one
__device__ __forceinline__ double mu2_exact(double T, double c, double g, double cinf, double RR) {
  const TTerms tt = t_terms(T, RR);
  const double D = 0.5 * (tt.dGs - tt.dGl);
  const double C0 = -D - 0.5 * (kL0Bcc - kL0Liq) * (1.0 - 2.0 * cinf);
  const double lam = log(c / (1.0 - c)) - log(cinf / (1.0 - cinf));
  return -(g + 1.0) * C0 - (c - cinf) * ((kL0Bcc + kL0Liq) + g * (kL0Bcc - kL0Liq)) + tt.RT * lam;
}

__device__ __forceinline__ double dG_exact(double T, double c, double RR) {
  const TTerms tt = t_terms(T, RR);
  return (1.0 - c) * tt.A_nb + c * tt.A_ti + c * (1.0 - c) * (kL0Liq - kL0Bcc);
}

// G_INPUT: the third input is g itself (3D model) instead of phi (2D model)
template <bool G_INPUT>
__global__ void sample_kernel(const double cinf, const double RR, const MlpBox box, const int64_t n,
                              const uint32_t seed_lo, const uint32_t seed_hi, float *__restrict__ x,
                              float *__restrict__ y) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  uint32_t r[4] = {(uint32_t)k, (uint32_t)((uint64_t)k >> 32), 0x4D4C5053u, 0u};
  philox4x32(r, seed_lo, seed_hi);
  const double u0 = u53(r[0], r[1]), u1 = u53(r[2], r[3]);
  uint32_t r2[4] = {(uint32_t)k, (uint32_t)((uint64_t)k >> 32), 0x4D4C5054u, 0u};
  philox4x32(r2, seed_lo, seed_hi);
  const double u2 = u53(r2[0], r2[1]);
  const double T = box.T_lo + (box.T_hi - box.T_lo) * u0;
  const double c = box.c_lo + (box.c_hi - box.c_lo) * u1;
  const double phi = -1.0 + 2.0 * u2;
  x[3 * k + 0] = (float)(2.0 * u0 - 1.0);
  x[3 * k + 1] = (float)(2.0 * u1 - 1.0);
  x[3 * k + 2] = (float)phi;
  const double g = G_INPUT ? phi : phi * (1.875 + phi * phi * (-1.25 + 0.375 * phi * phi));
  y[2 * k + 0] = (float)mu2_exact(T, c, g, cinf, RR);
  y[2 * k + 1] = (float)dG_exact(T, c, RR);
}

// The gradient of one call is computed by ONE cluster of CTAs (16, the opt-in
// size; 8 where the device cannot place 16), so that its sums have a fixed
// order and two trainings with the same seed give the same weights, with no
// scratch beyond shared memory.  The order, which does not depend on the
// cluster's size: each chunk of kChunk samples is summed sample by sample;
// kChains chains add the sums of the chunks r, r + kChains, ...; the chains are
// added in order.  A round takes two chunks per CTA:
//   samples: one thread per sample, forward, loss and backward; weights by
//     16-byte broadcasts from shared memory, the sigmoid of a unit evaluated
//     once for SiLU and its derivative; activations and deltas leave as
//     16-byte stores into rows of kRow floats (8 lanes x 16 bytes at a stride
//     of 36 words touch every bank once);
//   weights: four warps per chunk, W2's 32 x 32 gradient as 4 x 2 register
//     tiles, then the other 226 parameters one per thread and pass;
//   sums: the owner of a parameter (each CTA a share of them) adds the round's
//     chunk sums to its chains, read over distributed shared memory.
// At batch 4096 one thread per parameter and 32-way conflicting rows on 8 CTAs
// took 205 us; this takes 30.  Shared-memory bandwidth bounds it (the 16-byte
// weight broadcasts return 512 B each: 13 us), then the chain of its phases.
constexpr int kChunk = 128;
constexpr int kChains = 8;
constexpr int kRow = 36;
struct GradSmem {
  float w[kMlpNParams + 2];
  float part[2][kMlpNParams + 2];  // gradients of this CTA's two chunks
  alignas(16) float h1[kGradThreads][kRow];
  alignas(16) float h2[kGradThreads][kRow];
  alignas(16) float d1[kGradThreads][kRow];
  alignas(16) float d2[kGradThreads][kRow];
  float x[kGradThreads][4];  // inputs and 1
  float d3[kGradThreads][2];
  double wloss[kGradThreads / 32];
  double loss;
};
static_assert(sizeof(GradSmem) <= 227 * 1024, "one CTA per SM");
static_assert(kGradThreads == 2 * kChunk, "two chunks per CTA, a thread per sample");
static_assert(kOffW2 % 4 == 0 && kOffW3 % 4 == 0, "16-byte weight rows");

__device__ __forceinline__ float4 ld4s(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4s(float *p, const float (&v)[4]) {
  *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]);
}

__global__ void __launch_bounds__(kGradThreads, 1)
    grad_kernel(const MlpBox box, const float *__restrict__ w, const int64_t n,
                const float *__restrict__ x, const float *__restrict__ y, float *__restrict__ grad,
                double *__restrict__ loss) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  GradSmem &sm = *reinterpret_cast<GradSmem *>(smem_raw);
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank(), C = cluster.num_blocks();
  const int t = threadIdx.x, warp = t >> 5, lane = t & 31;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  for (int p = t; p < kMlpNParams; p += kGradThreads) sm.w[p] = w[p];
  __syncthreads();
  const MlpView W(sm.w);
  const float *W2 = sm.w + kOffW2, *W3 = sm.w + kOffW3;
  // this thread's chunk of a round, and its W2 tile (rows 4 ti.., columns 2 tj..) of it
  const int half = warp >> 2, id = t & (kChunk - 1), ti = id >> 4, tj = id & 15;
  float chain[kChains];  // the chains of the parameter this thread owns
#pragma unroll
  for (int r = 0; r < kChains; ++r) chain[r] = 0.f;
  const int share = (kMlpNParams + (int)C - 1) / (int)C, own = (int)rank * share + t;
  const bool owner = t < share && own < kMlpNParams;
  double l = 0.0;
  const int64_t round = (int64_t)2 * C * kChunk;
  for (int64_t first = 0; first < n; first += round) {
    // chunk `rank` + C half of the round
    const int64_t base = first + (int64_t)(rank + C * half) * kChunk;
    const bool some = base < n;
    const int64_t k = base + id;
    if (some) {
      const bool live = k < n;
      float xi[3] = {0.f, 0.f, 0.f};
      if (live)
        for (int q = 0; q < 3; ++q) xi[q] = x[3 * k + q];
      float a1[kMlpH], s1[kMlpH];  // activations and SiLU derivatives of layer 1
#pragma unroll
      for (int h = 0; h < kMlpH; ++h) {
        const float z = W.b1(h) + W.w1(h, 0) * xi[0] + W.w1(h, 1) * xi[1] + W.w1(h, 2) * xi[2];
        const float s = sigm(z);
        a1[h] = z * s;
        s1[h] = s * (1.f + z * (1.f - s));
      }
#pragma unroll
      for (int h = 0; h < kMlpH; h += 4) {
        const float v[4] = {a1[h], a1[h + 1], a1[h + 2], a1[h + 3]};
        st4s(&sm.h1[t][h], v);
      }
      float o[2] = {W.b3(0), W.b3(1)};
#pragma unroll 1
      for (int i = 0; i < kMlpH; i += 4) {
        float a2[4], s2[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          float z = W.b2(i + u);
#pragma unroll
          for (int j = 0; j < kMlpH; j += 4) {
            const float4 r = ld4s(W2 + (i + u) * kMlpH + j);
            z += r.x * a1[j];
            z += r.y * a1[j + 1];
            z += r.z * a1[j + 2];
            z += r.w * a1[j + 3];
          }
          const float s = sigm(z);
          a2[u] = z * s;
          s2[u] = s * (1.f + z * (1.f - s));
        }
        st4s(&sm.h2[t][i], a2);
        st4s(&sm.d2[t][i], s2);  // the derivative, until the delta replaces it
        const float4 r0 = ld4s(W3 + i), r1 = ld4s(W3 + kMlpH + i);
        const float w0[4] = {r0.x, r0.y, r0.z, r0.w}, w1[4] = {r1.x, r1.y, r1.z, r1.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {  // in the order of mlp_forward: the same outputs
          o[0] += w0[u] * a2[u];
          o[1] += w1[u] * a2[u];
        }
      }
      float e[2] = {0.f, 0.f};
      if (live) {
        for (int q = 0; q < 2; ++q) {
          e[q] = o[q] - (float)((y[2 * k + q] - box.y_mean[q]) / box.y_scale[q]);
          l += (double)e[q] * e[q];
        }
      }
      // backward: dL/do = 2 e (dead samples carry 0 deltas)
      const float g3[2] = {2.f * e[0], 2.f * e[1]};
      float g1[kMlpH];
#pragma unroll
      for (int j = 0; j < kMlpH; ++j) g1[j] = 0.f;
#pragma unroll 1
      for (int i = 0; i < kMlpH; i += 4) {
        const float4 r0 = ld4s(W3 + i), r1 = ld4s(W3 + kMlpH + i), s2 = ld4s(&sm.d2[t][i]);
        const float g2[4] = {(g3[0] * r0.x + g3[1] * r1.x) * s2.x, (g3[0] * r0.y + g3[1] * r1.y) * s2.y,
                             (g3[0] * r0.z + g3[1] * r1.z) * s2.z, (g3[0] * r0.w + g3[1] * r1.w) * s2.w};
        st4s(&sm.d2[t][i], g2);
#pragma unroll
        for (int u = 0; u < 4; ++u)
#pragma unroll
          for (int j = 0; j < kMlpH; j += 4) {
            const float4 r = ld4s(W2 + (i + u) * kMlpH + j);
            g1[j] += g2[u] * r.x;
            g1[j + 1] += g2[u] * r.y;
            g1[j + 2] += g2[u] * r.z;
            g1[j + 3] += g2[u] * r.w;
          }
      }
#pragma unroll
      for (int h = 0; h < kMlpH; h += 4) {
        const float v[4] = {g1[h] * s1[h], g1[h + 1] * s1[h + 1], g1[h + 2] * s1[h + 2], g1[h + 3] * s1[h + 3]};
        st4s(&sm.d1[t][h], v);
      }
      const float xv[4] = {xi[0], xi[1], xi[2], 1.f};
      st4s(sm.x[t], xv);
      sm.d3[t][0] = g3[0];
      sm.d3[t][1] = g3[1];
    }
    __syncthreads();
    if (some) {  // this chunk's weight gradients
      const int m0 = half * kChunk, m1 = m0 + kChunk, wq = warp & 3;
      float *part = sm.part[half];
      float acc[4][2] = {};
#pragma unroll 4
      for (int m = m0; m < m1; ++m) {
        const float4 d = ld4s(&sm.d2[m][4 * ti]);
        const float2 h = *reinterpret_cast<const float2 *>(&sm.h1[m][2 * tj]);
        const float dv[4] = {d.x, d.y, d.z, d.w};
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          acc[u][0] += dv[u] * h.x;
          acc[u][1] += dv[u] * h.y;
        }
      }
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        part[kOffW2 + (4 * ti + u) * kMlpH + 2 * tj] = acc[u][0];
        part[kOffW2 + (4 * ti + u) * kMlpH + 2 * tj + 1] = acc[u][1];
      }
      float one = 0.f, two = 0.f;
      if (wq < 3) {  // W1, column wq
#pragma unroll 8
        for (int m = m0; m < m1; ++m) one += sm.d1[m][lane] * sm.x[m][wq];
        part[kOffW1 + 3 * lane + wq] = one;
      } else {  // b1
#pragma unroll 8
        for (int m = m0; m < m1; ++m) one += sm.d1[m][lane];
        part[kOffB1 + lane] = one;
      }
      if (wq < 2) {  // W3
#pragma unroll 8
        for (int m = m0; m < m1; ++m) two += sm.d3[m][wq] * sm.h2[m][lane];
        part[kOffW3 + wq * kMlpH + lane] = two;
      } else if (wq == 2) {  // b2
#pragma unroll 8
        for (int m = m0; m < m1; ++m) two += sm.d2[m][lane];
        part[kOffB2 + lane] = two;
      } else if (lane < 2) {  // b3
#pragma unroll 8
        for (int m = m0; m < m1; ++m) two += sm.d3[m][lane];
        part[kOffB3 + lane] = two;
      }
    }
    cluster.sync();  // every CTA's chunk sums are in its shared memory
    if (owner) {
#pragma unroll
      for (int r = 0; r < kChains; ++r)
        for (unsigned c = r; c < 2 * C && first + (int64_t)c * kChunk < n; c += kChains)
          chain[r] += cluster.map_shared_rank(sm.part[c / C], c % C)[own];
    }
    cluster.sync();  // they are read before the next round, or the CTA's end
  }
  if (owner) {
    float s = 0.f;
#pragma unroll
    for (int r = 0; r < kChains; ++r) s += chain[r];
    grad[own] += s;
  }
  for (int off = 16; off > 0; off >>= 1) l += __shfl_down_sync(0xffffffffu, l, off);
  if (lane == 0) sm.wloss[warp] = l;
  __syncthreads();
  if (t == 0) {
    double s = 0.0;
    for (int q = 0; q < kGradThreads / 32; ++q) s += sm.wloss[q];
    sm.loss = s;
  }
  cluster.sync();
  if (rank == 0 && t == 0) {
    double s = 0.0;
    for (unsigned r = 0; r < C; ++r) s += *cluster.map_shared_rank(&sm.loss, r);
    *loss += s;
  }
  cluster.sync();  // the others' shared memory is read before they exit
}

// Adam (Kingma & Ba 2015) on the gradient scaled by `scale` (1 / batch size)
__global__ void adam_kernel(float *__restrict__ w, const float *__restrict__ grad, float *__restrict__ m,
                            float *__restrict__ v, const int64_t t, const float lr, const float scale) {
  const int p = blockIdx.x * blockDim.x + threadIdx.x;
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (p >= kMlpNParams) return;
  const float b1 = 0.9f, b2 = 0.999f, eps = 1e-8f;
  const float g = grad[p] * scale;
  const float mm = b1 * m[p] + (1.f - b1) * g;
  const float vv = b2 * v[p] + (1.f - b2) * g * g;
  m[p] = mm;
  v[p] = vv;
  const float mh = mm / (1.f - powf(b1, (float)t)), vh = vv / (1.f - powf(b2, (float)t));
  w[p] -= lr * mh / (sqrtf(vh) + eps);
}

__global__ void forward_kernel(const MlpBox box, const float *__restrict__ w, const int64_t n,
                               const float *__restrict__ x, float *__restrict__ out) {
  const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (k >= n) return;
  const MlpView W(w);
  const float xi[3] = {x[3 * k], x[3 * k + 1], x[3 * k + 2]};
  float o[2];
  mlp_forward(W, xi, o);
  out[2 * k] = (float)(o[0] * box.y_scale[0] + box.y_mean[0]);
  out[2 * k + 1] = (float)(o[1] * box.y_scale[1] + box.y_mean[1]);
}

}  // namespace

int launch_mlp_sample(double cinf, double RR, const MlpBox &box, int64_t n, uint64_t seed, float *x, float *y,
                      cudaStream_t st, bool g_input) {
  if (n <= 0) return 0;
  auto kfn = g_input ? sample_kernel<true> : sample_kernel<false>;
  kfn<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(cinf, RR, box, n, (uint32_t)seed, (uint32_t)(seed >> 32), x, y);
  return 0;
}

// CTAs of the gradient's cluster on the current device: 16 where it can place
// such a cluster, else 8 (the portable size); 0 on a CUDA error
static int grad_cluster() {
  static std::atomic<int> of[64];
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  int c = dev < 64 ? of[dev].load(std::memory_order_acquire) : 0;
  if (c) return c;
  if (cudaFuncSetAttribute(grad_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(GradSmem)) !=
          cudaSuccess ||
      cudaFuncSetAttribute(grad_kernel, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) != cudaSuccess)
    return 0;
  c = 8;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(16);
  cfg.blockDim = dim3(kGradThreads);
  cfg.dynamicSmemBytes = sizeof(GradSmem);
  cudaLaunchAttribute at[1];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {16, 1, 1};
  cfg.attrs = at;
  cfg.numAttrs = 1;
  int placed = 0;
  if (cudaOccupancyMaxActiveClusters(&placed, grad_kernel, &cfg) == cudaSuccess && placed > 0) c = 16;
  cudaGetLastError();
  if (dev < 64) of[dev].store(c, std::memory_order_release);
  return c;
}

int launch_mlp_grad(const MlpBox &box, const float *w, int64_t n, const float *x, const float *y, float *grad,
                    double *loss, cudaStream_t st) {
  if (n <= 0) return 0;
  const int C = grad_cluster();
  if (!C) return -3;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(C);  // one cluster
  cfg.blockDim = dim3(kGradThreads);
  cfg.dynamicSmemBytes = sizeof(GradSmem);
  cfg.stream = st;
  cudaLaunchAttribute at[2];
  at[0].id = cudaLaunchAttributeClusterDimension;
  at[0].val.clusterDim = {(unsigned)C, 1, 1};
  at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = at;
  cfg.numAttrs = 2;
  return cudaLaunchKernelEx(&cfg, grad_kernel, box, w, n, x, y, grad, loss) == cudaSuccess ? 0 : -3;
}

int launch_mlp_adam(float *w, const float *grad, float *m, float *v, int64_t t, float lr, float scale,
                    cudaStream_t st) {
  return launch_dep(adam_kernel, dim3((kMlpNParams + 255) / 256), dim3(256), st, w, grad, m, v, t, lr, scale) ==
                 cudaSuccess
             ? 0
             : -3;
}

int launch_mlp_forward(const MlpBox &box, const float *w, int64_t n, const float *x, float *out, cudaStream_t st) {
  if (n <= 0) return 0;
  forward_kernel<<<(unsigned)((n + 255) / 256), 256, 0, st>>>(box, w, n, x, out);
  return 0;
}

}  // namespace rs
