// rs_frame.cu — moving frame, grid reductions and the device tip tracker.
//
//  * pull_back (fun.cu:1469-1492): standalone column shift of every cell.
//  * grid partials: per-block FP64 sum of interior c, and per-block max tip
//    column; they replace the full-grid D2H copy + host scan of set_pull_back
//    (fun.cu:693-699, get_itip_all_grain fun.cu:1745-1754).
//  * precise tip (get_precise_tip, fun.cu:2895-2954): one warp per row finds
//    the last psi > 0 column; one block replays the reference's sequential row
//    scan (get_tip_int, fun.cu:2880-2893) over the per-row results and
//    performs the quartic and parabola least-squares fits (fun.cu:2648-2865)
//    in FP64.  This file is compiled with -fmad=false so that
//    the fits round like the reference's host code.
#include <cstdio>
#include <cstring>
#include <mutex>

#include "rs_kernels.cuh"

namespace rs {

// ---------------------------------------------------------------- pull_back
template <typename R>
__global__ void pull_back_kernel(const StepCoef K, const R *__restrict__ c, const R *__restrict__ psi,
                                 const R *__restrict__ phi, R *__restrict__ c_n,
                                 R *__restrict__ psi_n, R *__restrict__ phi_n, int i_offset,
                                 R c_fill) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  const int j = blockIdx.y * blockDim.y + threadIdx.y;
  if (i >= K.nx || j >= K.ny) return;
  int i_next = i + i_offset;
  i_next = max(i_next, 1);
  i_next = min(i_next, K.nx - 2);
  const int64_t d = (int64_t)j * K.pitch + i, s = (int64_t)j * K.pitch + i_next;
  c_n[d] = i_next < K.nx - 2 ? c[s] : c_fill;
  psi_n[d] = psi[s];
  if (phi_n) phi_n[d] = phi ? phi[s] : fmin(fmax(psi[s], R(-1)), R(1));
}

void launch_pull_back(int precision, const StepCoef &K, const void *c, const void *psi,
                      const void *phi, void *c_n, void *psi_n, void *phi_n, int i_offset,
                      cudaStream_t st) {
  dim3 b(64, 4), g((K.nx + 63) / 64, (K.ny + 3) / 4);
  if (precision == RS_F64)
    pull_back_kernel<double><<<g, b, 0, st>>>(K, (const double *)c, (const double *)psi,
                                              (const double *)phi, (double *)c_n, (double *)psi_n,
                                              (double *)phi_n, i_offset, K.cinf);
  else  // FP32 field sets hold c - cinf: the inflowing melt is 0
    pull_back_kernel<float><<<g, b, 0, st>>>(K, (const float *)c, (const float *)psi,
                                             (const float *)phi, (float *)c_n, (float *)psi_n,
                                             (float *)phi_n, i_offset, 0.0f);
}

// ---------------------------------------------------------------- reductions
// rs_itip, rs_mass and rs_precise_tip are two launches each: a pass over the
// one field the figure needs, and a small kernel that is a programmatic
// dependent of it.  The passes are programmatic dependents too: every kernel
// here waits (griddepcontrol.wait) before it touches memory, so its launch
// overlaps the kernel before it.  At 2048 x 2048 in FP64 (front at column 300)
// itip takes 9, the row pass of the precise tip 10 and the mass 9 us, their
// second kernels 3, 8 and 3, 296 together before: the tip's row scan was one
// thread's, and itip and mass read both fields.  16 loads a lane in flight
// instead of 32 make 14 and 13 of the row passes.
// The largest column in [0, hi] with psi > 0 of a row, or -1: the whole warp
// walks from the right end, kScan cells per lane and turn (their loads in
// flight together), and stops at the first turn that finds one, so it reads
// the melt ahead of the front only.
constexpr int kScan = 32;
// all of v in registers at once: without it the compiler loads and compares a
// few cells at a time (itip of 2048 x 2048 in FP64: 27 us)
#define RS_HOLD8(C, v, k)                                                                                  \
  "+" C(v[k]), "+" C(v[k + 1]), "+" C(v[k + 2]), "+" C(v[k + 3]), "+" C(v[k + 4]), "+" C(v[k + 5]), \
      "+" C(v[k + 6]), "+" C(v[k + 7])
__device__ __forceinline__ void hold(double (&v)[kScan]) {
  asm volatile("" : RS_HOLD8("d", v, 0), RS_HOLD8("d", v, 8), RS_HOLD8("d", v, 16));
  asm volatile("" : RS_HOLD8("d", v, 24));
}
__device__ __forceinline__ void hold(float (&v)[kScan]) {
  asm volatile("" : RS_HOLD8("f", v, 0), RS_HOLD8("f", v, 8), RS_HOLD8("f", v, 16));
  asm volatile("" : RS_HOLD8("f", v, 24));
}
#undef RS_HOLD8
template <typename R>
__device__ __forceinline__ int last_solid(const R *__restrict__ row, int hi, int lane) {
  int last = -1;
  for (; hi >= 0 && last < 0; hi -= 32 * kScan) {
    R v[kScan];
#pragma unroll
    for (int u = 0; u < kScan; ++u) {
      const int i = hi - 32 * u - lane;
      v[u] = i >= 0 ? row[i] : R(0);
    }
    hold(v);
#pragma unroll
    for (int u = kScan - 1; u >= 0; --u)
      if (v[u] > R(0)) last = hi - 32 * u - lane;
    last = __reduce_max_sync(0xffffffffu, last);
  }
  return last;
}

// coarse tip of four rows per block, a warp each (every cell, ghosts included)
constexpr int kRedRows = 4;
template <typename R>
__global__ void __launch_bounds__(32 * kRedRows) itip_partials_kernel(const StepCoef K, const R *__restrict__ psi,
                                                                      BlockPartial *out) {
  pdl_wait();
  pdl_trigger();
  const int j = blockIdx.x * kRedRows + (threadIdx.x >> 5);
  int it = 0;
  if (j < K.ny) it = last_solid(psi + (int64_t)j * K.pitch, K.nx - 1, threadIdx.x & 31);
  block_partial<32 * kRedRows>(0.0, it, out);
}

// FP64 sum of c (+ c_offset) over the interior cells of four rows per block,
// two warps per row, eight loads in flight per lane
template <typename R>
__global__ void __launch_bounds__(64 * kRedRows) mass_partials_kernel(const StepCoef K, const R *__restrict__ c,
                                                                      const double c_offset, BlockPartial *out) {
  pdl_wait();
  pdl_trigger();
  const int j = blockIdx.x * kRedRows + (threadIdx.x >> 6);
  double m = 0.0;
  if (j >= 1 && j <= K.ny - 2) {
    const R *__restrict__ row = c + (int64_t)j * K.pitch;
    constexpr int kU = 8;
    int i = 1 + (threadIdx.x & 63);
    for (; i + 64 * (kU - 1) <= K.nx - 2; i += 64 * kU) {
      R v[kU];
#pragma unroll
      for (int u = 0; u < kU; ++u) v[u] = row[i + 64 * u];
#pragma unroll
      for (int u = 0; u < kU; ++u) m += (double)v[u] + c_offset;
    }
    for (; i <= K.nx - 2; i += 64) m += (double)row[i] + c_offset;
  }
  block_partial<64 * kRedRows>(m, 0, out);
}

int launch_itip_partials(int precision, const StepCoef &K, const void *psi, BlockPartial *partials, int max_partials,
                         int *nblocks_out, cudaStream_t st) {
  const int nb = (K.ny + kRedRows - 1) / kRedRows;
  if (nb > max_partials) return -1;
  *nblocks_out = nb;
  return (precision == RS_F64
              ? launch_dep(itip_partials_kernel<double>, dim3(nb), dim3(32 * kRedRows), st, K, (const double *)psi, partials)
              : launch_dep(itip_partials_kernel<float>, dim3(nb), dim3(32 * kRedRows), st, K, (const float *)psi, partials)) ==
                 cudaSuccess
             ? 0
             : -3;
}

int launch_mass_partials(int precision, const StepCoef &K, const void *c, double c_offset, BlockPartial *partials,
                         int max_partials, int *nblocks_out, cudaStream_t st) {
  const int nb = (K.ny + kRedRows - 1) / kRedRows;
  if (nb > max_partials) return -1;
  *nblocks_out = nb;
  return (precision == RS_F64
              ? launch_dep(mass_partials_kernel<double>, dim3(nb), dim3(64 * kRedRows), st, K, (const double *)c, 0.0, partials)
              : launch_dep(mass_partials_kernel<float>, dim3(nb), dim3(64 * kRedRows), st, K, (const float *)c, c_offset,
                           partials)) == cudaSuccess
             ? 0
             : -3;
}

__global__ void __launch_bounds__(kRedThreads) reduce_partials_dep_kernel(const FinalRed FR) {
  pdl_wait();  // the kernel that wrote the partials has completed, its writes visible
  pdl_trigger();
  final_reduce(FR);
}

int launch_reduce_partials_dep(const FinalRed &FR, cudaStream_t st) {
  return launch_dep(reduce_partials_dep_kernel, dim3(1), dim3(kRedThreads), st, FR) == cudaSuccess ? 0 : -3;
}

// ---------------------------------------------------------------- precise tip
// per row j: last column i in [0, nx-2] with psi > 0 (or -1), and the two
// values get_tip_int can produce for the row: f_j at i0 = last, g_j at i0 = 0.
template <typename R>
__global__ void __launch_bounds__(128) tip_rows_kernel(const StepCoef K, const R *__restrict__ psi, int *row_last,
                                                       double *row_f, double *row_g) {
  pdl_wait();
  pdl_trigger();
  const int j = blockIdx.x * 4 + (threadIdx.x >> 5);
  const int lane = threadIdx.x & 31;
  if (j >= K.ny) return;
  const R *row = psi + (int64_t)j * K.pitch;
  const double g0 = (double)row[0], g1 = (double)row[1];
  const int last = last_solid(row, K.nx - 2, lane);
  if (lane == 0) {
    row_last[j] = last;
    if (last >= 0) {
      const double a = (double)row[last], b = (double)row[last + 1];
      row_f[j] = (b - a) * (0.0 - a) + last;
    } else {
      row_f[j] = 0.0;
    }
    row_g[j] = (g1 - g0) * (0.0 - g0) + 0;
  }
}

// solve_5x5 (fun.cu:2648-2691): Gaussian elimination with partial pivoting.
// The reference permutes row indices; here the rows themselves change places
// (the same operations on the same numbers in the same order), so that every
// index is a compile-time one and the system stays in registers.
__device__ __forceinline__ void solve_5x5_d(double A[5][5], double b[5], double c[5]) {
#pragma unroll
  for (int k = 0; k < 4; k++) {
    double max_val = fabs(A[k][k]);
    int max_idx = k;
#pragma unroll
    for (int i = k + 1; i < 5; i++)
      if (fabs(A[i][k]) > max_val) {
        max_val = fabs(A[i][k]);
        max_idx = i;
      }
#pragma unroll
    for (int i = k + 1; i < 5; i++)
      if (max_idx == i) {
#pragma unroll
        for (int j = 0; j < 5; j++) {
          const double t = A[k][j];
          A[k][j] = A[i][j];
          A[i][j] = t;
        }
        const double t = b[k];
        b[k] = b[i];
        b[i] = t;
      }
#pragma unroll
    for (int i = k + 1; i < 5; i++) {
      const double factor = A[i][k] / A[k][k];
#pragma unroll
      for (int j = k; j < 5; j++) A[i][j] -= factor * A[k][j];
      b[i] -= factor * b[k];
    }
  }
#pragma unroll
  for (int i = 4; i >= 0; i--) {
    double sum = 0.0;
#pragma unroll
    for (int j = i + 1; j < 5; j++) sum += A[i][j] * c[j];
    c[i] = (b[i] - sum) / A[i][i];
  }
}

// get_precise_x (fun.cu:2694-2738): quartic x(psi) through 5 points, x at psi = 0
__device__ __forceinline__ double precise_x_d(const double (&x)[5], const double (&y)[5]) {
  double A[5][5], b[5], c[5];
#pragma unroll
  for (int j = 0; j < 5; ++j) {
    b[j] = 0.0;
    c[j] = 0.0;
    for (int k = 0; k < 5; ++k) A[j][k] = 0.0;
  }
#pragma unroll
  for (int i = 0; i < 5; i++) {
    double yp[9];
    yp[0] = 1.0;
#pragma unroll
    for (int k = 1; k <= 8; k++) yp[k] = yp[k - 1] * y[i];
#pragma unroll
    for (int j = 0; j < 5; j++) {
      b[j] += x[i] * yp[j];
#pragma unroll
      for (int k = 0; k < 5; k++) A[j][k] += yp[j + k];
    }
  }
  solve_5x5_d(A, b, c);
  return c[0];  // c0 + c1 0 + ... evaluated at phi_interface = 0
}

// solve_3x3 (fun.cu:2740-2786)
__device__ int solve_3x3_d(double A[3][3], double cc[3], double x[3]) {
  for (int k = 0; k < 3; ++k) {
    int pivot = k;
    double maxval = fabs(A[k][k]);
    for (int i = k + 1; i < 3; ++i)
      if (fabs(A[i][k]) > maxval) {
        maxval = fabs(A[i][k]);
        pivot = i;
      }
    if (maxval < 1e-14) return -1;
    if (pivot != k) {
      for (int j = 0; j < 3; ++j) {
        const double t = A[k][j];
        A[k][j] = A[pivot][j];
        A[pivot][j] = t;
      }
      const double t = cc[k];
      cc[k] = cc[pivot];
      cc[pivot] = t;
    }
    const double piv = A[k][k];
    for (int i = k + 1; i < 3; ++i) {
      const double factor = A[i][k] / piv;
      A[i][k] = 0.0;
      for (int j = k + 1; j < 3; ++j) A[i][j] -= factor * A[k][j];
      cc[i] -= factor * cc[k];
    }
  }
  for (int i = 2; i >= 0; --i) {
    double sum = cc[i];
    for (int j = i + 1; j < 3; ++j) sum -= A[i][j] * x[j];
    x[i] = sum / A[i][i];
  }
  return 0;
}

// fit_parabola (fun.cu:2809-2865)
__device__ int fit_parabola_d(const double *x, const double *y, double *x0, double *y0, double *R) {
  double M[3][3] = {{0, 0, 0}, {0, 0, 0}, {0, 0, 0}}, cc[3] = {0, 0, 0}, aa[3] = {0, 0, 0};
  for (int i = 0; i < 5; ++i) {
    const double f0 = 1.0, f1 = y[i], f2 = y[i] * y[i];
    M[0][0] += f0 * f0; M[0][1] += f0 * f1; M[0][2] += f0 * f2;
    M[1][0] += f1 * f0; M[1][1] += f1 * f1; M[1][2] += f1 * f2;
    M[2][0] += f2 * f0; M[2][1] += f2 * f1; M[2][2] += f2 * f2;
    cc[0] += f0 * x[i]; cc[1] += f1 * x[i]; cc[2] += f2 * x[i];
  }
  if (solve_3x3_d(M, cc, aa) != 0) return -2;
  if (fabs(aa[2]) < 1e-14) return -3;
  const double R_loc = 1.0 / (2.0 * aa[2]);
  const double y0_loc = -aa[1] / (2.0 * aa[2]);
  *x0 = aa[0] - (y0_loc * y0_loc) / (2.0 * R_loc);
  *y0 = y0_loc;
  *R = R_loc;
  return 0;
}

// get_tip_int (fun.cu:2880-2893) is sequential over the rows: the scan start
// of row j is the running tip int(itip), so row j offers f_j if its last solid
// column is not behind that, else g_j, and becomes the tip if it is larger.
// Here the block reads kFitRows rows at a time and takes the larger of f_j and
// g_j over each group of 32.  Let M be the largest of them and m the first row
// that has it.  No row offers more than M, so where M does not exceed the tip no
// row raises it; and where m has it as f_m with a last solid column not behind
// int(M), row m is reached with a tip below M, offers f_m = M and becomes the
// tip, and no later row does: the scan's result at once.  Otherwise (f_j and g_j
// of odd fields) one warp visits the groups that can raise the tip, in order,
// and in a group the rows that do (ballots), with the comparisons of the
// sequential scan.  The five quartic fits run on five lanes.
constexpr int kFitThreads = 512;
constexpr int kFitRows = 2048;
constexpr int kFitGroups = kFitRows / 32;
template <typename R>
__global__ void __launch_bounds__(kFitThreads) tip_fit_kernel(const StepCoef K, const R *__restrict__ psi,
                                                              const int *__restrict__ row_last,
                                                              const double *__restrict__ row_f,
                                                              const double *__restrict__ row_g, rs_tip *out) {
  __shared__ int s_last[kFitRows];
  __shared__ double s_f[kFitRows], s_g[kFitRows], s_max[kFitGroups];
  static_assert(kFitGroups == 64, "two group maxima per lane");
  pdl_wait();
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ny = K.ny;
  double itip = 0.0;
  int ti = 0, tj = 0;
  for (int base = 0; base < ny; base += kFitRows) {
    if (base) __syncthreads();  // the warp has left the previous rows
#pragma unroll
    for (int q = 0; q < kFitRows / kFitThreads; ++q) {
      const int r = threadIdx.x + q * kFitThreads, j = base + r;
      const int last = j < ny ? __ldcg(row_last + j) : -1;
      const double f = j < ny ? __ldcg(row_f + j) : 0.0, g = j < ny ? __ldcg(row_g + j) : 0.0;
      s_last[r] = last;
      s_f[r] = f;
      s_g[r] = g;
      double m = fmax(f, g);
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) s_max[r >> 5] = m;
    }
    __syncthreads();
    if (warp != 0) continue;
    const double m0 = s_max[lane], m1 = s_max[32 + lane];
    double M = fmax(m0, m1);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) M = fmax(M, __shfl_xor_sync(0xffffffffu, M, o));
    if (!(M > itip)) continue;
    {
      const unsigned lo = __ballot_sync(0xffffffffu, m0 == M), hi = __ballot_sync(0xffffffffu, m1 == M);
      const int g = lo ? __ffs(lo) - 1 : 31 + __ffs(hi), r = 32 * g + lane;
      const unsigned at = __ballot_sync(0xffffffffu, fmax(s_f[r], s_g[r]) == M);
      const int l = __ffs(at) - 1;  // (a group's maximum is one of its rows')
      if (at && __shfl_sync(0xffffffffu, (int)(s_f[r] == M && s_last[r] >= 0 && (double)s_last[r] >= floor(M)), l)) {
        itip = M;
        ti = (int)M;
        tj = base + 32 * g + l;
        continue;
      }
    }
    for (int g = 0; g < kFitGroups; ++g) {  // the next group that can raise the tip
      const unsigned long long can = ((unsigned long long)__ballot_sync(0xffffffffu, m1 > itip) << 32) |
                                     __ballot_sync(0xffffffffu, m0 > itip);
      const unsigned long long left = can >> g;
      if (!left) break;
      g += __ffsll((long long)left) - 1;
      const int r = 32 * g + lane, last = s_last[r];
      const double f = s_f[r], gv = s_g[r];
      unsigned rest = 0xffffffffu;  // rows after the last one that raised it
      for (;;) {
        const int s = (int)itip;
        const double v = (last >= 0 && last >= s) ? f : gv;
        const unsigned hit = __ballot_sync(0xffffffffu, v > itip) & rest;
        if (!hit) break;
        const int l = __ffs(hit) - 1;
        itip = __shfl_sync(0xffffffffu, v, l);
        ti = (int)itip;
        tj = base + 32 * g + l;
        rest = l == 31 ? 0u : (0xffffffffu << (l + 1));
        if (!rest) break;
      }
    }
  }
  if (warp != 0) return;
  double xk = 0.0, yk = 0.0;
  if (lane < 5) {
    int j = tj - 2 + lane;
    // deal_with_boundary (fun.cu:2624-2641) with (jmin, jmax)
    const int nmin = min(K.jmin, K.jmax), nmax = max(K.jmin, K.jmax);
    if (K.jmin > K.jmax) {  // periodic
      if (j <= nmin - 1) j += (nmax - nmin + 1);
      else if (j >= nmax + 1) j -= (nmax - nmin + 1);
    } else {                // no-flux: mirror
      if (j < nmin) j = 2 * nmin - j;
      else if (j > nmax) j = 2 * nmax - j;
    }
    j = min(max(j, 0), ny - 1);
    const int s = max(ti - 5, 0);
    const int last = __ldcg(row_last + j);
    const int i0 = (last >= 0 && last >= s) ? last : 0;
    double id[5], pd[5];
#pragma unroll
    for (int m = 0; m < 5; ++m) {
      const int i = i0 - 2 + m;
      id[m] = i;
      pd[m] = (double)psi[(int64_t)j * K.pitch + min(max(i, 0), K.nx - 1)];
    }
    xk = precise_x_d(id, pd);
    yk = j;
  }
  double xd[5], yd[5];
#pragma unroll
  for (int k = 0; k < 5; ++k) {
    xd[k] = __shfl_sync(0xffffffffu, xk, k);
    yd[k] = __shfl_sync(0xffffffffu, yk, k);
  }
  if (lane != 0) return;
  double x0 = 0.0, y0 = 0.0, Rr = 0.0;
  const int status = fit_parabola_d(xd, yd, &x0, &y0, &Rr);
  rs_tip t;
  t.i = ti;
  t.j = tj;
  t.status = status;
  t.reserved = 0;
  t.x = x0;
  t.y = y0;
  double Rn = fabs(Rr) * K.dx * K.W0 * K.S;
  if (Rn > 1e5) Rn = 1e5;
  if (Rn < 1.0) Rn = 1.0;
  t.R = Rn;
  *out = t;
}

template <typename R>
static int launch_precise_tip_t(const StepCoef &K, const R *psi, int *row_last, double *row_f, double *row_g,
                                rs_tip *out, cudaStream_t st) {
  if (launch_dep(tip_rows_kernel<R>, dim3((K.ny + 3) / 4), dim3(128), st, K, psi, row_last, row_f, row_g) != cudaSuccess ||
      launch_dep(tip_fit_kernel<R>, dim3(1), dim3(kFitThreads), st, K, psi, row_last, row_f, row_g, out) != cudaSuccess)
    return -3;
  return 0;
}

int launch_precise_tip(int precision, const StepCoef &K, const void *psi, int *row_last, double *row_f, double *row_g,
                       rs_tip *out, cudaStream_t st) {
  return precision == RS_F64 ? launch_precise_tip_t(K, (const double *)psi, row_last, row_f, row_g, out, st)
                             : launch_precise_tip_t(K, (const float *)psi, row_last, row_f, row_g, out, st);
}

}  // namespace rs

// ---------------------------------------------------------------- no-allocation tip
// rs_precise_tip_noalloc: the precise tip for callers that cannot allocate
// device memory.  rs_precise_tip takes its per-row scratch (last psi > 0
// column and the two candidate tip values of every row) from a context that
// rs_create fills with cudaMalloc.  Some hosts cannot do that: a host that
// hands all device memory to its own pool allocator and forbids cudaMalloc
// once it runs, or a time-stepping loop that must not take the implicit
// device-wide synchronisation of cudaMalloc/cudaFree.  This entry point needs
// no context: its scratch is the file-scope array below, which every GPU that
// loads the library holds (RS_NOALLOC_TIP_MAX_ROWS rows, 20 bytes per row,
// 320 KiB) until the process exits.
//
// Host code cannot use the array's name as a device address (it names a host
// stand-in); the device address is looked up once per device with
// cudaGetSymbolAddress, with that device current, on the first call made on
// that device.  Make that first call before any stream capture.
//
// Every call shares the same scratch and it keeps the last call's contents.
// Nothing in it needs to start at zero: each call writes every row entry it
// later reads.  Calls whose kernels overlap on the GPU (different streams,
// different host threads) race on the scratch and must be ordered by the
// caller.
namespace rs {
namespace {

struct alignas(256) TipScratch {
  int last[RS_NOALLOC_TIP_MAX_ROWS];
  double f[RS_NOALLOC_TIP_MAX_ROWS];
  double g[RS_NOALLOC_TIP_MAX_ROWS];
};
static __device__ __align__(256) TipScratch g_tip_scratch;

constexpr int kMaxDevices = 64;
struct DeviceScratch {
  TipScratch *ptr;
  bool ready;
};
DeviceScratch g_dev_scratch[kMaxDevices];
std::mutex g_dev_scratch_mu;

int tip_scratch_for_current_device(TipScratch **out) {
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return rs::set_error(RS_E_CUDA, "rs_precise_tip_noalloc: no CUDA device");
  if (dev < 0 || dev >= kMaxDevices) return rs::set_error(RS_E_UNSUPPORTED, "rs_precise_tip_noalloc: device index too large");
  std::lock_guard<std::mutex> lock(g_dev_scratch_mu);
  DeviceScratch &d = g_dev_scratch[dev];
  if (!d.ready) {
    void *p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress(&p, g_tip_scratch);
    if (e != cudaSuccess) {
      char msg[256];
      snprintf(msg, sizeof(msg), "rs_precise_tip_noalloc: cudaGetSymbolAddress: %s", cudaGetErrorString(e));
      return rs::set_error(RS_E_CUDA, msg);
    }
    d.ptr = static_cast<TipScratch *>(p);
    d.ready = true;
  }
  *out = d.ptr;
  return RS_OK;
}

}  // namespace
}  // namespace rs

extern "C" int rs_precise_tip_noalloc(const rs_params *p, const rs_fields *f, rs_tip *d_tip, rs_stream_t stream) {
  if (!p || !f || !d_tip || !f->psi) return rs::set_error(RS_E_INVALID, "rs_precise_tip_noalloc: null argument");
  if (f->precision != RS_F64 && f->precision != RS_F32)
    return rs::set_error(RS_E_INVALID, "rs_precise_tip_noalloc: precision tag");
  if (p->nx_all < 8 || p->ny_all < 8) return rs::set_error(RS_E_INVALID, "rs_precise_tip_noalloc: grid below 8x8");
  if (p->band) return rs::set_error(RS_E_UNSUPPORTED, "rs_precise_tip_noalloc: needs the whole domain, not a band");
  if (p->ny_all > RS_NOALLOC_TIP_MAX_ROWS)
    return rs::set_error(RS_E_INVALID, "rs_precise_tip_noalloc: ny_all exceeds RS_NOALLOC_TIP_MAX_ROWS");
  const int pitch = f->pitch ? f->pitch : p->nx_all;
  if (pitch != p->nx_all) return rs::set_error(RS_E_UNSUPPORTED, "rs_precise_tip_noalloc: pitch must equal nx_all");
  if ((uintptr_t)f->psi % (f->precision == RS_F64 ? 8 : 4))
    return rs::set_error(RS_E_INVALID, "rs_precise_tip_noalloc: misaligned psi");
  rs::TipScratch *sc = nullptr;
  int rc = rs::tip_scratch_for_current_device(&sc);
  if (rc) return rc;
  // the tip kernels read only these geometry fields of the step coefficients
  rs::StepCoef K;
  memset(&K, 0, sizeof(K));
  K.nx = p->nx_all;
  K.ny = p->ny_all;
  K.pitch = pitch;
  K.jmin = p->periodic_j ? p->ny_all - 2 : 1;
  K.jmax = p->periodic_j ? 1 : p->ny_all - 2;
  K.dx = p->dx;
  K.W0 = p->W0;
  K.S = p->S;
  const int lr = rs::launch_precise_tip(f->precision, K, f->psi, sc->last, sc->f, sc->g, d_tip, (cudaStream_t)stream);
  const cudaError_t e = cudaGetLastError();
  if (lr || e != cudaSuccess) {
    char msg[256];
    snprintf(msg, sizeof(msg), "rs_precise_tip_noalloc: %s", cudaGetErrorString(e));
    return rs::set_error(RS_E_CUDA, msg);
  }
  return RS_OK;
}


