// rs_peri3d.cu — the 3D three-phase (peritectic) step on one GPU.
//
// Model: multi/peritectic_multiGPU/TiAg.cu — stored phi1 (liquid), phi2
// (solid alpha), phi3 = 1 - phi1 - phi2 (solid beta); mu = c - sum r_i g_i
// (computeMu, TiAg.cu:461-470); the update of phi1, phi2, c (diffuse,
// TiAg.cu:503-561); periodic x, y and no-flux z ghost layers (TiAg.cu:472-500,
// 565-605).  The reference runs five kernels per step (computeMu, three
// boundaryMu, diffuse) plus three boundary kernels and keeps mu as a field;
// here one kernel does the step and mu never leaves shared memory.
//
// The FP32 step runs on packed FP32 pairs (rs_peri3d_x2.cu); this file's
// step kernel is the FP64 one.
// Kernel: a CTA owns a column of 32 x 16 output cells (x, y) and marches
// through a chunk of z planes.  Every input plane (34 columns x 18 rows of
// phi1, phi2 and c) arrives by one 3D TMA box per field into a six-slot ring;
// the last warp that leaves plane z issues the load into the slot of plane
// z-1, so four planes are in flight while plane z is computed.  mu of each
// plane (tile plus x/y halo) is computed once into a four-slot ring, where the
// march is not in pure melt (there mu is c - r1).  Outputs go straight to
// global memory (32 consecutive x per warp), and each output that a ghost cell
// images (x = 1, nx-2; y = 1, ny-2; z = 1, nz-2) is written to its ghost cells
// too, which is what the reference's boundary kernels leave there.
// What bounds it (512 x 512 x 128): in melt the memory (333 us, 74 % of the
// copy rate), in fronts the FP64 pipe (605 us; 191 FP64 instructions per cell,
// 61 % of the pipe's rate at 16 warps per SM).  A front in two thirds of the
// planes: 546 -> 476 to 486 us.  Measured beside it: four slots 519, 14-row tiles
// with three CTAs per SM and four slots 532 (80 registers instead of 118).
// Algorithmic bytes per cell-step: 3 fields read + 3 written.
#include <cuda.h>

#include "rs_kernels.cuh"
#include "rs_peri3d_common.cuh"

namespace rs {
namespace {

struct D3 {  // the tile: 32 x 16 output cells, two rows of a column per thread
  static constexpr int BX = 32, BXin = 34, BY = 16, BYin = 18, kThreads = 256, K = BX * BY / kThreads;
  static constexpr int kSlots = 6;            // input plane ring: 6 x 15 KB, two CTAs per SM
  static constexpr int kPlane = BXin * BYin;  // elements of one field plane, 4896 bytes
  static constexpr int kPlaneAl = 624;        // TMA destinations stay 128-byte aligned
  static_assert(kPlaneAl >= kPlane && kPlaneAl * sizeof(double) % 128 == 0 && K == 2);
};

struct P3Smem {
  alignas(128) double in[D3::kSlots][3][D3::kPlaneAl];  // [slot][field][row][col]
  alignas(16) double mu[kP3MuSlots][D3::kPlane];
  uint64_t full[D3::kSlots];
  int melt[8];  // per plane (q mod 8): the box is pure melt inside the array (p3_melt_cell)
  uint32_t passed;  // warps that have left a plane, summed over the planes
};

// mu = c - sum_i r_i g_i (computeMu, TiAg.cu:461-470)
template <typename R>
__device__ __forceinline__ R mu_of(const K3<R> &k, R p1, R p2, R c) {
  const R p3 = R(1) - p1 - p2;
  return c - k.r1 * g3(p1, p2, p3) - k.r2 * g3(p2, p3, p1) - k.r3 * g3(p3, p1, p2);
}
// the same with the polynomials of g_i as multiply-adds about p = 1,
// 4 g = p^2 (4 + 8 q + 12 q^2 - 9 q^3 - 15 q d^2), q = 1 - p, d = p_k - p_j: near
// p = 1 and p = 0 its terms are small against 4 g, where the powers of p itself
// cancel (15 - 5 p - 15 p^2 + 9 p^3, one operation less per g: the new c 1.16e-16
// rms from 64 bits of the mantissa, this 0.70e-16, the reference's form 0.81e-16;
// mu rounded exactly would give 0.58e-16).  The r1 term first: in melt it is exact.
__device__ __forceinline__ double mu_step(const K3<double> &k, double p1, double p2, double c) {
  const double p3 = (1.0 - p1) - p2, d12 = p1 - p2, d23 = p2 - p3, d31 = p3 - p1;
  auto g = [](double p, double d) {
    const double q = 1.0 - p, a = fma(fma(fma(q, -9.0, 12.0), q, 8.0), q, 4.0);
    return p * p * fma(-15.0 * q, d * d, a);
  };
  return fma(g(p3, d12), -0.25 * k.r3, fma(g(p2, d31), -0.25 * k.r2, fma(g(p1, d23), -0.25 * k.r1, c)));
}

// A1: the a1 well terms are non-zero; SD: solid diffusivities Da or Db non-zero
// (the reference sets all of them to 0)
template <bool A1, bool SD>
__global__ void __launch_bounds__(D3::kThreads, 2)
    peri3d_kernel(const __grid_constant__ K3<double> k, const __grid_constant__ CUtensorMap m1,
                  const __grid_constant__ CUtensorMap m2, const __grid_constant__ CUtensorMap mc,
                  double *__restrict__ o1, double *__restrict__ o2, double *__restrict__ oc, const int64_t step,
                  int *err) {
  using C = D3;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  P3Smem &sm = *reinterpret_cast<P3Smem *>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31;
  const int xb = C::BX * blockIdx.x;   // first box column (array x); outputs xb+1 .. xb+BX
  const int yb = C::BY * blockIdx.y;   // first box row (array y); outputs yb+1 .. yb+BY
  const int zo0 = 1 + k.z_chunk * blockIdx.z;                 // first output plane
  const int zo1 = min(zo0 + k.z_chunk, k.nz - 1);            // one past the last
  if (zo0 >= zo1) return;
  const int zin0 = zo0 - 1, zin1 = zo1;  // input planes zin0 .. zin1
  pdl_wait();
  pdl_trigger();
  constexpr uint32_t kBytes = 3u * C::kPlane * sizeof(double);
  if (smem_u32(smem_raw) & 127u) {
    if (tid == 0) atomicExch(err, 2);
    return;
  }
  auto issue = [&](int z) {  // plane z into its ring slot
    const int q = z - zin0, s = q % C::kSlots;
    mbar_expect_tx(&sm.full[s], kBytes);
    tma_load_3d(&sm.in[s][0][0], &m1, &sm.full[s], xb, yb, z);
    tma_load_3d(&sm.in[s][1][0], &m2, &sm.full[s], xb, yb, z);
    tma_load_3d(&sm.in[s][2][0], &mc, &sm.full[s], xb, yb, z);
  };
  int issued = min(zin1, zin0 + C::kSlots - 1);  // last plane whose load was issued
  if (tid == 0) {
    for (int s = 0; s < C::kSlots; ++s) mbar_init(&sm.full[s], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    for (int z = zin0; z <= issued; ++z) issue(z);
    for (int s = 0; s < 8; ++s) sm.melt[s] = 1;
    sm.passed = 0u;
  }
  __syncthreads();
  // Planes of pure melt (p3_melt_cell; bit u: box element tid + C::kThreads u
  // lies outside the array); false if the plane's load never came
  constexpr int kElems = (C::kPlane + C::kThreads - 1) / C::kThreads;
  uint32_t outside = 0u;
#pragma unroll
  for (int u = 0; u < kElems; ++u) {
    const int e = tid + C::kThreads * u;
    if (e >= C::kPlane || xb + e % C::BXin >= k.nx || yb + e / C::BXin >= k.ny) outside |= 1u << u;
  }
  auto wait_plane = [&](int z) {
    const int q = z - zin0;
    return p3_wait<double>(&sm.full[q % C::kSlots], (uint32_t)((q / C::kSlots) & 1), err);
  };
  // the words in which a cell differs from pure melt (phi1 == 1, phi2 == 0 of
  // either sign), on the integer pipe
  auto off_melt = [](double p1, double p2) {
    return (uint32_t)(__double2hiint(p1) ^ 0x3FF00000) | (uint32_t)__double2loint(p1) |
           ((uint32_t)__double2hiint(p2) << 1) | (uint32_t)__double2loint(p2);
  };
  auto check_plane = [&](int z) {
    const int q = z - zin0, s = q % C::kSlots;
    uint32_t diff = 0u;
#pragma unroll
    for (int u = 0; u < kElems; ++u) {
      const int e = tid + C::kThreads * u;
      if (!((outside >> u) & 1u)) diff |= off_melt(sm.in[s][0][e], sm.in[s][1][e]);
    }
    if (diff) sm.melt[q & 7] = 0;
  };
  // mu of plane z (tile and halo, already loaded) into its slot, and its check
  auto mu_plane = [&](int z) {
    const int q = z - zin0, s = q % C::kSlots;
    double *mu = sm.mu[q % kP3MuSlots];
    const double *f1 = sm.in[s][0], *f2 = sm.in[s][1], *fc = sm.in[s][2];
    uint32_t diff = 0u;
#pragma unroll
    for (int u = 0; u < kElems; ++u) {
      const int e = tid + C::kThreads * u;
      if (e >= C::kPlane) break;
      const double p1 = f1[e], p2 = f2[e];
      mu[e] = mu_step(k, p1, p2, fc[e]);
      if (!((outside >> u) & 1u)) diff |= off_melt(p1, p2);
    }
    if (diff) sm.melt[q & 7] = 0;
  };
  // a load that did not arrive in time: wait (bounded) for every load still
  // in flight before the CTA leaves, so none lands in reused shared memory
  auto drain = [&](int from) {
    if (tid == 0)
      for (int z = from; z <= issued; ++z) {
        const int q = z - zin0;
        uint32_t tries = 0;
        while (!mbar_try_wait(&sm.full[q % C::kSlots], (uint32_t)((q / C::kSlots) & 1)) && ++tries < kP3WaitLimit) {
        }
      }
  };
  const bool ok = wait_plane(zin0) && wait_plane(zin0 + 1);
  if (ok) {
    check_plane(zin0);
    check_plane(zin0 + 1);
  }
  if (!__syncthreads_and(ok)) {
    drain(zin0);
    return;
  }

  // this thread's cells: column ix, a strip of K consecutive rows (the y
  // neighbours of the strip come from a register window)
  constexpr int K = C::K;
  const int ix = tid % C::BX, iy0 = (tid / C::BX) * K;
  const int gx = xb + 1 + ix;  // array x of the output
  const bool xin = gx <= k.nx - 2;
  const int xd = gx == k.nx - 2 ? 2 - k.nx : (gx == 1 ? k.nx - 2 : 0);  // to the ghost column it images
  const int e0 = (iy0 + 1) * C::BXin + ix + 1;                          // box element of the strip's first cell
  const int64_t plane = (int64_t)k.nx * k.ny;
  int64_t out0 = (int64_t)zo0 * plane + (int64_t)(yb + 1 + iy0) * k.nx + gx;  // the strip's first cell in plane z

  // mu is stored for the planes that the general form reads, ahead of the
  // barrier while the march is in it; a march that enters it from pure melt
  // makes up for the missing planes behind the barrier.  Uniform over the CTA.
  int mu_done = zin0 - 1;  // mu of planes .. mu_done stands, as far as the ring goes
  bool general = false;
  for (int z = zo0; z < zo1; ++z, out0 += plane) {
    // one barrier per plane: the flags and mu of planes .. z+1 stand behind it
    // (mu has four slots: mu(z+1) overwrites mu(z-3))
    const bool got = wait_plane(z + 1);
    if (got) {
      if (general) {
        mu_plane(z + 1);
        mu_done = z + 1;
      } else {
        check_plane(z + 1);
      }
    }
    if (!__syncthreads_and(got)) {
      issued = min(zin1, z + C::kSlots - 2);
      drain(z + 1);
      return;
    }
    const int q = z - zin0;
    // planes z-1 .. z+1 pure melt wherever a stencil of an output cell reaches
    // (p3_melt_cell); the flag of plane z+3 is re-armed here (check_plane(z+3),
    // before the barrier of iteration z+2, is separated from this write by the
    // barrier of z+1)
    const bool melt3 = sm.melt[(q - 1) & 7] && sm.melt[q & 7] && sm.melt[(q + 1) & 7];
    if (tid == 0) sm.melt[(q + 3) & 7] = 1;
    if (!melt3 && mu_done < z + 1) {
      for (int w = max(z - 1, mu_done + 1); w <= z + 1; ++w) mu_plane(w);
      mu_done = z + 1;
      __syncthreads();
    }
    general = !melt3;
    const double *c1 = sm.in[q % C::kSlots][0], *c2 = sm.in[q % C::kSlots][1], *cc = sm.in[q % C::kSlots][2];
    const int zd = z == 1 ? -1 : (z == k.nz - 2 ? 1 : 0);  // planes 0 and nz-1 copy their neighbours
    // the cell and every ghost cell that images it
    auto store_cell = [&](int r, double n1, double n2, double nc) {
      const int gy = yb + 1 + iy0 + r;
      if (gy > k.ny - 2) return;
      const int64_t o = out0 + (int64_t)r * k.nx;
      o1[o] = n1;
      o2[o] = n2;
      oc[o] = nc;
      const int yd = gy == k.ny - 2 ? 2 - k.ny : (gy == 1 ? k.ny - 2 : 0);
      if (xd | yd | zd) {
#pragma unroll 1
        for (int im = 1; im < 8; ++im) {
          if (((im & 1) && !xd) || ((im & 2) && !yd) || ((im & 4) && !zd)) continue;
          const int64_t og =
              o + (im & 1 ? xd : 0) + (im & 2 ? (int64_t)yd * k.nx : 0) + (im & 4 ? zd * plane : 0);
          o1[og] = n1;
          o2[og] = n2;
          oc[og] = nc;
        }
      }
    };
    if (xin && melt3) {
      // pure melt (p3_melt_cell): phi1, phi2 stay 1 and 0, mu is c - r1 (g_1 = 1,
      // g_2 = g_3 = 0) and the face mobilities are 2: the values the general
      // form gives bit for bit, without a mu plane
      const double *cd = sm.in[(q - 1) % C::kSlots][2], *cu = sm.in[(q + 1) % C::kSlots][2];
      const double r1 = k.r1;
      double w[K + 2];
#pragma unroll
      for (int r = 0; r < K + 2; ++r) w[r] = cc[e0 + (r - 1) * C::BXin];
#pragma unroll
      for (int r = 0; r < K; ++r) {
        const int e = e0 + r * C::BXin;
        const double m0 = w[r + 1] - r1;
        auto face = [&](double cp, double cm) { return 2.0 * (((cp - r1) - m0) + ((cm - r1) - m0)); };
        double dc = face(cc[e + 1], cc[e - 1]) * k.cfx;
        dc = fma(face(w[r + 2], w[r]), k.cfy, dc);
        dc = fma(face(cu[e], cd[e]), k.cfz, dc);
        store_cell(r, 1.0, 0.0, w[r + 1] + dc);
      }
    } else if (xin) {
      const double *d1 = sm.in[(q - 1) % C::kSlots][0], *d2 = sm.in[(q - 1) % C::kSlots][1];
      const double *u1 = sm.in[(q + 1) % C::kSlots][0], *u2 = sm.in[(q + 1) % C::kSlots][1];
      const double *mu = sm.mu[q % kP3MuSlots], *mud = sm.mu[(q - 1) % kP3MuSlots],
                   *muu = sm.mu[(q + 1) % kP3MuSlots];
      // the plane's B1, B2 (TiAg.cu:61-62) with the frozen T of this step
      const double Tz = k.G_T == 0.0 ? k.T_ref : k.T_ref + k.G_T * ((double)z - k.z_T - k.V_T * (double)step);
      const double B1 = k.B11 + k.B12 * Tz, B2 = k.B21 + k.B22 * Tz;
      const double s1 = B1, s2 = -B1 - B2, s3 = -B1 + B2;
      double w1[K + 2], w2[K + 2], wm[K + 2];  // the strip's column, rows iy0-1 .. iy0+K
#pragma unroll
      for (int r = 0; r < K + 2; ++r) {
        const int e = e0 + (r - 1) * C::BXin;
        w1[r] = c1[e];
        w2[r] = c2[e];
        wm[r] = mu[e];
      }
#pragma unroll
      for (int r = 0; r < K; ++r) {
        const int e = e0 + r * C::BXin;
        const double p1 = w1[r + 1], p2 = w2[r + 1], m0 = wm[r + 1], p3 = (1.0 - p1) - p2;
        const double d12 = p1 - p2, d23 = p2 - p3, d31 = p3 - p1;
        const double p1s = p1 * p1, p2s = p2 * p2, p3s = p3 * p3;
        // chemical driving forces (fcphi, TiAg.cu:514-516): gp2(pi, pj, pk) =
        // Q_i (pj - pk), Q_i = 7.5 (p_i - 1) p_i^2, and gp1(pi, pj, pk) = G_i =
        // 3.75 p_i (3 p_i^3 - 4 p_i^2 - p_i + 2 + (3 p_i - 2)(pj - pk)^2)
        const double Q1 = fma(p1, 7.5, -7.5) * p1s, Q2 = fma(p2, 7.5, -7.5) * p2s, Q3 = fma(p3, 7.5, -7.5) * p3s;
        auto G = [](double p, double d) {
          const double a = fma(fma(fma(p, 11.25, -15.0), p, -3.75), p, 7.5);
          return p * fma(fma(p, 11.25, -7.5), d * d, a);
        };
        const double G1 = G(p1, d23), G2 = G(p2, d31), G3 = G(p3, d12);
        const double o1w = fma(m0, -k.r1, s1), o2w = fma(m0, -k.r2, s2), o3w = fma(m0, -k.r3, s3);
        const double A = Q1 * d23 * o1w, Bq = Q2 * d31 * o2w, Cq = Q3 * d12 * o3w;
        // multi-well terms (fphi, TiAg.cu:522-527) with their shared factors
        const double s12 = p1 * p2, s13 = p1 * p3, s23 = p2 * p3;
        const double k2 = 2.0 * k.a2 * fma(s13, 3.0, p2 * fma(p2, k.b, 3.0));
        const double k3 = 2.0 * k.a3 * fma(s12, 3.0, p3 * fma(p3, k.b, 3.0));
        auto dw = [](double p) { return fma(fma(p, 4.0, -6.0), p, 2.0) * p; };  // 2p(1-p)(1-2p)
        double F1 = fma(p1 * p3s, k2, dw(p1));
        F1 = fma(p1 * p2s, k3, F1);
        F1 = fma(fma(G1, o1w, Cq - Bq), k.lam, F1);
        double F2 = fma(s13 * s13, fma(p2, 2.0 * k.b, 3.0) * k.a2, dw(p2));
        F2 = fma(p2 * p1s, k3, F2);
        F2 = fma(fma(G2, o2w, A - Cq), k.lam, F2);
        double F3 = fma(p3 * p1s, k2, dw(p3));
        F3 = fma(s12 * s12, fma(p3, 2.0 * k.b, 3.0) * k.a3, F3);
        F3 = fma(fma(G3, o3w, Bq - A), k.lam, F3);
        if constexpr (A1) {
          const double k1 = 2.0 * k.a1 * fma(s23, 3.0, p1 * fma(p1, k.b, 3.0));
          F1 = fma(s23 * s23, fma(p1, 2.0 * k.b, 3.0) * k.a1, F1);
          F2 = fma(p2 * p3s, k1, F2);
          F3 = fma(p3 * p2s, k1, F3);
        }
        // neighbours
        const double x1p = c1[e + 1], x1m = c1[e - 1], x2p = c2[e + 1], x2m = c2[e - 1];
        const double z1p = u1[e], z1m = d1[e], z2p = u2[e], z2m = d2[e];
        auto lap = [&](double p, double xp, double xm, double yp, double ym, double zp, double zm) {
          const double l = fma(fma(p, -2.0, yp + ym), k.dyi2, fma(p, -2.0, xp + xm) * k.dxi2);
          return fma(fma(p, -2.0, zp + zm), k.dzi2, l);
        };
        const double lap1 = lap(p1, x1p, x1m, w1[r + 2], w1[r], z1p, z1m);
        const double lap2 = lap(p2, x2p, x2m, w2[r + 2], w2[r], z2p, z2m);
        // phi_i' = phi_i + dt lap_i - dt (2 F_i - F_j - F_k) / 3 with mu_i = F_i - lap_i
        // and lap_3 = -lap_1 - lap_2 (TiAg.cu:529-537)
        const double T3 = ((F1 + F2) + F3) * (k.dt * (1.0 / 3.0));
        const double n1 = p1 + fma(lap1 - F1, k.dt, T3);
        const double n2 = p2 + fma(lap2 - F2, k.dt, T3);
        // solute: face mobility (phi1 + phi1') / 2 (+ solid terms), TiAg.cu:543-552
        auto mob = [&](double q1, double q2) {
          double m = p1 + q1;
          if constexpr (SD) m = fma(((p3 + 1.0) - q1) - q2, k.Db2, fma(p2 + q2, k.Da2, m));
          return m;
        };
        auto face2 = [&](double qp1, double qp2, double mp, double qm1, double qm2, double mm) {
          return fma(mob(qp1, qp2), mp - m0, mob(qm1, qm2) * (mm - m0));
        };
        double dc = face2(x1p, x2p, mu[e + 1], x1m, x2m, mu[e - 1]) * k.cfx;
        dc = fma(face2(w1[r + 2], w2[r + 2], wm[r + 2], w1[r], w2[r], wm[r]), k.cfy, dc);
        dc = fma(face2(z1p, z2p, muu[e], z1m, z2m, mud[e]), k.cfz, dc);
        store_cell(r, n1, n2, cc[e] + dc);
      }
    }
    // the last warp that leaves plane z hands the slot of plane z-1 to the load
    // of plane z+5, without waiting for plane z+2 first: four loads in flight
    __syncwarp();
    if (lane == 0 && arrive_count(&sm.passed) % (C::kThreads / 32) == C::kThreads / 32 - 1 && z + C::kSlots - 1 <= zin1)
      issue(z + C::kSlots - 1);
  }
}

// mu of every cell with image ghost layers (rs3_mu)
// (FP32 sets hold c - c_off: c_off is added back here and in the mass)
template <typename R>
__global__ void __launch_bounds__(256) peri3d_mu_kernel(const K3<R> k, const R *__restrict__ f1,
                                                        const R *__restrict__ f2, const R *__restrict__ fc,
                                                        R *__restrict__ mu, const double c_off) {
  const int64_t n = (int64_t)k.nx * k.ny * k.nz;
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    int x = (int)(i % k.nx), y = (int)((i / k.nx) % k.ny), z = (int)(i / ((int64_t)k.nx * k.ny));
    // image of a ghost cell: periodic x, y; no-flux z
    x = x == 0 ? k.nx - 2 : (x == k.nx - 1 ? 1 : x);
    y = y == 0 ? k.ny - 2 : (y == k.ny - 1 ? 1 : y);
    z = z == 0 ? 1 : (z == k.nz - 1 ? k.nz - 2 : z);
    const int64_t j = ((int64_t)z * k.ny + y) * k.nx + x;
    mu[i] = (R)((double)mu_of(k, f1[j], f2[j], fc[j]) + c_off);
  }
}

template <typename R>
__global__ void __launch_bounds__(256) peri3d_mass_kernel(const K3<R> k, const R *__restrict__ fc,
                                                          double *__restrict__ partial, const double c_off) {
  double s = 0.0;
  const int64_t nxi = k.nx - 2, nyi = k.ny - 2, n = nxi * nyi * (k.nz - 2);
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t x = 1 + i % nxi, y = 1 + (i / nxi) % nyi, z = 1 + i / (nxi * nyi);
    s += (double)fc[(z * k.ny + y) * k.nx + x] + c_off;
  }
  __shared__ double sh[8];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) s += __shfl_down_sync(0xffffffffu, s, o);
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += sh[w];
    partial[blockIdx.x] = t;
  }
}

__global__ void peri3d_sum_kernel(const double *__restrict__ partial, int n, double *__restrict__ out) {
  if (threadIdx.x == 0 && blockIdx.x == 0) {
    double t = 0.0;
    for (int i = 0; i < n; ++i) t += partial[i];
    *out = t;
  }
}

// initial state (rs3_initial); one thread per (x, y) column of the interior
template <typename R>
__global__ void peri3d_init_kernel(const K3<R> k, const P3Init ini, R *__restrict__ f1, R *__restrict__ f2,
                                   R *__restrict__ fc, const double c_off) {
  const int x = 1 + blockIdx.x * blockDim.x + threadIdx.x, y = 1 + blockIdx.y;
  if (x > k.nx - 2 || y > k.ny - 2) return;
  uint32_t r[4] = {(uint32_t)x, (uint32_t)y, 0u, 0x5A465254u};
  philox4x32(r, (uint32_t)ini.seed, (uint32_t)(ini.seed >> 32));
  const double zc = ini.z_front + ini.amp * (2.0 * u53(r[0], r[1]) - 1.0);
  const int64_t plane = (int64_t)k.nx * k.ny;
  for (int z = 1; z <= k.nz - 2; ++z) {
    bool cap = false;
    if (z >= zc)
      for (int c = 0; c < ini.n_alpha; ++c) {
        const double dx = x - ini.cx[c], dy = y - ini.cy[c], dz = z - (ini.z_front - ini.roff);
        if (dx * dx + dy * dy + dz * dz <= ini.radius * ini.radius) cap = true;
      }
    const int64_t o = (int64_t)z * plane + (int64_t)y * k.nx + x;
    if (cap) {
      f1[o] = R(0);
      f2[o] = R(1);
      fc[o] = (R)(ini.ca - c_off);
    } else if (z < zc) {
      f1[o] = R(0);
      f2[o] = R(0);
      fc[o] = (R)(ini.cb - c_off);
    } else {
      f1[o] = R(1);
      f2[o] = R(0);
      fc[o] = (R)(ini.clb - c_off);
    }
  }
}

// ghost layers as images, in the reference's order (x, then y, then z)
template <typename R>
__global__ void peri3d_ghost_kernel(const K3<R> k, int axis, R *__restrict__ f1, R *__restrict__ f2,
                                    R *__restrict__ fc) {
  const int a = blockIdx.x * blockDim.x + threadIdx.x, bidx = blockIdx.y;
  const int64_t plane = (int64_t)k.nx * k.ny;
  int64_t d0, s0, d1, s1;
  if (axis == 0) {  // (y, z) = (a, bidx)
    if (a >= k.ny || bidx >= k.nz) return;
    const int64_t base = (int64_t)bidx * plane + (int64_t)a * k.nx;
    d0 = base;
    s0 = base + k.nx - 2;
    d1 = base + k.nx - 1;
    s1 = base + 1;
  } else if (axis == 1) {  // (x, z)
    if (a >= k.nx || bidx >= k.nz) return;
    const int64_t base = (int64_t)bidx * plane + a;
    d0 = base;
    s0 = base + (int64_t)(k.ny - 2) * k.nx;
    d1 = base + (int64_t)(k.ny - 1) * k.nx;
    s1 = base + k.nx;
  } else {  // (x, y)
    if (a >= k.nx || bidx >= k.ny) return;
    const int64_t base = (int64_t)bidx * k.nx + a;
    d0 = base;
    s0 = base + plane;
    d1 = base + (int64_t)(k.nz - 1) * plane;
    s1 = base + (int64_t)(k.nz - 2) * plane;
  }
  f1[d0] = f1[s0];
  f2[d0] = f2[s0];
  fc[d0] = fc[s0];
  f1[d1] = f1[s1];
  f2[d1] = f2[s1];
  fc[d1] = fc[s1];
}

int launch_step(const rs3_params &p, const P3Maps &m, double *o1, double *o2, double *oc, int64_t step, int *err,
                cudaStream_t st) {
  using C = D3;
  K3<double> k = make_k3<double>(p);
  const size_t smem = sizeof(P3Smem) + 128;
  const bool a1 = p.a1 != 0.0, sd = p.Da != 0.0 || p.Db != 0.0;
  auto kfn = a1 ? (sd ? peri3d_kernel<true, true> : peri3d_kernel<true, false>)
                : (sd ? peri3d_kernel<false, true> : peri3d_kernel<false, false>);
  static std::atomic<unsigned long long> attr[4];
  if (!smem_limit_once((const void *)kfn, (int)smem, attr[(a1 ? 2 : 0) + (sd ? 1 : 0)])) return -3;
  dim3 grid((p.nx - 2 + C::BX - 1) / C::BX, (p.ny - 2 + C::BY - 1) / C::BY);
  k.z_chunk = p3_chunk(p, (int64_t)grid.x * grid.y, 2, false);
  grid.z = (p.nz - 2 + k.z_chunk - 1) / k.z_chunk;
  return launch_dep_smem(kfn, grid, dim3(C::kThreads), smem, st, k, m.phi1, m.phi2, m.c, o1, o2, oc, step, err) ==
                 cudaSuccess
             ? 0
             : -3;
}

}  // namespace

double peri3d_c_offset(const rs3_params &p) {  // clb at T_ref (TiAg.cu:67); c_ref for energy 1
  if (p.energy == 1) return p.c_ref;
  const double B1 = p.B11 + p.B12 * p.T_ref, B2 = p.B21 + p.B22 * p.T_ref;
  return (B1 - 0.5 * B2) / (p.A1 - 0.5 * p.A2) + p.A1;
}

int peri3d_box_width(int precision) { return precision == RS_F64 ? D3::BXin : peri3d_x2_box_width(); }
int peri3d_box_height(int precision) { return precision == RS_F64 ? D3::BYin : peri3d_x2_box_height(); }

int launch_peri3d_step(const rs3_params &p, const P3Maps &m, int precision, void *o1, void *o2, void *oc,
                       int64_t step, int *err, cudaStream_t st) {
  if (precision == RS_F64)
    return launch_step(p, m, (double *)o1, (double *)o2, (double *)oc, step, err, st);
  return launch_peri3d_step_x2(p, m, (float *)o1, (float *)o2, (float *)oc, step, err, st);
}

int launch_peri3d_mu(const rs3_params &p, int precision, const void *f1, const void *f2, const void *fc, void *mu,
                     cudaStream_t st) {
  const int64_t n = (int64_t)p.nx * p.ny * p.nz;
  const unsigned blocks = (unsigned)std::min<int64_t>((n + 255) / 256, 148 * 16);
  if (precision == RS_F64)
    peri3d_mu_kernel<double><<<blocks, 256, 0, st>>>(make_k3<double>(p), (const double *)f1, (const double *)f2,
                                                     (const double *)fc, (double *)mu, 0.0);
  else
    peri3d_mu_kernel<float><<<blocks, 256, 0, st>>>(make_k3<float>(p), (const float *)f1, (const float *)f2,
                                                    (const float *)fc, (float *)mu, peri3d_c_offset(p));
  return 0;
}

int launch_peri3d_mass(const rs3_params &p, int precision, const void *fc, double *partial, int nparts, double *out,
                       cudaStream_t st) {
  if (precision == RS_F64)
    peri3d_mass_kernel<double><<<nparts, 256, 0, st>>>(make_k3<double>(p), (const double *)fc, partial, 0.0);
  else
    peri3d_mass_kernel<float><<<nparts, 256, 0, st>>>(make_k3<float>(p), (const float *)fc, partial,
                                                      peri3d_c_offset(p));
  peri3d_sum_kernel<<<1, 32, 0, st>>>(partial, nparts, out);
  return 0;
}

int launch_peri3d_init(const rs3_params &p, int precision, const P3Init &ini, void *f1, void *f2, void *fc,
                       cudaStream_t st) {
  const dim3 g((p.nx - 2 + 127) / 128, p.ny - 2);
  if (precision == RS_F64)
    peri3d_init_kernel<double><<<g, 128, 0, st>>>(make_k3<double>(p), ini, (double *)f1, (double *)f2, (double *)fc,
                                                  0.0);
  else
    peri3d_init_kernel<float><<<g, 128, 0, st>>>(make_k3<float>(p), ini, (float *)f1, (float *)f2, (float *)fc,
                                                 peri3d_c_offset(p));
  return launch_peri3d_ghosts(p, precision, f1, f2, fc, st);
}

int launch_peri3d_ghosts(const rs3_params &p, int precision, void *f1, void *f2, void *fc, cudaStream_t st) {
  const int ext[3][2] = {{p.ny, p.nz}, {p.nx, p.nz}, {p.nx, p.ny}};
  for (int axis = 0; axis < 3; ++axis) {
    const dim3 gg((ext[axis][0] + 127) / 128, ext[axis][1]);
    if (precision == RS_F64)
      peri3d_ghost_kernel<double><<<gg, 128, 0, st>>>(make_k3<double>(p), axis, (double *)f1, (double *)f2,
                                                      (double *)fc);
    else
      peri3d_ghost_kernel<float><<<gg, 128, 0, st>>>(make_k3<float>(p), axis, (float *)f1, (float *)f2, (float *)fc);
  }
  return 0;
}

}  // namespace rs
