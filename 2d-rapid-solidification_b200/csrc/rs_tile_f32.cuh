// rs_tile_f32.cuh — the FP32 fused phase-field step on TMA-staged tiles: the
// phases (tile_body) and the one-tile-per-CTA kernels.  Included by rs_step_f32.cu
// (the column table, the exact kernels of aligned fields, the launch), the other
// rs_step_f32_*.cu and, by way of rs_ens_tile.cuh, the rs_ensemble*.cu.
//
// Same equations as the register-prefetch kernel of rs_step.cu
// (compute_phi / compute_psi / compute_c_CALPHAD, fun.cu:1143-1467).  One
// step is two launches:
//   * column_table_kernel: the per-column CALPHAD groups of this step's frozen
//     temperature (t_terms in FP64, get_delta fun.cu:1610-1619), rounded to
//     FP32, plus the FP64 column differences of the composition-independent
//     part of mu;
//   * tile_kernel.
// Both are programmatic dependent launches: they are scheduled while the
// kernel before them drains and wait for it on the device, so a run's steps
// follow one another without launch gaps.
//
// A CTA of 128 threads owns a tile of TR output rows x 128 output columns
// (x0 .. x0+127, x0 a multiple of 128; TR = 4, 8 or 16 by tile_rows_f32, 32 in
// ensembles too).  Its input, TR + 2 rows x 136 columns (x0-4 .. x0+131, so the
// TMA x coordinate stays 16-byte aligned), arrives in shared memory by one TMA
// box per field.  Four adjacent columns per lane.  The CTA votes on the tile's
// form: a tile of far melt takes its c update from registers straight to
// global memory, one of deep solid is copied; any other takes the phases:
//   phase 1  per-cell S = q(psi) c (1-c) and mu'' (below) of the input
//            rows into shared memory, with per-row flags "every psi == -1" /
//            "== +1" and per-lane phi masks; the halo columns x0-1 and
//            x0+128 are computed by 36 threads of warps 2 and 3 (one input
//            row fewer than warps 0 and 1);
//   phase 2  each warp computes its output rows: fluxes through the faces from
//            the shared S and mu'', the c update (kept in registers); cells
//            whose 3x3 phi neighbourhood is not uniformly +-1 are listed,
//            those that draw noise apart from the others;
//   phase 3  the listed interface cells are updated one per thread
//            (phi_cell), so a tile's interface work is spread over the CTA;
//   phase 4  new psi and c are written into the shared tile, ghost columns
//            copied there, and each output row leaves by one bulk async copy
//            per field (ghost rows by one more, except in row-band mode);
//   partials when the caller wants the solute mass or the coarse tip, each
//            CTA writes its partial sums and a dependent launch reduces them.
// What bounds it: a 2048^2 grid ahead of a planar front (20.6 us a step, 23.7
// without the melt form and the chained launches; floor 10.3, a plain copy of
// its fields by this tiling 17.3) its instruction issue (1150 instructions a
// warp for 512 cells of far melt, half of them arithmetic) and the chain of a
// CTA; small grids (256^2: 6.1 us, 12.0 with 16-row tiles) and fronts the chain
// of the phases.
// Arithmetic:
//   * mu = K(T) + C0(T) + mu'' with C0 = -D - (L0_BCC - L0_Liq)(1 - 2 cinf)/2
//     (D, K(T) as in rs_step.cu), so
//       mu'' = -(g+1) C0 - delta (L0_BCC + L0_Liq + g (L0_BCC - L0_Liq)) + RT lam,
//     which is small in the melt; K + C0 enters only through its FP64 column
//     differences dK;
//   * rows whose cells are all bulk liquid (psi = -1 exactly, |s| < 1/9) take
//     the short form: g(-1) = -1 and q(-1) = 1, so
//     mu'' = -2 L0_Liq delta + RT lam(delta) and S = c (1 - c);
//   * rows whose cells have psi = +1 exactly over their 3x3 neighbourhoods
//     (deep solid) store S = mu'' = 0: q(1) = 0, so every face weight touching
//     the row is 0 and its mu'' enters no flux (no network pass either);
//   * face weights use pair sums: the face (i, r+1/2) has
//     6 P_i + P_{i-1} + P_{i+1} with P_i = S(i,r) + S(i,r+1), and the face
//     (i+1/2, r) has 6 Q_r + Q_{r-1} + Q_{r+1} with Q_r = S(i,r) + S(i+1,r):
//     four times the 1.5 / 0.25 weights of rs_step.cu, the 4 folded into the
//     flux constant; face fluxes are rounded products, so a cell's result
//     does not depend on where the tiling puts it;
//   * interface noise is keyed by the global cell (row + j_offset in
//     row-band mode).
// Launch order: the tile columns from the one holding the front
// (front_first_block), whose interface and network work is the slowest.
// Once its own tile has arrived each CTA prefetches into L2 the input tile of
// the block launched one resident wave later, so the tiles of the next wave
// arrive while this wave computes (the CTAs of a wave otherwise load, compute
// and store in step).
// The coarse-grid temperature (TFC, interpolate_temperature fun.cu:1580-1608)
// takes tile_kernel_tfc alone: every cell evaluates its CALPHAD groups from its
// own bilinear temperature (K + C0 by its Taylor polynomial about the tile's
// centre temperature, kc_poly), keeps K + C0 in FP64 in shared memory, and the
// faces add its differences, rounded to FP32, along both axes; tiles of 8
// output rows, so that the FP64 array fits with five CTAs per SM.  Its only
// whole-tile form is the deep solid one.
// Fields store psi and delta = c - cinf (include/rs_b200.h).
#pragma once

#include <type_traits>

#include "rs_step_common.cuh"
#include "rs_surrogate.cuh"

namespace rs {
namespace {

constexpr int kW = kTileOutW;     // output columns of a tile
constexpr int kWin = kTmaBoxW32;  // input columns of a tile (kW + 8)
constexpr int kTR = kTileRows;    // output rows of a tile
constexpr int kTRin = kTmaBoxH;   // input rows of a tile
constexpr int kThreads = 128;
constexpr int kWarps = kThreads / 32;
constexpr int kRowsPerWarp = kTR / kWarps;
constexpr int kHaloL = 3, kHaloR = kW + 4;  // box columns of x0-1 and x0+kW
constexpr uint32_t kWaitLimit = 1u << 20;
constexpr unsigned FULL = 0xffffffffu;
static_assert(kW == 32 * 4, "four columns per lane");
static_assert(kTR % kWarps == 0 && kRowsPerWarp == 4, "four output rows per warp");
static_assert(kTRin <= 32, "row flags are 32-bit masks");
static_assert(64 + 2 * kTRin <= kThreads && 4 * kTR <= kThreads, "one thread per halo cell and per row copy");

// column table arrays (kColTabFields of them, col_tab_len floats each);
// entry k describes column k - 4
enum { kTabRT = 0, kTabC0 = 1, kTabDK = 2, kTabAnb = 3, kTabAti = 4 };

// Shared memory of one tile of TR output rows x kW output columns (input
// TR + 2 rows); the ensemble kernels take TR = 8, 16 or 32 (kTileShapes), the
// single-run kernels TR = 4, 8 or 16 (tile_rows_f32) and, with the coarse-grid
// temperature, kTfcTileRows32.
template <int TR, bool TFC = false>
struct alignas(128) TileSmemT {
  static constexpr int kRin = TR + 2;  // input rows
  using Mask = std::conditional_t<(kRin <= 32), uint32_t, unsigned long long>;  // one bit per input row
  // TMA destinations (128-byte aligned); rows 1..TR receive the new psi / c - cinf
  alignas(128) float psi[kRin][kWin];
  alignas(128) float d[kRin][kWin];
  alignas(16) float S[kRin][kWin];  // after phase 2: new psi of the listed cells
  alignas(16) float mu[kRin][kWin];
  // TFC: K + C0 of every cell in FP64 (the face terms are its differences)
  alignas(16) double kc[TFC ? kRin : 1][TFC ? kWin : 2];
  // interface cells (row << 8 | output column): those that draw noise from the
  // front, the others from the back, so that phase 3's warps are of one kind
  uint16_t list[TR * kW];
  uint8_t pmask[kRin][32];  // per lane: bits 0-3 psi <= -1, bits 4-7 psi >= 1 of its four cells
  uint8_t hmask[kRin][2];   // halo cells: bit 0 psi <= -1, bit 1 psi >= 1
  Mask liq, sol;            // bit r: every cell of input row r has psi == -1 / +1
  double ty[kRin];          // TFC: the row part of each input row's temperature
  int tj[kRin];             // (tfc_row), once per tile
  std::conditional_t<TFC, KcPoly, char> kp;  // TFC: K + C0 near the tile's temperature
  double hx[2];             // TFC: column part of the halo columns' temperatures
  int hiT[2];
  uint32_t nlist;  // how many of the first kind, and << 16 of the second
  uint32_t vote;   // the tile's form, OR of every thread's
  double part_mass[kWarps];
  int part_itip[kWarps];
  uint64_t full;
};
using TileSmem = TileSmemT<kTR>;

static_assert(offsetof(TileSmem, psi) % 128 == 0 && offsetof(TileSmem, d) % 128 == 0 &&
                  offsetof(TileSmemT<8>, d) % 128 == 0 && offsetof(TileSmemT<32>, d) % 128 == 0,
              "TMA destinations start on 128-byte boundaries");
static_assert((kWin * sizeof(float)) % 16 == 0, "rows stay 16-byte aligned for float4 and bulk copies");

__device__ __forceinline__ float4 ld4(const float *p) { return *reinterpret_cast<const float4 *>(p); }
__device__ __forceinline__ void st4(float *p, float a, float b, float c, float e) {
  *reinterpret_cast<float4 *>(p) = make_float4(a, b, c, e);
}
__device__ __forceinline__ float clamp1(float v) { return fminf(fmaxf(v, -1.f), 1.f); }

// general per-cell terms (fun.cu:1424-1452)
__device__ __forceinline__ void cell_terms(const Coef<float> &F, float pv, float dv, float RT, float C0, float &S,
                                           float &mu) {
  constexpr float L0sum = (float)(kL0Bcc + kL0Liq);
  constexpr float L0half = (float)(0.5 * (kL0Bcc - kL0Liq));
  const float c = F.cinf + dv, om = 1.f - c;
  const float a = 1.f - pv;
  S = (0.5f * F.AA * a - 0.25f * (F.AA - 1.f) * (a * a)) * c * om;
  const float p2 = pv * pv;
  const float g = pv * (1.875f + p2 * (-1.25f + 0.375f * p2));
  const float lam = Tr<float>::lam(c, om, dv, F.cinf, F.Lref);
  mu = -(g + 1.f) * C0 - dv * fmaf(2.f * L0half, g, L0sum) + RT * lam;
}

// A far-melt cell (psi = -1 exactly, |delta| <= melt_tiny): g = -1, q = 1, lam
// by its Taylor polynomial in delta (Coef::melt_a);
// mu'' = RT lam - 2 L0_Liq delta = delta (RT p + KL), lam = delta p.  Rounded
// products: the phases and the melt tiles give the same bits.
// M: its constants in registers (an ensemble's live in global memory, where
// the tile's own stores would have them read again for every row)
struct MeltC {
  float cinf, tiny, a0, a1, a2, a3;
  __device__ explicit MeltC(const Coef<float> &F)
      : cinf(F.cinf), tiny(F.melt_tiny), a0(F.melt_a[0]), a1(F.melt_a[1]), a2(F.melt_a[2]), a3(F.melt_a[3]) {}
};
__device__ __forceinline__ void far_cell(const MeltC &M, float dv, float RT, float &S, float &mu) {
  constexpr float KL = (float)(-2.0 * kL0Liq);
  const float c = M.cinf + dv, om = 1.f - c;
  float p = fmaf(M.a3, dv, M.a2);
  p = fmaf(p, dv, M.a1);
  p = fmaf(p, dv, M.a0);
  S = __fmul_rn(c, om);
  mu = __fmul_rn(dv, fmaf(RT, p, KL));
}
// A bulk-melt cell (psi = -1 exactly, delta in the series range): mu'' =
// -2 L0_Liq delta + RT 2 atanh(s), atanh to s^7 (relative truncation below
// 2.6e-9 for |s| < 1/9).
__device__ __forceinline__ void bulk_cell(const MeltC &M, float dv, float RT, float &S, float &mu) {
  constexpr float KL = (float)(-2.0 * kL0Liq);
  const float c = M.cinf + dv, om = 1.f - c;
  const float sv = __fdividef(dv, fmaf(M.cinf + M.cinf, om, dv));
  const float s2 = sv * sv;
  float p = fmaf(s2, 1.f / 7.f, 1.f / 5.f);
  p = fmaf(s2, p, 1.f / 3.f);
  const float ath = fmaf(sv * s2, p, sv);  // atanh(s); lam = 2 atanh(s)
  S = __fmul_rn(c, om);
  mu = fmaf(RT + RT, ath, __fmul_rn(dv, KL));
}
// a cell of the halo columns: the far-melt form where the cell has it, else
// the general one (a cell's form does not depend on the tile)
__device__ __forceinline__ void halo_cell(const Coef<float> &F, const MeltC &M, float pv, float dv, float RT, float C0,
                                          float &S, float &mu) {
  if (__float_as_uint(pv) == 0xBF800000u && fabsf(dv) <= M.tiny)
    far_cell(M, dv, RT, S, mu);
  else
    cell_terms(F, pv, dv, RT, C0, S, mu);
}

// shared -> global bulk copy (16-byte aligned addresses, size a multiple of 16)
__device__ __forceinline__ void bulk_store(void *gdst, const void *ssrc, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_u32(ssrc)),
               "r"(bytes)
               : "memory");
}

// One thread per column, one t_terms each (c/T terms by one reciprocal: the
// groups are rounded to FP32); K + C0 of the next column comes from the
// neighbouring thread, so blocks overlap by one column and write 127 entries.
constexpr int kTabBlock = 128;
// kc: kTabBlock doubles of shared scratch
// (griddepcontrol.wait before the table is written: the previous step's tiles
// have read it)
__device__ __forceinline__ void table_block(const StepCoef &K, const double d0, const double d1, const int len,
                                            float *__restrict__ tab, const int blk, double *kc) {
  const int k = blk * (kTabBlock - 1) + threadIdx.x;  // table entry; column k - 4
  const int gi = min(max(k - 4, 0), K.nx - 1);
  const double T = (d0 + d1 * gi) * K.deltaT0 + K.Tmelt;  // get_delta, fun.cu:1610-1619
  const TTerms tt = t_terms(T, K.RR, true);
  const double D = 0.5 * (tt.dGs - tt.dGl);
  const double C0 = -D - 0.5 * (kL0Bcc - kL0Liq) * (1.0 - 2.0 * K.cinf);
  kc[threadIdx.x] = 0.5 * (tt.dGs + tt.dGl) + 0.5 * (kL0Bcc + kL0Liq) * (1.0 - 2.0 * K.cinf) + tt.RT * K.Lref + C0;
  __syncthreads();
  pdl_wait();
  if (threadIdx.x == kTabBlock - 1 || k >= len) return;
  tab[kTabRT * len + k] = (float)tt.RT;
  tab[kTabC0 * len + k] = (float)C0;
  tab[kTabDK * len + k] = (float)(kc[threadIdx.x + 1] - kc[threadIdx.x]);  // (K + C0)(i+1) - (K + C0)(i)
  tab[kTabAnb * len + k] = (float)tt.A_nb;
  tab[kTabAti * len + k] = (float)tt.A_ti;
}

// SURR: mu'' and the driving force of in-box cells that are not bulk melt
// come from the learned surrogate (rs_surrogate.cuh) instead of the exact
// evaluation.  Bulk-melt cells (psi == -1 exactly, delta in the series range)
// keep the exact series form: it is exact and cheaper than the network.
// The work of one CTA on tile (row tile tr, column tile tc) of a field set;
// part: this tile's partial (mass, coarse tip), or nullptr.
// TR: output rows of the tile (8, 16 or 32; the tensor maps' box is TR + 2
// rows high).
// RAW: the fields' rows are not 16-byte aligned (any nx).
// AR: the surrogate's counters take every network cell as often as tiles of AR
// rows read its row (twice where two of them do), whatever TR is.
template <bool SURR, int TR, typename Prefetch, bool TFC = false, bool RAW = false, int AR = TR>
__device__ __forceinline__ void tile_body(const StepCoef &K, const Coef<float> &F, const StepScalars &PS,
                                          const CUtensorMap *tm_psi, const CUtensorMap *tm_c,
                                          const float *__restrict__ tab, const int tab_len, float *__restrict__ psi_n,
                                          float *__restrict__ c_n, float *__restrict__ phi_n, BlockPartial *part,
                                          int *err, const SurrArgs &SA, const int tr, const int tc,
                                          const Prefetch &prefetch) {
  // the tile's shape (these hide the single-run constants of the same names)
  constexpr int kTR = TR, kTRin = TR + 2, kRowsPerWarp = TR / kWarps;
  static_assert(TR % kWarps == 0 && kRowsPerWarp * 4 <= 32, "output rows split evenly over the warps");
  // halo-column threads: the last warps, which have one input row fewer
  constexpr int kHalo0 = (64 + 2 * kTRin <= kThreads) ? 64 : kThreads - 2 * kTRin;
  static_assert(kHalo0 >= 0 && 4 * kTR <= kThreads, "one thread per halo cell and per row copy");
  static_assert(!(SURR && TFC), "the surrogate takes the frozen temperature");
  using Smem = TileSmemT<TR, TFC>;
  using Mask = typename Smem::Mask;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  Smem &sm = *reinterpret_cast<Smem *>(smem_raw);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int x0 = kW * tc;       // first output column of the tile
  const int y0 = 1 + kTR * tr;  // first output row; input rows y0-1 .. y0+kTR
  constexpr uint32_t kTileBytes = 2u * kTRin * kWin * sizeof(float);

  if (smem_u32(smem_raw) & 127u) {  // TMA destinations must be 128-byte aligned
    if (threadIdx.x == 0) atomicExch(err, 2);
    return;
  }
  // a pull-back step reads column clamp(i + i_offset, 1, nx - 2) for column i
  // (pull_back, fun.cu:1469-1492): no TMA box has that shape, so the CTA
  // gathers its tile instead (same box, zeros outside the array, delta = 0
  // where the source is column nx - 2: the melt entering at the right edge)
  // (and so it does on rows that are not 16-byte aligned, unshifted)
  const bool pb = RAW || PS.pull_back != 0;
  if (threadIdx.x == 0) {
    mbar_init(&sm.full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sm.liq = 0;
    sm.sol = 0;
    sm.nlist = 0u;
    sm.vote = 0u;
  }

  const int col = 4 * lane;  // tile column of this lane's first cell
  const int gi = x0 + col;   // its global column
  const int bc = col + 4;    // its box column
  uint32_t outm = 0;         // per cell: an interior (output) cell
#pragma unroll
  for (int q = 0; q < 4; ++q)
    if (gi + q >= 1 && gi + q <= K.nx - 2) outm |= 1u << q;
  // launch constants of the row loops in registers (one read of the
  // arguments, which may live in global memory for the ensemble)
  const int ny = K.ny, nx = K.nx;
  const MeltC M(F);
  const float tiny = M.tiny;
  const float cflux4 = 0.25f * F.cflux;
  const float floor_d = F.c_floor - F.cinf;
  const float d_hi = F.ser_hi, d_lo = F.ser_lo;  // series range of delta (Coef)
  constexpr uint32_t kMinus1 = 0xBF800000u, kPlus1 = 0x3F800000u;

  // the kernel before this one in the stream (the column table's, and with it
  // every earlier one) has completed: its table and the fields are visible
  pdl_wait();
  if (threadIdx.x == 0 && !pb) {
    mbar_expect_tx(&sm.full, kTileBytes);
    tma_load_2d(&sm.psi[0][0], tm_psi, &sm.full, x0 - 4, y0 - 1);
    tma_load_2d(&sm.d[0][0], tm_c, &sm.full, x0 - 4, y0 - 1);
  }
  // dependents of this step (its reduction, the next step) may be scheduled now,
  // or (late) once the tile's listed cells are done
  if (!PS.late) pdl_trigger();
  const float *tRT = tab + kTabRT * tab_len + 4, *tC0 = tab + kTabC0 * tab_len + 4;
  const float *tDK = tab + kTabDK * tab_len + 4;
  float4 RTv = make_float4(0.f, 0.f, 0.f, 0.f), C0v = RTv, dKv = RTv;
  float dKl = 0.f;
  if constexpr (!TFC) {
    RTv = ld4(tRT + gi);
    C0v = ld4(tC0 + gi);
  }
  if constexpr (!TFC && !SURR) {
    // dK of the lane's faces, loaded now so that the load hides under the
    // tile's (the surrogate path, short of registers, loads them after phase 1)
    dKv = ld4(tDK + gi);
    dKl = tDK[gi - 1];
  }
  // TFC: RT and C0 per row, from each cell's own temperature
  float RTa[4] = {RTv.x, RTv.y, RTv.z, RTv.w}, C0a[4] = {C0v.x, C0v.y, C0v.z, C0v.w};
  // TFC: the column part of each cell's temperature (interpolate_temperature,
  // fun.cu:1580-1608); the row part and K + C0 about the tile's centre once
  // per tile, in shared memory
  int tiT[4] = {0, 0, 0, 0};
  double tx[4] = {0.0, 0.0, 0.0, 0.0};
  if constexpr (TFC) {
#pragma unroll
    for (int q = 0; q < 4; ++q) tfc_col(K, PS.i_left_end_T, gi + q, tiT[q], tx[q]);
    if (threadIdx.x < kTRin) tfc_row(K, y0 - 1 + (int)threadIdx.x, sm.tj[threadIdx.x], sm.ty[threadIdx.x]);
    if (threadIdx.x >= kTRin + 1 && threadIdx.x < kTRin + 3) {  // the halo columns x0-1, x0+kW
      const int side = (int)threadIdx.x - (kTRin + 1);
      tfc_col(K, PS.i_left_end_T, side ? x0 + kW : x0 - 1, sm.hiT[side], sm.hx[side]);
    }
    if (threadIdx.x == 64 || threadIdx.x == 96) {
      int iT, jT;
      double x, y;
      tfc_col(K, PS.i_left_end_T, x0 + kW / 2, iT, x);
      tfc_row(K, y0 + kTR / 2, jT, y);
      const double T0 = tfc_T(K, PS.T_coarse, iT, x, jT, y);
      if (threadIdx.x == 64) kc_poly(K, T0, sm.kp);
      else drive_poly(T0, sm.kp);
    }
  }
  // TFC: all groups of one cell, the logarithm exact (halo and interface cells)
  auto tfc_cell = [&](int gx, int row) {
    int iT, jT;
    double x, y;
    tfc_col(K, PS.i_left_end_T, gx, iT, x);
    tfc_row(K, row, jT, y);
    return groups_exact(K, tfc_T(K, PS.T_coarse, iT, x, jT, y));
  };
  // surrogate: per-lane fragments, and the scaled inputs as T(x) = TnA + TnB x
  // (tile column x; frozen T is linear in the column) and c = cnA + delta c_ihalf
  float TnA = 0.f, TnB = 0.f, cnA = 0.f;
  const float *tAnb = tab + kTabAnb * tab_len + 4, *tAti = tab + kTabAti * tab_len + 4;
  if constexpr (SURR) {
    const double T0 = (PS.d0 + PS.d1 * x0) * K.deltaT0 + K.Tmelt;
    TnA = (float)((T0 - SA.T_mid) * SA.T_ihalf);
    TnB = (float)(PS.d1 * K.deltaT0 * SA.T_ihalf);
    cnA = (F.cinf - SA.c_mid) * SA.c_ihalf;
  }
  // a cell the series form covers (the network is not used there)
  auto melt_cell = [&](int rr, int b) {
    const float dv = sm.d[rr][b];
    return __float_as_uint(sm.psi[rr][b]) == kMinus1 && dv < d_hi && dv > d_lo;
  };
  // the counters' tiling (AR): the input rows of this tile that it reads too, and
  // whether its last tile holds rows beyond the array, whose zeros leave no cell
  // of row ny-1 deep solid
  static_assert(AR % TR == 0, "the counters' tiles hold whole ones");
  auto counted = [&](int rr) {
    if (AR == TR || (rr >= 1 && rr <= kTR)) return true;
    return rr == 0 ? (y0 - 1) % AR == 0 : (y0 - 1 + kTR) % AR == 0 || y0 + kTR == ny - 1;
  };
  const bool open_end = SURR && (ny - 2) % AR != 0;
  auto open_row = [&](int rr) { return open_end && rr == kTR + 1 && y0 + kTR == ny - 1; };
  // a halo cell's mu'' enters only the face to the tile's edge column, whose
  // weight is 0 when psi is exactly +1 on both columns over rows rr-1..rr+1;
  // column -1 (left-most tile) enters no face at all (column 0 is a ghost)
  auto halo_mu_used = [&](int rr, int b) {
    if (b == kHaloL && x0 == 0) return false;
    if constexpr (AR != TR)
      if (open_row(rr)) return true;
    const int b2 = b == kHaloL ? b + 1 : b - 1;
    bool solid = true;
    for (int r2 = max(rr - 1, 0); r2 <= min(rr + 1, kTRin - 1); ++r2)
      solid = solid && __float_as_uint(sm.psi[r2][b]) == kPlus1 && __float_as_uint(sm.psi[r2][b2]) == kPlus1;
    return !solid;
  };
  // per lane, bit q: psi is exactly +1 over the 3x3 neighbourhood of cell
  // bc+q (rows of the box only: faces to rows outside it are not computed;
  // column -1 of the left-most tile enters no face, column 0 being a ghost).
  // S = q(1) c (1 - c) = 0 there, so every face weight touching the cell is 0
  // and its mu'' enters no flux (0 times a finite difference)
  auto solid3 = [&](int rr) -> uint32_t {
    if constexpr (AR != TR)
      if (open_row(rr)) return 0u;  // (warp-uniform)
    const int xh = lane == 0 ? kHaloL : kHaloR;
    uint32_t v = 0xFu;
    bool hs = true;  // the halo column beside lanes 0 and 31
    for (int r2 = max(rr - 1, 0); r2 <= min(rr + 1, kTRin - 1); ++r2) {
      const float4 q4 = ld4(&sm.psi[r2][bc]);
      v &= (__float_as_uint(q4.x) == kPlus1 ? 1u : 0u) | (__float_as_uint(q4.y) == kPlus1 ? 2u : 0u) |
           (__float_as_uint(q4.z) == kPlus1 ? 4u : 0u) | (__float_as_uint(q4.w) == kPlus1 ? 8u : 0u);
      hs = hs && __float_as_uint(sm.psi[r2][xh]) == kPlus1;
    }
    uint32_t lf = __shfl_up_sync(FULL, v >> 3, 1) & 1u, rt = __shfl_down_sync(FULL, v, 1) & 1u;
    if (lane == 0) lf = (hs || x0 == 0) ? 1u : 0u;
    if (lane == 31) rt = hs ? 1u : 0u;
    const uint32_t e = lf | (v << 1) | (rt << 5);  // bit k: box column bc-1+k
    return e & (e >> 1) & (e >> 2) & 0xFu;
  };
  auto net_inputs = [&](int rr, int b, float in[3]) {  // b: box column
    in[0] = fmaf(TnB, (float)(b - 4), TnA);
    in[1] = fmaf(sm.d[rr][b], SA.c_ihalf, cnA);
    in[2] = clamp1(sm.psi[rr][b]);
  };
  // box and audit of one cell (in: net_inputs of it)
  auto net_inbox = [&](int rr, int b, const float in[3]) {
    const float T = SA.T_mid + in[0] / SA.T_ihalf, c = F.cinf + sm.d[rr][b];
    return T >= SA.T_lo && T <= SA.T_hi && c >= SA.c_lo && c <= SA.c_hi;
  };
  auto net_audited = [&](int rr, int b) {
    return surr_audit_cell(PS.step, (int64_t)(y0 - 1 + rr + K.j_offset) * K.nx + x0 + b - 4);
  };
  auto audit_store = [&](int rr, int b, const float o[2]) {  // (the exact mu'' is in place)
    const int gx = x0 + b - 4;
    const float dG_ex = drive_dG<float>(F.cinf + sm.d[rr][b], tAnb[gx], tAti[gx]);
    const float mu_net = fmaf(o[0], SA.y_scale[0], SA.y_mean[0]), dG_net = fmaf(o[1], SA.y_scale[1], SA.y_mean[1]);
    atomicMax(&SA.audit[0], (unsigned long long)__float_as_uint(fabsf(mu_net - sm.mu[rr][b])));
    atomicMax(&SA.audit[1], (unsigned long long)__float_as_uint(fabsf(dG_net - dG_ex)));
    atomicAdd(&SA.audit[3], 1ull);
  };
  // store the surrogate mu'' of one cell, or keep the exact value already in
  // place (out-of-box and audited cells); audited cells record the errors
  auto net_store = [&](int rr, int b, const float in[3], const float o[2]) {
    const int gx = x0 + b - 4;
    const bool inbox = net_inbox(rr, b, in), real = gx >= 0 && gx <= K.nx - 1, audit = real && net_audited(rr, b);
    if (inbox && !audit) {
      sm.mu[rr][b] = fmaf(o[0], SA.y_scale[0], SA.y_mean[0]);
    } else if (real && counted(rr)) {
      if (!inbox) atomicAdd(&SA.audit[2], 1ull);
      if (audit) audit_store(rr, b, o);
    }
  };
  // the partial sums of this tile (a dependent launch reduces them)
  auto finish = [&](double mass, int itip) {
    if (!part) return;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mass += __shfl_down_sync(FULL, mass, o);
    itip = __reduce_max_sync(FULL, itip);
    if (lane == 0) {
      sm.part_mass[warp] = mass;
      sm.part_itip[warp] = itip;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      BlockPartial b;
      b.mass = 0.0;
      b.itip = 0;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        b.mass += sm.part_mass[w];
        b.itip = max(b.itip, sm.part_itip[w]);
      }
      b.pad = 0;
      *part = b;
    }
  };
  if (pb) {
    const float *__restrict__ gpsi = static_cast<const float *>(PS.src_psi);
    const float *__restrict__ gd = static_cast<const float *>(PS.src_c);
    if (!PS.pull_back) {
      // a warp per row, every fourth row; columns lane, lane + 32, ...
      for (int rr = warp; rr < kTRin; rr += kWarps) {
        const int row = y0 - 1 + rr;
        const int64_t o = (int64_t)min(row, ny - 1) * K.pitch + x0 - 4 + lane;
#pragma unroll
        for (int q = 0; q < (kWin + 31) / 32; ++q) {
          const int x = lane + 32 * q, g = x0 - 4 + x;
          const bool inside = row <= ny - 1 && g >= 0 && g <= nx - 1;
          if (x < kWin) {
            cp_async_elem(&sm.psi[rr][x], gpsi + (inside ? o + 32 * q : 0), inside);
            cp_async_elem(&sm.d[rr][x], gd + (inside ? o + 32 * q : 0), inside);
          }
        }
      }
      cp_async_wait();
    }
    else for (int k = threadIdx.x; k < kTRin * kWin; k += kThreads) {
      const int rr = k / kWin, x = k % kWin;
      const int row = y0 - 1 + rr, g = x0 - 4 + x;
      float pv = 0.f, dv = 0.f;
      if (row <= ny - 1 && g >= 0 && g <= nx - 1) {
        const int si = min(max(g + PS.i_offset, 1), nx - 2);
        const int64_t o = (int64_t)row * K.pitch + si;
        pv = gpsi[o];
        dv = si >= nx - 2 ? 0.f : gd[o];
      }
      sm.psi[rr][x] = pv;
      sm.d[rr][x] = dv;
    }
  }
  __syncthreads();  // barrier initialised, flags cleared (a pull-back tile gathered)
  // one interior cell by plain stores, with the ghost cells that copy it
  auto raw_cell = [&](int r, int g, float pv, float dv) {
    if (g < 1 || g > nx - 2) return;
    auto at = [&](int row, int col) {
      const int64_t o = (int64_t)row * K.pitch + col;
      psi_n[o] = pv;
      c_n[o] = dv;
      if (phi_n) phi_n[o] = clamp1(pv);
    };
    auto all = [&](int row) {
      at(row, g);
      if (g == 1) at(row, 0);
      if (g == nx - 2) at(row, nx - 1);
    };
    all(r);
    if (r == K.jmin) all(0);
    if (r == K.jmax) all(ny - 1);
  };
  bool gave_up = false;
  if (!pb) {  // bounded wait for the tile
    const uint32_t limit = PS.wait_limit ? PS.wait_limit : kWaitLimit;
    uint32_t tries = 0;
    while (!mbar_try(&sm.full, 0, PS.wait_limit != 0)) {
      if (++tries >= limit) {
        gave_up = true;
        break;
      }
    }
    // pull the tile of the CTA that will start about one resident wave later
    // into L2, so its loads overlap the rest of this wave's arithmetic
    if (threadIdx.x == 0 && !gave_up) prefetch();
  }
  // columns beyond the array (right-most tiles; zero-filled by TMA) become
  // bulk melt, so they never force the general path; no output reads them
  // (a thread that gave up leaves the tile alone)
  if (x0 + kW + 4 > nx) {
    if (!gave_up)
      for (int k = threadIdx.x; k < kTRin * kWin; k += kThreads) {
        const int rr = k / kWin, x = k % kWin;
        if (x0 - 4 + x >= nx) {
          sm.psi[rr][x] = -1.f;
          sm.d[rr][x] = 0.f;
        }
      }
    __syncthreads();
  }
  // ---- the tile's form: far melt (psi = -1 exactly, |delta| <= melt_tiny; melt
  // in the series range too, with its rows' votes, cost the far melt more than
  // it gained: 2048^2 all melt 18.3 -> 19.5 us) or deep solid (psi = +1 exactly) in every cell of the box that an output reads
  // (rows and columns outside the array are left out) needs no masks, list or
  // interface pass
  constexpr uint32_t kNotMinus1 = 1u, kNotPlus1 = 2u, kNotFar = 4u, kNotFinite = 8u, kGaveUp = 16u;
  {
    uint32_t m1 = 0u, p1 = 0u, dm = 0u;  // OR of psi's difference from -1 / +1, largest |delta| (bits)
    auto cell = [&](float p, float d) {
      m1 |= __float_as_uint(p) ^ kMinus1;
      p1 |= __float_as_uint(p) ^ kPlus1;
      dm = max(dm, __float_as_uint(d) & 0x7fffffffu);
    };
    uint32_t bad = gave_up ? kGaveUp : kNotMinus1 | kNotPlus1;
    // (the coarse-grid temperature has no melt form: its tiles vote only where the
    // first interior cell is solid; 2048^2 all melt, with the polynomials of K + C0
    // and of the driving force on two threads, 63.5 -> 59 us a step)
    if (!gave_up && (!TFC || __float_as_uint(sm.psi[1][5]) == kPlus1)) {
#pragma unroll
      for (int k = 0; k < (kTRin + kWarps - 1) / kWarps; ++k) {
        const int rr = warp + kWarps * k;
        if (rr < kTRin && rr <= ny - y0) {
          const float4 p4 = ld4(&sm.psi[rr][bc]), d4 = ld4(&sm.d[rr][bc]);
          cell(p4.x, d4.x);
          cell(p4.y, d4.y);
          cell(p4.z, d4.z);
          cell(p4.w, d4.w);
        }
      }
      if (threadIdx.x >= kHalo0 && threadIdx.x < kHalo0 + 2 * kTRin) {  // the halo columns, one cell per thread
        const int rr = ((int)threadIdx.x - kHalo0) >> 1, side = ((int)threadIdx.x - kHalo0) & 1;
        const int x = side ? kHaloR : kHaloL;
        if (rr <= ny - y0 && (side || x0 > 0)) cell(sm.psi[rr][x], sm.d[rr][x]);
      }
      bad = (m1 ? kNotMinus1 : 0u) | (p1 ? kNotPlus1 : 0u) | (dm <= __float_as_uint(tiny) ? 0u : kNotFar) |
            (dm < 0x3F800000u ? 0u : kNotFinite);
    }
    bad = __reduce_or_sync(FULL, bad);
    if (lane == 0 && bad) atomicOr(&sm.vote, bad);
  }
  __syncthreads();
  const uint32_t vote = sm.vote;
  const bool red = part != nullptr;
  double mass = 0.0;
  int itip = 0;
  if (vote & kGaveUp) {
    // if any thread gives up, the whole CTA skips the tile: nothing is
    // computed on a partly filled tile or stored.  Thread 0 first waits
    // (bounded again) for the load still in flight into this CTA's shared
    // memory, and the CTA still reports a (zero) partial
    if (threadIdx.x == 0) {
      atomicExch(err, 1);
      for (uint32_t t = 0; t < kWaitLimit && !mbar_try_wait(&sm.full, 0); ++t) {
      }
    }
    __syncthreads();
    finish(0.0, 0);
    return;
  }
  const bool melt = !TFC && !(vote & (kNotMinus1 | kNotFar));
  if (melt || !(vote & (kNotPlus1 | kNotFinite))) {
    // the warp's output rows straight from registers to global memory, with
    // the ghost columns and rows they copy to (nx is a multiple of 4: a lane's
    // cells are all inside the array or all beyond it)
    const int r0 = kRowsPerWarp * warp;  // input row before the warp's first output row
    const int64_t o0 = (int64_t)(y0 + r0) * K.pitch + gi;
    const bool inside = gi < nx, ghost = (K.jmin >= y0 + r0 && K.jmin < y0 + r0 + kRowsPerWarp) ||
                                         (K.jmax >= y0 + r0 && K.jmax < y0 + r0 + kRowsPerWarp);
    const float pv = melt ? -1.f : 1.f;
    auto put = [&](int j, float (&v)[4]) {
      if constexpr (RAW) {
        // through the warp's row of mu, so that each store is of 32 adjacent cells
        st4(&sm.mu[warp][4 * lane], v[0], v[1], v[2], v[3]);
        __syncwarp();
#pragma unroll
        for (int q = 0; q < 4; ++q) raw_cell(y0 + r0 + j, x0 + lane + 32 * q, pv, sm.mu[warp][lane + 32 * q]);
        __syncwarp();
        return;
      }
      if (gi == 0) v[0] = v[1];         // ghost column 0
      if (gi + 4 == nx) v[3] = v[2];    // ghost column nx-1
      if (!inside) return;
      auto row = [&](int64_t o) {
        st4(psi_n + o, pv, pv, pv, pv);
        st4(c_n + o, v[0], v[1], v[2], v[3]);
        if (phi_n) st4(phi_n + o, pv, pv, pv, pv);
      };
      row(o0 + (int64_t)j * K.pitch);
      if (ghost) {
        if (y0 + r0 + j == K.jmin) row(gi);
        if (y0 + r0 + j == K.jmax) row((int64_t)(ny - 1) * K.pitch + gi);
      }
    };
    if (!melt) {  // deep solid: S = 0 in every cell, so every flux is 0 and psi and c stay
#pragma unroll
      for (int j = 0; j < kRowsPerWarp; ++j) {
        if (y0 + r0 + j > ny - 2) break;
        const float4 d4 = ld4(&sm.d[r0 + 1 + j][bc]);
        float v[4] = {fmaxf(d4.x, floor_d), fmaxf(d4.y, floor_d), fmaxf(d4.z, floor_d), fmaxf(d4.w, floor_d)};
        if (red) {
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if ((outm >> q) & 1u) {
              mass += (double)v[q];
              itip = max(itip, gi + q == nx - 2 ? nx - 1 : gi + q);
            }
        }
        put(j, v);
      }
      if constexpr (SURR) {
        // row ny-1 at the counters' open end: its cells count, and the audited ones
        // take the network, as the phases would have them
        if (open_end && y0 + kTR >= ny - 1) {
          const int rr = ny - y0, own = 4 + 32 * warp;
          auto cells = [&](int b, bool real, int ba, int bb, uint32_t ma, uint32_t mb) {  // one lane's cell; two per pass
            float in0[3], in1[3], o0[2], o1[2], Sx, mx;
            bool audit = false;
            if (real) {
              net_inputs(rr, b, in0);
              audit = net_audited(rr, b);
              if (!net_inbox(rr, b, in0)) atomicAdd(&SA.audit[2], 1ull);
            }
            const uint32_t am = __ballot_sync(FULL, audit);
            if (!am) return;
            if (audit) {
              cell_terms(F, sm.psi[rr][b], sm.d[rr][b], tRT[x0 + b - 4], tC0[x0 + b - 4], Sx, mx);
              sm.mu[rr][b] = mx;
            }
            __syncwarp();
            const SurrConst SC = surr_load(SA, lane);
#pragma unroll 1
            for (int h = 0; h < 32; h += 16) {
              if (!(am >> h & 0xFFFFu)) continue;
              net_inputs(rr, ba + h, in0);
              net_inputs(rr, bb + h, in1);
              surr_tile16(SC, in0, in1, o0, o1);
              if ((lane & 3) == 0) {
                if (am >> h & ma) audit_store(rr, ba + h, o0);
                if (am >> h & mb) audit_store(rr, bb + h, o1);
              }
            }
          };
          const int g = lane >> 2;
          cells(own + lane, true, own + g, own + g + 8, 1u << g, 256u << g);
          if (warp == 3)  // the halo columns, lanes 0 and 1
            cells(lane ? kHaloR : kHaloL, lane == 1 || (lane == 0 && x0 > 0), kHaloL, kHaloR, g ? 0u : 1u, g ? 0u : 2u);
        }
      }
      finish(mass, itip);
      return;
    }
    if constexpr (!TFC) {
      // far melt: phases 1 and 2 with S and mu'' of the warp's rows in
      // registers (the same expressions, so the same bits); halo columns by a
      // lane per cell through scratch
      float *hs = &sm.S[warp][0], *hm = &sm.S[warp][kWin / 2];
      if (lane < 2 * (kRowsPerWarp + 2)) {
        const int rr = r0 + (lane >> 1), x = (lane & 1) ? kHaloR : kHaloL;
        float Sh = 0.f, mh = 0.f;
        if (rr <= ny - y0) far_cell(M, sm.d[rr][x], tRT[x0 - 4 + x], Sh, mh);
        hs[lane] = Sh;
        hm[lane] = mh;
      }
      __syncwarp();
      if constexpr (SURR) {
        dKv = ld4(tDK + gi);
        dKl = tDK[gi - 1];
      }
      const float dKm[5] = {dKl, dKv.x, dKv.y, dKv.z, dKv.w};
      struct MRow {
        float s[4], m[4], d[4], sl, sr, ml, mr, q[5];
      };
      auto melt_row = [&](int k, MRow &R) {
        const float4 d4 = ld4(&sm.d[r0 + k][bc]);
        R.d[0] = d4.x; R.d[1] = d4.y; R.d[2] = d4.z; R.d[3] = d4.w;
#pragma unroll
        for (int q = 0; q < 4; ++q) far_cell(M, R.d[q], RTa[q], R.s[q], R.m[q]);
        R.sl = __shfl_up_sync(FULL, R.s[3], 1);
        R.ml = __shfl_up_sync(FULL, R.m[3], 1);
        R.sr = __shfl_down_sync(FULL, R.s[0], 1);
        R.mr = __shfl_down_sync(FULL, R.m[0], 1);
        if (lane == 0) {
          R.sl = hs[2 * k];
          R.ml = hm[2 * k];
        }
        if (lane == 31) {
          R.sr = hs[2 * k + 1];
          R.mr = hm[2 * k + 1];
        }
        R.q[0] = R.sl + R.s[0];
        R.q[1] = R.s[0] + R.s[1];
        R.q[2] = R.s[1] + R.s[2];
        R.q[3] = R.s[2] + R.s[3];
        R.q[4] = R.s[3] + R.sr;
      };
      auto melt_face = [&](const MRow &A, const MRow &B, float jv[4]) {
        const float pp[6] = {A.sl + B.sl,         A.s[0] + B.s[0], A.s[1] + B.s[1],
                             A.s[2] + B.s[2], A.s[3] + B.s[3], A.sr + B.sr};
#pragma unroll
        for (int q = 0; q < 4; ++q) jv[q] = __fmul_rn(fmaf(6.f, pp[q + 1], pp[q] + pp[q + 2]), B.m[q] - A.m[q]);
      };
      MRow a, b, c;
      float lo[4], hi[4];
      melt_row(0, a);
      melt_row(1, b);
      melt_face(a, b, lo);
#pragma unroll
      for (int j = 0; j < kRowsPerWarp; ++j) {
        melt_row(j + 2, c);
        melt_face(b, c, hi);
        const float mm[6] = {b.ml, b.m[0], b.m[1], b.m[2], b.m[3], b.mr};
        float jh[5], v[4];
#pragma unroll
        for (int f = 0; f < 5; ++f) jh[f] = __fmul_rn(fmaf(6.f, b.q[f], a.q[f] + c.q[f]), mm[f + 1] - mm[f] + dKm[f]);
#pragma unroll
        for (int q = 0; q < 4; ++q) v[q] = fmaxf(fmaf(cflux4, (jh[q + 1] - jh[q]) + (hi[q] - lo[q]), b.d[q]), floor_d);
        if (y0 + r0 + j <= ny - 2) {
          if (red) {
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if ((outm >> q) & 1u) mass += (double)v[q];
          }
          put(j, v);
        }
        a = b;
        b = c;
#pragma unroll
        for (int q = 0; q < 4; ++q) lo[q] = hi[q];
      }
      finish(mass, 0);
      return;
    }
  }

  // ---- phase 1: per-cell terms; warp w takes input rows w, w+4, ...
  // The warp's row flags (warp-uniform) are OR-ed into sm.liq / sm.sol once;
  // rows flagged there store no phi masks (phase 2 takes 0x0F / 0xF0)
  Mask liq_rows = 0, sol_rows = 0;
#pragma unroll 1
  for (int rr = warp; rr < kTRin; rr += kWarps) {
    if (y0 - 1 + rr > ny - 1) {  // beyond the array (last tile): never read by an output
      st4(&sm.S[rr][bc], 0.f, 0.f, 0.f, 0.f);
      st4(&sm.mu[rr][bc], 0.f, 0.f, 0.f, 0.f);
      if constexpr (TFC) {
        *reinterpret_cast<double2 *>(&sm.kc[rr][bc]) = make_double2(0.0, 0.0);
        *reinterpret_cast<double2 *>(&sm.kc[rr][bc + 2]) = make_double2(0.0, 0.0);
      }
      liq_rows |= Mask(1) << rr;
      sol_rows |= Mask(1) << rr;
      continue;
    }
    const float4 pv4 = ld4(&sm.psi[rr][bc]), dv4 = ld4(&sm.d[rr][bc]);
    const float pv[4] = {pv4.x, pv4.y, pv4.z, pv4.w}, dv[4] = {dv4.x, dv4.y, dv4.z, dv4.w};
    float Sv[4], mv[4];
    // bulk melt: every psi exactly -1 (bit tests) and every delta in the
    // series range
    const uint32_t b0 = __float_as_uint(pv[0]), b1 = __float_as_uint(pv[1]), b2 = __float_as_uint(pv[2]),
                   b3 = __float_as_uint(pv[3]);
    const uint32_t band = b0 & b1 & b2 & b3, bor = b0 | b1 | b2 | b3;
    const float dmx = fmaxf(fmaxf(dv[0], dv[1]), fmaxf(dv[2], dv[3]));
    const float dmn = fminf(fminf(dv[0], dv[1]), fminf(dv[2], dv[3]));
    const bool liq4 = band == kMinus1 && bor == kMinus1;
    // the row's form (warp-uniform): far melt, bulk melt or general (voted
    // here with TFC, where it decides which groups to evaluate)
    bool far = false, bulk = false;
    if constexpr (TFC) {  // the melt forms need RT and K + C0 only
      far = __all_sync(FULL, liq4 && fmaxf(dmx, -dmn) <= tiny);
      bulk = !far && __all_sync(FULL, liq4 && dmx < d_hi && dmn > d_lo);
      const int jT = sm.tj[rr];
      const double y = sm.ty[rr];
      double kq[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        double RT, C0;
        cell_tfc(K, sm.kp, tfc_T(K, PS.T_coarse, tiT[q], tx[q], jT, y), !(far || bulk), RT, C0, kq[q]);
        RTa[q] = (float)RT;
        C0a[q] = (float)C0;
      }
      *reinterpret_cast<double2 *>(&sm.kc[rr][bc]) = make_double2(kq[0], kq[1]);
      *reinterpret_cast<double2 *>(&sm.kc[rr][bc + 2]) = make_double2(kq[2], kq[3]);
    }
    uint32_t code, s3 = 0u;
    if (TFC ? far : __all_sync(FULL, liq4 && fmaxf(dmx, -dmn) <= tiny)) {
      // far melt: lam by its Taylor polynomial in delta (Coef::melt_a);
      // mu'' = RT lam - 2 L0_Liq delta = delta (RT p + KL), lam = delta p
      code = 1u | 4u;  // 4: every cell in the exact melt form
#pragma unroll
      for (int q = 0; q < 4; ++q) far_cell(M, dv[q], RTa[q], Sv[q], mv[q]);
    } else if (TFC ? bulk : __all_sync(FULL, liq4 && dmx < d_hi && dmn > d_lo)) {
      code = 1u | 4u;  // 4: every cell in the series form
#pragma unroll
      for (int q = 0; q < 4; ++q) bulk_cell(M, dv[q], RTa[q], Sv[q], mv[q]);
    } else {
      const bool sol4 = band == kPlus1 && bor == kPlus1;
      code = (__all_sync(FULL, liq4) ? 1u : 0u) | (__all_sync(FULL, sol4) ? 2u : 0u);
      // deep solid row: no cell's mu'' enters a flux (solid3), so S = mu'' = 0
      // gives the same fluxes.  The surrogate also skips solid3 cells, which
      // pays only where a whole 16-cell network pass (lanes 4m .. 4m+3) is
      // solid
      bool want = (code & 2u) != 0u;
      if constexpr (SURR) {
        const uint32_t fs = __ballot_sync(FULL, sol4);
        want = want || (fs & (fs >> 1) & (fs >> 2) & (fs >> 3) & 0x11111111u) != 0u;
      }
      if (want) s3 = solid3(rr);
      const bool deep = (code & 2u) && __all_sync(FULL, s3 == 0xFu);
      if (deep) {
        code |= 8u;  // 8: mu'' not needed (no network pass either)
#pragma unroll
        for (int q = 0; q < 4; ++q) Sv[q] = mv[q] = 0.f;
      } else {
        uint32_t L = 0u, Sm = 0u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          if (pv[q] <= -1.f) L |= 1u << q;
          if (pv[q] >= 1.f) Sm |= 1u << q;
          cell_terms(F, pv[q], dv[q], RTa[q], C0a[q], Sv[q], mv[q]);
        }
        sm.pmask[rr][lane] = (uint8_t)(L | (Sm << 4));
      }
    }
    st4(&sm.S[rr][bc], Sv[0], Sv[1], Sv[2], Sv[3]);
    st4(&sm.mu[rr][bc], mv[0], mv[1], mv[2], mv[3]);
    liq_rows |= Mask(code & 1u) << rr;
    sol_rows |= Mask((code >> 1) & 1u) << rr;
    if constexpr (SURR) {  // the row's non-melt cells through the network, 16 at a time
      if (!(code & (4u | 8u))) {
        __syncwarp();
        const SurrConst SC = surr_load(SA, lane);
        const int g = lane >> 2;
        const bool any3 = __any_sync(FULL, s3 != 0u);
#pragma unroll 1
        for (int mt = 0; mt < kW / 16; ++mt) {
          const int ba = 4 + 16 * mt + g, bb = ba + 8;
          bool na = !melt_cell(rr, ba), nb = !melt_cell(rr, bb);
          if (any3) {  // warp-uniform
            const uint32_t sa = __shfl_sync(FULL, s3, (ba - 4) >> 2), sb = __shfl_sync(FULL, s3, (bb - 4) >> 2);
            na = na && !((sa >> ((ba - 4) & 3)) & 1u);
            nb = nb && !((sb >> ((bb - 4) & 3)) & 1u);
          }
          if (!__any_sync(FULL, na || nb)) continue;
          float in0[3], in1[3], o0[2], o1[2];
          net_inputs(rr, ba, in0);
          net_inputs(rr, bb, in1);
          surr_tile16(SC, in0, in1, o0, o1);
          if ((lane & 3) == 0) {
            if (na) net_store(rr, ba, in0, o0);
            if (nb) net_store(rr, bb, in1, o1);
          }
        }
      }
    }
  }
  if (lane == 0) {
    if (liq_rows) atomicOr(&sm.liq, liq_rows);
    if (sol_rows) atomicOr(&sm.sol, sol_rows);
  }
  // halo columns x0-1 and x0+kW, one thread per cell, on warps 2 and 3, which
  // have one input row fewer than warps 0 and 1 (surrogate: warp 3 alone,
  // then the same network pass as the rows)
  if (SURR ? warp == 3 : (threadIdx.x >= kHalo0 && threadIdx.x < kHalo0 + 2 * kTRin)) {
   for (int i = SURR ? lane : (int)threadIdx.x - kHalo0; i < 2 * kTRin; i += 32) {
    const int rr = i >> 1, side = i & 1;
    const int x = side ? kHaloR : kHaloL, g = x0 - 4 + x;
    float Sh = 0.f, mh = 0.f;
    double kh = 0.0;
    uint8_t hm = 3u;
    if (y0 - 1 + rr <= K.ny - 1) {
      const float pv = sm.psi[rr][x];
      if constexpr (TFC) {
        // C0 enters mu'' as (g + 1) C0, 0 at psi = -1 exactly: the liquid
        // groups suffice there
        double RT, C0;
        cell_tfc(K, sm.kp, tfc_T(K, PS.T_coarse, sm.hiT[side], sm.hx[side], sm.tj[rr], sm.ty[rr]),
                 __float_as_uint(pv) != kMinus1, RT, C0, kh);
        halo_cell(F, M, pv, sm.d[rr][x], (float)RT, (float)C0, Sh, mh);
      } else {
        halo_cell(F, M, pv, sm.d[rr][x], tRT[g], tC0[g], Sh, mh);
      }
      hm = (pv <= -1.f ? 1u : 0u) | (pv >= 1.f ? 2u : 0u);
    }
    sm.S[rr][x] = Sh;
    sm.mu[rr][x] = mh;
    if constexpr (TFC) sm.kc[rr][x] = kh;
    sm.hmask[rr][side] = hm;
    if (!SURR) break;
   }
   if constexpr (SURR) {
    __syncwarp();
    const int g = lane >> 2;
#pragma unroll 1
    for (int mt = 0; mt < (2 * kTRin + 15) / 16; ++mt) {
      const int ia = 16 * mt + g, ib = ia + 8;
      const int ra = ia < 2 * kTRin ? ia >> 1 : 0, rb = ib < 2 * kTRin ? ib >> 1 : 0;
      const int xa = (ia & 1) ? kHaloR : kHaloL, xb = (ib & 1) ? kHaloR : kHaloL;
      const bool na = ia < 2 * kTRin && y0 - 1 + ra <= K.ny - 1 && !melt_cell(ra, xa) && halo_mu_used(ra, xa);
      const bool nb = ib < 2 * kTRin && y0 - 1 + rb <= K.ny - 1 && !melt_cell(rb, xb) && halo_mu_used(rb, xb);
      if (!__any_sync(FULL, na || nb)) continue;
      const SurrConst SC = surr_load(SA, lane);
      float in0[3], in1[3], o0[2], o1[2];
      net_inputs(ra, xa, in0);
      net_inputs(rb, xb, in1);
      surr_tile16(SC, in0, in1, o0, o1);
      if ((lane & 3) == 0) {
        if (na) net_store(ra, xa, in0, o0);
        if (nb) net_store(rb, xb, in1, o1);
      }
    }
   }
  }
  if constexpr (SURR) {
    dKv = ld4(tDK + gi);
    dKl = tDK[gi - 1];
  }
  const float dKa[5] = {dKl, dKv.x, dKv.y, dKv.z, dKv.w};  // faces x-1|x for x = col .. col+4
  __syncthreads();

  // ---- phase 2: warp w computes output rows 1 + 4w .. 4 + 4w of the tile
  const Mask liq = sm.liq, sol = sm.sol;
  struct Row {
    float s[4], m[4], sl, sr, ml, mr, q[5];  // q[f]: S pair sum of the face left of cell f (f = 0..4)
    double k[4], kl, kr;                     // TFC: K + C0 of the cells and of their neighbours
  };
  auto load_row = [&](int rr, Row &R) {
    const float4 s = ld4(&sm.S[rr][bc]), m = ld4(&sm.mu[rr][bc]);
    R.s[0] = s.x; R.s[1] = s.y; R.s[2] = s.z; R.s[3] = s.w;
    R.m[0] = m.x; R.m[1] = m.y; R.m[2] = m.z; R.m[3] = m.w;
    R.sl = __shfl_up_sync(FULL, s.w, 1);
    R.ml = __shfl_up_sync(FULL, m.w, 1);
    R.sr = __shfl_down_sync(FULL, s.x, 1);
    R.mr = __shfl_down_sync(FULL, m.x, 1);
    if (lane == 0) {
      R.sl = sm.S[rr][kHaloL];
      R.ml = sm.mu[rr][kHaloL];
    }
    if (lane == 31) {
      R.sr = sm.S[rr][kHaloR];
      R.mr = sm.mu[rr][kHaloR];
    }
    if constexpr (TFC) {
      const double2 k01 = *reinterpret_cast<const double2 *>(&sm.kc[rr][bc]);
      const double2 k23 = *reinterpret_cast<const double2 *>(&sm.kc[rr][bc + 2]);
      R.k[0] = k01.x; R.k[1] = k01.y; R.k[2] = k23.x; R.k[3] = k23.y;
      R.kl = __shfl_up_sync(FULL, R.k[3], 1);
      R.kr = __shfl_down_sync(FULL, R.k[0], 1);
      if (lane == 0) R.kl = sm.kc[rr][kHaloL];
      if (lane == 31) R.kr = sm.kc[rr][kHaloR];
    }
    R.q[0] = R.sl + R.s[0];
    R.q[1] = R.s[0] + R.s[1];
    R.q[2] = R.s[1] + R.s[2];
    R.q[3] = R.s[2] + R.s[3];
    R.q[4] = R.s[3] + R.sr;
  };
  // fluxes through the faces between rows A and B = A+1 (compute_c_CALPHAD
  // F01/F0m).  Face fluxes are rounded products (__fmul_rn): a contracted
  // product would round a face differently depending on where the face falls
  // in a warp's rows, and so on the tiling (row bands must equal the whole
  // domain bit for bit).
  auto vface = [&](const Row &A, const Row &B, float jv[4]) {
    float pp[6];
    pp[0] = A.sl + B.sl;
#pragma unroll
    for (int q = 0; q < 4; ++q) pp[q + 1] = A.s[q] + B.s[q];
    pp[5] = A.sr + B.sr;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      float dm = B.m[q] - A.m[q];
      if constexpr (TFC) dm = dm + (float)(B.k[q] - A.k[q]);  // K + C0 differs along y too
      jv[q] = __fmul_rn(fmaf(6.f, pp[q + 1], pp[q] + pp[q + 2]), dm);
    }
  };

  const int rbase = 1 + kRowsPerWarp * warp;
  Row ra, rb, rc;
  float jv_lo[4], jv_hi[4];
  float dn[kRowsPerWarp][4];
  uint32_t needs_all = 0u;  // 4 bits per output row
  load_row(rbase - 1, ra);
  load_row(rbase, rb);
  vface(ra, rb, jv_lo);
#pragma unroll
  for (int j = 0; j < kRowsPerWarp; ++j) {
    const int rr = rbase + j;  // tile input row of the output row
    load_row(rr + 1, rc);
    vface(rb, rc, jv_hi);
    // fluxes through the faces (x-1/2, r) for x = col .. col+4
    const float mm[6] = {rb.ml, rb.m[0], rb.m[1], rb.m[2], rb.m[3], rb.mr};
    float jh[5], dKf[5];
    if constexpr (TFC) {  // the cells' own K + C0 differences, rounded from FP64
      const double kk[6] = {rb.kl, rb.k[0], rb.k[1], rb.k[2], rb.k[3], rb.kr};
#pragma unroll
      for (int f = 0; f < 5; ++f) dKf[f] = (float)(kk[f + 1] - kk[f]);
    } else {
#pragma unroll
      for (int f = 0; f < 5; ++f) dKf[f] = dKa[f];
    }
#pragma unroll
    for (int f = 0; f < 5; ++f) jh[f] = __fmul_rn(fmaf(6.f, rb.q[f], ra.q[f] + rc.q[f]), mm[f + 1] - mm[f] + dKf[f]);
    const float4 dv4 = ld4(&sm.d[rr][bc]);
    const float dv[4] = {dv4.x, dv4.y, dv4.z, dv4.w};
#pragma unroll
    for (int q = 0; q < 4; ++q)
      dn[j][q] = fmaxf(fmaf(cflux4, (jh[q + 1] - jh[q]) + (jv_hi[q] - jv_lo[q]), dv[q]), floor_d);
    const bool live = y0 - 1 + rr <= ny - 2;
    if (red && live) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if ((outm >> q) & 1u) mass += (double)dn[j][q];
    }
    // phi: cells whose 3x3 neighbourhood is not uniformly +-1 are listed
    const Mask w3 = Mask(7) << (rr - 1);
    if (live && (liq & w3) != w3 && (sol & w3) != w3) {
      auto pm = [&](int k) -> uint32_t {  // rows flagged all -1 / all +1 store no masks
        return ((liq >> k) & 1u) ? 0x0Fu : ((sol >> k) & 1u) ? 0xF0u : (uint32_t)sm.pmask[k][lane];
      };
      const uint32_t pk = pm(rr - 1) | (pm(rr) << 8) | (pm(rr + 1) << 16);
      uint32_t lf = __shfl_up_sync(FULL, pk, 1), rt = __shfl_down_sync(FULL, pk, 1);
      if (lane == 0) {
        lf = 0u;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const uint32_t h = sm.hmask[rr - 1 + k][0];
          lf |= ((h & 1u) << (8 * k + 3)) | (((h >> 1) & 1u) << (8 * k + 7));
        }
      }
      if (lane == 31) {
        rt = 0u;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const uint32_t h = sm.hmask[rr - 1 + k][1];
          rt |= ((h & 1u) << (8 * k)) | (((h >> 1) & 1u) << (8 * k + 4));
        }
      }
      uint32_t Lv = 0x3Fu, Sv = 0x3Fu;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const uint32_t L = (pk >> (8 * k)) & 0xFu, S = (pk >> (8 * k + 4)) & 0xFu;
        Lv &= (L << 1) | ((lf >> (8 * k + 3)) & 1u) | (((rt >> (8 * k)) & 1u) << 5);
        Sv &= (S << 1) | ((lf >> (8 * k + 7)) & 1u) | (((rt >> (8 * k + 4)) & 1u) << 5);
      }
      const uint32_t needs = ~((Lv & (Lv >> 1) & (Lv >> 2)) | (Sv & (Sv >> 1) & (Sv >> 2))) & outm;
      // cells that draw noise (phi_cell's own test; here it only sorts the list)
      uint32_t noisy = 0xFu;
      if (F.noise_amp > 0.f) {
        const float4 p4 = ld4(&sm.psi[rr][bc]);
        noisy = (fmaf(-p4.x, p4.x, 1.f) > 1.0e-3f ? 1u : 0u) | (fmaf(-p4.y, p4.y, 1.f) > 1.0e-3f ? 2u : 0u) |
                (fmaf(-p4.z, p4.z, 1.f) > 1.0e-3f ? 4u : 0u) | (fmaf(-p4.w, p4.w, 1.f) > 1.0e-3f ? 8u : 0u);
      }
      // inclusive warp scan of the counts of both kinds (packed as in nlist)
      const uint32_t cnt = __popc(needs & noisy) | (__popc(needs & ~noisy) << 16);
      uint32_t incl = cnt;
#pragma unroll
      for (int o = 1; o < 32; o <<= 1) {
        const uint32_t v = __shfl_up_sync(FULL, incl, o);
        if (lane >= o) incl += v;
      }
      uint32_t base = 0u;
      if (lane == 31 && incl) base = atomicAdd(&sm.nlist, incl);
      base = __shfl_sync(FULL, base, 31) + incl - cnt;
      uint32_t n_at = base & 0xFFFFu, t_at = kTR * kW - 1 - (base >> 16);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if ((needs >> q) & 1u) sm.list[((noisy >> q) & 1u) ? n_at++ : t_at--] = (uint16_t)((rr << 8) | (col + q));
      needs_all |= needs << (4 * j);
    }
    ra = rb;
    rb = rc;
#pragma unroll
    for (int q = 0; q < 4; ++q) jv_lo[q] = jv_hi[q];
  }
  __syncthreads();

  // ---- phase 3: interface cells, one per thread (compute_phi, fun.cu:1143-1218)
  const int na = (int)(sm.nlist & 0xFFFFu), nlist = na + (int)(sm.nlist >> 16);
  auto listed = [&](int idx) { return (uint32_t)sm.list[idx < na ? idx : kTR * kW - 1 - (idx - na)]; };
  if constexpr (SURR) {
    // network driving force of the listed cells, 16 per warp pass, into the
    // mu'' slots of those cells (mu'' is not read after phase 2)
    if (nlist > 16 * warp) {
      const SurrConst SC = surr_load(SA, lane);
      const int g = lane >> 2;
#pragma unroll 1
      for (int base = 16 * warp; base < nlist; base += 16 * kWarps) {
        const int ia = base + g, ib = ia + 8;
        const uint32_t ea = listed(min(ia, nlist - 1)), eb = listed(min(ib, nlist - 1));
        const int ra = (int)(ea >> 8), xa = (int)(ea & 0xFFu) + 4, rb = (int)(eb >> 8), xb = (int)(eb & 0xFFu) + 4;
        float in0[3], in1[3], o0[2], o1[2];
        net_inputs(ra, xa, in0);
        net_inputs(rb, xb, in1);
        surr_tile16(SC, in0, in1, o0, o1);
        __syncwarp();  // every lane has read its inputs before any slot is overwritten
        if ((lane & 3) == 0) {
          if (ia < nlist) sm.mu[ra][xa] = fmaf(o0[1], SA.y_scale[1], SA.y_mean[1]);
          if (ib < nlist) sm.mu[rb][xb] = fmaf(o1[1], SA.y_scale[1], SA.y_mean[1]);
        }
      }
    }
    __syncthreads();
  }
  for (int idx = threadIdx.x; idx < nlist; idx += kThreads) {
    const uint32_t e = listed(idx);
    const int rr = (int)(e >> 8), x = (int)(e & 0xFFu) + 4;  // box column
    const int r = y0 - 1 + rr, g = x0 + x - 4;
    const float c00 = F.cinf + sm.d[rr][x];
    float Anb, Ati;
    if constexpr (TFC) {
      const CellGroups cg = tfc_cell(g, r);
      Anb = (float)cg.Anb;
      Ati = (float)cg.Ati;
    } else {
      Anb = tAnb[g];
      Ati = tAti[g];
    }
    float dG = drive_dG<float>(c00, Anb, Ati);
    if constexpr (SURR) {  // driving force from the surrogate for in-box, unaudited cells
      float in[3];
      net_inputs(rr, x, in);
      const float T = SA.T_mid + in[0] / SA.T_ihalf;
      if (T >= SA.T_lo && T <= SA.T_hi && c00 >= SA.c_lo && c00 <= SA.c_hi &&
          !surr_audit_cell(PS.step, (int64_t)(r + K.j_offset) * K.nx + g))
        dG = sm.mu[rr][x];
    }
    const float res = phi_cell_dG<float>(
        &F, clamp1(sm.psi[rr][x]), clamp1(sm.psi[rr][x + 1]), clamp1(sm.psi[rr][x - 1]), clamp1(sm.psi[rr + 1][x]),
        clamp1(sm.psi[rr - 1][x]), clamp1(sm.psi[rr + 1][x + 1]), clamp1(sm.psi[rr + 1][x - 1]),
        clamp1(sm.psi[rr - 1][x + 1]), clamp1(sm.psi[rr - 1][x - 1]), dG, PS.step, (int64_t)(r + K.j_offset) * K.nx + g, K.seed_lo,
        K.seed_hi);
    sm.S[rr][x] = res;
    if (red && res > 0.f) itip = max(itip, g == K.nx - 2 ? K.nx - 1 : g);
  }
  __syncthreads();

  // (a whole-tile form, and a CTA that gave up, trigger by their end)
  if (PS.late) pdl_trigger();

  // ---- phase 4: new psi and c into the tile rows
#pragma unroll
  for (int j = 0; j < kRowsPerWarp; ++j) {
    const int rr = rbase + j;
    const float4 pv4 = ld4(&sm.psi[rr][bc]);
    // phi_next = phi where uniformly +-1: an output cell is not listed only
    // where psi <= -1 or >= 1 over its 3x3 neighbourhood, so clamp(psi) is
    // its sign (cells outside the interior are not stored or are overwritten
    // by the ghost copies); listed cells take phase 3's result
    float po[4] = {pv4.x > 0.f ? 1.f : -1.f, pv4.y > 0.f ? 1.f : -1.f, pv4.z > 0.f ? 1.f : -1.f,
                   pv4.w > 0.f ? 1.f : -1.f};
    const uint32_t lb = (needs_all >> (4 * j)) & 0xFu;
    if (lb) {
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if ((lb >> q) & 1u) po[q] = sm.S[rr][bc + q];
    }
    st4(&sm.psi[rr][bc], po[0], po[1], po[2], po[3]);
    st4(&sm.d[rr][bc], dn[j][0], dn[j][1], dn[j][2], dn[j][3]);
  }
  if (red) {  // coarse tip: the last column with phi > 0 (listed cells counted again, harmlessly)
#pragma unroll
    for (int j = 0; j < kRowsPerWarp; ++j) {
      const int rr = rbase + j;
      const float4 po4 = ld4(&sm.psi[rr][bc]);
      const float po[4] = {po4.x, po4.y, po4.z, po4.w};
      if (y0 - 1 + rr > ny - 2) continue;
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (((outm >> q) & 1u) && po[q] > 0.f) itip = max(itip, gi + q == nx - 2 ? nx - 1 : gi + q);
    }
  }
  const int nrow = min(kTR, K.ny - 1 - y0);  // output rows of this tile inside the interior
  if constexpr (RAW) {
    __syncthreads();
    for (int k = threadIdx.x; k < nrow * kW; k += kThreads) {
      const int j = k / kW, x = k % kW;
      raw_cell(y0 + j, x0 + x, sm.psi[1 + j][4 + x], sm.d[1 + j][4 + x]);
    }
    finish(mass, itip);
    return;
  }
  const int ncol = min(kW, K.nx - x0);       // columns of this tile inside the array (a multiple of 4)
  if (x0 == 0 || x0 + kW >= K.nx) {
    // ghost columns 0 and nx-1 (compute_boundary_individual, fun.cu:1220-1230)
    __syncthreads();
    if (threadIdx.x < nrow) {
      const int rr = 1 + threadIdx.x;
      if (x0 == 0) {
        sm.psi[rr][4] = sm.psi[rr][5];
        sm.d[rr][4] = sm.d[rr][5];
      }
      if (x0 + kW >= K.nx) {
        const int x = K.nx - 1 - x0 + 4;
        sm.psi[rr][x] = sm.psi[rr][x - 1];
        sm.d[rr][x] = sm.d[rr][x - 1];
      }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // tile writes -> bulk copies
  __syncthreads();

  // ---- bulk copies: thread (row j, field, kind): kind 0 the row itself,
  // kind 1 its ghost copies (row jmin -> 0, row jmax -> ny-1)
  if (threadIdx.x < 4 * kTR) {
    const int j = threadIdx.x >> 2, field = threadIdx.x & 1, kind = (threadIdx.x >> 1) & 1;
    const int r = y0 + j;
    if (j < nrow) {
      float *f = field ? c_n : psi_n;
      const float *src = field ? &sm.d[1 + j][4] : &sm.psi[1 + j][4];
      const uint32_t bytes = (uint32_t)ncol * 4u;
      bool any = false;
      if (kind == 0) {
        bulk_store(f + (int64_t)r * K.pitch + x0, src, bytes);
        any = true;
      } else {
        if (r == K.jmin) {
          bulk_store(f + x0, src, bytes);
          any = true;
        }
        if (r == K.jmax) {
          bulk_store(f + (int64_t)(K.ny - 1) * K.pitch + x0, src, bytes);
          any = true;
        }
      }
      if (any) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
  if (phi_n) {  // phi = clamp(psi) of the same rows, plain stores
    for (int k = threadIdx.x; k < nrow * ncol; k += kThreads) {
      const int j = k / ncol, x = k % ncol, r = y0 + j;
      const float v = clamp1(sm.psi[1 + j][4 + x]);
      phi_n[(int64_t)r * K.pitch + x0 + x] = v;
      if (r == K.jmin) phi_n[x0 + x] = v;
      if (r == K.jmax) phi_n[(int64_t)(K.ny - 1) * K.pitch + x0 + x] = v;
    }
  }

  finish(mass, itip);
  // shared memory stays allocated until the copies have read it
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

// the tile of the block launched one resident wave later (wave_y tile columns
// and wave_x tile rows on), into L2
struct WavePrefetch {
  const CUtensorMap *psi, *c;
  int f, wave_x, wave_y, TR;
  __device__ void operator()() const {
    int bx = (int)blockIdx.x + wave_x, by = (int)blockIdx.y + wave_y;
    if (bx >= (int)gridDim.x) {
      bx -= (int)gridDim.x;
      ++by;
    }
    if (by >= (int)gridDim.y) return;
    const int pc = front_first_block(by, f, (int)gridDim.y);
    tma_prefetch_2d(psi, kW * pc - 4, TR * bx);
    tma_prefetch_2d(c, kW * pc - 4, TR * bx);
  }
};

// (exact, 4 rows: 72 registers, so that seven CTAs fit on an SM; with 74 and six,
// 96 x 4000 took 14.0 us a step instead of 10.5)
template <bool SURR, int TR, bool RAW>
__global__ void __launch_bounds__(kThreads, SURR ? 4 : 5)
    tile_kernel(const __grid_constant__ StepCoef K, const __grid_constant__ Coef<float> F,
                const __grid_constant__ StepScalars PS, const __grid_constant__ CUtensorMap tm_psi,
                const __grid_constant__ CUtensorMap tm_c, const float *__restrict__ tab, const int tab_len,
                float *__restrict__ psi_n, float *__restrict__ c_n, float *__restrict__ phi_n, BlockPartial *partials,
                int *err, const __grid_constant__ SurrArgs SA, const int wave_x, const int wave_y) {
  // blockIdx.x walks the tile rows of one tile column (they share halo rows
  // in L2), blockIdx.y the tile columns, from the one holding column PS.i_front
  const int f = max(PS.i_front, 0) / kW;
  const int tr = blockIdx.x;
  const int tc = front_first_block((int)blockIdx.y, f, (int)gridDim.y);
  tile_body<SURR, TR, WavePrefetch, false, RAW, SURR ? kTileRows : TR>(K, F, PS, &tm_psi, &tm_c, tab, tab_len, psi_n, c_n, phi_n,
                      partials ? partials + ((int64_t)tc * gridDim.x + tr) : nullptr, err, SA, tr, tc,
                      WavePrefetch{&tm_psi, &tm_c, f, wave_x, wave_y, TR});
}

// The coarse-grid temperature (TFC): tiles of kTfcTileRows32 output rows, whose
// per-cell K + C0 (FP64) fits beside the tile with five CTAs per SM; per-cell
// CALPHAD groups instead of the column table.
constexpr int kTfcTR = kTfcTileRows32;
template <bool RAW>
__global__ void __launch_bounds__(kThreads, 5)
    tile_kernel_tfc(const __grid_constant__ StepCoef K, const __grid_constant__ Coef<float> F,
                    const __grid_constant__ StepScalars PS, const __grid_constant__ CUtensorMap tm_psi,
                    const __grid_constant__ CUtensorMap tm_c, const float *__restrict__ tab, const int tab_len,
                    float *__restrict__ psi_n, float *__restrict__ c_n, float *__restrict__ phi_n,
                    BlockPartial *partials, int *err, const int wave_x, const int wave_y) {
  const int f = max(PS.i_front, 0) / kW;
  const int tr = blockIdx.x;
  const int tc = front_first_block((int)blockIdx.y, f, (int)gridDim.y);
  const SurrArgs none = {};
  tile_body<false, kTfcTR, WavePrefetch, true, RAW>(
      K, F, PS, &tm_psi, &tm_c, tab, tab_len, psi_n, c_n, phi_n,
      partials ? partials + ((int64_t)tc * gridDim.x + tr) : nullptr, err, none, tr, tc,
      WavePrefetch{&tm_psi, &tm_c, f, wave_x, wave_y, kTfcTR});
}

}  // namespace

// The step kernels of the FP32 tiles and the shared memory they take; spread over
// the translation units as the FP64 ones (rs_tile_f64.cuh).
using StepFn32 = void (*)(StepCoef, Coef<float>, StepScalars, CUtensorMap, CUtensorMap, const float *, int, float *,
                          float *, float *, BlockPartial *, int *, SurrArgs, int, int);
struct StepKernel32 {
  StepFn32 fn;
  size_t smem;
};
using ExactFn32 = void (*)(StepCoef, Coef<float>, StepScalars, CUtensorMap, CUtensorMap, const float *, int, float *,
                           float *, float *, BlockPartial *, int *, int, int);  // (no surrogate argument)
struct ExactKernel32 {
  ExactFn32 fn;
  size_t smem;
};
StepKernel32 net_kernel_f32(int rows);       // rs_step_f32_net.cu
StepKernel32 raw_kernel_f32(int rows);       // rs_step_f32_raw.cu
ExactKernel32 tfc_kernel_f32(bool raw);      // rs_step_f32_tfc.cu
ExactKernel32 pipe_kernel_of_f32(int rows);  // rs_step_f32_pipe.cu
constexpr int kTileThreads32 = kThreads;
constexpr int kPipeThreads32 = 32 + 2 * kThreads;

}  // namespace rs
