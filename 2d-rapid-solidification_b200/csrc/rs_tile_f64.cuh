// rs_tile_f64.cuh — the FP64 (exact, drop-in) fused phase-field step on
// TMA-staged tiles: the phases and the one-tile-per-CTA kernel.  Included by
// rs_step_f64t.cu (the column table, the kernels of aligned fields, the launch),
// rs_step_f64t_raw.cu, rs_step_f64t_tfc.cu, rs_step_f64t_tfc_raw.cu and
// rs_step_f64t_pipe.cu.
//
// Same equations as the register-prefetch kernel of rs_step.cu
// (compute_phi / compute_psi / compute_c_CALPHAD, fun.cu:1143-1467) and the
// same tile organisation as the FP32 kernel of rs_tile_f32.cuh, in FP64 on the
// reference's own field layout (psi and c as doubles).  One step is two
// launches:
//   * column_table_kernel_f64: the per-column CALPHAD groups of this step's
//     frozen temperature (col_terms, get_delta fun.cu:1610-1619) in FP64;
//   * tile_kernel_f64.
// (Grids of one wave of CTAs: the second alone, its tiles computing their own
// columns' groups.)  Both are programmatic dependent launches: they are scheduled while the
// kernel before them drains and wait for it on the device, so a run's steps
// follow one another without launch gaps (2048^2, all solid: 28.7 -> 26.4 us).
//
// A CTA of 128 threads owns a tile of TR output rows x 64 output columns
// (x0 .. x0+63, x0 a multiple of 64; TR = 4, 8 or 16 by tile_rows_f64).  Its
// input, TR + 2 rows x 72 columns (x0-4 .. x0+67, so the TMA x coordinate stays
// 16-byte aligned), arrives in shared memory by one TMA box per field.  Two
// adjacent columns per lane (16-byte double2 shared-memory accesses).  The CTA
// votes on the tile's form:
//   * far melt everywhere (the bulk of a run ahead of its front): the c update
//     straight from registers to global memory (melt_tile), one barrier after
//     the load (frozen temperature only);
//   * deep solid everywhere: psi and c stay (solid_tile);
//   * anything else, the phases:
//   phase 1  per-cell S = q(psi) c (1-c) and mu'' of the input rows into
//            shared memory, with per-row flags "every psi == -1" / "== +1"
//            and per-lane phi masks; the halo columns x0-1 and x0+64 are
//            computed by 36 threads of warps 2 and 3 (one input row fewer);
//   phase 2  each warp computes its output rows: face fluxes from the shared S
//            and mu'' (neighbours straight from shared memory), the c update
//            (kept in registers); cells whose 3x3 phi neighbourhood is not
//            uniformly +-1 are listed;
//   phase 3  the listed interface cells are updated one per thread, those that
//            draw noise (a third of the tail cells of a planar front, at more
//            than twice the cost) apart from the others;
//   phase 4  new psi and c are written into the shared tile, ghost columns
//            copied there, and each output row leaves by one bulk async copy
//            per field (ghost rows by one more, except in row-band mode);
//   partials the solute mass (FP64) and coarse tip of the tile; a dependent
//            launch reduces them all.
// What bounds it: a 2048^2 grid ahead of a planar front (34.8 us a step, 43.0
// without the melt form and the chained launches, floor 20.5) its instruction
// issue and the load -> compute -> store chain of a CTA; small grids (256^2:
// 6.5 us, 12.1 with 16-row tiles and a table launch) and fronts the chain of the
// phases.
// Arithmetic (identical mathematics to the reference, regrouped as in the
// FP32 tile kernel):
//   * mu = K(T) + C0(T) + mu'', C0 = -D - (L0_BCC - L0_Liq)(1 - 2 cinf)/2, so
//       mu'' = -(g+1) C0 - delta (L0_BCC + L0_Liq + g (L0_BCC - L0_Liq)) + RT lam
//     and K + C0 enters only through its column differences dK;
//   * lam = log(c/(1-c)) - log(cinf/(1-cinf)) = 2 atanh(s),
//     s = delta / (2 cinf (1-c) + delta), by its series to s^15 where every
//     cell of the warp's row has |s| < 1/9 (truncation below 3.3e-17
//     relative), else by the logarithm;
//   * bulk melt rows (psi = -1 exactly, delta in the series range): g = -1,
//     q = 1, so mu'' = -2 L0_Liq delta + RT lam and S = c (1 - c); far-melt
//     rows (|delta| <= 1e-3 min(cinf, 1-cinf) as well) take lam as its
//     Taylor polynomial in delta (Coef::melt_a), without the division of s;
//   * deep solid rows (psi = +1 over the 3x3 neighbourhoods) store
//     S = mu'' = 0: every face weight touching them is 0;
//   * face weights by pair sums (6 P_i + P_{i-1} + P_{i+1}, four times the
//     1.5 / 0.25 weights, the 4 folded into the flux constant); face fluxes
//     are rounded products, so a cell's result does not depend on the tiling.
// Launch order: the tile columns from the one holding the front
// (front_first_block).  Once its own tile has arrived each CTA prefetches into
// L2 the input tile of the block launched one resident wave later.
// The coarse-grid temperature (TFC, interpolate_temperature
// fun.cu:1580-1608): no table kernel; every cell evaluates its CALPHAD groups
// from its own bilinear temperature (K + C0 by its Taylor polynomial about
// the tile's centre temperature, kc_poly, and C0 and the driving-force groups
// likewise, drive_poly on a second thread; cells out of the polynomials' range
// by the Gibbs functions) and
// stores mu = mu'' + (K + C0), so the faces take plain differences of mu.  Melt
// tiles take the phases and only tiles whose first interior cell is solid vote
// (2048^2 all melt: 59.2 us; 74.7 with the melt form and a vote in every
// tile, of which most fail).  768 x 832 with a cellular front: 22.7 to 25.6 us a
// step by where the front lies in its tile column (34.7 to 36.2 before the
// polynomials and the 8-row tiles).
//
// Two kernels run these phases (same functions, same results bit for bit):
//   * tile_kernel_f64: one tile per CTA of 128 threads, the phases in series
//     separated by CTA barriers, five CTAs per SM;
//   * pipe_kernel_f64: persistent CTAs of three warp roles that work on
//     three tiles at once -- one producer warp issuing the TMA loads of tile
//     k+2 into a three-slot input ring, four warps computing phase 1 of tile
//     k+1 into a two-slot staging ring, four warps doing phases 2-4 of tile k
//     and its bulk stores.  Hand-offs are mbarriers (full / empty per slot),
//     each role synchronises its own warps by a named barrier, every wait is
//     bounded (a wait that gives up sets the error flag and the CTA stops
//     after draining its loads and stores).
#pragma once

#include <type_traits>

#include "rs_step_common.cuh"

namespace rs {
namespace {

constexpr int kW = kTileOutW64;   // output columns of a tile
constexpr int kWin = kTmaBoxW64;  // input columns of a tile (kW + 8)
constexpr int kThreads = 128;     // threads of a phase group
constexpr int kWarps = kThreads / 32;
constexpr int kHaloL = 3, kHaloR = kW + 4;  // box columns of x0-1 and x0+kW
constexpr uint32_t kWaitLimit = 1u << 20;
constexpr unsigned FULL = 0xffffffffu;
constexpr unsigned long long kMinus1 = 0xBFF0000000000000ull, kPlus1 = 0x3FF0000000000000ull;
static_assert(kW == 32 * 2, "two columns per lane");
// column table arrays (kColTabFields of them, len doubles each); entry k
// describes column k - 4
enum { kTabRT = 0, kTabC0 = 1, kTabDK = 2, kTabAnb = 3, kTabAti = 4 };

__device__ __forceinline__ double2 ld2(const double *p) { return *reinterpret_cast<const double2 *>(p); }
__device__ __forceinline__ void st2(double *p, double a, double b) {
  *reinterpret_cast<double2 *>(p) = make_double2(a, b);
}
__device__ __forceinline__ double clamp1(double v) { return fmin(fmax(v, -1.0), 1.0); }
__device__ __forceinline__ unsigned long long bits(double v) { return (unsigned long long)__double_as_longlong(v); }
// barrier of one phase group of 128 threads (id 0 with 128-thread CTAs: the CTA)
__device__ __forceinline__ void gsync(int id) { asm volatile("bar.sync %0, 128;" ::"r"(id) : "memory"); }
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// 2 atanh(s) by its odd series to s^15 (|s| < 1/9: truncation below
// 3.3e-17 relative)
__device__ __forceinline__ double lam_series(double s) {
  const double s2 = s * s;
  double p = 1.0 / 15.0;
  p = fma(p, s2, 1.0 / 13.0);
  p = fma(p, s2, 1.0 / 11.0);
  p = fma(p, s2, 1.0 / 9.0);
  p = fma(p, s2, 1.0 / 7.0);
  p = fma(p, s2, 1.0 / 5.0);
  p = fma(p, s2, 1.0 / 3.0);
  return 2.0 * fma(s * s2, p, s);
}

// general per-cell terms (fun.cu:1424-1452); series: use 2 atanh(s)
__device__ __forceinline__ void cell_terms(const Coef<double> &F, double pv, double c, double s, bool series,
                                           double RT, double C0, double &S, double &mu) {
  constexpr double L0sum = kL0Bcc + kL0Liq;
  constexpr double L0half = 0.5 * (kL0Bcc - kL0Liq);
  const double om = 1.0 - c, dv = c - F.cinf;
  const double a = 1.0 - pv;
  S = (0.5 * F.AA * a - 0.25 * (F.AA - 1.0) * (a * a)) * c * om;
  const double p2 = pv * pv;
  const double g = pv * (1.875 + p2 * (-1.25 + 0.375 * p2));
  const double lam = series ? lam_series(s) : Tr<double>::lam(c, om, dv, F.cinf, F.Lref);
  mu = -(g + 1.0) * C0 - dv * fma(2.0 * L0half, g, L0sum) + RT * lam;
}

// A far-melt cell (psi = -1 exactly, |delta| <= melt_tiny): g = -1, q = 1, lam
// by its Taylor polynomial in delta (Coef::melt_a, six terms, ma),
// mu'' = RT lam - 2 L0_Liq delta = delta (RT p + KL), lam = delta p; with TFC
// plus the cell's K + C0.  Rounded products: phase 1 and the melt tiles give
// the same bits.
template <bool TFC>
__device__ __forceinline__ void far_cell(const double (&ma)[6], double c, double dv, double RT, double KC, double &S,
                                         double &mu) {
  constexpr double KL = -2.0 * kL0Liq;
  double p = ma[5];
#pragma unroll
  for (int k = 4; k >= 0; --k) p = fma(p, dv, ma[k]);
  S = __dmul_rn(c, 1.0 - c);
  const double w = fma(RT, p, KL);
  mu = TFC ? fma(dv, w, KC) : __dmul_rn(dv, w);
}
// a bulk-melt cell (psi = -1 exactly, delta in the series range)
template <bool TFC>
__device__ __forceinline__ void bulk_cell(double cinf, double c, double dv, double RT, double KC, double &S,
                                          double &mu) {
  const double om = 1.0 - c;
  const double sv = dv / fma(2.0 * cinf, om, dv);
  S = __dmul_rn(c, om);
  mu = fma(RT, lam_series(sv), __dmul_rn(dv, -2.0 * kL0Liq));
  if (TFC) mu += KC;
}

// shared -> global bulk copy (16-byte aligned addresses, size a multiple of 16)
__device__ __forceinline__ void bulk_store(void *gdst, const void *ssrc, uint32_t bytes) {
  asm volatile("cp.async.bulk.global.shared::cta.bulk_group [%0], [%1], %2;" ::"l"(gdst), "r"(smem_u32(ssrc)),
               "r"(bytes)
               : "memory");
}

// The table entries of the column at temperature T (dK by the caller, from KC,
// K + C0).  Out of line: the table kernel and the tiles that compute their own
// columns run one copy of it, so their entries are the same bits.
struct ColEntry {
  double RT, C0, KC, Anb, Ati;
};
__device__ __noinline__ ColEntry col_entry(const double T, const double RR, const double cinf, const double Lref) {
  StepCoef K;
  K.RR = RR;
  K.cinf = cinf;
  K.Lref = Lref;
  const ColT<double> ct = col_terms<double>(K, T);
  const double C0 = -ct.D - 0.5 * (kL0Bcc - kL0Liq) * (1.0 - 2.0 * cinf);
  return {ct.RT, C0, ct.Kc + C0, ct.A_nb, ct.A_ti};
}

// the column table, indexed by column
struct Tab {
  const double *RT, *C0, *DK, *Anb, *Ati;
  __device__ Tab(const double *tab, int len)
      : RT(tab + kTabRT * len + 4), C0(tab + kTabC0 * len + 4), DK(tab + kTabDK * len + 4),
        Anb(tab + kTabAnb * len + 4), Ati(tab + kTabAti * len + 4) {}
};

// Everything that depends on the tile's height: TR output rows (4, 8 or 16), a
// warp taking every fourth of them.  A tile's latency is the chain load ->
// phases -> stores of its four warps, and a tile at the front takes long (its
// phase 3 alone 6 to 8 rounds at 16 rows), so a grid whose 16-row tiles would
// leave SMs idle takes lower ones (tile_rows).
// RAW: the fields' rows are not 16-byte aligned (any nx): the tile is copied in
// element by element, the cells leave by plain stores.
template <int TR, bool RAW = false>
struct TileOps {
static constexpr int kTR = TR, kTRin = TR + 2;  // output and input rows
static constexpr int kRowsPerWarp = TR / kWarps;
static constexpr uint32_t kTileBytes = 2u * kTRin * kWin * sizeof(double);
static_assert(TR % kWarps == 0 && kRowsPerWarp * kWarps == TR, "output rows split evenly over the warps");
static_assert(kTRin <= 32, "row flags are 32-bit masks");
static_assert(64 + 2 * kTRin <= kThreads && 4 * kTR <= kThreads, "one thread per halo cell and per row copy");

// the input tile: TMA destinations (128-byte aligned); after phase 3 rows
// 1..16 receive the new psi / c for the bulk stores
struct alignas(128) InSlot {  // both arrays are TMA destinations: 128-byte aligned
  alignas(128) double psi[kTRin][kWin];
  alignas(128) double c[kTRin][kWin];
};
// phase 1 -> phases 2-4: per-cell terms
struct alignas(128) StArr {
  double S[kTRin][kWin];  // after phase 2: new psi of the listed cells
  double mu[kTRin][kWin];
};
// and row flags
struct alignas(16) StFlags {
  uint8_t pmask[kTRin][32];  // per lane: bits 0-1 psi <= -1, bits 4-5 psi >= 1 of its two cells
                             // (rows flagged in liq / sol store none)
  uint8_t hmask[kTRin][2];   // halo cells: bit 0 psi <= -1, bit 1 psi >= 1
  uint32_t liq, sol;         // bit r: every cell of input row r has psi == -1 / +1
};
// TFC: what a tile's temperatures need, once per tile
struct TfcTile {
  double ty[kTRin];  // the row part of each input row's temperature (tfc_row)
  int tj[kTRin];
  KcPoly kp;         // K + C0 near the tile's temperature
  double hx[2];      // column part of the halo columns' temperatures
  int hiT[2];
  double tx[kW];     // and of the tile's columns (tfc_col)
  int ti[kW];
};
// phases 2-4: the interface list and the partial sums
struct P2Smem {
  // interface cells (row << 8 | output column): those that draw noise from the
  // front, the others from the back, so that phase 3's warps are of one kind
  uint16_t list[kTR * kW];
  uint32_t nlist;  // how many of the first kind, and << 16 of the second
  double part_mass[kWarps];
  int part_itip[kWarps];
};
// melt tiles: S and mu of the halo columns of each warp's rows
static constexpr int kHaloTerms = 2 * (kRowsPerWarp + 2);
struct MeltHalo {
  double s[kWarps][kHaloTerms], m[kWarps][kHaloTerms];
};
static_assert(sizeof(MeltHalo) <= sizeof(uint16_t) * kTR * kW, "a melt tile's halo terms use the list's room");
template <bool TFC>
struct alignas(128) TileSmem {
  InSlot in;
  StArr st;
  StFlags fl;
  alignas(16) P2Smem p2;
  std::conditional_t<TFC, TfcTile, char> tf;
  uint64_t full;
  uint32_t vote;  // the tile's form (tile_vote), OR of every thread's
};
// Everything one phase group needs about a tile and its own lane.
struct TileView {
  const StepCoef &K;
  const Coef<double> &F;
  const StepScalars &PS;
  Tab T;
  int x0, y0;  // first output column, first output row (input rows y0-1 .. y0+kTR)
  int gw, lane, gtid;  // warp and lane within the group, thread of the group
  int col, gi, bc;     // the lane's first cell: tile column, global column, box column
  uint32_t outm;       // per cell of the lane: an interior (output) cell
  __device__ TileView(const StepCoef &K_, const Coef<double> &F_, const StepScalars &PS_, const double *tab,
                      int tab_len, int x0_, int y0_, int gtid_)
      : K(K_), F(F_), PS(PS_), T(tab, tab_len), x0(x0_), y0(y0_), gw(gtid_ >> 5), lane(gtid_ & 31), gtid(gtid_) {
    col = 2 * lane;
    gi = x0 + col;
    bc = col + 4;
    outm = 0;
#pragma unroll
    for (int q = 0; q < 2; ++q)
      if (gi + q >= 1 && gi + q <= K.nx - 2) outm |= 1u << q;
  }
};

// The column table entries a lane uses: RT and C0 of its two columns, dK of
// the faces left of its columns and of the next one.  The tile kernel loads
// them before it waits for its tile, so their latency hides under the load.
struct LaneCols {
  double RT[2], C0[2], dK[3];
};
template <bool TFC>
static __device__ __forceinline__ LaneCols lane_cols(const TileView &V) {
  LaneCols L;
  if constexpr (TFC) {  // per cell (cell_tfc); no column differences
    L.RT[0] = L.RT[1] = L.C0[0] = L.C0[1] = 0.0;
    L.dK[0] = L.dK[1] = L.dK[2] = 0.0;
    return L;
  }
  const double2 RTv = ld2(V.T.RT + V.gi), C0v = ld2(V.T.C0 + V.gi);
  L.RT[0] = RTv.x;
  L.RT[1] = RTv.y;
  L.C0[0] = C0v.x;
  L.C0[1] = C0v.y;
  L.dK[0] = V.T.DK[V.gi - 1];  // faces x-1|x for x = col .. col+2
  L.dK[1] = V.T.DK[V.gi];
  L.dK[2] = V.T.DK[V.gi + 1];
  return L;
}

// columns beyond the array (right-most tiles; zero-filled by TMA) become
// bulk melt, so they never force the general path; no output reads them.
// Returns whether it wrote (the group then synchronises).
static __device__ __forceinline__ bool fix_beyond(const TileView &V, InSlot &in) {
  if (V.x0 + kW + 4 <= V.K.nx) return false;
  for (int k = V.gtid; k < kTRin * kWin; k += kThreads) {
    const int rr = k / kWin, x = k % kWin;
    if (V.x0 - 4 + x >= V.K.nx) {
      in.psi[rr][x] = -1.0;
      in.c[rr][x] = V.F.cinf;
    }
  }
  return true;
}

// S and mu of a cell of the halo columns x0-1 (side 0), x0+kW (side 1), at
// global column g: the far-melt form where the cell has it, else the general
// one (a cell's form does not depend on the tile)
template <bool TFC>
static __device__ __forceinline__ void halo_cell(const TileView &V, const TfcTile *tf, const double (&ma)[6], double pv,
                                          double cv, int rr, int side, int g, double &Sh, double &mh) {
  const Coef<double> &F = V.F;
  const double dv = cv - F.cinf;
  double RT, C0, KC = 0.0;
  if constexpr (TFC) {
    // C0 enters mu'' as (g + 1) C0, 0 at psi = -1 exactly: the liquid
    // groups suffice there
    cell_tfc(V.K, tf->kp, tfc_T(V.K, V.PS.T_coarse, tf->hiT[side], tf->hx[side], tf->tj[rr], tf->ty[rr]),
             bits(pv) != kMinus1, RT, C0, KC);
  } else {
    RT = V.T.RT[g];
    C0 = V.T.C0[g];
  }
  if (bits(pv) == kMinus1 && fabs(dv) <= F.melt_tiny) {
    far_cell<TFC>(ma, cv, dv, RT, KC, Sh, mh);
    return;
  }
  const double sv = dv / fma(2.0 * F.cinf, 1.0 - cv, dv);
  cell_terms(F, pv, cv, sv, fabs(sv) < 1.0 / 9.0, RT, C0, Sh, mh);
  if (TFC) mh += KC;
}

// ---- phase 1: per-cell terms of the input rows of group warp gw (rows gw,
// gw+4, ...) and of the halo columns (group threads 64..99); st.liq and
// st.sol must be 0 on entry
template <bool TFC>
static __device__ __forceinline__ void phase1(const TileView &V, const LaneCols &LC, const InSlot &in, StArr &sa, StFlags &st,
                                       const TfcTile *tf) {
  const Coef<double> &F = V.F;
  const int lane = V.lane, bc = V.bc;
  const double cinf = F.cinf;
  const double d_hi = F.ser_hi, d_lo = F.ser_lo;  // series range of delta (Coef)
  double RTa[2] = {LC.RT[0], LC.RT[1]}, C0a[2] = {LC.C0[0], LC.C0[1]}, KCa[2] = {0.0, 0.0};
  // per lane, bit q: psi is exactly +1 over the 3x3 neighbourhood of cell
  // bc+q (rows of the box only; column -1 of the left-most tile enters no
  // face, column 0 being a ghost).  S = q(1) c (1 - c) = 0 there, so every
  // face weight touching the cell is 0 and its mu'' enters no flux
  auto solid3 = [&](int rr) -> uint32_t {
    const int xh = lane == 0 ? kHaloL : kHaloR;
    uint32_t v = 0x3u;
    bool hs = true;  // the halo column beside lanes 0 and 31
    for (int r2 = max(rr - 1, 0); r2 <= min(rr + 1, kTRin - 1); ++r2) {
      const double2 q2 = ld2(&in.psi[r2][bc]);
      v &= (bits(q2.x) == kPlus1 ? 1u : 0u) | (bits(q2.y) == kPlus1 ? 2u : 0u);
      hs = hs && bits(in.psi[r2][xh]) == kPlus1;
    }
    uint32_t lf = __shfl_up_sync(FULL, v >> 1, 1) & 1u, rt = __shfl_down_sync(FULL, v, 1) & 1u;
    if (lane == 0) lf = (hs || V.x0 == 0) ? 1u : 0u;
    if (lane == 31) rt = hs ? 1u : 0u;
    const uint32_t e = lf | (v << 1) | (rt << 3);  // bit k: box column bc-1+k
    return e & (e >> 1) & (e >> 2) & 0x3u;
  };
  // constants of the row loop in registers (one read of the launch
  // arguments, not one per row)
  double ma[6];
#pragma unroll
  for (int k = 0; k < 6; ++k) ma[k] = F.melt_a[k];
  const double tiny = F.melt_tiny;
  const int rows_in = V.K.ny - V.y0;  // input rows inside the array: rr <= ny - y0
  // this warp's row flags (warp-uniform), OR-ed into st.liq / st.sol once
  uint32_t liq_rows = 0u, sol_rows = 0u;
  // TFC: along a column the bilinear temperature is P + Q y within one coarse
  // row band jT; the lane keeps P and Q of its two columns for the band of
  // its last row (rows of a warp are 4 apart, bands `ratio` rows high)
  int band_jT = -1;
  double Pb[2] = {0.0, 0.0}, Qb[2] = {0.0, 0.0};
#pragma unroll 1
  for (int rr = V.gw; rr < kTRin; rr += kWarps) {
    if (rr > rows_in) {  // beyond the array (last tile): never read by an output
      st2(&sa.S[rr][bc], 0.0, 0.0);
      st2(&sa.mu[rr][bc], 0.0, 0.0);
      liq_rows |= 1u << rr;
      sol_rows |= 1u << rr;
      continue;
    }
    const double2 pv2 = ld2(&in.psi[rr][bc]), cv2 = ld2(&in.c[rr][bc]);
    const double pv[2] = {pv2.x, pv2.y}, cv[2] = {cv2.x, cv2.y};
    const double dv[2] = {cv[0] - cinf, cv[1] - cinf};
    double Sv[2], mv[2];
    const unsigned long long b0 = bits(pv[0]), b1 = bits(pv[1]);
    const bool liq2 = b0 == kMinus1 && b1 == kMinus1;
    const bool sol2 = b0 == kPlus1 && b1 == kPlus1;
    // the row's form (warp-uniform): far melt, bulk melt or general
    const bool far = __all_sync(FULL, liq2 && fmax(fabs(dv[0]), fabs(dv[1])) <= tiny);
    const bool bulk = !far && __all_sync(FULL, liq2 && fmax(dv[0], dv[1]) < d_hi && fmin(dv[0], dv[1]) > d_lo);
    if constexpr (TFC) {  // the melt forms need RT and K + C0 only
      const int jT = tf->tj[rr];
      const double y = tf->ty[rr];
      if (jT != band_jT) {  // warp-uniform: jT depends on the row only
        band_jT = jT;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          const double tx = tf->tx[V.col + q];
          const double *r0 = V.PS.T_coarse + (int64_t)jT * V.K.NxT_all + tf->ti[V.col + q], *r1 = r0 + V.K.NxT_all;
          const double f00 = r0[0], f10 = r0[1], f01 = r1[0], f11 = r1[1];
          Pb[q] = fma(f10 - f00, tx, f00);
          Qb[q] = fma(f11 - f10 - f01 + f00, tx, f01 - f00);
        }
      }
#pragma unroll
      for (int q = 0; q < 2; ++q)
        cell_tfc(V.K, tf->kp, fma(Qb[q], y, Pb[q]), !(far || bulk), RTa[q], C0a[q], KCa[q]);
    }
    uint32_t code;
    bool deep = false;
    if (far) {
      code = 1u;
#pragma unroll
      for (int q = 0; q < 2; ++q) far_cell<TFC>(ma, cv[q], dv[q], RTa[q], KCa[q], Sv[q], mv[q]);
    } else if (bulk) {
      code = 1u;
#pragma unroll
      for (int q = 0; q < 2; ++q) bulk_cell<TFC>(cinf, cv[q], dv[q], RTa[q], KCa[q], Sv[q], mv[q]);
    } else {
      code = (__all_sync(FULL, liq2) ? 1u : 0u) | (__all_sync(FULL, sol2) ? 2u : 0u);
      // deep solid row: no cell's mu'' enters a flux, so S = mu'' = 0 gives
      // the same fluxes
      const uint32_t s3 = (code & 2u) ? solid3(rr) : 0u;
      if ((code & 2u) && __all_sync(FULL, s3 == 0x3u)) {
        Sv[0] = Sv[1] = mv[0] = mv[1] = 0.0;
        deep = true;
      } else {
        double sv[2];
        bool small = true;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          sv[q] = dv[q] / fma(2.0 * cinf, 1.0 - cv[q], dv[q]);
          small = small && fabs(sv[q]) < 1.0 / 9.0;
        }
        const bool series = __all_sync(FULL, small);
        uint32_t L = 0u, Sm = 0u;
#pragma unroll
        for (int q = 0; q < 2; ++q) {
          if (pv[q] <= -1.0) L |= 1u << q;
          if (pv[q] >= 1.0) Sm |= 1u << q;
          cell_terms(F, pv[q], cv[q], sv[q], series, RTa[q], C0a[q], Sv[q], mv[q]);
        }
        st.pmask[rr][lane] = (uint8_t)(L | (Sm << 4));
      }
    }
    if (TFC && !deep && !far && !bulk) {  // mu = mu'' + (K + C0) of the cell itself
      mv[0] += KCa[0];
      mv[1] += KCa[1];
    }
    st2(&sa.S[rr][bc], Sv[0], Sv[1]);
    st2(&sa.mu[rr][bc], mv[0], mv[1]);
    liq_rows |= (code & 1u) << rr;
    sol_rows |= ((code >> 1) & 1u) << rr;
  }
  if (lane == 0) {
    if (liq_rows) atomicOr(&st.liq, liq_rows);
    if (sol_rows) atomicOr(&st.sol, sol_rows);
  }
  // halo columns x0-1 and x0+kW, one thread per cell, on group warps 2 and
  // 3, which have one input row fewer than warps 0 and 1
  if (V.gtid >= 64 && V.gtid < 64 + 2 * kTRin) {
    const int i = V.gtid - 64;
    const int rr = i >> 1, side = i & 1;
    const int x = side ? kHaloR : kHaloL, g = V.x0 - 4 + x;
    double Sh = 0.0, mh = 0.0;
    uint8_t hm = 3u;
    if (V.y0 - 1 + rr <= V.K.ny - 1) {
      const double pv = in.psi[rr][x], cv = in.c[rr][x];
      halo_cell<TFC>(V, tf, ma, pv, cv, rr, side, g, Sh, mh);
      hm = (pv <= -1.0 ? 1u : 0u) | (pv >= 1.0 ? 2u : 0u);
    }
    sa.S[rr][x] = Sh;
    sa.mu[rr][x] = mh;
    st.hmask[rr][side] = hm;
  }
}

// ---- phase 2: group warp gw computes output rows 1 + 4gw .. 4 + 4gw:
// fluxes, the c update into dn, the interface cells into the list (nlist
// must be 0 on entry).  Returns the listed cells, 2 bits per output row.
static __device__ __forceinline__ uint32_t phase2(const TileView &V, const LaneCols &LC, const InSlot &in,
                                           const StArr &sa, const StFlags &st, P2Smem &p2,
                                           double dn[kRowsPerWarp][2], double &mass, bool red) {
  const Coef<double> &F = V.F;
  const int lane = V.lane, bc = V.bc;
  const double cflux4 = 0.25 * F.cflux, c_floor = F.c_floor;
  const int rows_live = V.K.ny - 1 - V.y0;  // output rows inside the interior: rr <= ny - 1 - y0
  const uint32_t liq = st.liq, sol = st.sol;
  const double dKa[3] = {LC.dK[0], LC.dK[1], LC.dK[2]};  // faces x-1|x for x = col .. col+2
  struct Row {
    double s[2], m[2], sl, sr, ml, mr;
  };
  // S pair sums of the faces left of cell f (f = 0..2) of a row
  struct Pairs {
    double q[3];
  };
  auto load_row = [&](int rr, Row &R) {
    const double2 s = ld2(&sa.S[rr][bc]), m = ld2(&sa.mu[rr][bc]);
    R.s[0] = s.x;
    R.s[1] = s.y;
    R.m[0] = m.x;
    R.m[1] = m.y;
    R.sl = sa.S[rr][bc - 1];  // lane 0: the halo column x0-1
    R.ml = sa.mu[rr][bc - 1];
    R.sr = sa.S[rr][bc + 2];  // lane 31: the halo column x0+kW
    R.mr = sa.mu[rr][bc + 2];
  };
  auto pairs = [](const Row &R) {
    Pairs P;
    P.q[0] = R.sl + R.s[0];
    P.q[1] = R.s[0] + R.s[1];
    P.q[2] = R.s[1] + R.sr;
    return P;
  };
  // fluxes through the faces between rows A and B = A+1 (compute_c_CALPHAD
  // F01/F0m), rounded products so that a face rounds the same wherever the
  // tiling puts it
  auto vface = [&](const Row &A, const Row &B, double jv[2]) {
    const double pp[4] = {A.sl + B.sl, A.s[0] + B.s[0], A.s[1] + B.s[1], A.sr + B.sr};
#pragma unroll
    for (int q = 0; q < 2; ++q) jv[q] = __dmul_rn(fma(6.0, pp[q + 1], pp[q] + pp[q + 2]), B.m[q] - A.m[q]);
  };

  const int rbase = 1 + kRowsPerWarp * V.gw;
  Row rb, rc;
  Pairs pa, pb, pc;
  double jv_lo[2], jv_hi[2];
  uint32_t needs_all = 0u;
  {
    Row ra;
    load_row(rbase - 1, ra);
    load_row(rbase, rb);
    vface(ra, rb, jv_lo);
    pa = pairs(ra);
    pb = pairs(rb);
  }
#pragma unroll
  for (int j = 0; j < kRowsPerWarp; ++j) {
    const int rr = rbase + j;  // tile input row of the output row
    load_row(rr + 1, rc);
    pc = pairs(rc);
    vface(rb, rc, jv_hi);
    // fluxes through the faces (x-1/2, r) for x = col .. col+2
    const double mm[4] = {rb.ml, rb.m[0], rb.m[1], rb.mr};
    double jh[3];
#pragma unroll
    for (int fc = 0; fc < 3; ++fc)
      jh[fc] = __dmul_rn(fma(6.0, pb.q[fc], pa.q[fc] + pc.q[fc]), mm[fc + 1] - mm[fc] + dKa[fc]);
    const double2 cv2 = ld2(&in.c[rr][bc]);
    const double cv[2] = {cv2.x, cv2.y};
#pragma unroll
    for (int q = 0; q < 2; ++q)
      dn[j][q] = fmax(fma(cflux4, (jh[q + 1] - jh[q]) + (jv_hi[q] - jv_lo[q]), cv[q]), c_floor);
    const bool live = rr <= rows_live;
    if (red && live) {
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if ((V.outm >> q) & 1u) mass += dn[j][q];
    }
    // phi: cells whose 3x3 neighbourhood is not uniformly +-1 are listed
    const uint32_t w3 = 7u << (rr - 1);
    if (live && (liq & w3) != w3 && (sol & w3) != w3) {
      // per input row k: bits 0-1 psi <= -1, bits 4-5 psi >= 1 of the lane's cells
      // (rows flagged all -1 / all +1 store no masks: 0x03 / 0x30)
      auto pm = [&](int k) -> uint32_t {
        return ((liq >> k) & 1u) ? 0x03u : ((sol >> k) & 1u) ? 0x30u : (uint32_t)st.pmask[k][lane];
      };
      const uint32_t pk = pm(rr - 1) | (pm(rr) << 8) | (pm(rr + 1) << 16);
      const uint32_t lf = __shfl_up_sync(FULL, pk, 1), rt = __shfl_down_sync(FULL, pk, 1);
      // left neighbour's second cell: its bits 1 and 5; right neighbour's first: bits 0 and 4
      uint32_t lL = 0u, lS = 0u, rL = 0u, rS = 0u;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        lL |= ((lf >> (8 * k + 1)) & 1u) << k;
        lS |= ((lf >> (8 * k + 5)) & 1u) << k;
        rL |= ((rt >> (8 * k)) & 1u) << k;
        rS |= ((rt >> (8 * k + 4)) & 1u) << k;
      }
      if (lane == 0) {
        lL = lS = 0u;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const uint32_t h = st.hmask[rr - 1 + k][0];
          lL |= (h & 1u) << k;
          lS |= ((h >> 1) & 1u) << k;
        }
      }
      if (lane == 31) {
        rL = rS = 0u;
#pragma unroll
        for (int k = 0; k < 3; ++k) {
          const uint32_t h = st.hmask[rr - 1 + k][1];
          rL |= (h & 1u) << k;
          rS |= ((h >> 1) & 1u) << k;
        }
      }
      // over the three rows, bit b: box column bc-1+b is liquid / solid
      uint32_t Lv = 0xFu, Sv = 0xFu;
#pragma unroll
      for (int k = 0; k < 3; ++k) {
        const uint32_t L = (pk >> (8 * k)) & 0x3u, S = (pk >> (8 * k + 4)) & 0x3u;
        Lv &= ((lL >> k) & 1u) | (L << 1) | (((rL >> k) & 1u) << 3);
        Sv &= ((lS >> k) & 1u) | (S << 1) | (((rS >> k) & 1u) << 3);
      }
      const uint32_t needs = ~((Lv & (Lv >> 1) & (Lv >> 2)) | (Sv & (Sv >> 1) & (Sv >> 2))) & V.outm;
      // cells that draw noise (phi_cell's own test; here it only sorts the list)
      const double2 ps2 = ld2(&in.psi[rr][bc]);
      const uint32_t noisy =
          F.noise_amp > 0.0 ? (fma(-ps2.x, ps2.x, 1.0) > 1.0e-3 ? 1u : 0u) | (fma(-ps2.y, ps2.y, 1.0) > 1.0e-3 ? 2u : 0u)
                            : 3u;
      // the lanes with such a cell (n) and with another listed one (t), per cell
      const uint32_t n0 = __ballot_sync(FULL, needs & noisy & 1u), n1 = __ballot_sync(FULL, needs & noisy & 2u);
      const uint32_t t0 = __ballot_sync(FULL, needs & ~noisy & 1u), t1 = __ballot_sync(FULL, needs & ~noisy & 2u);
      const uint32_t add = (__popc(n0) + __popc(n1)) | ((__popc(t0) + __popc(t1)) << 16);
      uint32_t base = 0u;
      if (lane == 0 && add) base = atomicAdd(&p2.nlist, add);
      base = __shfl_sync(FULL, base, 0);
      const uint32_t below = (1u << lane) - 1u;
      const uint32_t n_at = base & 0xFFFFu, t_at = kTR * kW - 1 - (base >> 16);
      if (needs & 1u)
        p2.list[(noisy & 1u) ? n_at + __popc(n0 & below) : t_at - __popc(t0 & below)] =
            (uint16_t)((rr << 8) | V.col);
      if (needs & 2u)
        p2.list[(noisy & 2u) ? n_at + __popc(n0) + __popc(n1 & below) : t_at - __popc(t0) - __popc(t1 & below)] =
            (uint16_t)((rr << 8) | (V.col + 1));
      needs_all |= needs << (2 * j);
    }
    rb = rc;
    pa = pb;
    pb = pc;
#pragma unroll
    for (int q = 0; q < 2; ++q) jv_lo[q] = jv_hi[q];
  }
  return needs_all;
}

// ---- phase 3: the listed interface cells, one per group thread
// (compute_phi, fun.cu:1143-1218); new psi into np[rr][x]
template <bool TFC>
static __device__ __forceinline__ void phase3(const TileView &V, const InSlot &in, const P2Smem &p2, const TfcTile *tf,
                                       double (*np)[kWin], bool red, int &itip) {
  const int na = (int)(p2.nlist & 0xFFFFu), nlist = na + (int)(p2.nlist >> 16);
  for (int idx = V.gtid; idx < nlist; idx += kThreads) {
    const uint32_t e = p2.list[idx < na ? idx : kTR * kW - 1 - (idx - na)];
    const int rr = (int)(e >> 8), x = (int)(e & 0xFFu) + 4;  // box column
    const int r = V.y0 - 1 + rr, g = V.x0 + x - 4;
    const double c00 = in.c[rr][x];
    double Anb, Ati;
    if constexpr (TFC) {
      const double T = tfc_T(V.K, V.PS.T_coarse, tf->ti[x - 4], tf->tx[x - 4], tf->tj[rr], tf->ty[rr]);
      drive_tfc(V.K, tf->kp, T, Anb, Ati);
    } else {
      Anb = V.T.Anb[g];
      Ati = V.T.Ati[g];
    }
    const double dG = drive_dG<double>(c00, Anb, Ati);
    const double res = phi_cell_dG<double>(
        &V.F, clamp1(in.psi[rr][x]), clamp1(in.psi[rr][x + 1]), clamp1(in.psi[rr][x - 1]),
        clamp1(in.psi[rr + 1][x]), clamp1(in.psi[rr - 1][x]), clamp1(in.psi[rr + 1][x + 1]),
        clamp1(in.psi[rr + 1][x - 1]), clamp1(in.psi[rr - 1][x + 1]), clamp1(in.psi[rr - 1][x - 1]), dG,
        V.PS.step, (int64_t)(r + V.K.j_offset) * V.K.nx + g, V.K.seed_lo, V.K.seed_hi);
    np[rr][x] = res;
    if (red && res > 0.0) itip = max(itip, g == V.K.nx - 2 ? V.K.nx - 1 : g);
  }
}

// ---- phase 4: new psi and c of group warp gw's rows into the input tile
// (after every group thread has finished phase 3)
static __device__ __forceinline__ void phase4_rows(const TileView &V, InSlot &in, const double (*np)[kWin],
                                            uint32_t needs_all, const double dn[kRowsPerWarp][2], bool red,
                                            int &itip) {
  const int rbase = 1 + kRowsPerWarp * V.gw, bc = V.bc;
#pragma unroll
  for (int j = 0; j < kRowsPerWarp; ++j) {
    const int rr = rbase + j;
    const double2 pv2 = ld2(&in.psi[rr][bc]);
    // phi_next = phi where uniformly +-1: an output cell is not listed only
    // where psi <= -1 or >= 1 over its 3x3 neighbourhood, so clamp(psi) is
    // its sign (cells outside the interior are not stored or are overwritten
    // by the ghost copies); listed cells take phase 3's result
    double po[2] = {pv2.x > 0.0 ? 1.0 : -1.0, pv2.y > 0.0 ? 1.0 : -1.0};
    const uint32_t lb = (needs_all >> (2 * j)) & 3u;
    if (lb) {
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if ((lb >> q) & 1u) po[q] = np[rr][bc + q];
    }
    st2(&in.psi[rr][bc], po[0], po[1]);
    st2(&in.c[rr][bc], dn[j][0], dn[j][1]);
  }
  if (red) {  // coarse tip: the last column with phi > 0 (listed cells counted again, harmlessly)
    const int rows_live = V.K.ny - 1 - V.y0, nx = V.K.nx;
#pragma unroll
    for (int j = 0; j < kRowsPerWarp; ++j) {
      const int rr = rbase + j;
      const double2 po2 = ld2(&in.psi[rr][bc]);
      const double po[2] = {po2.x, po2.y};
      if (rr > rows_live) continue;
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if (((V.outm >> q) & 1u) && po[q] > 0.0) itip = max(itip, V.gi + q == nx - 2 ? nx - 1 : V.gi + q);
    }
  }
}

// ghost columns, then the tile's rows out by bulk copies (group threads
// < 64: row j, field, kind) and phi by plain stores; returns whether this
// thread committed a bulk group (it then waits for its reads before the
// tile's shared memory is reused)
static __device__ __forceinline__ bool store_tile(const TileView &V, InSlot &in, double *__restrict__ psi_n,
                                           double *__restrict__ c_n, double *__restrict__ phi_n, int bar) {
  const StepCoef &K = V.K;
  const int x0 = V.x0, y0 = V.y0;
  const int nrow = min(kTR, K.ny - 1 - y0);  // output rows of this tile inside the interior
  if constexpr (RAW) {
    gsync(bar);
    for (int k = V.gtid; k < nrow * kW; k += kThreads) {
      const int j = k / kW, x = k % kW;
      raw_cell(V, y0 + j, x0 + x, in.psi[1 + j][4 + x], in.c[1 + j][4 + x], psi_n, c_n, phi_n);
    }
    return false;
  }
  const int ncol = min(kW, K.nx - x0);       // columns of this tile inside the array (even)
  if (x0 == 0 || x0 + kW >= K.nx) {
    // ghost columns 0 and nx-1 (compute_boundary_individual, fun.cu:1220-1230)
    gsync(bar);
    if (V.gtid < nrow) {
      const int rr = 1 + V.gtid;
      if (x0 == 0) {
        in.psi[rr][4] = in.psi[rr][5];
        in.c[rr][4] = in.c[rr][5];
      }
      if (x0 + kW >= K.nx) {
        const int x = K.nx - 1 - x0 + 4;
        in.psi[rr][x] = in.psi[rr][x - 1];
        in.c[rr][x] = in.c[rr][x - 1];
      }
    }
  }
  asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // tile writes -> bulk copies
  gsync(bar);
  bool any = false;
  if (V.gtid < 4 * kTR) {
    const int j = V.gtid >> 2, field = V.gtid & 1, kind = (V.gtid >> 1) & 1;
    const int r = y0 + j;
    if (j < nrow) {
      double *fo = field ? c_n : psi_n;
      const double *src = field ? &in.c[1 + j][4] : &in.psi[1 + j][4];
      const uint32_t bytes = (uint32_t)ncol * 8u;
      if (kind == 0) {
        bulk_store(fo + (int64_t)r * K.pitch + x0, src, bytes);
        any = true;
      } else {
        if (r == K.jmin) {
          bulk_store(fo + x0, src, bytes);
          any = true;
        }
        if (r == K.jmax) {
          bulk_store(fo + (int64_t)(K.ny - 1) * K.pitch + x0, src, bytes);
          any = true;
        }
      }
      if (any) asm volatile("cp.async.bulk.commit_group;" ::: "memory");
    }
  }
  if (phi_n) {  // phi = clamp(psi) of the same rows, plain stores
    for (int k = V.gtid; k < nrow * ncol; k += kThreads) {
      const int j = k / ncol, x = k % ncol, r = y0 + j;
      const double v = clamp1(in.psi[1 + j][4 + x]);
      phi_n[(int64_t)r * K.pitch + x0 + x] = v;
      if (r == K.jmin) phi_n[x0 + x] = v;
      if (r == K.jmax) phi_n[(int64_t)(K.ny - 1) * K.pitch + x0 + x] = v;
    }
  }
  return any;
}

// the tile's partial sums (a dependent launch reduces them)
static __device__ __forceinline__ void finish_tile(const TileView &V, P2Smem &p2, double mass, int itip,
                                            BlockPartial *part, int bar) {
  if (!part) return;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mass += __shfl_down_sync(FULL, mass, o);
  itip = __reduce_max_sync(FULL, itip);
  if (V.lane == 0) {
    p2.part_mass[V.gw] = mass;
    p2.part_itip[V.gw] = itip;
  }
  gsync(bar);
  if (V.gtid == 0) {
    BlockPartial b;
    b.mass = 0.0;
    b.itip = 0;
#pragma unroll
    for (int w = 0; w < kWarps; ++w) {
      b.mass += p2.part_mass[w];
      b.itip = max(b.itip, p2.part_itip[w]);
    }
    b.pad = 0;
    *part = b;
  }
}

// ---- whole-tile forms: a tile whose input box is far melt (psi = -1 exactly,
// |delta| <= melt_tiny) or deep solid (psi = +1 exactly) throughout needs
// no masks, list or interface pass.  The CTA votes over every cell of the box
// that an output reads (rows and columns outside the array are left out).  The ranges of delta are compared
// by the high words of the doubles, on the safe side.  (Melt within the series
// range only, the solute layer ahead of the front, keeps the phases: its rows
// choose their form one by one, and a register form of that took 50 us on a
// 2048^2 grid of such melt against 45.)
enum : uint32_t { kNotMinus1 = 1u, kNotPlus1 = 2u, kNotFar = 4u, kNotFinite = 8u, kGaveUp = 16u };
static __device__ __forceinline__ uint32_t hi_abs(double v) { return (uint32_t)__double2hiint(v) & 0x7fffffffu; }
static __device__ __forceinline__ uint32_t tile_vote(const TileView &V, const InSlot &in) {
  const Coef<double> &F = V.F;
  const double cinf = F.cinf;
  const int rows_in = V.K.ny - V.y0;
  uint32_t m1 = 0u, p1 = 0u, dm = 0u;  // OR of psi's difference from -1 / +1, largest |delta| (high word)
  auto cell = [&](double p, double c) {
    const uint32_t lo = (uint32_t)__double2loint(p), hi = (uint32_t)__double2hiint(p);
    m1 |= lo | (hi ^ 0xBFF00000u);
    p1 |= lo | (hi ^ 0x3FF00000u);
    dm = max(dm, hi_abs(c - cinf));
  };
#pragma unroll
  for (int k = 0; k < (kTRin + kWarps - 1) / kWarps; ++k) {
    const int rr = V.gw + kWarps * k;
    if (rr < kTRin && rr <= rows_in) {
      const double2 p = ld2(&in.psi[rr][V.bc]), c = ld2(&in.c[rr][V.bc]);
      cell(p.x, c.x);
      cell(p.y, c.y);
    }
  }
  // the halo columns, one cell per thread, on the warps with a row fewer
  if (V.gtid >= 64 && V.gtid < 64 + 2 * kTRin) {
    const int rr = (V.gtid - 64) >> 1, side = V.gtid & 1;
    if (rr <= rows_in && (side || V.x0 > 0)) cell(in.psi[rr][side ? kHaloR : kHaloL], in.c[rr][side ? kHaloR : kHaloL]);
  }
  return (m1 ? kNotMinus1 : 0u) | (p1 ? kNotPlus1 : 0u) | (dm < hi_abs(F.melt_tiny) ? 0u : kNotFar) |
         (dm < 0x3FF00000u ? 0u : kNotFinite);
}

// one interior cell by plain stores, with the ghost cells that copy it (others
// are left out)
static __device__ __forceinline__ void raw_cell(const TileView &V, int r, int g, double pv, double c,
                                                double *__restrict__ psi_n, double *__restrict__ c_n,
                                                double *__restrict__ phi_n) {
  const StepCoef &K = V.K;
  if (g < 1 || g > K.nx - 2) return;
  auto put = [&](int row, int col) {
    const int64_t o = (int64_t)row * K.pitch + col;
    psi_n[o] = pv;
    c_n[o] = c;
    if (phi_n) phi_n[o] = clamp1(pv);
  };
  auto row = [&](int rw) {
    put(rw, g);
    if (g == 1) put(rw, 0);
    if (g == K.nx - 2) put(rw, K.nx - 1);
  };
  row(r);
  if (r == K.jmin) row(0);
  if (r == K.jmax) row(K.ny - 1);
}

// new psi (constant pv) and c of the lane's two cells of the output rows of
// its warp straight to global memory, with the ghost columns and rows they
// copy to
// (raw: rows not 16-byte aligned, any nx; cell by cell)
struct CellStore {
  double *pr, *cr, *fr;  // the lane's cells of the row to store next
  int64_t pitch;
  double *stage;  // RAW: a row of shared memory of the warp's own
  bool live, left, right, ghost;
  __device__ CellStore(const TileView &V, double *stage_, double *psi_n, double *c_n, double *phi_n)
      : stage(stage_) {
    const StepCoef &K = V.K;
    const int r = V.y0 + kRowsPerWarp * V.gw;
    pitch = K.pitch;
    const int64_t o = (int64_t)r * pitch + V.gi;
    pr = psi_n + o;
    cr = c_n + o;
    fr = phi_n ? phi_n + o : nullptr;
    live = V.gi < K.nx;          // (nx is even: both cells or neither)
    left = V.gi == 0;            // ghost column 0
    right = V.gi + 2 == K.nx;    // ghost column nx-1
    ghost = (K.jmin >= r && K.jmin < r + kRowsPerWarp) || (K.jmax >= r && K.jmax < r + kRowsPerWarp);
  }
  // row r = y0 - 1 + rr, the next one of the warp
  __device__ void put(const TileView &V, int rr, double pv, double c0, double c1, double *psi_n, double *c_n,
                      double *phi_n) {
    if constexpr (RAW) {
      const int r = V.y0 - 1 + rr;
      st2(stage + V.col, c0, c1);  // so that each store is of 32 adjacent cells
      __syncwarp();
      raw_cell(V, r, V.x0 + V.lane, pv, stage[V.lane], psi_n, c_n, phi_n);
      raw_cell(V, r, V.x0 + V.lane + 32, pv, stage[V.lane + 32], psi_n, c_n, phi_n);
      __syncwarp();
      return;
    }
    if (left) c0 = c1;
    if (right) c1 = c0;
    if (live) {
      st2(pr, pv, pv);
      st2(cr, c0, c1);
      if (fr) st2(fr, pv, pv);
      if (ghost) {
        const int r = V.y0 - 1 + rr;
        auto copy = [&](int row) {
          const int64_t o = (int64_t)row * pitch + V.gi;
          st2(psi_n + o, pv, pv);
          st2(c_n + o, c0, c1);
          if (phi_n) st2(phi_n + o, pv, pv);
        };
        if (r == V.K.jmin) copy(0);
        if (r == V.K.jmax) copy(V.K.ny - 1);
      }
    }
    pr += pitch;
    cr += pitch;
    if (fr) fr += pitch;
  }
};

// a far-melt tile: psi stays -1; the c update of phases 1 and 2 with S and mu'' of
// a warp's rows in registers (neighbour columns by shuffles, halo columns by
// twelve lanes through scratch), stored straight to global memory.  The same
// expressions as phases 1 and 2, so the same bits.  No row votes on its form,
// so the arithmetic of the rows overlaps.  Returns the warp's part of the mass.
static __device__ __forceinline__ double melt_tile(const TileView &V, const LaneCols &LC, const InSlot &in, MeltHalo &mh,
                                            bool red, double *stage, double *__restrict__ psi_n,
                                            double *__restrict__ c_n,
                                            double *__restrict__ phi_n) {
  const Coef<double> &F = V.F;
  const int lane = V.lane, r0 = kRowsPerWarp * V.gw;
  const double cinf = F.cinf, cflux4 = 0.25 * F.cflux, c_floor = F.c_floor;
  const int rows_live = V.K.ny - 1 - V.y0;
  const double(&ma)[6] = F.melt_a;
  double *hs = mh.s[V.gw], *hm = mh.m[V.gw];  // halo terms of the warp's six rows, 2 per row
  if (lane < kHaloTerms) {
    const int rr = r0 + (lane >> 1), side = lane & 1;
    double S = 0.0, m = 0.0;
    if (rr <= V.K.ny - V.y0) {
      const int x = side ? kHaloR : kHaloL;
      halo_cell<false>(V, nullptr, ma, in.psi[rr][x], in.c[rr][x], rr, side, V.x0 - 4 + x, S, m);
    }
    hs[lane] = S;
    hm[lane] = m;
  }
  __syncwarp();
  struct Row {
    double s[2], m[2], sl, sr, ml, mr;
  };
  auto load_row = [&](int k, Row &R) {
    const int rr = r0 + k;
    const double2 cv = ld2(&in.c[rr][V.bc]);
    const double cc[2] = {cv.x, cv.y};
    const double dv[2] = {cv.x - cinf, cv.y - cinf};
#pragma unroll
    for (int q = 0; q < 2; ++q) far_cell<false>(ma, cc[q], dv[q], LC.RT[q], 0.0, R.s[q], R.m[q]);
    R.sl = __shfl_up_sync(FULL, R.s[1], 1);
    R.ml = __shfl_up_sync(FULL, R.m[1], 1);
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
  };
  struct Pairs {
    double q[3];
  };
  auto pairs = [](const Row &R) {
    Pairs P;
    P.q[0] = R.sl + R.s[0];
    P.q[1] = R.s[0] + R.s[1];
    P.q[2] = R.s[1] + R.sr;
    return P;
  };
  auto vface = [](const Row &A, const Row &B, double jv[2]) {
    const double pp[4] = {A.sl + B.sl, A.s[0] + B.s[0], A.s[1] + B.s[1], A.sr + B.sr};
#pragma unroll
    for (int q = 0; q < 2; ++q) jv[q] = __dmul_rn(fma(6.0, pp[q + 1], pp[q] + pp[q + 2]), B.m[q] - A.m[q]);
  };
  CellStore out(V, stage, psi_n, c_n, phi_n);
  double mass = 0.0, jv_lo[2], jv_hi[2];
  Row rb, rc;
  Pairs pa, pb, pc;
  {
    Row ra;
    load_row(0, ra);
    load_row(1, rb);
    vface(ra, rb, jv_lo);
    pa = pairs(ra);
    pb = pairs(rb);
  }
#pragma unroll
  for (int j = 0; j < kRowsPerWarp; ++j) {
    load_row(j + 2, rc);
    pc = pairs(rc);
    vface(rb, rc, jv_hi);
    const double mm[4] = {rb.ml, rb.m[0], rb.m[1], rb.mr};
    const double2 cv2 = ld2(&in.c[r0 + 1 + j][V.bc]);
    const double cv[2] = {cv2.x, cv2.y};
    double jh[3], dn[2];
#pragma unroll
    for (int fc = 0; fc < 3; ++fc)
      jh[fc] = __dmul_rn(fma(6.0, pb.q[fc], pa.q[fc] + pc.q[fc]), mm[fc + 1] - mm[fc] + LC.dK[fc]);
#pragma unroll
    for (int q = 0; q < 2; ++q)
      dn[q] = fmax(fma(cflux4, (jh[q + 1] - jh[q]) + (jv_hi[q] - jv_lo[q]), cv[q]), c_floor);
    if (r0 + 1 + j <= rows_live) {
      if (red) {
#pragma unroll
        for (int q = 0; q < 2; ++q)
          if ((V.outm >> q) & 1u) mass += dn[q];
      }
      out.put(V, r0 + 1 + j, -1.0, dn[0], dn[1], psi_n, c_n, phi_n);
    }
    rb = rc;
    pa = pb;
    pb = pc;
#pragma unroll
    for (int q = 0; q < 2; ++q) jv_lo[q] = jv_hi[q];
  }
  return mass;
}

// a deep solid tile: S = 0 in every cell, so every flux is 0 and psi and c
// stay (itip: the last interior column, as phase 4 counts it)
static __device__ __forceinline__ double solid_tile(const TileView &V, const InSlot &in, bool red, double *stage,
                                             double *__restrict__ psi_n, double *__restrict__ c_n,
                                             double *__restrict__ phi_n, int &itip) {
  const int r0 = kRowsPerWarp * V.gw, rows_live = V.K.ny - 1 - V.y0, nx = V.K.nx;
  const double c_floor = V.F.c_floor;
  CellStore out(V, stage, psi_n, c_n, phi_n);
  double mass = 0.0;
#pragma unroll
  for (int j = 0; j < kRowsPerWarp; ++j) {
    const int rr = r0 + 1 + j;
    if (rr > rows_live) break;
    const double2 c = ld2(&in.c[rr][V.bc]);
    const double dn[2] = {fmax(c.x, c_floor), fmax(c.y, c_floor)};
    if (red) {
#pragma unroll
      for (int q = 0; q < 2; ++q)
        if ((V.outm >> q) & 1u) {
          mass += dn[q];
          itip = max(itip, V.gi + q == nx - 2 ? nx - 1 : V.gi + q);
        }
    }
    out.put(V, rr, 1.0, dn[0], dn[1], psi_n, c_n, phi_n);
  }
  return mass;
}

// the input tile of a pull-back step: the same box as the TMA load (columns
// x0-4 .. x0+kW+3, rows y0-1 .. y0+kTR, zeros outside the array), each
// column i read from clamp(i + i_offset, 1, nx - 2), with c = cinf where that
// is nx - 2 (the melt entering at the right edge)
// A step on unaligned rows (RAW) copies the same box, unshifted.
static __device__ __forceinline__ void gather_box(const StepCoef &K, const StepScalars &PS, int x0, int y0,
                                                  InSlot &in) {
  const double *__restrict__ psi = static_cast<const double *>(PS.src_psi);
  const double *__restrict__ c = static_cast<const double *>(PS.src_c);
  if (!PS.pull_back) {
    // a warp per row, every fourth row; columns lane, lane + 32, lane + 64
    const int lane = threadIdx.x & 31;
    for (int rr = threadIdx.x >> 5; rr < kTRin; rr += kWarps) {
      const int row = y0 - 1 + rr;
      const int64_t o = (int64_t)min(row, K.ny - 1) * K.pitch + x0 - 4 + lane;
#pragma unroll
      for (int q = 0; q < (kWin + 31) / 32; ++q) {
        const int x = lane + 32 * q, g = x0 - 4 + x;
        const bool inside = row <= K.ny - 1 && g >= 0 && g <= K.nx - 1;
        if (x < kWin) {
          cp_async_elem(&in.psi[rr][x], psi + (inside ? o + 32 * q : 0), inside);
          cp_async_elem(&in.c[rr][x], c + (inside ? o + 32 * q : 0), inside);
        }
      }
    }
    cp_async_wait();
    return;
  }
  for (int k = threadIdx.x; k < kTRin * kWin; k += kThreads) {
    const int rr = k / kWin, x = k % kWin;
    const int row = y0 - 1 + rr, g = x0 - 4 + x;
    double pv = 0.0, cv = 0.0;
    if (row <= K.ny - 1 && g >= 0 && g <= K.nx - 1) {
      const int si = min(max(g + PS.i_offset, 1), K.nx - 2);
      const int64_t o = (int64_t)row * K.pitch + si;
      pv = psi[o];
      cv = si >= K.nx - 2 ? K.cinf : c[o];
    }
    in.psi[rr][x] = pv;
    in.c[rr][x] = cv;
  }
}

};

// tile (row tr, column tc) of the launch order: tile columns from the one
// holding the front, tile rows of a column consecutive (they share halo rows
// in L2)
__device__ __forceinline__ void tile_of(int t, int nrt, int ncb, int f, int &tr, int &tc) {
  tr = t % nrt;
  tc = front_first_block(t / nrt, f, ncb);
}

// ---------------------------------------------------------------- one tile per CTA
// OWN: the CTA computes the table entries of its 72 columns itself, before it
// waits for the kernel before it, and the step is one launch.  For grids whose
// CTAs are all resident at once: theirs are scheduled, and compute the entries,
// while the step before is still at work (256^2: 8.1 -> 6.5 us a step; 352 x 1568
// with a cellular front on 16-row tiles: 18.5 -> 16.2); on larger ones every wave
// would compute them again.
template <int TR, bool TFC, bool RAW, bool OWN = false>
__global__ void __launch_bounds__(kThreads, 5)
    tile_kernel_f64(const __grid_constant__ StepCoef K, const __grid_constant__ Coef<double> F,
                    const __grid_constant__ StepScalars PS, const __grid_constant__ CUtensorMap tm_psi,
                    const __grid_constant__ CUtensorMap tm_c, const double *__restrict__ tab, const int tab_len,
                    double *__restrict__ psi_n, double *__restrict__ c_n, double *__restrict__ phi_n,
                    BlockPartial *partials, int *err, const int wave_x, const int wave_y) {
  using Ops = TileOps<TR, RAW>;
  extern __shared__ __align__(128) unsigned char smem_raw[];
  auto &sm = *reinterpret_cast<typename Ops::template TileSmem<TFC> *>(smem_raw);
  // blockIdx.x walks the tile rows of one tile column, blockIdx.y the tile
  // columns, from the one holding column PS.i_front
  const int f = max(PS.i_front, 0) / kW;
  const int tr = (int)blockIdx.x, tc = front_first_block((int)blockIdx.y, f, (int)gridDim.y);
  const int x0 = kW * tc, y0 = 1 + TR * tr;
  BlockPartial *part = partials ? partials + ((int64_t)tc * gridDim.x + tr) : nullptr;

  if (smem_u32(smem_raw) & 127u) {  // TMA destinations must be 128-byte aligned
    if (threadIdx.x == 0) atomicExch(err, 2);
    return;
  }
  // a pull-back step reads column clamp(i + i_offset, 1, nx - 2) for column i
  // (pull_back, fun.cu:1469-1492): no TMA box has that shape, so the CTA
  // gathers its tile (gather_box) instead; so it does on unaligned rows
  const bool pb = RAW || PS.pull_back != 0;
  if (threadIdx.x == 0) {
    mbar_init(&sm.full, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    sm.fl.liq = sm.fl.sol = 0u;
    sm.vote = 0u;
    sm.p2.nlist = 0u;
  }
  __shared__ alignas(16) double own_tab[OWN ? kColTabFields * kWin : 1];
  if constexpr (OWN) {
    // (as column_table_kernel_f64, entry k the column x0 - 4 + k; the last dK is
    // no lane's)
    __shared__ double kc[kWin];
    const int k = (int)threadIdx.x;
    ColEntry ct = {};
    if (k < kWin) {
      const int gi = min(max(x0 - 4 + k, 0), K.nx - 1);
      ct = col_entry((PS.d0 + PS.d1 * gi) * K.deltaT0 + K.Tmelt, K.RR, K.cinf, K.Lref);
      kc[k] = ct.KC;
    }
    __syncthreads();
    if (k < kWin) {
      own_tab[kTabRT * kWin + k] = ct.RT;
      own_tab[kTabC0 * kWin + k] = ct.C0;
      own_tab[kTabDK * kWin + k] = k + 1 < kWin ? kc[k + 1] - ct.KC : 0.0;
      own_tab[kTabAnb * kWin + k] = ct.Anb;
      own_tab[kTabAti * kWin + k] = ct.Ati;
    }
    __syncthreads();
  }
  // the kernel before this one in the stream (the column table's, and with it
  // every earlier one) has completed: its table and the fields are visible
  asm volatile("griddepcontrol.wait;" ::: "memory");
  if (threadIdx.x == 0 && !pb) {
    mbar_expect_tx(&sm.full, Ops::kTileBytes);
    tma_load_2d(&sm.in.psi[0][0], &tm_psi, &sm.full, x0 - 4, y0 - 1);
    tma_load_2d(&sm.in.c[0][0], &tm_c, &sm.full, x0 - 4, y0 - 1);
  }
  // dependents of this step (its reduction, the next step) may be scheduled now,
  // or (late) once the tile's phase 3 is done
  if (!PS.late) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  const typename Ops::TileView V(K, F, PS, OWN ? own_tab - x0 : tab, OWN ? kWin : tab_len, x0, y0,
                                 (int)threadIdx.x);
  const typename Ops::LaneCols LC = Ops::template lane_cols<TFC>(V);
  const typename Ops::TfcTile *tf = nullptr;
  if constexpr (TFC) {
    typename Ops::TfcTile &T = sm.tf;
    tf = &T;
    // the column parts of the cells' temperatures, the row parts, and K + C0
    // about the temperature of the tile's centre, once per tile
    const int t = (int)threadIdx.x;
    if (t < kW) tfc_col(K, PS.i_left_end_T, x0 + t, T.ti[t], T.tx[t]);
    else if (t < kW + 2) tfc_col(K, PS.i_left_end_T, t == kW ? x0 - 1 : x0 + kW, T.hiT[t - kW], T.hx[t - kW]);
    else if (t >= 96 && t < 96 + Ops::kTRin) tfc_row(K, y0 - 1 + t - 96, T.tj[t - 96], T.ty[t - 96]);
    else if (t == 80 || t == 127) {  // (two warps)
      int iT, jT;
      double x, y;
      tfc_col(K, PS.i_left_end_T, x0 + kW / 2, iT, x);
      tfc_row(K, y0 + TR / 2, jT, y);
      const double T0 = tfc_T(K, PS.T_coarse, iT, x, jT, y);
      if (t == 127) kc_poly(K, T0, T.kp);
      else drive_poly(T0, T.kp);
    }
  }
  if (pb) Ops::gather_box(K, PS, x0, y0, sm.in);
  __syncthreads();  // barrier initialised, flags cleared (and the TFC tables written)
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
  }
  if constexpr (RAW) {
    // as below, line by line
    int bx = (int)blockIdx.x + wave_x, by = (int)blockIdx.y + wave_y;
    if (bx >= (int)gridDim.x) {
      bx -= (int)gridDim.x;
      ++by;
    }
    if (by < (int)gridDim.y && !PS.pull_back) {
      const int px = max(kW * front_first_block(by, f, (int)gridDim.y) - 4, 0), py = TR * bx;
      for (int k = threadIdx.x; k < Ops::kTRin * 6 * 2; k += kThreads) {
        const int row = min(py + (k >> 1) / 6, K.ny - 1), x = min(px + 16 * ((k >> 1) % 6), K.nx - 1);
        const double *q = static_cast<const double *>((k & 1) ? PS.src_psi : PS.src_c) + (int64_t)row * K.pitch + x;
        asm volatile("prefetch.global.L2 [%0];" ::"l"(q));
      }
    }
  }
  // pull the tile of the CTA that will start about one resident wave later
  // (wave_y tile columns and wave_x tile rows on) into L2, so its loads
  // overlap the rest of this wave's arithmetic
  if (threadIdx.x == 0 && !pb && !gave_up) {
    int nx = (int)blockIdx.x + wave_x, ny = (int)blockIdx.y + wave_y;
    if (nx >= (int)gridDim.x) {
      nx -= (int)gridDim.x;
      ++ny;
    }
    if (ny < (int)gridDim.y) {
      const int pc = front_first_block(ny, f, (int)gridDim.y);
      tma_prefetch_2d(&tm_psi, kW * pc - 4, TR * nx);
      tma_prefetch_2d(&tm_c, kW * pc - 4, TR * nx);
    }
  }
  if (x0 + kW + 4 > K.nx) {  // (CTA-uniform) a thread that gave up leaves the tile alone
    if (!gave_up) Ops::fix_beyond(V, sm.in);
    __syncthreads();
  }
  {
    // (the coarse-grid temperature has no melt form: a tile votes only where its
    // first interior cell is solid)
    uint32_t bad = gave_up ? (uint32_t)Ops::kGaveUp
                   : TFC && bits(sm.in.psi[1][5]) != kPlus1 ? (uint32_t)(Ops::kNotMinus1 | Ops::kNotPlus1)
                                                            : Ops::tile_vote(V, sm.in);
    bad = __reduce_or_sync(FULL, bad);
    if (V.lane == 0 && bad) atomicOr(&sm.vote, bad);
  }
  __syncthreads();
  const uint32_t vote = sm.vote;
  const bool red = part != nullptr;
  double mass = 0.0;
  int itip = 0;
  if (vote & Ops::kGaveUp) {
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
    Ops::finish_tile(V, sm.p2, 0.0, 0, part, 0);
    return;
  }
  const bool melt = !TFC && !(vote & (Ops::kNotMinus1 | Ops::kNotFar));
  if (melt || !(vote & (Ops::kNotPlus1 | Ops::kNotFinite))) {
    if (melt)
      mass = Ops::melt_tile(V, LC, sm.in, *reinterpret_cast<typename Ops::MeltHalo *>(sm.p2.list), red, sm.st.S[V.gw], psi_n,
                            c_n, phi_n);
    else
      mass = Ops::solid_tile(V, sm.in, red, sm.st.S[V.gw], psi_n, c_n, phi_n, itip);
    Ops::finish_tile(V, sm.p2, mass, itip, part, 0);
    return;
  }
  Ops::template phase1<TFC>(V, LC, sm.in, sm.st, sm.fl, tf);
  __syncthreads();
  double dn[Ops::kRowsPerWarp][2];
  const uint32_t needs_all = Ops::phase2(V, LC, sm.in, sm.st, sm.fl, sm.p2, dn, mass, red);
  __syncthreads();
  Ops::template phase3<TFC>(V, sm.in, sm.p2, tf, sm.st.S, red, itip);  // S is free after phase 2
  __syncthreads();
  // (a whole-tile form, and a CTA that gave up, trigger by their end)
  if (PS.late) asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  Ops::phase4_rows(V, sm.in, sm.st.S, needs_all, dn, red, itip);
  Ops::store_tile(V, sm.in, psi_n, c_n, phi_n, 0);
  Ops::finish_tile(V, sm.p2, mass, itip, part, 0);
  // shared memory stays allocated until the copies have read it
  asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");
}

}  // namespace

// A step kernel of the FP64 tiles and the shared memory it takes.  The kernels
// are spread over the translation units, a module of the device each, by what a
// run uses together: the first launch of a kernel loads its whole module.
using StepFn64 = void (*)(StepCoef, Coef<double>, StepScalars, CUtensorMap, CUtensorMap, const double *, int, double *,
                          double *, double *, BlockPartial *, int *, int, int);
struct StepKernel64 {
  StepFn64 fn;
  size_t smem;
};
template <int TR, bool RAW>
StepKernel64 frozen_kernel(bool own) {
  return {own ? tile_kernel_f64<TR, false, RAW, true> : tile_kernel_f64<TR, false, RAW>,
          sizeof(typename TileOps<TR>::template TileSmem<false>)};
}
StepKernel64 raw_kernel_f64(int rows, bool own);  // rs_step_f64t_raw.cu
StepKernel64 tfc_kernel_f64(int rows);            // rs_step_f64t_tfc.cu
StepKernel64 tfc_raw_kernel_f64(int rows);        // rs_step_f64t_tfc_raw.cu
StepKernel64 pipe_kernel_of_f64(int rows);        // rs_step_f64t_pipe.cu
constexpr int kTileThreads64 = kThreads;
constexpr int kPipeThreads64 = 32 + 2 * kThreads;  // producer warp, phase-1 group, phases 2-4 group

}  // namespace rs
