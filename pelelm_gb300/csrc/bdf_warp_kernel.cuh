// Persistent, work-stealing, warp-per-cell BDF reactor kernel for mechanisms whose per-cell state
// no longer fits a thread: an option for drm19-sized mechanisms (21 species, 84 reactions) and
// the only mapping for GRI-Mech-sized ones (53 species, 325 reactions, N = 54 unknowns), there
// also with a team of warps per cell.
//
// Same contract and algorithm as bdf_kernel.cuh (the PelePhysics reactor called at
// Source/PeleLM.cpp:5752; CVODE-class fixed-leading-coefficient variable-order Nordsieck BDF,
// modified Newton with analytic Jacobian and dense partial-pivot LU, CVODE's documented
// step/order heuristics): each warp runs the step loop of oracle/bdf_oracle.cpp for one cell at a
// time, with the length-N vectors split over the lanes (element i in lane i % 32, slot i / 32).
//
// GB300 mapping:
//  * the scalar step logic runs redundantly in every lane (uniform values, no divergence): an
//    FP64 warp instruction costs the same whatever its active mask, so this is free next to a
//    lane-parallel right-hand side;
//  * RHS: lanes over species (concentrations, g/RT, h, cp), then over reactions (rates of
//    progress, from global-memory tables read through L1: lanes read different entries), then
//    over species again gathering their reactions (species-major lists: a deterministic order,
//    no atomics), with warp-shuffle sums for the energy closure;
//  * Jacobian (type JR: FP32 in mixed precision): NASA-7 terms once per species, per-reaction
//    partials lane-parallel, then an assembly by a generated program in reaction order with lanes
//    over matrix entries (each entry has one owner, so the result does not depend on scheduling);
//    constant-pressure energy row by column;
//  * LU and triangular solves: lanes own rows; pivot search by warp arg-max (FP32: one max-
//    reduction over the |a| bit patterns); matrix rows padded to N+1 so a column access is
//    bank-conflict free;
//  * per-warp state (Nordsieck history, forcing, rates, matrix) in shared memory; a warp takes
//    the next cell index with one atomic when its cell is done (work stealing across all boxes);
//  * with few cells a warp of its own leaves three of the four schedulers of an SM idle and a cell
//    waits for one warp's dependent latencies: teams of W = 4 warps share its right-hand side
//    (team_rates) and its Jacobian (partials and contribution program), the first warp leading.
//    Used for launches of up to two cells per SM, for the last four cells per SM of a longer one
//    (its warps hand them over) and for the FP64 pass over failed cells. Every sum keeps the order
//    of the one-warp form, so the results are bit for bit the same. Measured (53 species, 60 cells
//    mixed / 125 cells FP64): only the right-hand side shared 3.2 / 9.3 ms, the Jacobian too 2.5 / 7.5;
//  * with a retry list (mixed precision), a failed cell is listed and left untouched for the
//    FP64 pass that follows on the same stream.
#ifndef PGB_BDF_WARP_KERNEL_CUH
#define PGB_BDF_WARP_KERNEL_CUH

#include "bdf_kernel.cuh"
#include "mech_tables.cuh"

namespace pgb {

namespace wbdf {
constexpr int RXW = 8;  // Jacobian scratch per reaction: dq/dT, 3 reactant partials, 3 product partials, [M] partial
// Partials of the whole mechanism: RXW per reaction, then the [M] partials times each listed
// collider's efficiency.
template <class M>
__host__ __device__ constexpr int rx_len() {
  return RXW * M::NR + M::TabG::JAC_X;
}
}

// Shared memory of one warp (one cell) for mechanism M and Jacobian type JR: the FP64 state
// (Nordsieck history, forcing, l, tau), one scratch region and the matrix. The scratch region
// holds the RHS scratch (concentrations, g/RT, rates of progress) inside warp_rhs and the setup
// scratch (per-reaction partials, NASA-7 terms) inside warp_setup: never both live.
template <class M>
__host__ __device__ constexpr int bdf_warp_state_bytes() {
  return (((QMAX + 2) * M::N + M::N + (QMAX + 1) + (QMAX + 2)) * 8 + 15) / 16 * 16;
}
template <class M, class JR>
__host__ __device__ constexpr int bdf_warp_scratch_bytes() {
  constexpr int NS = M::NS, NR = M::NR;
  constexpr int rhs = (2 * NS + NR) * 8, setup = (wbdf::rx_len<M>() + 4 * NS) * (int)sizeof(JR);
  return ((rhs > setup ? rhs : setup) + 15) / 16 * 16;
}
template <class M, class JR>
__host__ __device__ constexpr int bdf_warp_smem_per_warp() {
  constexpr int N = M::N;
  constexpr int nj = N * (N + 1) + N;
  return (bdf_warp_state_bytes<M>() + bdf_warp_scratch_bytes<M, JR>() + nj * (int)sizeof(JR) + N * 4 + 15) / 16 * 16;
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}

// K quotients (K <= 8 <= G) in one division: lane i of the group forms the i-th, and all lanes get
// all of them. The step logic is the same in every lane of a group, and an FP64 division takes ten of
// its slots, so its quotients are formed side by side wherever they do not depend on one another.
template <int K>
__device__ __forceinline__ void group_div(const double (&num)[K], const double (&den)[K], double (&quot)[K],
                                          unsigned gm, int gbase) {
  const int sub = (threadIdx.x & 31) - gbase;
  double a = num[0], b = den[0];
#pragma unroll
  for (int i = 1; i < K; ++i)
    if (sub == i) { a = num[i]; b = den[i]; }
  const double d = pgb_div64(a, b);
#pragma unroll
  for (int i = 0; i < K; ++i) quot[i] = __shfl_sync(gm, d, gbase + i);
}

// The lane-distributed part of a length-N vector (element i in lane i % 32, slot i / 32).
template <class M>
struct WVec {
  double v[(M::N + 31) / 32];
};

// Rate of progress of reaction j (table order) at one state, FP64: the equations of the table
// RHS in mech_tables.cuh (Arrhenius forward rate, third-body and Lindemann/Troe fall-off
// factors, reverse rate from K_c with the exponent capped at 700), the same operations in the
// same order. Shared by the warp and lane-group right-hand sides; the reaction's data comes
// from its two packed records (TabRxArr, TabRxPk: three loads instead of one per field).
template <class Tab>
__device__ __forceinline__ double rate_of_progress(int j, double T, double invT, double lnT, double lnP0RT,
                                                   double Ctot, const double* CS, const double* GS) {
  const TabRxArr& ar = Tab::rx_arr(j);
  const TabRxPk pk = Tab::rx_pk(j);
  const int kind = pk.x & 3u, nr = (pk.x >> 3) & 3u, np = (pk.x >> 5) & 3u;
  const bool rev = (pk.x >> 2) & 1u;
  const int dnu = (int)((pk.x >> 7) & 15u) - 8, tbi = (int)((pk.x >> 11) & 2047u) - 1;
  const int troe = (int)(pk.x >> 22) - 1;
  auto rs = [&](int s) { return (int)((pk.y >> (10 * s)) & 1023u); };
  auto ps = [&](int s) { return (int)((pk.z >> (10 * s)) & 1023u); };
  const double lnkf = fma(ar.beta, lnT, fma(ar.mEaR, invT, ar.lnA));
  double kf = pgb_exp64(lnkf);
  double Mc = 1.0;
  if (tbi >= 0) {
    const TabThirdBody<double>& tb = Tab::template tb<double>(tbi);
    Mc = Ctot;
#pragma unroll
    for (int e = 0; e < 8; ++e)
      if (e < tb.n) Mc = fma(tb.effm1[e], CS[tb.sp[e]], Mc);
  }
  if (kind == 2) {
    const TabTroe<double>& fo = Tab::template troe<double>(troe);
    const double lnk0 = fma(fo.beta0, lnT, fma(fo.mEa0R, invT, fo.lnA0));
    const double Pr = __dmul_rn(Mc, pgb_exp64(lnk0 - lnkf));
    double blend = pgb_div64(Pr, __dadd_rn(1.0, Pr));
    if (fo.ntroe > 0) {
      double Fcent = fma(fo.one_m_a, pgb_exp64(T * fo.m_invT3), fo.a * pgb_exp64(T * fo.m_invT1));
      if (fo.ntroe > 3) Fcent += pgb_exp64(invT * fo.m_T2);
      const double lFc = pgb_log64(Fcent) * 0.4342944819032518;
      const double cc = fma(-0.67, lFc, -0.4), nn = fma(-1.27, lFc, 0.75);
      const double lPr = fma(pgb_log64(fmax(Pr, 1e-300)), 0.4342944819032518, cc);
      const double f1 = pgb_div64(lPr, fma(-0.14, lPr, nn));
      blend *= pgb_exp64(pgb_div64(2.302585092994046 * lFc, fma(f1, f1, 1.0)));
    }
    kf *= blend;
  }
  // both sides hold at least one species, and no reaction more slots than MAXR / MAXP: a predicated
  // multiply that no lane takes still costs its FP64 slot
  double Pf = CS[rs(0)], Pp = CS[ps(0)];
#pragma unroll
  for (int s = 1; s < Tab::MAXR; ++s) if (s < nr) Pf *= CS[rs(s)];
#pragma unroll
  for (int s = 1; s < Tab::MAXP; ++s) if (s < np) Pp *= CS[ps(s)];
  double q;
  if (rev) {
    // -dnu ln(P0/RT): a sign for dnu = -1, 0, 1
    double dG = dnu == 0 ? 0.0 : dnu == -1 ? lnP0RT : dnu == 1 ? -lnP0RT : -dnu * lnP0RT;
    dG += GS[ps(0)];
#pragma unroll
    for (int s = 1; s < Tab::MAXP; ++s) if (s < np) dG += GS[ps(s)];
    dG -= GS[rs(0)];
#pragma unroll
    for (int s = 1; s < Tab::MAXR; ++s) if (s < nr) dG -= GS[rs(s)];
    const double kr = kf * pgb_exp64(fmin(dG, 700.0));  // finite: Pp = 0 gives 0, not NaN
    q = fma(kf, Pf, -kr * Pp);
  } else {
    q = kf * Pf;
  }
  if (kind == 1) q *= Mc;
  return q;
}

// Right-hand side f = [W_k wdot_k + F_k, dT/dt] at y, one warp cooperating (see the kernel
// below). One non-inlined copy serves every call site: the step loop calls it from five places
// and inlined copies of this exp/log-heavy body overflow the instruction cache.
//
// W > 1: the warp leads a team of W warps (TP: T, 1/T, ln T, ln(P0/RT), [M] and the order, for the
// others), which share the reactions and the species sums (team_rates).
template <int W>
__device__ __forceinline__ void team_sync(int id) {
  asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(32 * W) : "memory");
}
// Rates of progress and production rates (into CS) of one right-hand side, warp `role` of W.
template <class M, int W>
__device__ __forceinline__ void team_rates(int role, int id, double T, double invT, double lnT, double lnP0RT,
                                           double Ctot, double* CS, const double* GS, double* QS) {
  using Tab = typename M::TabG;
  constexpr int NS = M::NS, NR = M::NR, R = (M::N + 31) / 32;
  const int first = 32 * role + (threadIdx.x & 31);
  for (int j = first; j < NR; j += 32 * W) QS[j] = rate_of_progress<Tab>(j, T, invT, lnT, lnP0RT, Ctot, CS, GS);
  if constexpr (W > 1) team_sync<W>(id);
  else __syncwarp();
  // production rates, the longest sums together (their FP64 time is the longest lane's of a round)
#pragma unroll 1
  for (int i = first; i < NS; i += 32 * W) {
    const int k = R > 1 ? Tab::sprx_by_len(i) : i;
    double wdot = 0.0;
    const int e1 = Tab::sprx_end(k);
#pragma unroll 4
    for (int e = Tab::sprx_begin(k); e < e1; ++e) wdot = fma(Tab::sprx_nu(e), QS[Tab::sprx_j(e)], wdot);
    CS[k] = wdot;
  }
  if constexpr (W > 1) team_sync<W>(id);
  else __syncwarp();
}

template <class M, int W = 1>
__device__ __noinline__ WVec<M> warp_rhs(const WVec<M> yv, double* CS, double* GS, double* QS,
                                         const double* FRC, double* TP = nullptr, int id = 0) {
  using Tab = typename M::TabG;
  constexpr int N = M::N, NS = M::NS;
  constexpr int R = (N + 31) / 32;
  const int lane = threadIdx.x & 31;
  auto idx = [&](int r) { return lane + 32 * r; };
  const double (&y)[R] = yv.v;
  WVec<M> fv;
  double (&f)[R] = fv.v;
  auto bcast = [&](const double (&v)[R], int i) -> double {
    return __shfl_sync(0xffffffffu, v[i >> 5], i & 31);
  };
  const double T = bcast(y, NS);
  const double invT = pgb_div64(1.0, T);
  const double lnT = pgb_log64(T);
  const double lnT1 = 1.0 - lnT;
  const double lnP0RT = kLnP0OverR - lnT;
  double c_loc = 0.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int k = idx(r);
    if (k < NS) {
      const TabSpecies<double>& s = Tab::template sp<double>(k);
      const double c = __dmul_rn(y[r], s.invW);
      CS[k] = c;
      c_loc += c;
      const double* g = below_positive(T, s.Tmid) ? s.glo : s.ghi;
      GS[k] = fma(g[0], lnT1, fma(T, fma(T, fma(T, fma(T, g[4], g[3]), g[2]), g[1]), fma(g[5], invT, g[6])));
    }
  }
  const double Ctot = warp_sum(c_loc);
  __syncwarp();
  if constexpr (W > 1) {
    if (lane == 0) {
      TP[0] = T; TP[1] = invT; TP[2] = lnT; TP[3] = lnP0RT; TP[4] = Ctot; TP[5] = 1.0;
    }
    team_sync<W>(id);
  }
  team_rates<M, W>(0, id, T, invT, lnT, lnP0RT, Ctot, CS, GS, QS);
  double hs = 0.0, rcp = 0.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int k = idx(r);
    f[r] = 0.0;
    if (k < NS) {
      const double wdot = CS[k];
      const TabSpecies<double>& s = Tab::template sp<double>(k);
      const double wm = fma(wdot, s.W, FRC[k]);
      f[r] = wm;
      const bool lo = below_positive(T, s.Tmid);
      const double* a = lo ? s.lo : s.hi;
      const double* hc = lo ? s.hlo : s.hhi;
      const double hRT = fma(T, fma(T, fma(T, fma(T, hc[4], hc[3]), hc[2]), hc[1]), fma(hc[5], invT, hc[0]));
      const double cpR = fma(T, fma(T, fma(T, fma(T, a[4], a[3]), a[2]), a[1]), a[0]);
      hs = fma(hRT * s.invW, wm, hs);
      rcp = fma(y[r] * s.invW, cpR, rcp);
    }
  }
  hs = warp_sum(hs);
  rcp = warp_sum(rcp);
  const double fT = pgb_div64(fma(-hs, kRerg * T, FRC[NS]), rcp * kRerg);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (idx(r) == NS) f[r] = fT;
  __syncwarp();  // CS/GS/QS are reused by the next evaluation
  return fv;
}

// Sign flip by the top bit of `top`, and a test for zero, on the integer pipe (an FP64 compare
// takes an FP64 slot).
__device__ __forceinline__ float flip_sign(float x, unsigned top) {
  return __uint_as_float(__float_as_uint(x) ^ (top & 0x80000000u));
}
__device__ __forceinline__ double flip_sign(double x, unsigned top) {
  return __hiloint2double(__double2hiint(x) ^ (int)(top & 0x80000000u), __double2loint(x));
}
__device__ __forceinline__ bool not_zero(float x) { return (__float_as_uint(x) << 1) != 0u; }
__device__ __forceinline__ bool not_zero(double x) {
  return (((unsigned)__double2hiint(x) << 1) | (unsigned)__double2loint(x)) != 0u;
}

// Largest |a| over the warp's candidates (`ok`), NaN never: true in the slots that hold it; false
// everywhere if no candidate is above 0. A non-negative float orders as its bit pattern, so the
// search is warp max-reductions of integers (FP64: high words, then low words).
template <int R>
__device__ __forceinline__ bool warp_abs_max(const float (&a)[R], const bool (&ok)[R], bool (&is_max)[R]) {
  unsigned bits[R], m = 0u;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float v = fabsf(a[r]);
    bits[r] = ok[r] && v == v ? __float_as_uint(v) : 0u;
    m = max(m, bits[r]);
  }
  m = __reduce_max_sync(0xffffffffu, m);
#pragma unroll
  for (int r = 0; r < R; ++r) is_max[r] = m != 0u && bits[r] == m;
  return m != 0u;
}
template <int R>
__device__ __forceinline__ bool warp_abs_max(const double (&a)[R], const bool (&ok)[R], bool (&is_max)[R]) {
  unsigned hi[R], lo[R], mh = 0u, ml = 0u;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    hi[r] = (unsigned)__double2hiint(a[r]) & 0x7fffffffu;
    lo[r] = (unsigned)__double2loint(a[r]);
    if (!ok[r] || hi[r] > 0x7ff00000u || (hi[r] == 0x7ff00000u && lo[r])) hi[r] = lo[r] = 0u;
    mh = max(mh, hi[r]);
  }
  mh = __reduce_max_sync(0xffffffffu, mh);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (hi[r] == mh) ml = max(ml, lo[r]);
  ml = __reduce_max_sync(0xffffffffu, ml);
#pragma unroll
  for (int r = 0; r < R; ++r) is_max[r] = (mh | ml) != 0u && hi[r] == mh && lo[r] == ml;
  return (mh | ml) != 0u;
}

// Partial-pivot LU of I - g J, J in shared memory rows of N + 1, one warp: L below the diagonal,
// U above, reciprocal pivots on it, rows in pivot order, PIV[i] the row of J that row i came from.
// False: singular. Each lane keeps its rows (lane + 32 r) in registers and the step loop rotates
// them left by one, so the pivot column is always element 0 and one rolled loop body serves every
// step; after N steps the rows are back in place. Rows are not moved between lanes: `pos` is a
// row's place in the pivot order. The pivot row reaches the lanes by shuffles; the columns already
// eliminated are skipped four at a time. The shared-memory form it replaces paid about a thousand
// cycles a step in dependent loads and stores (21 species: 22k cycles a matrix).
template <int N, class JR>
__device__ __forceinline__ bool warp_lu_factor_regs(JR* A, int* PIV, const JR g) {
  constexpr int R = (N + 31) / 32, LDA = N + 1;
  const int lane = threadIdx.x & 31;
  JR a[R][N];
  int pos[R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int i = lane + 32 * r;
    pos[r] = i < N ? i : 2 * N;
#pragma unroll
    for (int j = 0; j < N; ++j) a[r][j] = i < N ? fma(-g, A[i * LDA + j], i == j ? JR(1) : JR(0)) : JR(0);
  }
#pragma unroll 1
  for (int k = 0; k < N; ++k) {
    // pivot: first row of largest |a_ik|, i >= k
    JR head[R];
    bool ok[R], is_max[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      head[r] = a[r][0];
      ok[r] = pos[r] >= k && pos[r] < N;
    }
    if (!warp_abs_max(head, ok, is_max)) return false;
    int p = 2 * N;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (is_max[r]) p = min(p, pos[r]);
    p = __reduce_min_sync(0xffffffffu, p);
    int src = 0, slot = 0;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const unsigned b = __ballot_sync(0xffffffffu, pos[r] == p);
      if (b) { src = __ffs(b) - 1; slot = r; }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      if (pos[r] == p) pos[r] = k;
      else if (pos[r] == k) pos[r] = p;
    }
    auto pivot_row = [&](int j) -> JR {
      JR v = a[0][j];
#pragma unroll
      for (int r = 1; r < R; ++r)
        if (slot == r) v = a[r][j];
      return __shfl_sync(0xffffffffu, v, src);
    };
    const JR inv = JR(1) / pivot_row(0);
    JR l[R];
    bool below[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      below[r] = pos[r] > k && pos[r] < N;
      l[r] = head[r] * inv;
      head[r] = below[r] ? l[r] : pos[r] == k ? inv : head[r];
    }
    const int live = N - k;  // columns k..N-1 are elements 0..live-1
#pragma unroll
    for (int j0 = 1; j0 < N; j0 += 4) {
      if (j0 < live) {
#pragma unroll
        for (int j = j0; j < j0 + 4 && j < N; ++j) {
          const JR u = pivot_row(j);
#pragma unroll
          for (int r = 0; r < R; ++r) a[r][j - 1] = below[r] && j < live ? fma(-l[r], u, a[r][j]) : a[r][j];
        }
      } else {
#pragma unroll
        for (int j = j0; j < j0 + 4 && j < N; ++j)
#pragma unroll
          for (int r = 0; r < R; ++r) a[r][j - 1] = a[r][j];
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r) a[r][N - 1] = head[r];
  }
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (pos[r] < N) {
      PIV[pos[r]] = lane + 32 * r;
#pragma unroll
      for (int j = 0; j < N; ++j) A[pos[r] * LDA + j] = a[r][j];
    }
  __syncwarp();
  return true;
}

// The same factors for matrices whose rows do not fit registers (FP64, 53 species: 216 a lane): in
// shared memory, the trailing block's elements dealt to the lanes one by one, so that no lane idles
// on a row above the pivot (FP64 multiply-adds bound this: 1,670 warp instructions against 2,610
// with a row per lane).
template <int N, class JR>
__device__ __forceinline__ bool warp_lu_factor_shared(JR* A, int* PIV, const JR g) {
  constexpr int R = (N + 31) / 32, LDA = N + 1;
  const int lane = threadIdx.x & 31;
  for (int e = lane; e < N * LDA; e += 32) {
    const int i = e / LDA, j = e - i * LDA;
    if (j < N) A[e] = fma(-g, A[e], i == j ? JR(1) : JR(0));
  }
  for (int i = lane; i < N; i += 32) PIV[i] = i;
  __syncwarp();
#pragma unroll 1
  for (int k = 0; k < N; ++k) {
    JR col[R];
    bool ok[R], is_max[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = lane + 32 * r;
      ok[r] = i >= k && i < N;
      col[r] = ok[r] ? A[i * LDA + k] : JR(0);
    }
    if (!warp_abs_max(col, ok, is_max)) return false;
    int p = 2 * N;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (is_max[r]) p = min(p, lane + 32 * r);
    p = __reduce_min_sync(0xffffffffu, p);
    __syncwarp();
    if (p != k) {
      for (int j = lane; j < N; j += 32) {
        const JR tmp = A[k * LDA + j];
        A[k * LDA + j] = A[p * LDA + j];
        A[p * LDA + j] = tmp;
      }
      if (lane == 0) {
        const int tmp = PIV[k];
        PIV[k] = PIV[p];
        PIV[p] = tmp;
      }
      __syncwarp();
    }
    const JR inv = JR(1) / A[k * LDA + k];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = lane + 32 * r;
      if (i > k && i < N) A[i * LDA + k] *= inv;
    }
    __syncwarp();
    const int m = N - 1 - k;
    if (m > 0) {
      int i = k + 1 + lane / m, j = k + 1 + lane % m;
#pragma unroll 4
      for (int e = lane; e < m * m; e += 32) {
        A[i * LDA + j] = fma(-A[i * LDA + k], A[k * LDA + j], A[i * LDA + j]);
        j += 32;
        while (j >= N) { j -= m; ++i; }
      }
    }
    if (lane == 0) A[k * LDA + k] = inv;
    __syncwarp();
  }
  return true;
}

template <int N, class JR>
__device__ __forceinline__ bool warp_lu_factor(JR* A, int* PIV, const JR g) {
  // up to 128 registers of rows a lane: FP32 to N = 64, FP64 to N = 64 / 2 rows
  if constexpr ((N + 31) / 32 * N * (int)sizeof(JR) <= 512) return warp_lu_factor_regs<N>(A, PIV, g);
  else return warp_lu_factor_shared<N>(A, PIV, g);
}

// Jacobian (equations of jac_table, mech_tables.cuh) into A, one warp cooperating. Inlined: each
// kernel calls it from one place, so inlining adds no copy and removes the call's register save and
// restore (measured: 1 to 3 %).
// Every rounding is written out (fma, pgb_mul, pgb_add): kernels of different widths hand cells to one another.
// W > 1: by the warps of a team (role 0 leads and has y; TJ: four numbers it tells the others; QN: [NR]
// the reactions' net rates, whose energy sums the leader then forms in its own order).
template <class M, class JR, int W = 1>
__device__ __forceinline__ void warp_jacobian(const WVec<M> yv, const double* FRC, JR* A, JR* XS, JR* RX, JR* TH,
                                              int role = 0, int id = 0, JR* TJ = nullptr, JR* QN = nullptr) {
  using Tab = typename M::TabG;
  constexpr int N = M::N, NS = M::NS, NR = M::NR;
  constexpr int R = (N + 31) / 32;
  constexpr int LDA = N + 1;
  const int lane = threadIdx.x & 31, first = 32 * role + lane;
  const double (&y)[R] = yv.v;
  auto idx = [&](int r) { return lane + 32 * r; };
  auto bcast = [&](const double (&v)[R], int i) -> double {
    return __shfl_sync(0xffffffffu, v[i >> 5], i & 31);
  };
  using namespace jac_detail;
  JR T = (JR)bcast(y, NS);
  if constexpr (W > 1) {
    if (role > 0) T = TJ[0];
  }
  const JR invT = JR(1) / T;
  const JR lnT = pgb_logT<JR>(T);
  const JR lnT1 = pgb_add(JR(1), -lnT);
  const JR lnP0RT = pgb_add(JR(kLnP0OverR), -lnT);
  const JR RT = JR(kRerg) * T;
  // per species, once: concentration (the solve vector is free during the setup) and the
  // NASA-7 terms g/RT, h/RT, cp/R, d(cp/R)/dT that the reaction and energy terms reuse
  JR* TG = TH;
  JR* TH_ = TH + NS;
  JR* TC = TH + 2 * NS;
  JR* TD = TH + 3 * NS;
  JR c_loc = JR(0);
  if (W == 1 || role == 0)
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int k = idx(r);
    if (k < NS) {
      const JR c = pgb_mul((JR)y[r], Tab::template sp<JR>(k).invW);
      XS[k] = c;
      c_loc += c;
      JR g, h, cp, d;
      nasa_exact<JR>(Tab::template sp<JR>(k), T, invT, lnT1, g, h, cp, d);
      TG[k] = g;
      TH_[k] = h;
      TC[k] = cp;
      TD[k] = d;
    }
  }
  JR Ctot = warp_sum(c_loc);
  for (int e = first; e < N * LDA; e += 32 * W) A[e] = JR(0);
  if constexpr (W > 1) {
    if (role == 0 && lane == 0) TJ[1] = Ctot;
    team_sync<W>(id);
    Ctot = TJ[1];
  } else {
    __syncwarp();
  }
  // (1) per-reaction partials, lanes over reactions; energy-closure sums
  JR Qw = JR(0), cpw = JR(0);
  for (int j = first; j < NR; j += 32 * W) {
    const TabReaction<JR>& r = Tab::template rx<JR>(j);
    const JR eT = pgb_mul(r.mEaR, invT);
    const JR lnkinf = pgb_add(fma(r.beta, lnT, eT), r.lnA);
    JR dlnkf = pgb_mul(pgb_add(r.beta, -eT), invT);
    JR kf = pgb_expT<JR>(lnkinf);
    JR Mc = JR(1), alpha = JR(1), dkeff_dM = JR(0);
    if (r.tb >= 0) {
      const TabThirdBody<JR>& t = Tab::template tb<JR>(r.tb);
      Mc = Ctot;
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (e < t.n) Mc = fma(t.effm1[e], XS[t.sp[e]], Mc);
      if (r.kind == 1) alpha = Mc;
    }
    if (r.kind == 2) {
      const TabTroe<JR>& fo = Tab::template troe<JR>(r.troe);
      const JR eT0 = pgb_mul(fo.mEa0R, invT);
      const JR lnk0 = pgb_add(fma(fo.beta0, lnT, eT0), fo.lnA0);
      const JR dlnk0_T = pgb_add(fo.beta0, -eT0);  // times 1/T: d ln k0 / dT
      const JR k0 = pgb_expT<JR>(lnk0);
      const JR Pr = pgb_mul(Mc, pgb_expT<JR>(lnk0 - lnkinf));
      JR Fb = JR(1);
      if (fo.ntroe > 0) {
        JR Fcent = fma(fo.one_m_a, pgb_expT<JR>(T * fo.m_invT3), pgb_mul(fo.a, pgb_expT<JR>(T * fo.m_invT1)));
        if (fo.ntroe > 3) Fcent = pgb_add(Fcent, pgb_expT<JR>(fo.m_T2 * invT));
        const JR lFc = pgb_mul(pgb_logT<JR>(Fcent), JR(0.4342944819032518));
        const JR cc = fma(JR(-0.67), lFc, JR(-0.4)), nn = fma(JR(-1.27), lFc, JR(0.75));
        const JR lPr = fma(pgb_logT<JR>(Pr > JR(1e-30) ? Pr : JR(1e-30)), JR(0.4342944819032518), cc);
        const JR f1 = lPr / fma(JR(-0.14), lPr, nn);
        Fb = pgb_expT<JR>(pgb_mul(JR(2.302585092994046), lFc) / fma(f1, f1, JR(1)));
      }
      const JR onePr = pgb_add(JR(1), Pr);
      kf = pgb_mul(pgb_mul(kf, Pr) / onePr, Fb);
      dkeff_dM = pgb_mul(Fb, k0) / pgb_mul(onePr, onePr);
      // (the FP64 form fuses the difference: what each type's code did before its roundings were written out)
      const JR dln = sizeof(JR) == sizeof(double) ? fma(dlnk0_T, invT, -dlnkf) : pgb_add(pgb_mul(dlnk0_T, invT), -dlnkf);
      dlnkf = pgb_add(dlnkf, dln / onePr);
    }
    JR cr[3], cp[3];
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      cr[s] = s < r.nr ? XS[r.rs[s]] : JR(1);
      cp[s] = s < r.np ? XS[r.ps[s]] : JR(1);
    }
    const JR Pf = cr[0] * cr[1] * cr[2];
    const JR Pp = cp[0] * cp[1] * cp[2];
    JR kr = JR(0), dlnkr = JR(0);
    if (r.rev) {
      JR dG = -(JR)r.dnu * lnP0RT, dH = JR(0);
#pragma unroll
      for (int s = 0; s < 3; ++s)
        if (s < r.np) {
          dG += TG[r.ps[s]];
          dH += TH_[r.ps[s]];
        }
#pragma unroll
      for (int s = 0; s < 3; ++s)
        if (s < r.nr) {
          dG -= TG[r.rs[s]];
          dH -= TH_[r.rs[s]];
        }
      kr = kf * pgb_expT<JR>(fmin(dG, JR(700)));
      dlnkr = fma(-(dH - (JR)r.dnu), invT, dlnkf);
    }
    const JR net = fma(kf, Pf, -pgb_mul(kr, Pp));
    const JR q = pgb_mul(alpha, net);
    JR* out = RX + j * wbdf::RXW;
    out[0] = pgb_mul(alpha, fma(pgb_mul(kf, dlnkf), Pf, -pgb_mul(pgb_mul(kr, dlnkr), Pp)));
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      out[1 + s] = alpha * kf * (s == 0 ? cr[1] * cr[2] : s == 1 ? cr[0] * cr[2] : cr[0] * cr[1]);
      out[4 + s] = -alpha * kr * (s == 0 ? cp[1] * cp[2] : s == 1 ? cp[0] * cp[2] : cp[0] * cp[1]);
    }
    JR bm = JR(0);
    if (r.kind == 1) bm = net;
    else if (r.kind == 2) bm = pgb_mul(dkeff_dM, fma(-(kf > JR(0) ? kr / kf : JR(0)), Pp, Pf));
    out[7] = bm;
    if (r.tb >= 0) {  // the collider terms of the listed species read these
      const TabThirdBody<JR>& t = Tab::template tb<JR>(r.tb);
      JR* ox = RX + Tab::jac_x0(r.tb);
#pragma unroll
      for (int e = 0; e < 8; ++e)
        if (e < t.n) ox[e] = bm * (JR(1) + t.effm1[e]);
    }
    if constexpr (W > 1) {
      QN[j] = q;
    } else {
#pragma unroll
      for (int row = 0; row < 6; ++row)
        if (row < r.nr + r.np) {
          const bool isr = row < r.nr;
          const int i = isr ? r.rs[row] : r.ps[row - r.nr];
          Qw = fma(pgb_mul(isr ? -q : q, TH_[i]), RT, Qw);
          cpw = fma(pgb_mul(isr ? -q : q, TC[i]), JR(kRerg), cpw);
        }
    }
  }
  if constexpr (W > 1) {
    team_sync<W>(id);
    if (role == 0)
      for (int j = lane; j < NR; j += 32) {
        const TabReaction<JR>& r = Tab::template rx<JR>(j);
        const JR q = QN[j];
#pragma unroll
        for (int row = 0; row < 6; ++row)
          if (row < r.nr + r.np) {
            const bool isr = row < r.nr;
            const int i = isr ? r.rs[row] : r.ps[row - r.nr];
            Qw = fma(pgb_mul(isr ? -q : q, TH_[i]), RT, Qw);
            cpw = fma(pgb_mul(isr ? -q : q, TC[i]), JR(kRerg), cpw);
          }
      }
  }
  Qw = warp_sum(Qw);
  cpw = warp_sum(cpw);
  __syncwarp();
  // (2) assembly by the generated contribution program: each lane owns whole entries A[i][k]
  // (species rows; k = NS: the T column) and sums their terms in a register, in the order of
  // the reaction walk (reactions ascending, then row slots): a term of reaction j is c v,
  // c = -+W_i / W_k (-+W_i in the T column) and v the partials of j that land in column k
  // (dq/dT in the T column). The lanes' 4-byte term codes are interleaved in the table (one
  // contiguous line per warp load); each entry has one writer, so the result does not depend
  // on the lane schedule.
  // A lane reads four terms per 16-byte load, one load ahead, and an entry's coefficient and
  // target one entry ahead: with shared memory taking almost all of the L1, each of these loads
  // is an L2 round trip, and a load per term made the program the setup's longest part.
  {
    constexpr int L = 32 * W;
    auto quad_of = [&](int c) -> uint4 {
      if constexpr (W > 1) return Tab::team_quad(c);
      else return Tab::jac_quad(c);
    };
    auto ent_of = [&](int c) -> TabJacEnt<JR> {
      if constexpr (W > 1) return Tab::template team_ent<JR>(c);
      else return Tab::template jac_ent<JR>(c);
    };
    // efficiency of a term that adds its collider slot to other partials (few do)
    auto eff_of = [&](unsigned c, int term, int k) -> JR {
      if constexpr (W == 1) {
        return Tab::template jac_eff<JR>(term);
      } else {
        const TabThirdBody<JR>& t = Tab::template tb<JR>(Tab::template rx<JR>((c & 0x1fff) / wbdf::RXW).tb);
        JR v = JR(1);
        for (int e = 0; e < t.n; ++e)
          if (t.sp[e] == k) v = JR(1) + t.effm1[e];
        return v;
      }
    };
    int quads, ents;
    if constexpr (W > 1) { quads = Tab::TEAM_QUADS; ents = Tab::TEAM_ENTS; }
    else { quads = Tab::JAC_QUADS; ents = Tab::JAC_ENTS; }
    JR acc = JR(0);
    int ent = first;
    TabJacEnt<JR> cur = ent_of(ent), ahead = ent_of(ent + L);
    uint4 quad = quad_of(first);
#pragma unroll 1
    for (int q = 0; q < quads; ++q) {
      const unsigned code[4] = {quad.x, quad.y, quad.z, quad.w};
      if (q + 1 < quads) quad = quad_of(L * (q + 1) + first);
      JR v[4];
#pragma unroll
      for (int u = 0; u < 4; ++u) v[u] = RX[code[u] & 0x1fff];
#pragma unroll
      for (int u = 0; u < 4; ++u) {
        const unsigned c = code[u];
        if (c & 0xfe000) {  // species on several slots of the reaction
          const JR* pj = RX + (c & 0x1ff8);
#pragma unroll
          for (int s = 1; s < 7; ++s)
            if (c & (1u << (12 + s))) v[u] += pj[s];
          if (c & (1u << 19))
            v[u] = fma(pj[7], (c & (1u << 22)) ? eff_of(c, L * (4 * q + u) + first, cur.target % LDA) : JR(1), v[u]);
        }
        if (not_zero(v[u]) || (c & (1u << 23))) acc = fma(flip_sign(cur.w, c << 11), v[u], acc);
        if (c & (1u << 21)) {  // last term of the entry
          A[cur.target] = acc;
          acc = JR(0);
          cur = ahead;
          ent += L;
          ahead = ent_of(min(ent + L, L * (ents - 1) + first));
        }
      }
    }
  }
  if constexpr (W > 1) {
    team_sync<W>(id);
    if (role > 0) return;
  } else {
    __syncwarp();
  }
  // (3) constant-pressure energy row: dT/dt = (Fh - sum h_k wm_k) / (rho cp)
  JR D = JR(0), dD = JR(0), Qf = JR(0), cpf = JR(0);
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int k = idx(r);
    if (k < NS) {
      const JR h = TH_[k], c = TC[k], d = TD[k];
      const JR iw = Tab::template sp<JR>(k).invW;
      const JR cpm = c * JR(kRerg) * iw, hm = h * RT * iw;
      const JR yk = (JR)y[r];
      const JR fk = (JR)FRC[k];
      D = fma(yk, cpm, D);
      dD = fma(pgb_mul(pgb_mul(yk, d), JR(kRerg)), iw, dD);
      Qf = fma(-hm, fk, Qf);
      cpf = fma(cpm, fk, cpf);
    }
  }
  D = warp_sum(D);
  dD = warp_sum(dD);
  const JR Q = (JR)FRC[NS] - Qw + warp_sum(Qf);
  const JR cpwm = cpw + warp_sum(cpf);
  const JR invD = JR(1) / D;
  const JR QD2 = Q * invD * invD;
#pragma unroll
  for (int cc = 0; cc < R; ++cc) {
    const int k = idx(cc);
    if (k > NS) continue;
    JR acc = JR(0);
#pragma unroll 1
    for (int i = 0; i < NS; ++i) acc = fma(pgb_mul(pgb_mul(TH_[i], RT), Tab::template sp<JR>(i).invW), A[i * LDA + k], acc);
    if (k < NS) {
      A[NS * LDA + k] = fma(-pgb_mul(pgb_mul(QD2, TC[k]), JR(kRerg)), Tab::template sp<JR>(k).invW, pgb_mul(-acc, invD));
    } else {
      A[NS * LDA + NS] = fma(-(acc + cpwm), invD, -pgb_mul(QD2, dD));
    }
  }
  __syncwarp();
}

// The Jacobian and the LU of I - gamma J. False: singular. With FACTOR false it stops after the
// Jacobian, which A then holds (the diagnostic entry point).
template <class M, class JR, bool FACTOR = true, int W = 1>
__device__ __forceinline__ bool warp_setup(const WVec<M> yv, const double gamma, const double* FRC, JR* A,
                                        JR* XS, JR* RX, JR* TH, int* PIV, double* TP = nullptr, int id = 0,
                                        JR* QN = nullptr) {
  if constexpr (W > 1) {
    JR* const TJ = reinterpret_cast<JR*>(TP);
    const double T = __shfl_sync(0xffffffffu, yv.v[M::NS >> 5], M::NS & 31);
    if ((threadIdx.x & 31) == 0) {
      TJ[0] = (JR)T;
      TP[5] = 2.0;
    }
    team_sync<W>(id);
    warp_jacobian<M, JR, W>(yv, FRC, A, XS, RX, TH, 0, id, TJ, QN);
  } else {
    warp_jacobian<M, JR>(yv, FRC, A, XS, RX, TH);
  }
  if constexpr (FACTOR) return warp_lu_factor<M::N>(A, PIV, (JR)gamma);
  else return true;
}

// Substitution steps of (I - gamma J) x = b, L lanes per cell with row i in lane i % L, slot i / L,
// of the cell's lanes (mask, first lane gbase): the solution moves by shuffles, so a step costs one
// shuffle and one multiply-add and the matrix loads run ahead of it (the staged shared-memory form
// waited for a store, a barrier and a load at each step: 200 cycles instead of 40).
// BACK false: the forward half alone.
template <int N, int L, class JR, bool BACK = true>
__device__ __forceinline__ void lu_substitute(const JR* A, unsigned mask, int gbase, JR (&x)[(N + L - 1) / L]) {
  constexpr int R = (N + L - 1) / L, LDA = N + 1;
  const int sub = (threadIdx.x & 31) - gbase;
#pragma unroll
  for (int s = 0; s < R; ++s)
#pragma unroll 2
    for (int q = 0; q < (s + 1 < R ? L : N - s * L); ++q) {
      const int k = s * L + q;
      const JR bk = __shfl_sync(mask, x[s], gbase + q);
#pragma unroll
      for (int r = s; r < R; ++r) {
        const int i = sub + L * r;
        if (i > k && i < N) x[r] = fma(-A[i * LDA + k], bk, x[r]);
      }
    }
  if constexpr (!BACK) return;
#pragma unroll
  for (int s = R - 1; s >= 0; --s)
#pragma unroll 2
    for (int q = (s + 1 < R ? L : N - s * L) - 1; q >= 0; --q) {
      const int k = s * L + q;
      const JR xk = __shfl_sync(mask, x[s], gbase + q) * A[k * LDA + k];
#pragma unroll
      for (int r = 0; r <= s; ++r) {
        const int i = sub + L * r;
        if (i == k) x[r] = xk;
        else if (i < k) x[r] = fma(-A[i * LDA + k], xk, x[r]);
      }
    }
}

// (I - gamma J) x = b with the factors warp_setup left in A / PIV: one warp, rows over lanes, b
// distributed like the state (element i in lane i mod 32) and overwritten with x; XS is the
// N-element staging vector.
template <class M, class JR>
__device__ __forceinline__ void warp_lu_solve(const JR* A, const int* PIV, JR* XS, double (&b)[(M::N + 31) / 32]) {
  constexpr int N = M::N, R = (N + 31) / 32;
  const int lane = threadIdx.x & 31;
  JR x[R];
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (lane + 32 * r < N) XS[lane + 32 * r] = (JR)b[r];
  __syncwarp();
#pragma unroll
  for (int r = 0; r < R; ++r) x[r] = lane + 32 * r < N ? XS[PIV[lane + 32 * r]] : JR(0);
  lu_substitute<N, 32>(A, 0xffffffffu, 0, x);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (lane + 32 * r < N) b[r] = (double)x[r];
  __syncwarp();
}

// W > 1: teams of W warps per cell (WPB / W cells a block), the first warp leading: for few cells.
template <class M, class JR, int WPB, int W = 1>
__global__ void __launch_bounds__(WPB * 32, 1) bdf_warp_kernel(const ReactParams P) {
  using namespace bdf;
  using Tab = typename M::TabG;
  constexpr int N = M::N, NS = M::NS;
  constexpr int R = (N + 31) / 32;   // vector elements per lane
  constexpr int LDA = N + 1;         // padded matrix row
  constexpr bool MIXED = sizeof(JR) == sizeof(float);
  extern __shared__ __align__(16) unsigned char wsmem[];
  const int lane = threadIdx.x & 31, wid = (threadIdx.x >> 5) / W;  // wid: the cell's place in the block
  __shared__ double team_par[W > 1 ? WPB / W : 1][6];
  double* const TP = team_par[W > 1 ? wid : 0];
  unsigned char* base = wsmem + (size_t)wid * bdf_warp_smem_per_warp<M, JR>();
  double* Z = reinterpret_cast<double*>(base);   // [(QMAX+2)][N]
  double* FRC = Z + (QMAX + 2) * N;              // [N] forcing (rhoY, then rho h)
  double* LC = FRC + N;                          // [QMAX+1] l coefficients
  double* TAU = LC + (QMAX + 1);                 // [QMAX+2] step history
  unsigned char* const scratch = base + bdf_warp_state_bytes<M>();  // RHS | setup scratch
  double* CS = reinterpret_cast<double*>(scratch);  // [NS] concentrations
  double* GS = CS + NS;                          // [NS] g/RT
  double* QS = GS + NS;                          // [NR] rates of progress
  JR* RX = reinterpret_cast<JR*>(scratch);       // Jacobian partials
  JR* TH = RX + wbdf::rx_len<M>();               // [4][NS] NASA-7 terms of the setup
  JR* A = reinterpret_cast<JR*>(scratch + bdf_warp_scratch_bytes<M, JR>());  // [N][LDA] Jacobian, then its LU
  JR* XS = A + N * LDA;                          // [N] solve vector
  int* PIV = reinterpret_cast<int*>(XS + N);
  // teams: [NR] net rates, after the cells' memory
  JR* const QN = reinterpret_cast<JR*>(wsmem + (size_t)(WPB / W) * bdf_warp_smem_per_warp<M, JR>()) + (W > 1 ? wid * M::NR : 0);

  if constexpr (W > 1) {
    const int role = (threadIdx.x >> 5) % W;
    if (role > 0) {  // follow the leader's right-hand sides until it has no more cells
      for (;;) {
        team_sync<W>(1 + wid);
        if (TP[5] == 0.0) return;
        if (TP[5] == 2.0) {
          const WVec<M> none = {};
          warp_jacobian<M, JR, W>(none, FRC, A, XS, RX, TH, role, 1 + wid, reinterpret_cast<JR*>(TP), QN);
          continue;
        }
        team_rates<M, W>(role, 1 + wid, TP[0], TP[1], TP[2], TP[3], TP[4], CS, GS, QS);
      }
    }
  }

  const long long ncell = P.ncell_dev ? (long long)*P.ncell_dev : P.ncell;
  const int qmax = max(1, min(P.max_order, QMAX));
  const double tout = P.dt;
  auto cell_done = [&]() {
    if (P.done && lane == 0) atomicAdd(P.done, 1ull);
  };

  // ---- lane-distributed vectors: element i = lane + 32 r ----
  auto idx = [&](int r) { return lane + 32 * r; };
  auto bcast = [&](const double (&v)[R], int i) -> double {
    return __shfl_sync(0xffffffffu, v[i >> 5], i & 31);
  };
  double ewt[R];
  auto wms = [&](const double (&v)[R]) -> double {  // squared WRMS norm
    double s = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (idx(r) < N) { const double x = v[r] * ewt[r]; s = fma(x, x, s); }
    return warp_sum(s) * (1.0 / N);
  };

  // ---- right-hand side: f = [W_k wdot_k + F_k, dT/dt] at y ----
  auto rhs = [&](const double (&y)[R], double (&f)[R]) {
    WVec<M> yv;
#pragma unroll
    for (int r = 0; r < R; ++r) yv.v[r] = y[r];
    const WVec<M> fv = warp_rhs<M, W>(yv, CS, GS, QS, FRC, TP, 1 + wid);
#pragma unroll
    for (int r = 0; r < R; ++r) f[r] = fv.v[r];
  };

  // ---- analytic Jacobian into A (equations of jac_table, mech_tables.cuh), in type JR ----
  auto solve = [&](double (&b)[R]) { warp_lu_solve<M, JR>(A, PIV, XS, b); };

  for (;;) {
    // ---------------------------------------------- next cell (work stealing, one per warp)
    unsigned long long cnext = 0;
    if (lane == 0) cnext = atomicAdd(P.next_cell, 1ull);
    cnext = __shfl_sync(0xffffffffu, cnext, 0);
    if ((long long)cnext >= ncell) break;
    const bool resuming = W > 1 && P.resuming;
    const ResumeRec<N, JR> rec(P.resume, resuming ? cnext : 0);
    const long long cell = resuming ? rec.head->cell : P.cell_list ? P.cell_list[cnext] : (long long)cnext;
    int lo = 0, hi = P.nbox - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (P.boxes[mid].cell_offset <= cell) lo = mid; else hi = mid - 1;
    }
    const BoxDev& B = P.boxes[lo];
    long long rr = cell - B.cell_offset;
    const int ci = B.lo0 + (int)(rr % B.len0);
    rr /= B.len0;
    const int cj = B.lo1 + (int)(rr % B.len1);
    const int ck = B.lo2 + (int)(rr / B.len1);
    auto elem = [&](const ArrDev& a, int n) -> double& {
      return a.p[(long long)(ci - a.begin0) + (long long)(cj - a.begin1) * a.jstride +
                 (long long)(ck - a.begin2) * a.kstride + (long long)n * a.nstride];
    };
    if (B.mask.p && B.mask.p[(long long)(ci - B.mask.begin0) + (long long)(cj - B.mask.begin1) * B.mask.jstride +
                             (long long)(ck - B.mask.begin2) * B.mask.kstride] < 0) {
      if (lane == 0) elem(B.FC, 0) = 0.0;
      if (B.IR.p)
        for (int k = lane; k < NS; k += 32) elem(B.IR, k) = -elem(B.rYsrc, k);
      cell_done();
      continue;
    }
    double y[R], f[R], acor[R], tmp[R], acor_saved[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = idx(r);
      y[r] = 0.0; f[r] = 0.0; acor[r] = 0.0; tmp[r] = 0.0; acor_saved[r] = 0.0; ewt[r] = 1.0;
      if (i < NS) { y[r] = elem(B.rY, i) * B.sY_in; FRC[i] = elem(B.rYsrc, i) * B.sY_in; }
      else if (i == NS) { y[r] = elem(B.T, 0); FRC[NS] = elem(B.rEsrc, 0) * B.sE_in; }
      if (i < N) Z[i] = y[r];
    }
    const double rE0 = elem(B.rE, 0) * B.sE_in;
    if (lane < QMAX + 2) TAU[lane] = 0.0;
    __syncwarp();
    auto zget = [&](int j, int r) -> double& { return Z[j * N + idx(r)]; };
    auto set_ewt = [&]() {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) {
          const double d = fma(P.rtol, fabs(zget(0, r)), P.atol[idx(r)]);
          ewt[r] = MIXED ? recip_fast(d) : 1.0 / d;
        }
    };

    double t = 0.0, h = 0.0, hscale = 0.0, etamax = ETAMX1, eta = 1.0;
    double gamma = 0.0, gammap = 0.0, gamrat = 1.0, crate2 = 1.0, rl1 = 1.0, acnrm2 = 0.0;
    double tq1 = 1.0, tq2 = 1.0, tq3 = 1.0, tq5 = 1.0, tq5_saved = 1.0, inv_tq4_sq = 1.0;
    int q = 1, qwait = 2, nef = 0, ncf = 0, status = OK;
    long long nst = 0, nfe = 0, nje = 0, nstlp = 0, netf = 0, ncfn = 0;
    bool force_setup = true;

    auto rescale = [&](double e) {
      double fac = e;
#pragma unroll 1
      for (int j = 1; j <= q; ++j) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (idx(r) < N) zget(j, r) *= fac;
        fac *= e;
      }
      h = __dmul_rn(hscale, e);
      hscale = h;
    };
    auto predict = [&]() {
      t += h;
#pragma unroll 1
      for (int k = 1; k <= q; ++k)
#pragma unroll 1
        for (int j = q; j >= k; --j)
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (idx(r) < N) zget(j - 1, r) += zget(j, r);
    };
    auto retract = [&]() {
      t -= h;
#pragma unroll 1
      for (int k = 1; k <= q; ++k)
#pragma unroll 1
        for (int j = q; j >= k; --j)
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (idx(r) < N) zget(j - 1, r) -= zget(j, r);
    };
    // l coefficients and error constants, gamma and its ratio: the arithmetic of the per-thread kernel's
    // set_coeffs, coefficient l_i in lane i and independent quotients formed side by side
    auto set_coeffs = [&]() {
      const double alpha0 = alpha0_of(q);
      double hs = h;  // lane i: h + tau_1 + ... + tau_i
#pragma unroll 1
      for (int i = 1; i <= min(lane, QMAX); ++i) hs += TAU[i];
      const double xi = pgb_div64(h, hs);
      double sum_xi_inv = 0.0, l = lane == 0 ? 1.0 : 0.0;
#pragma unroll 1
      for (int i = 1; i <= q - 1; ++i) {
        const double xi_inv = __shfl_sync(0xffffffffu, xi, i - 1);
        sum_xi_inv += xi_inv;
        const double below = __shfl_up_sync(0xffffffffu, l, 1);
        if (lane >= 1 && lane <= i) l = fma(below, xi_inv, l);
      }
      const double xistar_inv = -alpha0 - sum_xi_inv;
      {
        const double below = __shfl_up_sync(0xffffffffu, l, 1);
        if (lane >= 1 && lane <= q) l = fma(below, xistar_inv, l);
      }
      const double xiq_inv = __shfl_sync(0xffffffffu, xi, q - 1), xiq1_inv = __shfl_sync(0xffffffffu, xi, q);
      const double alpha0_hat = -(sum_xi_inv + xiq_inv);
      const double A1 = 1.0 - alpha0_hat + alpha0;
      const double A2 = fma((double)q, A1, 1.0);
      const double lq = __shfl_sync(0xffffffffu, l, q), l1 = __shfl_sync(0xffffffffu, l, 1);
      const double A3 = alpha0 + inv_int(q), A4 = alpha0_hat + xiq_inv;
      const double A5 = alpha0 - inv_int(q + 1), A6 = alpha0_hat - xiq1_inv;
      double d[5];
      group_div<5>({A1, A2 * xistar_inv, xistar_inv, 1.0 - A6 + A5, 1.0}, {alpha0 * A2, lq * xiq_inv, lq, A2, l1}, d,
                   0xffffffffu, 0);
      tq2 = fabs(d[0]);
      tq5 = fabs(d[1]);
      rl1 = d[4];
      gamma = h * rl1;
      double e[3];
      group_div<3>({d[2] * (1.0 - A4 + A3), d[3], gamma}, {A3, xiq1_inv * (q + 2) * A5, gammap}, e, 0xffffffffu, 0);
      if (qwait == 1) {
        tq1 = q > 1 ? fabs(e[0]) : 1.0;
        tq3 = fabs(e[1]);
      }
      gamrat = nst > 0 ? e[2] : 1.0;
      if (nst == 0) gammap = gamma;
      inv_tq4_sq = (tq2 * (1.0 / NLSCOEF)) * (tq2 * (1.0 / NLSCOEF));
      __syncwarp();
      if (lane <= QMAX) LC[lane] = l;
      __syncwarp();
    };
    auto adjust_order = [&](int dq) {
      double hs = 0.0;  // lane i: tau_1 + ... + tau_{i+1}
#pragma unroll 1
      for (int i = 0; i <= min(lane, QMAX - 1); ++i) hs += TAU[i + 1];
      const double xis = pgb_div64(hs, hscale), rxis = pgb_div64(1.0, xis);
      double w = lane == 2 ? 1.0 : 0.0, alpha1 = 0.0, prod = 1.0;  // lane i: w_i
      const int top = dq > 0 ? q : q - 2;
#pragma unroll 1
      for (int j = 1; j <= top; ++j) {
        const double xi = __shfl_sync(0xffffffffu, xis, j - 1);
        prod *= xi;
        alpha1 += __shfl_sync(0xffffffffu, rxis, j - 1);
        const double below = __shfl_up_sync(0xffffffffu, w, 1);
        if (lane >= 2 && lane <= j + 2 && (dq < 0 || j <= q - 1)) w = fma(w, xi, below);
      }
      if (dq > 0) {
        const double A1 = pgb_div64(-alpha0_of(q) - alpha1, prod);
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (idx(r) < N) zget(q + 1, r) = A1 * acor_saved[r];
      }
      const int from = dq > 0 ? q + 1 : q, last = dq > 0 ? q : q - 1;
#pragma unroll 1
      for (int j = 2; j <= last; ++j) {
        double wj = __shfl_sync(0xffffffffu, w, j);
        if (dq < 0) wj = -wj;
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (idx(r) < N) zget(j, r) = fma(wj, zget(from, r), zget(j, r));
      }
      if (dq < 0) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (idx(r) < N) zget(q, r) = 0.0;
      }
    };
    // modified Newton on the corrector; 0 converged, 1 convergence failure, 2 singular matrix
    auto newton = [&]() -> int {
      bool call_setup = force_setup || nst == 0 || nst >= nstlp + MSBP || fabs(gamrat - 1.0) > DGMAX;
      force_setup = false;
      for (;;) {
#pragma unroll
        for (int r = 0; r < R; ++r) { y[r] = idx(r) < N ? zget(0, r) : 0.0; acor[r] = 0.0; }
        rhs(y, f);
        ++nfe;
        bool jcur = false;
        if (call_setup) {
          WVec<M> yv;
#pragma unroll
          for (int r = 0; r < R; ++r) yv.v[r] = y[r];
          ++nje;
          const bool ok = warp_setup<M, JR, true, W>(yv, gamma, FRC, A, XS, RX, TH, PIV, TP, 1 + wid, QN);
          gammap = gamma;
          gamrat = 1.0;
          crate2 = 1.0;
          nstlp = nst;
          if (!ok) return 2;
          jcur = true;
          call_setup = false;
        }
        double delp2 = 0.0, del2 = 0.0;
        int mm = 0;
        bool ok = false;
        for (;;) {
#pragma unroll
          for (int r = 0; r < R; ++r)
            tmp[r] = idx(r) < N ? fma(gamma, f[r], -fma(rl1, zget(1, r), acor[r])) : 0.0;
          solve(tmp);
          if (gamrat != 1.0) {
            const double s = pgb_div64(2.0, 1.0 + gamrat);
#pragma unroll
            for (int r = 0; r < R; ++r) tmp[r] = __dmul_rn(tmp[r], s);
          }
          del2 = wms(tmp);
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (idx(r) < N) { acor[r] += tmp[r]; y[r] = zget(0, r) + acor[r]; }
          if (mm > 0) crate2 = fmax((CRDOWN * CRDOWN) * crate2, pgb_div64(del2, delp2));
          if (del2 * fmin(1.0, crate2) * inv_tq4_sq <= 1.0) {
            acnrm2 = (mm == 0) ? del2 : wms(acor);
            ok = true;
            break;
          }
          ++mm;
          if (mm == MAXCOR || (mm >= 2 && del2 > (RDIV * RDIV) * delp2)) break;
          delp2 = del2;
          rhs(y, f);
          ++nfe;
          if (!isfinite(bcast(f, 0))) break;
        }
        if (ok) return 0;
        if (!jcur) { call_setup = true; continue; }
        return 1;
      }
    };

    // ---------------------------------------------- initial step size
    if (!resuming) {
      rhs(y, f);
      ++nfe;
      set_ewt();
      {
        const double tround = UROUND * tout;
        const double hlb = 100.0 * tround;
        double hub_inv = 0.0;
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (idx(r) < N) hub_inv = fmax(hub_inv, pgb_div64(fabs(f[r]), fma(0.1, fabs(zget(0, r)), P.atol[idx(r)])));
        hub_inv = warp_max(hub_inv);
        double hub = 0.1 * tout;
        if (hub * hub_inv > 1.0) hub = pgb_div64(1.0, hub_inv);
        double hg = sqrt(hlb * hub), hnew = hg;
        if (hub > hlb) {
#pragma unroll 1
          for (int count = 1; count <= 4; ++count) {
            double yy[R], fy[R];
#pragma unroll
            for (int r = 0; r < R; ++r) yy[r] = idx(r) < N ? fma(hg, f[r], zget(0, r)) : 0.0;
            rhs(yy, fy);
            ++nfe;
#pragma unroll
            for (int r = 0; r < R; ++r) tmp[r] = pgb_div64(fy[r] - f[r], hg);
            const double ydd = sqrt(wms(tmp));
            hnew = sqrt((ydd * hub * hub > 2.0) ? pgb_div64(2.0, ydd) : hg * hub);
            if (count == 4) break;
            const double hrat = pgb_div64(hnew, hg);
            if (hrat > 0.5 && hrat < 2.0) break;
            if (count >= 2 && hrat > 2.0) { hnew = hg; break; }
            hg = hnew;
          }
        }
        h = fmin(fmax(0.5 * hnew, hlb), hub);
      }
      hscale = h;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) zget(1, r) = h * f[r];
      q = 1; qwait = 2; etamax = ETAMX1;
      if (lane == 0) TAU[1] = h;
      __syncwarp();
    } else {  // or the state another launch left
      const ResumeHead& H = *rec.head;
#pragma unroll 1
      for (int e = lane; e < (QMAX + 1) * N; e += 32) Z[e] = rec.Z[e];
#pragma unroll
      for (int r = 0; r < R; ++r) acor_saved[r] = idx(r) < N ? rec.Z[(QMAX + 1) * N + idx(r)] : 0.0;
      if (lane < QMAX + 2) TAU[lane] = rec.tau[lane];
#pragma unroll 1
      for (int e = lane; e < N * N; e += 32) A[e + e / N] = rec.lu[e];
#pragma unroll 1
      for (int e = lane; e < N; e += 32) PIV[e] = rec.piv[e];
      t = H.t; h = H.h; hscale = H.hscale; etamax = H.etamax; gammap = H.gammap; crate2 = H.crate2;
      tq5_saved = H.tq5_saved;
      q = H.q; qwait = H.qwait;
      nst = H.nst; nfe = H.nfe; nje = H.nje; nstlp = H.nstlp; netf = H.netf; ncfn = H.ncfn;
      force_setup = H.force_setup != 0;
      __syncwarp();
    }

    // ---------------------------------------------- step loop
    bool handed_over = false;
    for (;;) {
      if (nst >= P.max_steps) { status = MAX_STEPS; break; }
      if (W == 1 && P.drain > 0) {  // few cells left in the whole launch: leave this one to a team
        unsigned long long done = 0;
        if (lane == 0) done = *static_cast<volatile unsigned long long*>(P.done);
        done = __shfl_sync(0xffffffffu, done, 0);
        if (ncell - (long long)done <= P.drain) {
          unsigned long long at = 0;
          if (lane == 0) at = atomicAdd(P.resume_count, 1ull);
          const ResumeRec<N, JR> out(P.resume, __shfl_sync(0xffffffffu, at, 0));
          if (lane == 0) {
            ResumeHead H;
            H.t = t; H.h = h; H.hscale = hscale; H.etamax = etamax; H.gammap = gammap; H.crate2 = crate2;
            H.tq5_saved = tq5_saved;
            H.cell = cell;
            H.box = lo; H.ci = ci; H.cj = cj; H.ck = ck;
            H.q = q; H.qwait = qwait; H.nst = (int)nst; H.nfe = (int)nfe; H.nje = (int)nje; H.nstlp = (int)nstlp;
            H.netf = (int)netf; H.ncfn = (int)ncfn;
            H.force_setup = force_setup;
            H.full_swaps = 1;
            *out.head = H;
          }
#pragma unroll 1
          for (int e = lane; e < (QMAX + 1) * N; e += 32) out.Z[e] = Z[e];
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (idx(r) < N) out.Z[(QMAX + 1) * N + idx(r)] = acor_saved[r];
          if (lane < QMAX + 2) out.tau[lane] = TAU[lane];
#pragma unroll 1
          for (int e = lane; e < N * N; e += 32) out.lu[e] = A[e + e / N];
#pragma unroll 1
          for (int e = lane; e < N; e += 32) out.piv[e] = PIV[e];
          handed_over = true;
          break;
        }
      }
      if ((t + h - tout) * h > 0.0) rescale(pgb_div64((tout - t) * (1.0 - 4.0 * UROUND), h));
      set_ewt();
      nef = 0; ncf = 0;
      double dsm2 = 0.0;
      bool failed = false;
      for (;;) {
        predict();
        set_coeffs();
        const int nflag = newton();
        if (nflag != 0) {
          retract();
          ++ncf; ++ncfn;
          if (nflag == 2 || ncf >= MXNCF || fabs(h) <= 100.0 * UROUND * fabs(t)) { status = CONV; failed = true; break; }
          force_setup = true;
          etamax = 1.0;
          rescale(ETACF);
          continue;
        }
        dsm2 = acnrm2 * (tq2 * tq2);
        if (!(dsm2 <= 1.0)) {
          retract();
          ++nef; ++netf;
          if (nef >= MXNEF || !isfinite(dsm2)) { status = isfinite(dsm2) ? ERRTEST : NONFINITE; failed = true; break; }
          etamax = 1.0;
          if (nef <= MXNEF1) {
            double e = pgb_div64(1.0, pgb_pow64((BIAS2 * BIAS2) * dsm2, 0.5 * inv_int(q + 1)) + ADDON);
            e = fmax(ETAMIN, e);
            if (nef >= SMALL_NEF) e = fmin(e, ETAMXF);
            rescale(e);
          } else if (q > 1) {
            adjust_order(-1);
            --q;
            qwait = q + 1;
            rescale(ETAMIN);
          } else {
            rescale(ETAMIN);
#pragma unroll
            for (int r = 0; r < R; ++r) y[r] = idx(r) < N ? zget(0, r) : 0.0;
            rhs(y, f);
            ++nfe;
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (idx(r) < N) zget(1, r) = h * f[r];
            qwait = 10;
          }
          if (fabs(h) <= 100.0 * UROUND * fabs(t)) { status = HSMALL; failed = true; break; }
          continue;
        }
        break;
      }
      if (failed) break;
      // ---- complete the step ----
      ++nst;
      __syncwarp();
      if (lane == 0) {
#pragma unroll 1
        for (int i = q + 1; i >= 2; --i) TAU[i] = TAU[i - 1];
        TAU[1] = h;
      }
#pragma unroll 1
      for (int j = 0; j <= q; ++j) {
        const double lj = LC[j];
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (idx(r) < N) zget(j, r) = fma(lj, acor[r], zget(j, r));
      }
      __syncwarp();
      --qwait;
      if (qwait == 1 && q != qmax) {
#pragma unroll
        for (int r = 0; r < R; ++r) acor_saved[r] = acor[r];
        tq5_saved = tq5;
      }
      if (fabs(t - tout) <= 100.0 * UROUND * (fabs(t) + fabs(h)) || t >= tout) break;
      // ---- next step size and order ----
      // step-size factors of orders q, q - 1 and q + 1: one power and one quotient, lane 1 takes q - 1,
      // lane 2 q + 1
      const bool orders = etamax != 1.0 && qwait == 0;
      double ddn2 = 0.0, dup2 = 0.0;
      if (orders) {
        if (q > 1) {
          double zq[R];
#pragma unroll
          for (int r = 0; r < R; ++r) zq[r] = idx(r) < N ? zget(q, r) : 0.0;
          ddn2 = wms(zq) * (tq1 * tq1);
        }
        if (q != qmax) {
          double d[2];
          group_div<2>({h, tq5}, {TAU[2], tq5_saved}, d, 0xffffffffu, 0);
          double hrp = d[0];
#pragma unroll 1
          for (int k = 0; k < q; ++k) hrp *= d[0];
          const double cquot = d[1] * hrp;
#pragma unroll
          for (int r = 0; r < R; ++r) tmp[r] = fma(-cquot, acor_saved[r], acor[r]);
          dup2 = wms(tmp) * (tq3 * tq3);
        }
      }
      double etaq, etaqm1 = 0.0, etaqp1 = 0.0;
      {
        const double x = lane == 1 ? (BIAS1 * BIAS1) * ddn2 : lane == 2 ? (BIAS3 * BIAS3) * dup2 : (BIAS2 * BIAS2) * dsm2;
        const double a = 0.5 * inv_int(lane == 1 ? q : lane == 2 ? q + 2 : q + 1);
        const double e = pgb_div64(1.0, pgb_pow64(x, a) + ADDON);
        etaq = __shfl_sync(0xffffffffu, e, 0);
        const double em = __shfl_sync(0xffffffffu, e, 1), ep = __shfl_sync(0xffffffffu, e, 2);
        if (orders && q > 1) etaqm1 = em;
        if (orders && q != qmax) etaqp1 = ep;
      }
      int qprime = q;
      if (etamax == 1.0) {
        qwait = max(qwait, 2);
        eta = 1.0;
      } else {
        eta = etaq;
        if (qwait == 0) {
          qwait = 2;
          const double etam = fmax(etaqm1, fmax(etaq, etaqp1));
          if (etam < THRESH) {
            eta = 1.0;
          } else if (etam == etaq) {
            eta = etaq;
          } else if (etam == etaqm1) {
            eta = etaqm1;
            qprime = q - 1;
          } else {
            eta = etaqp1;
            qprime = q + 1;
#pragma unroll
            for (int r = 0; r < R; ++r) acor_saved[r] = acor[r];
          }
        } else if (eta < THRESH) {
          eta = 1.0;
        }
        if (eta >= THRESH || qprime != q) eta = fmin(eta, etamax);
        else eta = 1.0;
      }
      etamax = (nst <= SMALL_NST) ? ETAMX2 : ETAMX3;
      if (qprime != q) {
        adjust_order(qprime - q);
        q = qprime;
        qwait = q + 1;
      }
      if (eta != 1.0) rescale(eta);
      __syncwarp();
    }

    // ---------------------------------------------- finish: rho h(t), T from (h, Y)
    __syncwarp();
    if (handed_over) continue;
    cell_done();
    if (status != OK && P.retry_list) {  // hand the cell to the retry pass, arrays untouched
      if (lane == 0) {
        P.retry_list[atomicAdd(P.retry_count, 1ull)] = cell;
        ReactStats* S = P.stats;
        atomicAdd(&S->nst, (unsigned long long)nst);
        atomicAdd(&S->nfe, (unsigned long long)nfe);
        atomicAdd(&S->nje, (unsigned long long)nje);
        atomicAdd(&S->netf, (unsigned long long)netf);
        atomicAdd(&S->ncfn, (unsigned long long)ncfn);
        atomicAdd(&S->nretry, 1ull);
      }
      __syncwarp();
      continue;
    }
    const double rE = fma(tout, FRC[NS], rE0);
    double rho_l = 0.0;
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (idx(r) < NS) rho_l += zget(0, r);
    const double inv_rho = pgb_div64(1.0, warp_sum(rho_l));
    const double htarget = __dmul_rn(rE, inv_rho);
    double Tn = Z[NS];
    if (!(Tn > 90.0 && Tn < 5000.0)) Tn = 1000.0;
#pragma unroll 1
    for (int it = 0; it < 50; ++it) {
      double hl = 0.0, cl = 0.0;
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const int k = idx(r);
        if (k < NS) {
          const TabSpecies<double>& s = Tab::template sp<double>(k);
          const bool lo = Tn < s.Tmid;
          const double* a = lo ? s.lo : s.hi;
          const double* hc = lo ? s.hlo : s.hhi;
          const double invTn = pgb_div64(1.0, Tn);
          const double hRT = fma(Tn, fma(Tn, fma(Tn, fma(Tn, hc[4], hc[3]), hc[2]), hc[1]), fma(hc[5], invTn, hc[0]));
          const double cpR = fma(Tn, fma(Tn, fma(Tn, fma(Tn, a[4], a[3]), a[2]), a[1]), a[0]);
          const double Yk = zget(0, r) * inv_rho;
          hl = fma(Yk * s.invW, hRT * kRerg * Tn, hl);
          cl = fma(Yk * s.invW, cpR * kRerg, cl);
        }
      }
      const double hh = warp_sum(hl), cp = warp_sum(cl);
      double dT = pgb_div64(htarget - hh, cp);
      dT = fmax(-100.0, fmin(100.0, dT));
      Tn = fmax(90.0, fmin(5000.0, Tn + dT));
      if (fabs(dT) < 1e-10 * Tn) break;
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (idx(r) < NS) {
        const double rYn = __dmul_rn(zget(0, r), B.sY_out);
        if (B.IR.p)  // separate roundings, as separate passes over arrays give
          elem(B.IR, idx(r)) = __dsub_rn(__dmul_rn(-__dsub_rn(elem(B.rY, idx(r)), rYn), 1.0 / tout),
                                         elem(B.rYsrc, idx(r)));
        elem(B.rY, idx(r)) = rYn;
      }
    if (lane == 0) {
      elem(B.T, 0) = Tn;
      elem(B.rE, 0) = rE * B.sE_out;
      elem(B.FC, 0) = (status == OK) ? (double)nfe : -(double)status;
      ReactStats* S = P.stats;
      atomicAdd(&S->nst, (unsigned long long)nst);
      atomicAdd(&S->nfe, (unsigned long long)nfe);
      atomicAdd(&S->nje, (unsigned long long)nje);
      atomicAdd(&S->netf, (unsigned long long)netf);
      atomicAdd(&S->ncfn, (unsigned long long)ncfn);
      if (status != OK) atomicAdd(&S->nfail, 1ull);
      atomicMax(&S->max_nst, (unsigned long long)nst);
      const int bin = min(15, 31 - __clz((int)max(nst, 1LL)));
      atomicAdd(&S->hist[bin], 1ull);
    }
    __syncwarp();
  }
  if constexpr (W > 1) {  // dismiss the team
    if (lane == 0) TP[5] = 0.0;
    team_sync<W>(1 + wid);
  }
}

}  // namespace pgb

#endif  // PGB_BDF_WARP_KERNEL_CUH
