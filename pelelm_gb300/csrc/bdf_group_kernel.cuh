// Persistent, work-stealing BDF reactor kernel with one cell per group of G lanes (32 / G cells
// per warp): the default for drm19-sized mechanisms (21 species, 84 reactions, N = 22).
//
// Same contract and algorithm as bdf_kernel.cuh and bdf_warp_kernel.cuh (the PelePhysics reactor
// called at Source/PeleLM.cpp:5752; CVODE-class fixed-leading-coefficient variable-order
// Nordsieck BDF, modified Newton with analytic Jacobian and dense partial-pivot LU, CVODE's
// documented step/order heuristics; its CPU statement is oracle/bdf_oracle.cpp).
//
// Why groups on GB300: an FP64 warp instruction occupies the FP64 pipe for the same time whatever
// its active mask, so FP64 work should fill lanes with different cells. A warp per cell leaves
// the scalar step logic (coefficients, error test, step and order selection: about half of the
// FP64 instructions for drm19) on one useful lane in 32 and rounds 84 reactions up to 96 lane
// slots; a thread per cell cannot hold a 22-unknown cell's state in registers and shared memory
// at useful occupancy. A group of G lanes per cell runs the scalar logic for 32 / G cells per
// instruction, spreads reactions and species over G lanes, and keeps each lane's share of the
// state vectors (ceil(N / G) elements) in registers.
//
//  * every group runs the flattened state machine of bdf_kernel.cuh: each pass evaluates one
//    FP64 right-hand side per active cell (group-parallel: species, then reactions, then a
//    species-major gather; group sums by xor shuffles inside the group's lane mask);
//  * Jacobian and LU (type JR: FP32 in mixed precision) are built one cell at a time by the
//    whole warp (warp_setup of bdf_warp_kernel.cuh, the same arithmetic as the warp mapping)
//    into the cell's matrix in shared memory; the triangular solves run per group (rows over
//    the group's lanes), the same operations in the same order as the warp mapping's solve;
//  * per cell in shared memory: Nordsieck history (+ saved correction), forcing, l and tau,
//    the matrix and its pivots; per warp one region that holds the cells' RHS scratch
//    (concentrations, g/RT, rates of progress) during the RHS and the Jacobian scratch
//    (per-reaction partials, NASA-7 terms) during the setups;
//  * a group whose cell is done takes the next cell index from the global queue (one atomic
//    per warp for all groups that need a cell: work stealing across all boxes);
//  * with a retry list (mixed precision), a failed cell is listed and left untouched for the
//    FP64 pass that follows on the same stream.
#ifndef PGB_BDF_GROUP_KERNEL_CUH
#define PGB_BDF_GROUP_KERNEL_CUH

#include "bdf_warp_kernel.cuh"

namespace pgb {

// Bytes of shared memory per cell (state that lives across passes), per cell of RHS scratch
// (concentrations, g/RT, rates of progress: live only inside group_rhs) and per warp. The RHS
// scratch of the warp's cells and the Jacobian scratch of the cooperative setup share one region:
// every pass evaluates the right-hand sides first and runs the setups after them, never both at
// once, and 3.3 KB less per warp (drm19) leaves room for more cells or more L1 for the tables.
template <class M, class JR>
__host__ __device__ constexpr int gbdf_cell_bytes() {
  constexpr int N = M::N;
  constexpr int nd = (QMAX + 2) * N + N + (QMAX + 1) + (QMAX + 2);
  constexpr int nj = N * (N + 1) + N;
  return (nd * 8 + nj * (int)sizeof(JR) + N * 4 + 15) / 16 * 16;
}
template <class M>
__host__ __device__ constexpr int gbdf_rhs_bytes() {
  return (2 * M::NS + M::NR + (M::RHS_TABLE ? 0 : M::NR)) * 8;  // unrolled: and each reaction's [M]
}
template <class M, class JR>
__host__ __device__ constexpr int gbdf_setup_bytes() {
  constexpr int N = M::N, NS = M::NS;
  if (!M::RHS_TABLE) return 0;  // unrolled: the Jacobian goes straight into the cell's matrix
  return N * 8 + (N + wbdf::rx_len<M>() + 4 * NS) * (int)sizeof(JR);
}
template <class M, class JR, int G>
__host__ __device__ constexpr int gbdf_shared_scratch_bytes() {
  constexpr int a = (32 / G) * gbdf_rhs_bytes<M>(), b = gbdf_setup_bytes<M, JR>();
  return ((a > b ? a : b) + 15) / 16 * 16;
}
template <class M, class JR, int G>
__host__ __device__ constexpr int gbdf_smem_per_warp() {
  return (32 / G) * gbdf_cell_bytes<M, JR>() + gbdf_shared_scratch_bytes<M, JR, G>();
}

// The group-distributed part of a length-N vector (element i in sub-lane i % G, slot i / G).
template <class M, int G>
struct GVec {
  double v[(M::N + G - 1) / G];
};

template <int G>
__device__ __forceinline__ unsigned group_mask() {
  if constexpr (G == 32) {
    return 0xffffffffu;
  } else {
    const int lane = threadIdx.x & 31;
    return ((1u << G) - 1u) << (lane - lane % G);
  }
}
// Out of line: the kernel sums at fourteen places, and a shuffle with a run-time mask is several
// instructions (17 KB of code inlined).
template <int G>
__device__ __noinline__ double group_sum(double v, unsigned gm) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(gm, v, o);
  return v;
}
template <int G>
__device__ __forceinline__ double group_max(double v, unsigned gm) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(gm, v, o));
  return v;
}

// Sum over elements 0..NV-1, element i in lane i of the cell's lanes, in the order that a group of S
// lanes adds them: sub-lane s of S takes elements s, s + S, ... in turn, then the S partial sums meet
// by xor shuffles (S = 1: one sequential sum). Lets a wider group of lanes repeat a narrower
// mapping's bits. lane_dot accumulates a_i b_i with multiply-adds.
template <int NV, int S>
__device__ __noinline__ double lane_dot(double a, double b, unsigned gm, int gbase) {
  const int s0 = ((threadIdx.x & 31) - gbase) % S;
  double s = 0.0;
#pragma unroll 1
  for (int i = s0, r = 0; r < (NV + S - 1) / S; ++r, i += S) {
    const double x = __shfl_sync(gm, a, gbase + i), y = __shfl_sync(gm, b, gbase + i);
    if (i < NV) s = fma(x, y, s);
  }
#pragma unroll
  for (int o = S / 2; o > 0; o >>= 1) s += __shfl_xor_sync(gm, s, o);
  return s;
}

// Rate of progress of reaction j with the operations and their order of the unrolled right-hand
// side (mech/codegen.py): Gibbs sum over products, then reactants, then pressure; the reverse product
// multiplied into the rate coefficient factor by factor.
template <class Tab>
__device__ __forceinline__ double rate_of_progress_unrolled(int j, double T, double invT, double lnT, double lnP0RT,
                                                            double Ctot, const double* CS, const double* GS,
                                                            double& Mthird) {
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
      double Fcent = fma(fo.one_m_a, pgb_exp64(T * fo.m_invT3), __dmul_rn(fo.a, pgb_exp64(T * fo.m_invT1)));
      if (fo.ntroe > 3) Fcent = __dadd_rn(Fcent, pgb_exp64(invT * fo.m_T2));
      constexpr double kInvLn10 = 0.43429448190325176;  // 1 / ln 10 as the generator rounds it
      const double lFc = __dmul_rn(pgb_log64(Fcent), kInvLn10);
      const double cc = fma(-0.67, lFc, -0.4), nn = fma(-1.27, lFc, 0.75);
      const double lPr = fma(pgb_log64(fmax(Pr, 1e-300)), kInvLn10, cc);
      const double f1 = pgb_div64(lPr, fma(-0.14, lPr, nn));
      blend = __dmul_rn(blend, pgb_exp64(pgb_div64(__dmul_rn(2.302585092994046, lFc), fma(f1, f1, 1.0))));
    }
    kf = __dmul_rn(kf, blend);
  }
  double Pf = CS[rs(0)];
#pragma unroll
  for (int s = 1; s < Tab::MAXR; ++s)
    if (s < nr) Pf = __dmul_rn(Pf, CS[rs(s)]);
  double q;
  if (rev) {
    double dG = 0.0;
    bool first = true;
#pragma unroll
    for (int side = 0; side < 2; ++side) {
      const int n = side ? nr : np;
#pragma unroll
      for (int s = 0; s < (side ? Tab::MAXR : Tab::MAXP); ++s) {
        if (s >= n) continue;
        const int k = side ? rs(s) : ps(s);
        if (s > 0 && (side ? rs(s - 1) : ps(s - 1)) == k) continue;  // counted with its first slot
        int same = 1;  // the coefficient: slots of one species are neighbours
#pragma unroll
        for (int u = s + 1; u < (side ? Tab::MAXR : Tab::MAXP); ++u)
          if (u < n && (side ? rs(u) : ps(u)) == k) ++same;
        const double one = side ? -1.0 : 1.0, nu = same == 1 ? one : same == 2 ? 2.0 * one : 3.0 * one;
        dG = first ? __dmul_rn(nu, GS[k]) : fma(nu, GS[k], dG);
        first = false;
      }
    }
    if (dnu != 0) dG = fma(-(double)dnu, lnP0RT, dG);
    double kr = -__dmul_rn(kf, pgb_exp64(fmin(dG, 700.0)));  // finite: an absent product gives 0, not NaN
#pragma unroll
    for (int s = 0; s < Tab::MAXP; ++s)
      if (s < np) kr = __dmul_rn(kr, CS[ps(s)]);
    q = fma(kf, Pf, kr);
  } else {
    q = __dmul_rn(kf, Pf);
  }
  Mthird = kind == 1 ? Mc : 1.0;
  return q;
}

// Right-hand side f = [W_k wdot_k + F_k, dT/dt] at y for one cell, its group of G lanes
// cooperating (the equations of warp_rhs with G lanes in place of 32), every sum over species in the
// order of S lanes. Inlined: the kernel calls it from one place, so inlining adds no copy and
// removes the call's register save and restore (measured: no spills left, +5 %).
template <class M, int G, int S>
__device__ __forceinline__ GVec<M, G> group_rhs(const GVec<M, G> yv, double* CS, double* GS, double* QS,
                                             const double* FRC) {
  using Tab = typename M::TabG;
  constexpr int N = M::N, NS = M::NS, NR = M::NR;
  constexpr int R = (N + G - 1) / G;
  constexpr bool UNROLLED = !M::RHS_TABLE;  // the operations of the unrolled per-thread code
  static_assert(S == G || R == 1, "another summation order needs an element per lane");
  static_assert(!UNROLLED || S == 1, "the unrolled code sums in sequence");
  const int lane = threadIdx.x & 31, sub = lane % G, gbase = lane - sub;
  const unsigned gm = group_mask<G>();
  auto idx = [&](int r) { return sub + G * r; };
  const double (&y)[R] = yv.v;
  GVec<M, G> fv;
  double (&f)[R] = fv.v;
  const double T = __shfl_sync(gm, y[NS / G], gbase + NS % G);
  const double invT = pgb_div64(1.0, T);
  const double lnT = pgb_log64(T);
  const double lnT1 = 1.0 - lnT;
  const double lnP0RT = kLnP0OverR - lnT;
  double c_loc = 0.0, c_fac = 1.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int k = idx(r);
    if (k < NS) {
      double invW, Tmid;
      bool fused = false;
      const double* g;
      if constexpr (UNROLLED) {
        const TabUnrolled& s = Tab::un(k);
        invW = s.invW;
        Tmid = s.Tmid;
        fused = s.only_total != 0;
        g = below_positive(T, Tmid) ? s.glo : s.ghi;
      } else {
        const TabSpecies<double>& s = Tab::template sp<double>(k);
        invW = s.invW;
        Tmid = s.Tmid;
        g = below_positive(T, Tmid) ? s.glo : s.ghi;
      }
      const double c = y[r] * invW;
      CS[k] = c;
      c_loc = __dadd_rn(c_loc, c);
      if (fused) { c_loc = y[r]; c_fac = invW; }
      GS[k] = fma(g[0], lnT1, fma(T, fma(T, fma(T, fma(T, g[4], g[3]), g[2]), g[1]), fma(g[5], invT, g[6])));
    }
  }
  double Ctot;
  if constexpr (S == G) Ctot = group_sum<G>(c_loc, gm);
  else Ctot = lane_dot<NS, S>(c_loc, c_fac, gm, gbase);
  __syncwarp(gm);
#pragma unroll 1
  for (int j = sub; j < NR; j += G) {
    if constexpr (UNROLLED) QS[j] = rate_of_progress_unrolled<Tab>(j, T, invT, lnT, lnP0RT, Ctot, CS, GS, QS[NR + j]);
    else QS[j] = rate_of_progress<Tab>(j, T, invT, lnT, lnP0RT, Ctot, CS, GS);
  }
  __syncwarp(gm);
  if constexpr (!UNROLLED) {
    // production rates, the longest sums together (their FP64 time is the longest lane's of a round)
#pragma unroll 1
    for (int i = sub; i < NS; i += G) {
      const int k = R > 1 ? Tab::sprx_by_len(i) : i;
      double wdot = 0.0;
      const int e1 = Tab::sprx_end(k);
#pragma unroll 4
      for (int e = Tab::sprx_begin(k); e < e1; ++e) wdot = fma(Tab::sprx_nu(e), QS[Tab::sprx_j(e)], wdot);
      CS[k] = wdot;
    }
    __syncwarp(gm);
  }
  double hs = 0.0, rcp = 0.0, h_one = 0.0, cp_one = 0.0, c_one = 0.0;
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const int k = idx(r);
    f[r] = 0.0;
    if (k < NS) {
      double wdot = 0.0;
      if constexpr (UNROLLED) {
        const TabUnrolled& s = Tab::un(k);
        const int e1 = Tab::un_begin(k + 1);
#pragma unroll 2
        for (int e = Tab::un_begin(k); e < e1; ++e) {
          const int j = Tab::un_j(e);
          const double nu = Tab::un_nu(e), qj = QS[j], mj = QS[NR + j];
          wdot = Tab::un_m(e) ? fma(nu * qj, mj, wdot) : fma(nu, __dmul_rn(qj, mj), wdot);  // un_m: nu is 1 or -1
        }
        f[r] = fma(wdot, s.W, FRC[k]);
        const bool lo = below_positive(T, s.Tmid);
        const double* a = lo ? s.clo : s.chi;
        const double* hc = lo ? s.hlo : s.hhi;
        h_one = fma(T, fma(T, fma(T, fma(T, hc[4], hc[3]), hc[2]), hc[1]), fma(hc[5], invT, hc[0]));
        cp_one = fma(T, fma(T, fma(T, fma(T, a[4], a[3]), a[2]), a[1]), a[0]);
        c_one = y[r];
      } else {
        wdot = CS[k];
        const TabSpecies<double>& s = Tab::template sp<double>(k);
        const double wm = fma(wdot, s.W, FRC[k]);
        f[r] = wm;
        const bool lo = below_positive(T, s.Tmid);
        const double* a = lo ? s.lo : s.hi;
        const double* hc = lo ? s.hlo : s.hhi;
        const double hRT = fma(T, fma(T, fma(T, fma(T, hc[4], hc[3]), hc[2]), hc[1]), fma(hc[5], invT, hc[0]));
        const double cpR = fma(T, fma(T, fma(T, fma(T, a[4], a[3]), a[2]), a[1]), a[0]);
        if constexpr (S == G) {
          hs = fma(hRT * s.invW, wm, hs);
          rcp = fma(y[r] * s.invW, cpR, rcp);
        } else {
          h_one = hRT * s.invW;
          cp_one = cpR;
          c_one = y[r] * s.invW;
        }
      }
    }
  }
  if constexpr (S == G) {
    hs = group_sum<G>(hs, gm);
    rcp = group_sum<G>(rcp, gm);
  } else {
    hs = lane_dot<NS, S>(h_one, f[0], gm, gbase);
    rcp = lane_dot<NS, S>(c_one, cp_one, gm, gbase);
  }
  if constexpr (!UNROLLED) rcp *= kRerg;
  const double fT = pgb_div64(fma(-hs, kRerg * T, FRC[NS]), rcp);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (idx(r) == NS) f[r] = fT;
  __syncwarp(gm);  // CS/GS/QS are reused by the next evaluation
  return fv;
}

template <class M, class JR, int G, int WPB, int S = G>
__global__ void __launch_bounds__(WPB * 32, 1) bdf_group_kernel(const ReactParams P) {
  using namespace bdf;
  using Tab = typename M::TabG;
  static_assert(G == 4 || G == 8 || G == 16 || G == 32, "group size must divide the warp");
  constexpr int N = M::N, NS = M::NS;
  constexpr int R = (N + G - 1) / G;  // vector elements per lane
  constexpr int LDA = N + 1;          // padded matrix row
  constexpr int CPW = 32 / G;         // cells per warp
  constexpr bool MIXED = sizeof(JR) == sizeof(float);
  constexpr int RW = (N + 31) / 32;   // slots of the warp-wide setup vector
  // mechanisms whose per-thread kernel runs unrolled code: same bits here (its Jacobian evaluated by
  // one lane, its orders of summation)
  constexpr bool UNROLLED = !M::RHS_TABLE;
  static_assert(!UNROLLED || (S == 1 && R == 1), "an element per lane, summed in sequence");
  extern __shared__ __align__(16) unsigned char gsmem[];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
  const int sub = lane % G, grp = lane / G, gbase = lane - sub;
  const unsigned gm = group_mask<G>();
  unsigned char* wbase = gsmem + (size_t)wid * gbdf_smem_per_warp<M, JR, G>();
  auto cell_base = [&](int g) { return wbase + (size_t)g * gbdf_cell_bytes<M, JR>(); };
  unsigned char* const wscratch = cell_base(CPW);  // RHS scratch of the cells | setup scratch
  struct CellMem {
    double *Z, *FRC, *CS, *GS, *QS, *LC, *TAU;
    JR *A, *XS;
    int* PIV;
  };
  auto cell_mem = [&](int g) {
    CellMem c;
    c.Z = reinterpret_cast<double*>(cell_base(g));  // [(QMAX+2)][N]; column QMAX+1: saved acor
    c.FRC = c.Z + (QMAX + 2) * N;                   // [N] forcing (rhoY, then rho h)
    c.CS = reinterpret_cast<double*>(wscratch + (size_t)g * gbdf_rhs_bytes<M>());  // [NS] concentrations
    c.GS = c.CS + NS;                               // [NS] g/RT
    c.QS = c.GS + NS;                               // [NR] rates of progress
    c.LC = c.FRC + N;                               // [QMAX+1] l coefficients
    c.TAU = c.LC + (QMAX + 1);                      // [QMAX+2] step history
    c.A = reinterpret_cast<JR*>(c.TAU + (QMAX + 2));  // [N][LDA] matrix, then its LU
    c.XS = c.A + N * LDA;                           // [N] solve vector
    c.PIV = reinterpret_cast<int*>(c.XS + N);       // [N] pivots
    return c;
  };
  const CellMem C = cell_mem(grp);
  double* const YS = reinterpret_cast<double*>(wscratch);         // [N] setup input staging
  JR* const WXS = reinterpret_cast<JR*>(YS + N);                  // [N] setup concentrations
  JR* const WRX = WXS + N;                                        // Jacobian partials
  JR* const WTH = WRX + wbdf::rx_len<M>();                        // [4][NS] NASA-7 terms

  const long long ncell = P.ncell_dev ? (long long)*P.ncell_dev : P.ncell;
  const int qmax = max(1, min(P.max_order, QMAX));
  const double tout = P.dt;
  auto idx = [&](int r) { return sub + G * r; };
  auto Z = [&](int j, int r) -> double& { return C.Z[j * N + idx(r)]; };

  // ---- per-group state (scalars replicated in the group's lanes; vectors distributed) ----
  // a small launch spreads its cells over the SMs: the first P.cells_per_warp groups of a warp work
  int phase = P.cells_per_warp > 0 && grp >= P.cells_per_warp ? IDLE : NEED;
  long long cell = -1;
  int box = 0, ci = 0, cj = 0, ck = 0;
  double y[R], acor[R], ewt[R];
  double t = 0.0, h = 0.0, hscale = 0.0, etamax = ETAMX1, eta = 1.0;
  double gamma = 0.0, gammap = 0.0, gamrat = 1.0, crate2 = 1.0, rl1 = 1.0;
  double tq1 = 1.0, tq2 = 1.0, tq3 = 1.0, tq5 = 1.0, tq5_saved = 1.0, inv_tq4_sq = 1.0;
  double del2 = 0.0, delp2 = 0.0, hg = 0.0, hub = 0.0, hlb = 0.0, rE0 = 0.0;
  int q = 1, qwait = 2, nef = 0, ncf = 0, m = 0, hin_count = 0, status = OK;
  int nst = 0, nfe = 0, nje = 0, nstlp = 0, netf = 0, ncfn = 0;  // bounded by ode.max_steps
  bool new_step = true, need_setup = true, force_setup = true, jcur = false, setup_ok = true, fresh = false;
#pragma unroll
  for (int r = 0; r < R; ++r) { y[r] = 0.0; acor[r] = 0.0; ewt[r] = 1.0; }

  auto wms = [&](const double (&v)[R]) -> double {  // squared WRMS norm
    if constexpr (S != G) {
      const double x = v[0] * ewt[0];
      return lane_dot<N, S>(x, x, gm, gbase) * (1.0 / N);
    } else {
      double s = 0.0;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) { const double x = v[r] * ewt[r]; s = fma(x, x, s); }
      return group_sum<G>(s, gm) * (1.0 / N);
    }
  };
  auto set_ewt = [&]() {
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (idx(r) < N) {
        const double d = fma(P.rtol, fabs(Z(0, r)), P.atol[idx(r)]);
        ewt[r] = MIXED ? recip_fast(d) : 1.0 / d;
      }
  };
  auto rescale = [&](double e) {
    double fac = e;
#pragma unroll 1
    for (int j = 1; j <= q; ++j) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) Z(j, r) *= fac;
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
          if (idx(r) < N) Z(j - 1, r) += Z(j, r);
  };
  auto retract = [&]() {  // t goes back where the outcome is found
#pragma unroll 1
    for (int k = 1; k <= q; ++k)
#pragma unroll 1
      for (int j = q; j >= k; --j)
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (idx(r) < N) Z(j - 1, r) -= Z(j, r);
  };
  auto tau = [&](int j) -> double { return C.TAU[j]; };
  // l coefficients and error constants (the arithmetic of bdf_kernel.cuh's set_coeffs); l is
  // computed in registers by every lane of the group and stored once
  // With eight lanes or more the coefficients are spread over them (l_i in lane i) and independent
  // quotients are formed side by side; the operations and their order are those of the form below.
  auto set_coeffs_lanes = [&]() {
    const double alpha0 = alpha0_of(q);
    double hs = h;  // lane i: h + tau_1 + ... + tau_i
#pragma unroll 1
    for (int i = 1; i <= min(sub, QMAX); ++i) hs += tau(i);
    const double xi = pgb_div64(h, hs);
    double sum_xi_inv = 0.0, l = sub == 0 ? 1.0 : 0.0;
#pragma unroll 1
    for (int i = 1; i <= q - 1; ++i) {
      const double xi_inv = __shfl_sync(gm, xi, gbase + i - 1);
      sum_xi_inv += xi_inv;
      const double below = __shfl_sync(gm, l, gbase + max(sub - 1, 0));
      if (sub >= 1 && sub <= i) l = fma(below, xi_inv, l);
    }
    const double xistar_inv = -alpha0 - sum_xi_inv;
    {
      const double below = __shfl_sync(gm, l, gbase + max(sub - 1, 0));
      if (sub >= 1 && sub <= q) l = fma(below, xistar_inv, l);
    }
    const double xiq_inv = __shfl_sync(gm, xi, gbase + q - 1), xiq1_inv = __shfl_sync(gm, xi, gbase + q);
    const double alpha0_hat = -(sum_xi_inv + xiq_inv);
    const double A1 = 1.0 - alpha0_hat + alpha0;
    const double A2 = fma((double)q, A1, 1.0);
    const double lq = __shfl_sync(gm, l, gbase + q), l1 = __shfl_sync(gm, l, gbase + 1);
    const double A3 = alpha0 + inv_int(q), A4 = alpha0_hat + xiq_inv;
    const double A5 = alpha0 - inv_int(q + 1), A6 = alpha0_hat - xiq1_inv;
    double d[5];  // 1/tq2's and 1/tq5's quotients, Cq, Cpp, 1/l_1
    group_div<5>({A1, A2 * xistar_inv, xistar_inv, 1.0 - A6 + A5, 1.0}, {alpha0 * A2, lq * xiq_inv, lq, A2, l1}, d, gm,
                 gbase);
    tq2 = fabs(d[0]);
    tq5 = fabs(d[1]);
    rl1 = d[4];
    gamma = h * rl1;
    double e[3];
    group_div<3>({d[2] * (1.0 - A4 + A3), d[3], gamma}, {A3, xiq1_inv * (q + 2) * A5, gammap}, e, gm, gbase);
    if (qwait == 1) {
      tq1 = q > 1 ? fabs(e[0]) : 1.0;
      tq3 = fabs(e[1]);
    }
    gamrat = nst > 0 ? e[2] : 1.0;
    inv_tq4_sq = (tq2 * (1.0 / NLSCOEF)) * (tq2 * (1.0 / NLSCOEF));
    __syncwarp(gm);
    if (sub <= QMAX) C.LC[sub] = l;
    __syncwarp(gm);
  };
  auto set_coeffs = [&]() {
    double l[QMAX + 1];
#pragma unroll
    for (int i = 0; i <= QMAX; ++i) l[i] = 0.0;
    l[0] = 1.0;
    double alpha0 = 0.0;
#pragma unroll 1
    for (int j = 1; j <= q; ++j) alpha0 -= inv_int(j);
    double hsum = h, sum_xi_inv = 0.0;
#pragma unroll 1
    for (int i = 1; i <= q - 1; ++i) {
      if (i > 1) hsum += tau(i - 1);
      const double xi_inv = pgb_div64(h, hsum);
      sum_xi_inv += xi_inv;
#pragma unroll
      for (int k = QMAX; k >= 1; --k)
        if (k <= i) l[k] += l[k - 1] * xi_inv;
    }
    const double xistar_inv = -alpha0 - sum_xi_inv;
#pragma unroll
    for (int k = QMAX; k >= 1; --k)
      if (k <= q) l[k] += l[k - 1] * xistar_inv;
    if (q > 1) hsum += tau(q - 1);
    const double xiq_inv = pgb_div64(h, hsum);
    const double alpha0_hat = -(sum_xi_inv + xiq_inv);
    const double A1 = 1.0 - alpha0_hat + alpha0;
    const double A2 = fma((double)q, A1, 1.0);
    double lq = 0.0;
#pragma unroll
    for (int k = 0; k <= QMAX; ++k) if (k == q) lq = l[k];
    tq2 = fabs(pgb_div64(A1, alpha0 * A2));
    tq5 = fabs(pgb_div64(A2 * xistar_inv, lq * xiq_inv));
    if (qwait == 1) {
      if (q > 1) {
        const double Cq = pgb_div64(xistar_inv, lq);
        const double A3 = alpha0 + inv_int(q);
        const double A4 = alpha0_hat + xiq_inv;
        tq1 = fabs(pgb_div64(Cq * (1.0 - A4 + A3), A3));
      } else {
        tq1 = 1.0;
      }
      const double xiq1_inv = pgb_div64(h, hsum + tau(q));
      const double A5 = alpha0 - inv_int(q + 1);
      const double A6 = alpha0_hat - xiq1_inv;
      const double Cpp = pgb_div64(1.0 - A6 + A5, A2);
      tq3 = fabs(pgb_div64(Cpp, xiq1_inv * (q + 2) * A5));
    }
    inv_tq4_sq = (tq2 * (1.0 / NLSCOEF)) * (tq2 * (1.0 / NLSCOEF));
    rl1 = pgb_div64(1.0, l[1]);
    __syncwarp(gm);
    for (int e = sub; e <= QMAX; e += G) {
      double v = 0.0;
#pragma unroll
      for (int k = 0; k <= QMAX; ++k) if (k == e) v = l[k];
      C.LC[e] = v;
    }
    __syncwarp(gm);
  };
  auto adjust_order_lanes = [&](int dq) {
    double hs = 0.0;  // lane i: tau_1 + ... + tau_{i+1}
#pragma unroll 1
    for (int i = 0; i <= min(sub, QMAX - 1); ++i) hs += tau(i + 1);
    const double xis = pgb_div64(hs, hscale), rxis = pgb_div64(1.0, xis);
    double w = sub == 2 ? 1.0 : 0.0, alpha1 = 0.0, prod = 1.0;  // lane i: w_i
    const int top = dq > 0 ? q : q - 2;
#pragma unroll 1
    for (int j = 1; j <= top; ++j) {
      const double xi = __shfl_sync(gm, xis, gbase + j - 1);
      prod *= xi;
      alpha1 += __shfl_sync(gm, rxis, gbase + j - 1);
      const double below = __shfl_sync(gm, w, gbase + max(sub - 1, 0));
      if (sub >= 2 && sub <= j + 2 && (dq < 0 || j <= q - 1)) w = fma(w, xi, below);
    }
    if (dq > 0) {
      const double A1 = pgb_div64(-alpha0_of(q) - alpha1, prod);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) Z(q + 1, r) = A1 * Z(QMAX + 1, r);
    }
    const int from = dq > 0 ? q + 1 : q, last = dq > 0 ? q : q - 1;
#pragma unroll 1
    for (int j = 2; j <= last; ++j) {
      double wj = __shfl_sync(gm, w, gbase + j);
      if (dq < 0) wj = -wj;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) Z(j, r) = fma(wj, Z(from, r), Z(j, r));
    }
    if (dq < 0) {
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) Z(q, r) = 0.0;
    }
  };
  auto adjust_order = [&](int dq) {
    double w[QMAX + 2];
#pragma unroll
    for (int i = 0; i < QMAX + 2; ++i) w[i] = 0.0;
    w[2] = 1.0;
    if (dq > 0) {
      double alpha0 = 0.0, alpha1 = 0.0, prod = 1.0, hsum = 0.0;
#pragma unroll 1
      for (int j = 1; j <= q; ++j) {
        hsum += tau(j);
        const double xi = pgb_div64(hsum, hscale);
        prod *= xi;
        alpha0 -= inv_int(j);
        alpha1 += pgb_div64(1.0, xi);
        if (j <= q - 1)
#pragma unroll
          for (int i = QMAX + 1; i >= 2; --i)
            if (i <= j + 2) w[i] = w[i] * xi + w[i - 1];
      }
      const double A1 = pgb_div64(-alpha0 - alpha1, prod);
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) Z(q + 1, r) = A1 * Z(QMAX + 1, r);
#pragma unroll
      for (int j = 2; j <= QMAX; ++j)
        if (j <= q)
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (idx(r) < N) Z(j, r) = fma(w[j], Z(q + 1, r), Z(j, r));
    } else {
      double hsum = 0.0;
#pragma unroll 1
      for (int j = 1; j <= q - 2; ++j) {
        hsum += tau(j);
        const double xi = pgb_div64(hsum, hscale);
#pragma unroll
        for (int i = QMAX + 1; i >= 2; --i)
          if (i <= j + 2) w[i] = w[i] * xi + w[i - 1];
      }
#pragma unroll
      for (int j = 2; j <= QMAX; ++j)
        if (j < q)
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (idx(r) < N) Z(j, r) = fma(-w[j], Z(q, r), Z(j, r));
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) Z(q, r) = 0.0;
    }
  };
  // (I - gamma J) x = b with the cell's factors: rows over the group's lanes, the operations and
  // their order of the warp mapping's solve
  auto solve = [&](double (&b)[R]) {
    JR x[R];
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (idx(r) < N) C.XS[idx(r)] = (JR)b[r];
    __syncwarp(gm);
#pragma unroll
    for (int r = 0; r < R; ++r) x[r] = idx(r) < N ? C.XS[C.PIV[idx(r)]] : JR(0);
    if constexpr (UNROLLED) {
      // the per-thread kernel's order: rows from the last up, each a sum over ascending columns
      lu_substitute<N, G, JR, false>(C.A, gm, gbase, x);
      if (idx(0) < N) C.XS[idx(0)] = x[0];
      __syncwarp(gm);
      JR xs[N];
#pragma unroll
      for (int k = N - 1; k >= 0; --k) {
        JR v = C.XS[k];
#pragma unroll
        for (int j = k + 1; j < N; ++j) v = fma(-C.A[k * LDA + j], xs[j], v);
        xs[k] = v * C.A[k * LDA + k];
        if (k == idx(0)) x[0] = xs[k];
      }
    } else {
      lu_substitute<N, G>(C.A, gm, gbase, x);
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (idx(r) < N) b[r] = (double)x[r];
    __syncwarp(gm);
  };
  // ---- cell I/O ----
  auto elem = [&](const ArrDev& a, int n) -> double& {
    return a.p[(long long)(ci - a.begin0) + (long long)(cj - a.begin1) * a.jstride +
               (long long)(ck - a.begin2) * a.kstride + (long long)n * a.nstride];
  };
  auto add_stats = [&](bool retried) {
    if (sub != 0) return;
    ReactStats* T = P.stats;
    atomicAdd(&T->nst, (unsigned long long)nst);
    atomicAdd(&T->nfe, (unsigned long long)nfe);
    atomicAdd(&T->nje, (unsigned long long)nje);
    atomicAdd(&T->netf, (unsigned long long)netf);
    atomicAdd(&T->ncfn, (unsigned long long)ncfn);
    if (retried) {
      atomicAdd(&T->nretry, 1ull);
      return;
    }
    if (status != OK) atomicAdd(&T->nfail, 1ull);
    atomicMax(&T->max_nst, (unsigned long long)nst);
    const int bin = min(15, 31 - __clz(max(nst, 1)));
    atomicAdd(&T->hist[bin], 1ull);
  };
  auto finish_cell = [&]() {
    const BoxDev& B = P.boxes[box];
    if (status != OK && P.retry_list) {  // hand the cell to the retry pass, arrays untouched
      if (sub == 0) P.retry_list[atomicAdd(P.retry_count, 1ull)] = cell;
      add_stats(true);
      phase = NEED;
      return;
    }
    // rho h(t) = rho h0 + F_h t ; T from (h, Y) by Newton with the integrated T as guess
    const double rE = fma(tout, C.FRC[NS], rE0);
    double Tn = C.Z[NS];
    if (!(Tn > 90.0 && Tn < 5000.0)) Tn = 1000.0;
    if constexpr (UNROLLED) {  // as the per-thread kernel does
      double rho = 0.0, hm = 0.0;
#pragma unroll 1
      for (int k = 0; k < NS; ++k) {
        rho += C.Z[k];
        hm = fma(C.Z[k], M::Tab::h_mid(k), hm);
      }
      Tn = hy2t_mixture<typename M::Tab>(__dmul_rn(rE, 1.0 / kRerg), [&](int k) { return C.Z[k]; }, rho, hm, Tn, 90.0,
                                         5000.0);
    } else {
      // sums over species in the order of S lanes
      auto sum_of = [&](const double (&u)[R], const double (&v)[R]) -> double {
        if constexpr (S == G) {
          double x = 0.0;
#pragma unroll
          for (int r = 0; r < R; ++r)
            if (idx(r) < NS) x = fma(u[r], v[r], x);
          return group_sum<G>(x, gm);
        } else {
          return lane_dot<NS, S>(u[0], v[0], gm, gbase);
        }
      };
      double y0[R], one[R];
#pragma unroll
      for (int r = 0; r < R; ++r) {
        y0[r] = idx(r) < NS ? Z(0, r) : 0.0;
        one[r] = 1.0;
      }
      const double inv_rho = pgb_div64(1.0, sum_of(y0, one));
      const double htarget = __dmul_rn(rE, inv_rho);
#pragma unroll 1
      for (int it = 0; it < 50; ++it) {
        const double invTn = pgb_div64(1.0, Tn);
        double yw[R], hk[R], ck[R];
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int k = idx(r);
          yw[r] = hk[r] = ck[r] = 0.0;
          if (k < NS) {
            const TabSpecies<double>& s = Tab::template sp<double>(k);
            const bool lo = below_positive(Tn, s.Tmid);
            const double* a = lo ? s.lo : s.hi;
            const double* hc = lo ? s.hlo : s.hhi;
            const double hRT = fma(Tn, fma(Tn, fma(Tn, fma(Tn, hc[4], hc[3]), hc[2]), hc[1]), fma(hc[5], invTn, hc[0]));
            const double cpR = fma(Tn, fma(Tn, fma(Tn, fma(Tn, a[4], a[3]), a[2]), a[1]), a[0]);
            yw[r] = y0[r] * inv_rho * s.invW;
            hk[r] = hRT * kRerg * Tn;
            ck[r] = cpR * kRerg;
          }
        }
        const double hh = sum_of(yw, hk), cp = sum_of(yw, ck);
        double dT = pgb_div64(htarget - hh, cp);
        dT = fmax(-100.0, fmin(100.0, dT));
        Tn = fmax(90.0, fmin(5000.0, Tn + dT));
        if (fabs(dT) < 1e-10 * Tn) break;
      }
    }
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (idx(r) < NS) {
        const double rYn = __dmul_rn(Z(0, r), B.sY_out);
        if (B.IR.p)  // separate roundings, as separate passes over arrays give
          elem(B.IR, idx(r)) = __dsub_rn(__dmul_rn(-__dsub_rn(elem(B.rY, idx(r)), rYn), 1.0 / tout),
                                         elem(B.rYsrc, idx(r)));
        elem(B.rY, idx(r)) = rYn;
      }
    if (sub == 0) {
      elem(B.T, 0) = Tn;
      elem(B.rE, 0) = rE * B.sE_out;
      elem(B.FC, 0) = (status == OK) ? (double)nfe : -(double)status;
    }
    add_stats(false);
    phase = NEED;
  };
  auto fail_cell = [&](int st) {
    status = st;
    phase = FINISH;
  };
  // loads flat cell c into the group; false for a covered cell (FC = 0, I_R = -F written)
  auto load_cell = [&](long long c) -> bool {
    int lo = 0, hi = P.nbox - 1;
    while (lo < hi) {
      const int mid = (lo + hi + 1) >> 1;
      if (P.boxes[mid].cell_offset <= c) lo = mid; else hi = mid - 1;
    }
    box = lo;
    const BoxDev& B = P.boxes[box];
    long long rr = c - B.cell_offset;
    ci = B.lo0 + (int)(rr % B.len0);
    rr /= B.len0;
    cj = B.lo1 + (int)(rr % B.len1);
    ck = B.lo2 + (int)(rr / B.len1);
    if (B.mask.p && B.mask.p[(long long)(ci - B.mask.begin0) + (long long)(cj - B.mask.begin1) * B.mask.jstride +
                             (long long)(ck - B.mask.begin2) * B.mask.kstride] < 0) {
      if (sub == 0) elem(B.FC, 0) = 0.0;
      if (B.IR.p)
        for (int k = sub; k < NS; k += G) elem(B.IR, k) = -elem(B.rYsrc, k);
      return false;
    }
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int i = idx(r);
      if (i < NS) { Z(0, r) = elem(B.rY, i) * B.sY_in; C.FRC[i] = elem(B.rYsrc, i) * B.sY_in; }
      else if (i == NS) { Z(0, r) = elem(B.T, 0); C.FRC[NS] = elem(B.rEsrc, 0) * B.sE_in; }
    }
    for (int e = sub; e < (QMAX + 1) * N; e += G) C.Z[N + e] = 0.0;  // columns 1..QMAX+1
    for (int e = sub; e < QMAX + 2; e += G) C.TAU[e] = 0.0;
    rE0 = elem(B.rE, 0) * B.sE_in;
    t = 0.0; h = 0.0; hscale = 0.0; etamax = ETAMX1; eta = 1.0;
    gamma = 0.0; gammap = 0.0; gamrat = 1.0; crate2 = 1.0; rl1 = 1.0;
    tq1 = tq2 = tq3 = tq5 = tq5_saved = inv_tq4_sq = 1.0;
    q = 1; qwait = 2; nef = 0; ncf = 0; m = 0; status = OK;
    nst = 0; nfe = 0; nje = 0; nstlp = 0; netf = 0; ncfn = 0;
    new_step = true; need_setup = true; force_setup = true; jcur = false; fresh = false;
    __syncwarp(gm);
    return true;
  };

  // hands the group's cell over at the start of a step; the group rests
  auto hand_over = [&]() {
    unsigned long long at = 0;
    if (sub == 0) at = atomicAdd(P.resume_count, 1ull);
    const ResumeRec<N, JR> rec(P.resume, __shfl_sync(gm, at, gbase));
    if (sub == 0) {
      ResumeHead H;
      H.t = t; H.h = h; H.hscale = hscale; H.etamax = etamax; H.gammap = gammap; H.crate2 = crate2;
      H.tq5_saved = tq5_saved;
      H.cell = cell;
      H.box = box; H.ci = ci; H.cj = cj; H.ck = ck;
      H.q = q; H.qwait = qwait; H.nst = nst; H.nfe = nfe; H.nje = nje; H.nstlp = nstlp; H.netf = netf; H.ncfn = ncfn;
      H.force_setup = force_setup;
      H.full_swaps = 1;
      *rec.head = H;
    }
#pragma unroll 1
    for (int e = sub; e < (QMAX + 2) * N; e += G) rec.Z[e] = C.Z[e];
#pragma unroll 1
    for (int e = sub; e < QMAX + 2; e += G) rec.tau[e] = C.TAU[e];
#pragma unroll 1
    for (int e = sub; e < N * N; e += G) rec.lu[e] = C.A[e + e / N];  // rows of N + 1
#pragma unroll 1
    for (int e = sub; e < N; e += G) rec.piv[e] = C.PIV[e];
    phase = IDLE;
  };
  // takes over record i
  auto take_over = [&](unsigned long long i) {
    const ResumeRec<N, JR> rec(P.resume, i);
    const ResumeHead& H = *rec.head;
    cell = H.cell;
    box = H.box; ci = H.ci; cj = H.cj; ck = H.ck;
    const BoxDev& B = P.boxes[box];
#pragma unroll 1
    for (int e = sub; e < (QMAX + 2) * N; e += G) C.Z[e] = rec.Z[e];
#pragma unroll 1
    for (int e = sub; e < QMAX + 2; e += G) C.TAU[e] = rec.tau[e];
#pragma unroll 1
    for (int e = sub; e < N * N; e += G) C.A[e + e / N] = rec.lu[e];
#pragma unroll 1
    for (int e = sub; e < N; e += G) {
      C.PIV[e] = H.full_swaps ? rec.piv[e] : e;
      C.FRC[e] = e < NS ? elem(B.rYsrc, e) * B.sY_in : elem(B.rEsrc, 0) * B.sE_in;
    }
    rE0 = elem(B.rE, 0) * B.sE_in;
    t = H.t; h = H.h; hscale = H.hscale; etamax = H.etamax; eta = 1.0;
    gamma = 0.0; gammap = H.gammap; gamrat = 1.0; crate2 = H.crate2; rl1 = 1.0;
    tq1 = tq2 = tq3 = tq5 = inv_tq4_sq = 1.0;
    tq5_saved = H.tq5_saved;
    q = H.q; qwait = H.qwait; nef = 0; ncf = 0; m = 0; status = OK;
    nst = H.nst; nfe = H.nfe; nje = H.nje; nstlp = H.nstlp; netf = H.netf; ncfn = H.ncfn;
    new_step = true; need_setup = false; force_setup = H.force_setup != 0; jcur = false; fresh = false;
    __syncwarp(gm);
    if (!H.full_swaps) {
      // the per-thread kernel exchanges rows right of the pivot: exchange the multipliers too
      if (sub == 0) {
#pragma unroll 1
        for (int k = 0; k < N; ++k) {
          const int p = rec.piv[k];
          if (p <= k || p >= N) continue;
          const int i0 = C.PIV[k];
          C.PIV[k] = C.PIV[p];
          C.PIV[p] = i0;
#pragma unroll 1
          for (int j = 0; j < k; ++j) {
            const JR a = C.A[k * LDA + j];
            C.A[k * LDA + j] = C.A[p * LDA + j];
            C.A[p * LDA + j] = a;
          }
        }
      }
      __syncwarp(gm);
    }
    phase = STEP;
  };
  bool queue_empty = false;

  for (;;) {
    // ------------------------------------------------ (A) work stealing, one atomic per warp
    {
      const unsigned need = __ballot_sync(0xffffffffu, phase == NEED && sub == 0);
      if (need) {
        const int leader = __ffs(need) - 1;
        unsigned long long base = 0;
        if (lane == leader) base = atomicAdd(P.next_cell, (unsigned long long)__popc(need));
        base = __shfl_sync(0xffffffffu, base, leader);
        const long long c = (long long)base + __popc(need & ((1u << gbase) - 1u));
        bool past_end = false;
        if (phase == NEED) {
          if (c >= ncell) {
            phase = IDLE;
            past_end = true;
          } else if (S != G && P.resuming) {
            take_over((unsigned long long)c);
          } else {
            cell = P.cell_list ? P.cell_list[c] : c;
            if (load_cell(cell)) phase = START;  // covered cells stay NEED and refetch next pass
          }
        }
        queue_empty = __any_sync(0xffffffffu, past_end) || queue_empty;
      }
      if (S == G && queue_empty && P.drain > 0) {
        const unsigned left = __ballot_sync(0xffffffffu, phase != IDLE && sub == 0);
        if (__popc(left) <= P.drain && phase == STEP && new_step && nst > 0 && nst < P.max_steps) hand_over();
        __syncwarp();
      }
      if (__all_sync(0xffffffffu, phase == IDLE)) break;
    }

    // ------------------------------------------------ (B) prepare the RHS argument
    if (phase == STEP && new_step && nst >= P.max_steps) fail_cell(MAX_STEPS);
    if ((phase == STEP && new_step) || (phase == HIN && hin_count == 1)) set_ewt();
    if (phase == STEP) {
      if (new_step) {
        nef = 0; ncf = 0;
        new_step = false;
      }
      predict();
      if constexpr (G >= 8) {
        set_coeffs_lanes();
      } else {
        set_coeffs();
        gamma = h * rl1;
        gamrat = (nst > 0) ? pgb_div64(gamma, gammap) : 1.0;
      }
      if (nst == 0) gammap = gamma;
      need_setup = force_setup || nst == 0 || nst >= nstlp + MSBP || fabs(gamrat - 1.0) > DGMAX;
      force_setup = false;
      jcur = false;
      m = 0;
      phase = NEWTON;
      fresh = true;
    }
    if (fresh || phase == START || phase == RESETD) {  // from the prediction
#pragma unroll
      for (int r = 0; r < R; ++r) { y[r] = idx(r) < N ? Z(0, r) : 0.0; acor[r] = 0.0; }
      fresh = false;
    } else if (phase == HIN) {
#pragma unroll
      for (int r = 0; r < R; ++r) y[r] = idx(r) < N ? fma(hg, Z(1, r), Z(0, r)) : 0.0;
    }

    // ------------------------------------------------ (C) one FP64 RHS per active cell
    double f[R];
    const bool active = phase >= START;
    if (active) {
      GVec<M, G> yv;
#pragma unroll
      for (int r = 0; r < R; ++r) yv.v[r] = y[r];
      const GVec<M, G> fv = group_rhs<M, G, S>(yv, C.CS, C.GS, C.QS, C.FRC);
#pragma unroll
      for (int r = 0; r < R; ++r) f[r] = fv.v[r];
      ++nfe;
    } else {
#pragma unroll
      for (int r = 0; r < R; ++r) f[r] = 0.0;
    }

    // ------------------------------------------------ (E) Jacobian setups, one cell at a time
    // by the whole warp (cells that start a Newton iteration with a stale or missing matrix)
    __syncwarp();
    {
      const bool wanted = phase == NEWTON && m == 0 && need_setup;
      unsigned todo = __ballot_sync(0xffffffffu, sub == 0 && wanted);
      if constexpr (UNROLLED) {
        if (wanted && idx(0) < N) C.CS[idx(0)] = y[0];  // the RHS scratch is free
        __syncwarp();
        if (wanted && sub == 0) M::template jac<JR>(C.CS, C.FRC, C.FRC[NS], C.A, LDA, 1);
        __syncwarp();
      }
      while (todo) {
        const int g = (__ffs(todo) - 1) / G;
        todo &= todo - 1;
        const double gam = __shfl_sync(0xffffffffu, gamma, g * G);
        const CellMem Cg = cell_mem(g);
        bool ok;
        if constexpr (UNROLLED) {
          ok = warp_lu_factor<N>(Cg.A, Cg.PIV, (JR)gam);
        } else {
          if (grp == g) {
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (idx(r) < N) YS[idx(r)] = y[r];
          }
          __syncwarp();
          WVec<M> yv;
#pragma unroll
          for (int s = 0; s < RW; ++s) {
            const int i = lane + 32 * s;
            yv.v[s] = i < N ? YS[i] : 0.0;
          }
          ok = warp_setup<M, JR>(yv, gam, Cg.FRC, Cg.A, WXS, WRX, WTH, Cg.PIV);
        }
        __syncwarp();
        if (grp == g) {
          setup_ok = ok;
          ++nje;
          gammap = gamma;
          gamrat = 1.0;
          crate2 = 1.0;
          nstlp = nst;
        }
      }
    }

    // ------------------------------------------------ (D) consume it
    // The step's vector work that more than one outcome needs (undoing the prediction, changing
    // the order, rescaling the history) is only noted here and done once, below, for every
    // cell that needs it: one copy of its code, and one pass of its FP64 instructions instead of
    // one per outcome (this kernel is bound by instruction fetch as much as by the FP64 pipe).
    bool undo = false, check_h = false, first_step = false;
    int dq = 0;
    double scale = 1.0;
    if (phase == START || phase == RESETD) {
      const double fac = phase == START ? 1.0 : h;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) Z(1, r) = fac * f[r];  // START: f0 parked until h is known
    }
    if (phase == START) {
      // initial step size: difference-quotient estimate of y'' (bounded)
      const double tround = UROUND * tout;
      hlb = 100.0 * tround;
      double hub_inv = 0.0;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) hub_inv = fmax(hub_inv, pgb_div64(fabs(f[r]), fma(0.1, fabs(Z(0, r)), P.atol[idx(r)])));
      hub_inv = group_max<G>(hub_inv, gm);
      hub = 0.1 * tout;
      if (hub * hub_inv > 1.0) hub = pgb_div64(1.0, hub_inv);
      hg = sqrt(hlb * hub);
      if (hub > hlb) {
        hin_count = 1;
        phase = HIN;
      } else {
        h = fmin(fmax(0.5 * hg, hlb), hub);
        first_step = true;
      }
    } else if (phase == HIN) {
      double d[R];
#pragma unroll
      for (int r = 0; r < R; ++r) d[r] = idx(r) < N ? pgb_div64(f[r] - Z(1, r), hg) : 0.0;
      const double ydd = sqrt(wms(d));
      double hnew = sqrt((ydd * hub * hub > 2.0) ? pgb_div64(2.0, ydd) : hg * hub);
      bool done = false;
      if (hin_count == 4) {
        done = true;
      } else {
        const double hrat = pgb_div64(hnew, hg);
        if (hrat > 0.5 && hrat < 2.0) done = true;
        else if (hin_count >= 2 && hrat > 2.0) { hnew = hg; done = true; }
        else { hg = hnew; ++hin_count; }
      }
      if (done) {
        h = fmin(fmax(0.5 * hnew, hlb), hub);
        first_step = true;
      }
    } else if (phase == RESETD) {
      phase = STEP;
    } else if (phase == NEWTON) {
      bool singular = false;
      if (m == 0 && need_setup) {
        singular = !setup_ok;
        need_setup = false;
        jcur = true;
      }
      int outcome = 0;  // 0 continue, 1 converged, 2 convergence failure
      if (singular) {
        outcome = 3;
      } else {
        double b[R];
#pragma unroll
        for (int r = 0; r < R; ++r) b[r] = idx(r) < N ? fma(gamma, f[r], -fma(rl1, Z(1, r), acor[r])) : 0.0;
        solve(b);
        if (gamrat != 1.0) {
          const double s = pgb_div64(2.0, 1.0 + gamrat);
#pragma unroll
          for (int r = 0; r < R; ++r) b[r] = __dmul_rn(b[r], s);
        }
        del2 = wms(b);
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (idx(r) < N) { acor[r] += b[r]; y[r] = Z(0, r) + acor[r]; }
        if (m > 0) crate2 = fmax((CRDOWN * CRDOWN) * crate2, pgb_div64(del2, delp2));
        // convergence: del * min(1, crate) / tq4 <= 1, in squares
        const double dcon2 = del2 * fmin(1.0, crate2) * inv_tq4_sq;
        if (dcon2 <= 1.0) {
          outcome = 1;
        } else {
          ++m;
          if (m == MAXCOR || (m >= 2 && del2 > (RDIV * RDIV) * delp2)) outcome = 2;
          else delp2 = del2;
        }
      }
      if (outcome == 2 && !jcur) {
        // stale Jacobian: refresh it and restart the iteration from the prediction
        need_setup = true;
        m = 0;
        fresh = true;
      } else if (outcome >= 2) {
        undo = true;
        t -= h;
        ++ncf; ++ncfn;
        if (outcome == 3 || ncf >= MXNCF || fabs(h) <= 100.0 * UROUND * fabs(t)) {
          fail_cell(CONV);
        } else {
          force_setup = true;
          etamax = 1.0;
          scale = ETACF;
          phase = STEP;
        }
      } else if (outcome == 1) {
        const double acnrm2 = (m == 0) ? del2 : wms(acor);
        const double dsm2 = acnrm2 * (tq2 * tq2);  // squared local error estimate
        const bool accepted = dsm2 <= 1.0;
        bool save = false, ended = false, orders = false;  // orders: q - 1 and q + 1 are weighed too
        double ddn2 = 0.0, dup2 = 0.0;
        if (accepted) {
          // ---- step accepted: complete it ----
          ++nst;
          __syncwarp(gm);
          if (sub == 0) {
#pragma unroll 1
            for (int i = q + 1; i >= 2; --i) C.TAU[i] = C.TAU[i - 1];
            C.TAU[1] = h;
          }
#pragma unroll 1
          for (int j = 0; j <= q; ++j) {
            const double lj = C.LC[j];
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (idx(r) < N) Z(j, r) = fma(lj, acor[r], Z(j, r));
          }
          __syncwarp(gm);
          --qwait;
          if (qwait == 1 && q != qmax) {
            save = true;
            tq5_saved = tq5;
          }
          ended = fabs(t - tout) <= 100.0 * UROUND * (fabs(t) + fabs(h)) || t >= tout;
          orders = !ended && etamax != 1.0 && qwait == 0;
          if (orders) {
            if (q > 1) {
              double zq[R];
#pragma unroll
              for (int r = 0; r < R; ++r) zq[r] = idx(r) < N ? Z(q, r) : 0.0;
              ddn2 = wms(zq) * (tq1 * tq1);
            }
            if (q != qmax) {
              double hr, tq;
              if constexpr (G >= 8) {
                double d[2];
                group_div<2>({h, tq5}, {tau(2), tq5_saved}, d, gm, gbase);
                hr = d[0];
                tq = d[1];
              } else {
                hr = pgb_div64(h, tau(2));
                tq = pgb_div64(tq5, tq5_saved);
              }
              double hrp = hr;
#pragma unroll 1
              for (int k = 0; k < q; ++k) hrp *= hr;  // (h / tau2)^(q+1)
              const double cquot = tq * hrp;
              double tv[R];
              // the order test's difference: a group of 8 rounds the product of elements 8..15 and
              // fuses the others (as the compiler chose when this was one expression; kept, so
              // that every width of group takes the same steps)
#pragma unroll
              for (int r = 0; r < R; ++r) {
                const double saved = idx(r) < N ? Z(QMAX + 1, r) : 0.0;
                if (S == 1) tv[r] = fma(-cquot, saved, acor[r]);
                else if (idx(r) / S == 1) tv[r] = __dsub_rn(acor[r], __dmul_rn(cquot, saved));
                else tv[r] = fma(-cquot, saved, acor[r]);
              }
              dup2 = wms(tv) * (tq3 * tq3);
            }
          }
        }
        // step-size factors of orders q, q - 1 and q + 1
        double etaq, etaqm1, etaqp1;
        if constexpr (G >= 8) {  // one power and one quotient: lane 1 takes q - 1, lane 2 q + 1
          const double x = sub == 1 ? (BIAS1 * BIAS1) * ddn2 : sub == 2 ? (BIAS3 * BIAS3) * dup2 : (BIAS2 * BIAS2) * dsm2;
          const double a = 0.5 * inv_int(sub == 1 ? q : sub == 2 ? q + 2 : q + 1);
          const double e = pgb_div64(1.0, pgb_pow64(x, a) + ADDON);
          etaq = __shfl_sync(gm, e, gbase);
          etaqm1 = __shfl_sync(gm, e, gbase + 1);
          etaqp1 = __shfl_sync(gm, e, gbase + 2);
        } else {
          etaq = pgb_div64(1.0, pgb_pow64((BIAS2 * BIAS2) * dsm2, 0.5 * inv_int(q + 1)) + ADDON);
          etaqm1 = pgb_div64(1.0, pgb_pow64((BIAS1 * BIAS1) * ddn2, 0.5 * inv_int(q)) + ADDON);
          etaqp1 = pgb_div64(1.0, pgb_pow64((BIAS3 * BIAS3) * dup2, 0.5 * inv_int(q + 2)) + ADDON);
        }
        if (!orders || q == 1) etaqm1 = 0.0;
        if (!orders || q == qmax) etaqp1 = 0.0;
        if (!accepted) {
          // ---- local error test failed ----
          undo = true;
          t -= h;
          ++nef; ++netf;
          if (nef >= MXNEF || !isfinite(dsm2)) {
            fail_cell(isfinite(dsm2) ? ERRTEST : NONFINITE);
          } else {
            check_h = true;
            etamax = 1.0;
            phase = STEP;
            scale = ETAMIN;
            if (nef <= MXNEF1) {
              scale = fmax(ETAMIN, etaq);
              if (nef >= SMALL_NEF) scale = fmin(scale, ETAMXF);
            } else if (q > 1) {
              dq = -1;
            } else {
              qwait = 10;
              phase = RESETD;
            }
          }
        } else {
          if (ended) {
            phase = FINISH;
          } else {
            // ---- next step size and order ----
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
                  save = true;
                }
              } else if (eta < THRESH) {
                eta = 1.0;
              }
              if (eta >= THRESH || qprime != q) eta = fmin(eta, etamax);
              else eta = 1.0;
            }
            etamax = (nst <= SMALL_NST) ? ETAMX2 : ETAMX3;
            dq = qprime - q;
            scale = eta;
            new_step = true;
            phase = STEP;
          }
          if (save) {
#pragma unroll
            for (int r = 0; r < R; ++r)
              if (idx(r) < N) Z(QMAX + 1, r) = acor[r];
          }
        }
      }
    }
    if (undo) retract();
    if (dq != 0) {
      if constexpr (G >= 8) adjust_order_lanes(dq);
      else adjust_order(dq);
      q += dq;
      qwait = q + 1;
    }
    if (first_step) {
      hscale = h;
#pragma unroll
      for (int r = 0; r < R; ++r)
        if (idx(r) < N) Z(1, r) *= h;
      q = 1; qwait = 2; etamax = ETAMX1; new_step = true;
      __syncwarp(gm);
      if (sub == 0) C.TAU[1] = h;
      phase = STEP;
    }
    // the new step size, then a cut to end at tout
#pragma unroll 1
    for (int pass = 0; pass < 2; ++pass) {
      if (pass == 1) {
        scale = 1.0;
        if (phase == STEP && new_step && (t + h - tout) * h > 0.0)
          scale = pgb_div64((tout - t) * (1.0 - 4.0 * UROUND), h);
      }
      if (scale != 1.0) rescale(scale);
    }
    if (check_h && fabs(h) <= 100.0 * UROUND * fabs(t)) fail_cell(HSMALL);
    // ------------------------------------------------ (F) write back a finished cell
    if (phase == FINISH) finish_cell();
    __syncwarp();
  }
}

}  // namespace pgb

#endif  // PGB_BDF_GROUP_KERNEL_CUH
