#pragma once
// Latency kernel: one mode per SM on eight warps, for launches of a few modes per SM (spectra,
// single modes), whose run time is that of their slowest mode.
//
// The generic kernel (sbz_pt_impl.cuh) with four warps per mode spends a step of the massive-ν
// model at the default tolerances in 115k cycles, 35 % of them with the FP64 pipe of its busiest
// sub-partition occupied; the rest is dependent latency (shared memory, shuffles, barriers, the
// controller, the coefficient tables).  Here four solver warps (one per sub-partition) own the
// state and everything on the stage-to-stage critical path, and four companion warps (the second
// warp of each sub-partition) run beside them:
//   * error norm, PI controller and step publication, while the solver warps already form f(t1, y1);
//   * the coefficients of the step's five later stage times, while the solver warps factorise and
//     solve stage 1;
//   * the inverse of the 8x8 head, while the solver warps tabulate their scan multipliers;
//   * the stage sums y + Σ A_ij U_j and Σ C_ij U_j except for their last term, while the solver
//     warps are in the FP32 solve (the FP64 pipe idle), so a stage adds one term instead of up to six.
// On the critical path itself:
//   * row descriptors, scan multipliers, the head inverse and the rank-2 columns live in registers
//     for the kernel or the step (the generic kernel reads 22 multipliers per lane from shared memory
//     in each of the 9 to 17 solves of a step);
//   * the metric functionals of an operator product are formed once, by the solver warp with the least
//     FP64 work, and reach the others through shared memory (each FP64 warp instruction holds a
//     sub-partition for 64 cycles: 8 of warp 0's 23 instructions per product leave it);
//   * scans and sums stop at the level that the longest chain or sum of the model needs.
// Every sum keeps the order and the fusion of the generic kernel, so both give the same bits in mixed
// precision (the stage sums use explicit fma: a product left unfused by the compiler in one
// of the two kernels changes an FP32 rounding somewhere and then every later step).  In all-FP64
// solves the pivots' reciprocals differ from the generic kernel's by a unit in the last place.
// 20 modes, generic kernel -> here, ms: n = 47 83.6 -> 48.6, n = 82 80.8 -> 48.5, n = 133 85.7 -> 56.0, n = 133 at rtol
// 1e-6 / atol 3e-8 (10 modes) 484 -> 309; all-FP64 n = 38 158 -> 108, n = 133 (10 modes) 108 -> 84.  Bound: the
// dependent FP64 instructions and shuffles of a stage, about 4.2k cycles of them.
#include "sbz_pt_impl.cuh"

namespace sbz {
namespace ptk {

constexpr int kSolvers = 128, kLatThreads = 256;
// named barriers of the block (0 is __syncthreads)
enum : int {
  LB_MAIN = 1,  // solver warps
  LB_COMP,      // companion warps
  LB_STEP,      // the step's last stage and y1 are in shared memory (both sides)
  LB_CTL,       // step size and decision published (control warp arrives, solvers wait)
  LB_COEF,      // coefficients of the later stage times ready (coefficient warps arrive, solvers wait)
  LB_RHS,       // a stage's right-hand side is in shared memory; companions may add the previous stage (both)
  LB_SUM,       // next stage's sums ready (companions arrive, solvers wait)
  LB_DD,        // factorisation diagonals ready (solvers arrive, control warp waits)
  LB_LU,        // chain pivots ready (control warp arrives, solvers wait)
  LB_HROW,      // head rows ready (solver warp 3 arrives, control warp waits)
  LB_HEAD,      // head inverse ready (control warp arrives, solvers wait)
  LB_FUN,       // metric functionals ready (functional warp arrives, the others wait)
  LB_REJ,       // a rejected step: the solvers have left the step-end set (both)
  LB_CO3,       // the three coefficient warps
  LB_ERR        // error-norm parts (companion warps 0..2 arrive, the control warp waits)
};
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) { asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory"); }

template <int NSL, typename ST>
struct LatMem {
  static constexpr int NM = kSolvers * NSL;
  double x[NM + 1];  // operator input; x[n..NM] stay 0
  double f[NM + 1];
  double Us[TB::S][NM];          // stage solutions of the step
  double PA[NM], PC[NM];         // next stage's sums without their last term
  ST r[NM + 1];                  // structured-solve right-hand side / work vector
  ST dd[NM], sup[NM], sub[NM], dinv[NM], mfw[NM], bP[NM];
  ST Z1[NM + 1], Z2[NM + 1];
  ST H[64], Hinv[64];
  ST hmul[2], hcorr[2];   // couplings of the photon tails to the head
  ST wS[kWF], fS[4];
  CSet cs[kNSets];
  double B[kMaxT][B_COUNT], dB[kMaxT][B_COUNT];  // base scalars of the companions' times
  double Bo[B_COUNT], dBo[B_COUNT];              // and of the solver warps' (initial, output, final times)
  double src[4];
  double fun[4];                 // Ψ, Φ̇ and their derivative parts of the current operator product
  double red[4];                 // solver-warp reductions
  double rede[4];                // companion-warp reductions
  float redf[2][4];
  double ctl[4 + kMaxT];
  int ctlf, accept;
  double tA[TB::S], tC[TB::S], td[TB::S];  // tableau: last A and C of each stage, d
  double hd[TB::S];                        // h d of the step
  int tq[TB::S], tinc[TB::S];              // stage time set, incremental input
  CosmoDesc cdesc;
  int item;
};

struct LGrp {
  int gt, lane, wq;   // within the solver (or companion) warps
  int fc;             // component of this lane's metric-functional term
  int fw;             // solver warp that forms the metric functionals
  int ftop;           // first butterfly distance of a metric functional's sum
  unsigned pp, act;   // bit s: some row of slot s in this warp carries a Φ̇ or Ψ coupling / exists
  int rp;             // ping-pong buffer of group_max
};

// A thread's rows in registers.  Slot 1 of the solver warps starts at warp 2: warp 0 has the head
// rows, warp 1 the functionals.
__device__ __forceinline__ int lat_comp(int gt, int s) { return s * kSolvers + ((gt + 64 * s) & (kSolvers - 1)); }
template <int NSL>
struct Rows {
  double A[NSL], C[NSL];
  int i[NSL], ip[NSL], in[NSL], sp[NSL], dg[NSL];
  int fd[NSL], fx[NSL];  // coupling to the metric functionals: coefficient, and 0 for Ψ or 1 for Φ̇ (no row has both)
  int e0, e0c, e1, e1c, e3, e3a, e3b;  // head rows (slot 0): cv[e0] x[e0c] + cv[e1] x[e1c] + cv[e3] (x[e3a] - (3k/4) x[e3b])
  bool extra;
};
template <int NSL>
__device__ __forceinline__ Rows<NSL> load_rows(const LGrp& g, const ModelDesc& M, const CompDesc* comps) {
  Rows<NSL> R;
#pragma unroll
  for (int s = 0; s < NSL; ++s) {
    const int i = lat_comp(g.gt, s);
    const bool on = i < M.n;
    const CompDesc& D = comps[on ? i : 0];
    R.i[s] = i;
    R.A[s] = on ? D.A : 0.0; R.C[s] = on ? D.C : 0.0;
    R.ip[s] = on ? D.ip : M.n; R.in[s] = on ? D.inx : M.n;
    R.sp[s] = on ? D.sp : 0; R.dg[s] = on ? D.dg : 0; 
    R.fx[s] = on && D.psid != CV_ZERO ? 0 : 1; R.fd[s] = on ? (R.fx[s] ? D.phid : D.psid) : 0;
  }
  const CompDesc& D = comps[R.i[0] < M.n ? R.i[0] : 0];
  R.extra = g.gt < 32;
  // no row has both an e2 and a drag term: one product serves either
  const bool drag = D.dx != CV_ZERO;
  R.e0 = D.e0; R.e0c = D.e0c; R.e1 = D.e1; R.e1c = D.e1c;
  R.e3 = drag ? D.dx : D.e2; R.e3a = drag ? D.dxa : D.e2c; R.e3b = drag ? D.dxb : M.n;
  return R;
}

// Sum over the solver or companion warps; the caller guarantees that no warp still reads red.
__device__ __forceinline__ double lat_sum(const LGrp& g, double* red, int bar, double v) {
  v = warp_sum(v);
  if (g.lane == 0) red[g.wq] = v;
  bar_sync(bar, kSolvers);
  double s = 0;
#pragma unroll
  for (int w = 0; w < 4; ++w) s += red[w];
  return s;
}
template <int NSL, typename ST>
__device__ __forceinline__ float lat_max(LGrp& g, LatMem<NSL, ST>& W, float v) {  // v >= 0
  const unsigned m = __reduce_max_sync(FULL, __float_as_uint(v));
  if (g.lane == 0) W.redf[g.rp][g.wq] = __uint_as_float(m);
  bar_sync(LB_MAIN, kSolvers);
  float s = 0;
#pragma unroll
  for (int w = 0; w < 4; ++w) s = fmaxf(s, W.redf[g.rp][w]);
  g.rp ^= 1;
  return s;
}

// Coefficient set of one time by the solver warps (base scalars in Bo); ends with a solver barrier.
template <int NSL, typename ST>
__device__ __forceinline__ void lat_coef1(const LGrp& g, LatMem<NSL, ST>& W, CSet& C, double tau, bool deriv, bool source, const CosmoDesc* cd,
                                          const double* __restrict__ tab, const ModelDesc& M, const ModeK& mk) {
  if (g.wq == 0) coef_base(g.lane, g.lane < 16, g.lane < 16 && deriv, source, tau, cd, tab, M.nx, mk, W.Bo, W.dBo, W.src);
  bar_sync(LB_MAIN, kSolvers);
  for (int e = g.gt; e < M.nexpr_t; e += kSolvers) coef_expr(cd->expr[e], W.Bo, W.dBo, deriv, C);
  bar_sync(LB_MAIN, kSolvers);
}

// Ψ(v) and the δρ sum, as ptk::functionals with the butterfly started at the distance the model's
// terms need (the skipped levels only add zeros); valid on lane 0.
__device__ __forceinline__ void lat_functionals(const LGrp& g, const double* v, const double* w, double& psi, double& rho) {
  double t = w[g.lane] * v[g.fc];
#pragma unroll
  for (int o = 8; o; o >>= 1)
    if (o <= g.ftop) t += __shfl_xor_sync(FULL, t, o);
  psi = t;
  rho = __shfl_down_sync(FULL, t, 16);
}

// Metric functionals as every thread that uses them sees them.
struct Fun { double psi, phd, dpsi, dphd; };

// out = J(τ) x for the thread's rows; DT: also dout = (dJ/dτ) x, with the metric terms added before the
// head rows' extra ones when DSRC (the order of the output pass), after them otherwise.  x complete
// in shared memory; the functional warp publishes Ψ, Φ̇ through LB_FUN, warps that need neither only
// arrive there.  want: the calling thread's warp reads them although no row of it is coupled.
template <int NSL, typename ST, bool DT, bool DSRC>
__device__ __forceinline__ Fun lat_matvec(const LGrp& g, LatMem<NSL, ST>& W, const Rows<NSL>& R, const double* x, const CSet& C, double k34,
                                          double (&out)[NSL], double (&dout)[NSL], bool want) {
  const double* cv = C.cv; const double* cvd = C.cvd;
  const bool isf = g.wq == g.fw, uses = g.pp != 0 || want;
  Fun F{0, 0, 0, 0};
  if (isf) {
    double psi, rho, dpsi = 0, drho = 0;
    lat_functionals(g, x, C.w, psi, rho);
    if (DT) lat_functionals(g, x, C.wd, dpsi, drho);
    F.psi = psi;
    F.phd = phidot(cv, rho, x[0], psi);
    if (DT) {
      F.dpsi = dpsi;
      F.dphd = cvd[CV_PA] * rho + cv[CV_PA] * drho + cvd[CV_PB] * x[0] + cvd[CV_MH] * psi + cv[CV_MH] * dpsi;
    }
    if (g.lane == 0) {
      W.fun[0] = F.psi; W.fun[1] = F.phd;
      if (DT) { W.fun[2] = F.dpsi; W.fun[3] = F.dphd; }
    }
    __syncwarp();
    bar_arrive(LB_FUN, kSolvers);
  } else if (!uses) {
    bar_arrive(LB_FUN, kSolvers);
  }
#pragma unroll
  for (int s = 0; s < NSL; ++s) {
    double o = 0, d = 0;
    if ((g.act >> s) & 1u) {
      const double ax = R.A[s] * x[R.ip[s]] + R.C[s] * x[R.in[s]], xi = x[R.i[s]];
      o = cv[R.sp[s]] * ax + cv[R.dg[s]] * xi;
      if (DT) d = cvd[R.sp[s]] * ax + cvd[R.dg[s]] * xi;
      if (s == 0 && R.extra) {
        const double x0 = x[R.e0c], x1 = x[R.e1c], x3 = x[R.e3a] - k34 * x[R.e3b];
        o += cv[R.e0] * x0 + cv[R.e1] * x1 + cv[R.e3] * x3;
        if (DT && !DSRC) d += cvd[R.e0] * x0 + cvd[R.e1] * x1 + cvd[R.e3] * x3;
      }
    }
    out[s] = o;
    if (DT) dout[s] = d;
  }
  if (uses) {
    if (!isf) bar_sync(LB_FUN, kSolvers);
    if (want) {
      F.psi = W.fun[0]; F.phd = W.fun[1];
      if (DT) { F.dpsi = W.fun[2]; F.dphd = W.fun[3]; }
    }
#pragma unroll
    for (int s = 0; s < NSL; ++s)
      if ((g.pp >> s) & 1u) {
        // one product per row (the generic kernel's other one has a zero coefficient), rounded by itself as there
        const double v = W.fun[R.fx[s]], c = cv[R.fd[s]];
        out[s] = __dadd_rn(out[s], __dmul_rn(c, v));
        if (DT) dout[s] = __dadd_rn(dout[s], fma(c, W.fun[2 + R.fx[s]], __dmul_rn(cvd[R.fd[s]], v)));
      }
  }
  if (DT && DSRC && R.extra) {
    const double x0 = x[R.e0c], x1 = x[R.e1c], x3 = x[R.e3a] - k34 * x[R.e3b];
    dout[0] += cvd[R.e0] * x0 + cvd[R.e1] * x1 + cvd[R.e3] * x3;
  }
  return F;
}

// Reciprocal of a pivot.  FP32: the hardware approximation (pivots are far from the subnormals that the
// non-ftz form would handle).  FP64: its 20-bit seed and two Newton steps r += r (1 - v r), each squaring
// the error: a unit in the last place at most (the division's bits in 2e9 random values) for a fifth of a division's
// FP64 instructions.
template <typename ST>
__device__ __forceinline__ ST lat_rcp(ST v);
template <>
__device__ __forceinline__ float lat_rcp<float>(float v) {
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(v));
  return r;
}
template <>
__device__ __forceinline__ double lat_rcp<double>(double v) {
  double r;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(v));
  r = fma(r, fma(-v, r, 1.0), r);
  return fma(r, fma(-v, r, 1.0), r);
}
// Magnitudes in order as integers (an FP64 comparison holds the FP64 pipe like a product).
__device__ __forceinline__ unsigned mag_key(float v) { return __float_as_uint(v) & 0x7fffffffu; }
__device__ __forceinline__ unsigned long long mag_key(double v) { return (unsigned long long)__double_as_longlong(v) & 0x7fffffffffffffffull; }

// ---- structured solve with the step's factorisation in registers -----------------------------------
// Warp p eliminates chains 2p and 2p + 1 (lane j: row last - j), as in sbz_pt_impl.cuh.
template <typename ST>
struct LatScan {
  int i0, i1, j0, j1, n0, n1;  // rows, rows clamped into the arrays, chain lengths
  bool on0, on1, pair, more;   // more: a chain has more than eight rows (levels 3 and 4 have nonzero multipliers)
  ST f0[5], f1[5], b0[5], b1[5], d0, d1;
};
template <typename ST>
struct LatFactor {
  ST is, ihc, S00, S01, S10, S11;
  ST hv[8], hm;     // head inverse row and chain coupling of warp 0's lanes
  ST wS, fS[3];     // functional weight of the lane, Φ̇ coefficients
};

template <int NV, int NSL, typename ST>
__device__ __forceinline__ void lat_solve_M(const LGrp& g, const LatScan<ST>& S, const LatFactor<ST>& F, ST* v0, ST* v1) {
  const int lane = g.lane;
  if (g.wq == 3) {  // Φ and CDM ([[s, 1], [0, s+ℋ]]), on every lane of the warp with fewest rows
    const ST a2 = v0[2] * F.ihc, a1 = (v0[1] - a2) * F.is, a0 = v0[0] * F.is;
    ST c0 = 0, c1 = 0, c2 = 0;
    if (NV > 1) { c2 = v1[2] * F.ihc; c1 = (v1[1] - c2) * F.is; c0 = v1[0] * F.is; }
    __syncwarp();
    if (lane == 0) {
      v0[0] = a0; v0[1] = a1; v0[2] = a2;
      if (NV > 1) { v1[0] = c0; v1[1] = c1; v1[2] = c2; }
    }
  }
  if (S.pair) {
    const ST r0 = v0[S.j0], r1 = v0[S.j1];
    ST x0 = S.on0 ? r0 : ST(0), x1 = S.on1 ? r1 : ST(0);
    ST y0 = ST(0), y1 = ST(0);
    if (NV > 1) { const ST s0 = v1[S.j0], s1 = v1[S.j1]; y0 = S.on0 ? s0 : ST(0); y1 = S.on1 ? s1 : ST(0); }
    ST hb0 = v0[3 + (lane & 7)], hb1 = NV > 1 ? v1[3 + (lane & 7)] : ST(0);
    // levels 0..2 always, the others where a chain of the warp has more than eight rows: one branch per
    // direction (a branch per level cost as much as the level it skipped)
    auto fwd = [&](int q) {
      const int d = 1 << q;
      const ST px0 = shfl_up_(x0, d), px1 = shfl_up_(x1, d);
      x0 += S.f0[q] * px0; x1 += S.f1[q] * px1;
      if (NV > 1) { const ST py0 = shfl_up_(y0, d), py1 = shfl_up_(y1, d); y0 += S.f0[q] * py0; y1 += S.f1[q] * py1; }
    };
    auto bwd = [&](int q) {
      const int d = 1 << q;
      const ST px0 = __shfl_down_sync(FULL, x0, d), px1 = __shfl_down_sync(FULL, x1, d);
      x0 += S.b0[q] * px0; x1 += S.b1[q] * px1;
      if (NV > 1) {
        const ST py0 = __shfl_down_sync(FULL, y0, d), py1 = __shfl_down_sync(FULL, y1, d);
        y0 += S.b0[q] * py0; y1 += S.b1[q] * py1;
      }
    };
    auto back = [&]() {
      x0 *= S.d0; x1 *= S.d1;
      if (NV > 1) { y0 *= S.d0; y1 *= S.d1; }
      bwd(0); bwd(1); bwd(2);
      if (S.more) { bwd(3); bwd(4); }
      if (S.on0) { v0[S.i0] = x0; if (NV > 1) v1[S.i0] = y0; }
      if (S.on1) { v0[S.i1] = x1; if (NV > 1) v1[S.i1] = y1; }
    };
    fwd(0); fwd(1); fwd(2);
    if (S.more) { fwd(3); fwd(4); }
    if (g.wq == 0) {
      // head: chain 0 (photon T tail) ends at F2 (lane 4), chain 1 (P tail) at G2 (lane 7); hm is zero on
      // the other lanes.  Its shuffles and the back substitution's are one straight run of code.
      const ST c0 = __shfl_sync(FULL, x0, S.n0 - 1), c1 = __shfl_sync(FULL, x1, S.n1 - 1);
      hb0 -= F.hm * (lane == 4 ? c0 : c1);
      if (NV > 1) {
        const ST e0 = __shfl_sync(FULL, y0, S.n0 - 1), e1 = __shfl_sync(FULL, y1, S.n1 - 1);
        hb1 -= F.hm * (lane == 4 ? e0 : e1);
      }
      ST q0[8], q1[8];
#pragma unroll
      for (int q = 0; q < 8; ++q) { q0[q] = __shfl_sync(FULL, hb0, q); q1[q] = NV > 1 ? __shfl_sync(FULL, hb1, q) : ST(0); }
      x0 *= S.d0; x1 *= S.d1;
      if (NV > 1) { y0 *= S.d0; y1 *= S.d1; }
      ST o0 = 0, o1 = 0;
      bwd(0);
#pragma unroll
      for (int q = 0; q < 4; ++q) { o0 += F.hv[q] * q0[q]; if (NV > 1) o1 += F.hv[q] * q1[q]; }
      bwd(1);
#pragma unroll
      for (int q = 4; q < 8; ++q) { o0 += F.hv[q] * q0[q]; if (NV > 1) o1 += F.hv[q] * q1[q]; }
      bwd(2);
      if (lane < 8) { v0[3 + lane] = o0; if (NV > 1) v1[3 + lane] = o1; }
      if (S.more) { bwd(3); bwd(4); }
      if (S.on0) { v0[S.i0] = x0; if (NV > 1) v1[S.i0] = y0; }
      if (S.on1) { v0[S.i1] = x1; if (NV > 1) v1[S.i1] = y1; }
    } else {
      back();
    }
  }
  bar_sync(LB_MAIN, kSolvers);
}

template <typename ST>
__device__ __forceinline__ void lat_functionals_st(const LGrp& g, const LatFactor<ST>& F, const ST* v, ST& psi, ST& phd) {
  ST t = F.wS * v[g.fc];
#pragma unroll
  for (int o = 8; o; o >>= 1)
    if (o <= g.ftop) t += __shfl_xor_sync(FULL, t, o);
  psi = __shfl_sync(FULL, t, 0);
  const ST rho = __shfl_sync(FULL, t, 16);
  phd = F.fS[0] * rho + F.fS[1] * v[0] + F.fS[2] * psi;
}

// What of the factorisation depends on the Jacobian set alone (no step size).
template <int NSL, typename ST>
__device__ __forceinline__ void lat_factor_inputs(const LGrp& g, LatMem<NSL, ST>& W, LatFactor<ST>& F, const Rows<NSL>& R, const CSet& C, int n,
                                                  double (&dg)[NSL]) {
  const double* cv = C.cv;
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) {
    dg[sl] = cv[R.dg[sl]];
    const int i = R.i[sl];
    if (i < n) {
      const double spv = cv[R.sp[sl]];
      W.sup[i] = to_st<ST>(-spv * R.C[sl]);
      W.sub[i] = to_st<ST>(-spv * R.A[sl]);
      const ST c = to_st<ST>(cv[R.fd[sl]]);
      W.Z1[i] = R.fx[sl] ? c : ST(0);
      W.Z2[i] = R.fx[sl] ? ST(0) : c;
    }
  }
  F.wS = to_st<ST>(C.w[g.lane]);
  F.fS[0] = to_st<ST>(cv[CV_PA]); F.fS[1] = to_st<ST>(cv[CV_PB]); F.fS[2] = to_st<ST>(cv[CV_MH]);
}

// Chain LU from the truncation ends, one chain per lane of the control warp (precision ST); four rows are
// read ahead of the serial pivot recurrence.  Then the photon tails' couplings to the head.
template <int NSL, typename ST>
__device__ __forceinline__ void lat_chain_lu(int lane, LatMem<NSL, ST>& W, const ModelDesc& M) {
  if (lane >= M.nchain) return;
  const int first = M.chFirst[lane], last = M.chLast[lane];
  ST dn = lat_rcp<ST>(W.dd[last]);
  W.dinv[last] = dn; W.mfw[last] = 0;
  for (int i = last - 1; i >= first; i -= 4) {
    ST sp[4], sb[4], d[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const int r = i - q > first ? i - q : first;
      sp[q] = W.sup[r]; sb[q] = W.sub[r + 1]; d[q] = W.dd[r];
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (i - q >= first) {
        const ST di = lat_rcp<ST>(d[q] - sp[q] * sb[q] * dn);
        W.dinv[i - q] = di; W.mfw[i - q] = sp[q] * dn;
        dn = di;
      }
  }
  if (lane < 2) {  // coupling of x[first] into the head row (F2, G2)
    const ST hs = W.sup[M.chAttach[lane]];
    const ST hm = hs * dn;
    W.hmul[lane] = hm;
    W.hcorr[lane] = hm * W.sub[first];
  }
}

// Factorisation for the step size s = 1/(hγ), first part: diagonals to the control warp, which runs the
// chain LU and inverts the head, and the head rows (solver warp 3).
template <int NSL, typename ST>
__device__ __forceinline__ void lat_factor_start(const LGrp& g, LatMem<NSL, ST>& W, LatFactor<ST>& F, const Rows<NSL>& R, const CSet& C,
                                                 const CompDesc* __restrict__ comps, int n, double k, double h, double s, const double (&dg)[NSL]) {
  const int lane = g.lane;
  const double* cv = C.cv;
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) { const int i = R.i[sl]; if (i < n) W.dd[i] = to_st<ST>(s - dg[sl]); }
  bar_arrive(LB_DD, kSolvers + 32);
  if (g.wq == 3) {
    if (lane >= 16 && lane < 24) {  // assemble head row 3 + j
      const int j = lane - 16, r = 3 + j;
      const double k34 = 0.75 * k;
      const CompDesc& D = comps[r];
      double row[8];
#pragma unroll
      for (int c = 0; c < 8; ++c) row[c] = 0;
      row[j] += s - cv[D.dg];
      const double spv = cv[D.sp];
      int c;
      if ((c = head_local(D.ip)) >= 0) row[c] -= spv * D.A;
      if ((c = head_local(D.inx)) >= 0) row[c] -= spv * D.C;
      if ((c = head_local(D.e0c)) >= 0) row[c] -= cv[D.e0];
      if ((c = head_local(D.e1c)) >= 0) row[c] -= cv[D.e1];
      if ((c = head_local(D.e2c)) >= 0) row[c] -= cv[D.e2];
      if ((c = head_local(D.dxa)) >= 0) row[c] -= cv[D.dx];
      if ((c = head_local(D.dxb)) >= 0) row[c] += k34 * cv[D.dx];
#pragma unroll
      for (int q = 0; q < 8; ++q) W.H[j * 8 + q] = to_st<ST>(row[q]);
    }
    __syncwarp();
    bar_arrive(LB_HROW, 64);
  }
  F.is = to_st<ST>(h * TB::gam);
  F.ihc = lat_rcp<ST>(to_st<ST>(s - cv[CV_MH]));
}

// Second part, from the chain pivots: ends with the rank-2 columns z1, z2 and the head-value factors P of
// the thread's rows in registers.
template <int NSL, typename ST>
__device__ __forceinline__ void lat_factor_finish(const LGrp& g, LatMem<NSL, ST>& W, LatFactor<ST>& F, LatScan<ST>& S, const Rows<NSL>& R,
                                                  const ModelDesc& M, const int (&at)[NSL], ST (&z1)[NSL], ST (&z2)[NSL], ST (&P)[NSL]) {
  const int lane = g.lane;
  bar_sync(LB_LU, kSolvers + 32);
  if (S.pair) {  // Kogge-Stone multipliers of both recurrences of the warp's two chains, side by side
    const ST e0 = W.dinv[S.j0], e1 = W.dinv[S.j1], m0 = W.mfw[S.j0], m1 = W.mfw[S.j1], u0 = W.sub[S.j0], u1 = W.sub[S.j1];
    ST a0 = (S.on0 && lane > 0) ? -m0 : ST(0), a1 = (S.on1 && lane > 0) ? -m1 : ST(0);
    ST c0 = S.on0 ? -e0 * u0 : ST(0), c1 = S.on1 ? -e1 * u1 : ST(0);
    auto level = [&](int q) {
      const int d = 1 << q;
      const ST p0 = shfl_up_(a0, d), p1 = shfl_up_(a1, d);
      const ST q0 = __shfl_down_sync(FULL, c0, d), q1 = __shfl_down_sync(FULL, c1, d);
      const bool up = lane >= d, in0 = lane + d < S.n0, in1 = lane + d < S.n1;
      S.f0[q] = (S.on0 && up) ? a0 : ST(0); S.f1[q] = (S.on1 && up) ? a1 : ST(0);
      S.b0[q] = (S.on0 && in0) ? c0 : ST(0); S.b1[q] = (S.on1 && in1) ? c1 : ST(0);
      if (up) { a0 *= p0; a1 *= p1; }
      if (in0) c0 *= q0;
      if (in1) c1 *= q1;
    };
    level(0); level(1); level(2);
    if (S.more) { level(3); level(4); }
    S.d0 = S.on0 ? e0 : ST(0); S.d1 = S.on1 ? e1 : ST(0);
    if (S.on0) W.bP[S.j0] = c0;  // ∂z_i/∂h
    if (S.on1) W.bP[S.j1] = c1;
  }
  bar_sync(LB_HEAD, kSolvers + 32);
  if (g.wq == 0) {
#pragma unroll
    for (int q = 0; q < 8; ++q) F.hv[q] = W.Hinv[(lane & 7) * 8 + q];
    F.hm = lane == 4 ? W.hmul[0] : lane == 7 ? W.hmul[1] : ST(0);
  }
  // rank-2 correction: Z1 = M⁻¹ c_Φ̇, Z2 = M⁻¹ c_Ψ
  lat_solve_M<2, NSL, ST>(g, S, F, W.Z1, W.Z2);
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) {  // own rows, with the head-value terms of the chain back substitutions
    const int ic = R.i[sl] < M.n ? R.i[sl] : 0, a = at[sl];
    ST u1 = W.Z1[ic], u2 = W.Z2[ic];
    P[sl] = W.bP[ic];
    if (a >= 0) { u1 += P[sl] * W.Z1[a]; u2 += P[sl] * W.Z2[a]; }
    z1[sl] = u1; z2[sl] = u2;
  }
  ST psi1, p1, psi2, p2;
  lat_functionals_st(g, F, W.Z1, psi1, p1);
  lat_functionals_st(g, F, W.Z2, psi2, p2);
  const ST a = 1 - p1, b = -p2, c = -psi1, d = 1 - psi2;
  const ST idet = sizeof(ST) == 8 ? lat_rcp<ST>(a * d - b * c) : ST(1) / (a * d - b * c);
  F.S00 = d * idet; F.S01 = -b * idet; F.S10 = -c * idet; F.S11 = a * idet;
}

// One output time (sources, factors or state) for state y: solver warps only.
template <int NSL, typename ST>
__device__ void lat_emit(const LGrp& g, LatMem<NSL, ST>& W, const Rows<NSL>& R, const PtArgs& A, const CosmoDesc* cd, const double* tab,
                         const ModelDesc& M, const ModeK& mk, double tau, const double (&y)[NSL], int item, int j) {
  if (A.output == SBZ_OUT_STATE) {
    double* o = A.out + ((size_t)item * A.ntau + j) * M.n;
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < M.n) o[R.i[sl]] = y[sl];
    return;
  }
  if (A.output != SBZ_OUT_SOURCES && A.output != SBZ_OUT_SOURCES4 && A.output != SBZ_OUT_FACTORS) return;
  CSet& C = W.cs[kNSets - 1];
  const double k34 = 0.75 * mk.k;
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < M.n) W.x[R.i[sl]] = y[sl];
  lat_coef1(g, W, C, tau, true, true, cd, tab, M, mk);
  double fy[NSL], dJy[NSL], Jf[NSL], un[NSL];
  const Fun F = lat_matvec<NSL, ST, true, true>(g, W, R, W.x, C, k34, fy, dJy, g.wq == 0);
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < M.n) W.f[R.i[sl]] = fy[sl];
  bar_sync(LB_MAIN, kSolvers);
  const Fun Ff = lat_matvec<NSL, ST, false, false>(g, W, R, W.f, C, k34, Jf, un, g.wq == 0);
  if (g.wq == 0) {
    // second derivative of Π = F2 + G0 + G2 along the flow: (J'y + J f) restricted to those rows, in
    // the order of a butterfly sum over the warp
    const double gv = dJy[0] + Jf[0];
    const double g7 = __shfl_sync(FULL, gv, 7), g8 = __shfl_sync(FULL, gv, 8), g10 = __shfl_sync(FULL, gv, 10);
    if (g.gt == 0) write_output(A, cd, mk, tau, W.x, W.f, W.src, W.Bo[B_KD], F.psi, F.phd, F.dpsi + Ff.psi, (g8 + g10) + g7, item, j);
  }
  bar_sync(LB_MAIN, kSolvers);
}

// Step control as ptk::pt_body publishes it, in two parts: flags, h, 1/h and 1/(hγ) (what the solver warps
// wait for; the divisions one per lane), then the step end and the stage times.  Returns the step end.  Each FP64
// instruction of this chain is 65 cycles of every warp's wait: times are positive and compared as integers, and
// left = tend - tc and tmin = 1e-14 tc come from the caller.
template <int NSL, typename ST>
__device__ __forceinline__ double lat_publish(int lane, LatMem<NSL, ST>& W, double& hp, double tc, double tend, double left, double tmin) {
  // the divisions start before the clamp to the end point, which is rare, is decided
  double inv = 1.0 / (lane == 1 ? hp * TB::gam : hp);
  const bool done = dkey(tc) >= dkey(tend);
  if (dkey(tc + 1.01 * hp) >= dkey(tend)) {
    hp = left;
    inv = 1.0 / (lane == 1 ? hp * TB::gam : hp);
  }
  const bool tiny = dkey(hp) <= dkey(tmin);
  if (lane == 0) { W.ctlf = (done ? 1 : 0) | (tiny ? 2 : 0); W.ctl[0] = hp; W.ctl[1] = inv; }
  if (lane == 1) W.ctl[2] = inv;
  return dkey(hp) == dkey(left) ? tend : tc + hp;
}
template <int NSL, typename ST>
__device__ __forceinline__ void lat_publish_times(int lane, LatMem<NSL, ST>& W, double hp, double tc, double te) {
  double c = 0;  // stage time lane - 4 + 1 of the tableau
#pragma unroll
  for (int q = 1; q < TB::NTIME; ++q) {
    int st = 1;
#pragma unroll
    for (int i = 1; i < TB::S; ++i) if (TB::tslot(i) == q) st = i;
    if (lane == 3 + q) c = TB::c(st);
  }
  const double ts = tc + c * hp;
  if (lane < TB::S) W.hd[lane] = hp * W.td[lane];
  if (lane == 0) { W.ctl[3] = te; W.ctl[4 + TB::NTIME - 1] = te; }
  if (lane >= 4 && lane < 4 + TB::NTIME - 1) W.ctl[lane] = ts;
}

// ---- solver warps -------------------------------------------------------------------------------------
template <int NSL, typename ST>
__device__ void lat_solver(const PtArgs& A, const ModelDesc& M, const CompDesc* __restrict__ comps, LatMem<NSL, ST>& W, LGrp& g,
                           const Rows<NSL>& R, LatScan<ST>& S, const int (&at)[NSL], const double* tab, const double* taus, int item,
                           const ModeK& mk) {
  const int gt = g.gt, n = M.n;
  const CosmoDesc* cd = &W.cdesc;
  const double k = mk.k, k34 = 0.75 * k, rtol = A.rtol, atol = A.atol, inv_n = 1.0 / n;
  const double tend = cd->tau0;
  double t = fmin(fmax(A.item_tau_ini[item], cd->tau_start), tend);
  int status = SBZ_OK;
  int64_t nacc = 0, nrej = 0;
  double y[NSL], f0[NSL], ft[NSL];
  int sJ = 0, sE = TB::NTIME;

  lat_coef1(g, W, W.cs[kNSets - 1], t, false, false, cd, tab, M, mk);
  {
    const IcScal ic = ic_scalars(g.lane, M, cd, W.Bo, k, t);
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) {
      const int i = R.i[sl];
      const double v = i < n ? ic_value(i, M, cd, W.Bo, ic, k) : 0.0;
      y[sl] = v;
      if (i < n) W.x[i] = v;
    }
    bar_sync(LB_MAIN, kSolvers);
    // Φ from k²(Φ - Ψ) = 12πa²Π with the initial shears: Ψ(y) is linear with unit weight on Φ
    double psi0, rho0;
    lat_functionals(g, W.x, W.cs[kNSets - 1].w, psi0, rho0);  // Φ slot still 0
    bar_sync(LB_MAIN, kSolvers);
    if (gt == 0) { y[0] = ic.Psi - psi0; W.x[0] = y[0]; }
    bar_sync(LB_MAIN, kSolvers);
  }
  int jout = 0;
  if (taus) {
    while (jout < A.ntau && taus[jout] <= t) {
      if (taus[jout] < t) zero_output(A, gt, kSolvers, n, item, jout);  // before the mode starts
      else lat_emit(g, W, R, A, cd, tab, M, mk, t, y, item, jout);
      ++jout;
    }
  }
  if (t < tend) {
    lat_coef1(g, W, W.cs[sJ], t, true, false, cd, tab, M, mk);
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n) W.x[R.i[sl]] = y[sl];
    bar_sync(LB_MAIN, kSolvers);
    lat_matvec<NSL, ST, true, false>(g, W, R, W.x, W.cs[sJ], k34, f0, ft, false);  // f(t, y) and ∂f/∂τ
    // initial step (Hairer-Nørsett-Wanner II.4), its norms summed in the companions' row order
    double h;
    {
      auto norm = [&](const double (&v)[NSL]) {  // Σ v² over all rows
        bar_sync(LB_MAIN, kSolvers);
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) W.Us[0][R.i[sl]] = v[sl];
        bar_sync(LB_MAIN, kSolvers);
        double e = 0;
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) { const int i = comp_of<4>(gt, sl); if (i < n) { const double q = W.Us[0][i]; e += q * q; } }
        return lat_sum(g, W.red, LB_MAIN, e);
      };
      double q0[NSL], q1[NSL];
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) {
        const double sk = atol + fabs(y[sl]) * rtol;
        q0[sl] = y[sl] / sk; q1[sl] = f0[sl] / sk;
      }
      const double d0 = sqrt(norm(q0) * inv_n), d1 = sqrt(norm(q1) * inv_n);
      double h0 = (d0 < 1e-5 || d1 < 1e-5) ? 1e-6 : 0.01 * d0 / d1;
      h0 = fmin(h0, tend - t);
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n) W.x[R.i[sl]] = y[sl] + h0 * f0[sl];
      const double th = t + h0;
      lat_coef1(g, W, W.cs[sE], th, false, false, cd, tab, M, mk);
      double f1[NSL], un[NSL];
      lat_matvec<NSL, ST, false, false>(g, W, R, W.x, W.cs[sE], k34, f1, un, false);
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) { const double sk = atol + fabs(y[sl]) * rtol; q0[sl] = (f1[sl] - f0[sl]) / (h0 * sk); }
      const double d2 = sqrt(norm(q0) * inv_n);
      const double mx = fmax(d1, d2);
      const double h1 = (mx <= 1e-15 || !isfinite(mx)) ? fmax(1e-6, 1e-3 * h0) : pow(0.01 / mx, 0.2);
      h = fmin(100 * h0, h1);
      if (!isfinite(h) || h <= 0) h = 1e-6 * fmax(1.0, t);
    }
    bar_sync(LB_MAIN, kSolvers);
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n) W.x[R.i[sl]] = y[sl];
    if (g.wq == 1) {
      const double te = lat_publish(g.lane, W, h, t, tend, tend - t, 1e-14 * t);
      lat_publish_times(g.lane, W, h, t, te);
    }
    bool nonfinite = false, moved = false;  // moved: y is new since f0 and ft were formed
    LatFactor<ST> F;
    double dg[NSL];
    int64_t iters = 0;
    lat_factor_inputs(g, W, F, R, W.cs[sJ], n, dg);
    bar_sync(LB_STEP, kLatThreads);
    bar_sync(LB_CTL, kSolvers + 32);
    for (;;) {
      // step control published by companion warp 3
      const int fl = W.ctlf;  // bit 0: t reached the end; bit 1: the step is below 1e-14 t
      if (fl & 1) break;
      if (++iters > A.maxiters) { status = SBZ_MAXITERS; break; }
      if (fl & 2) { status = nonfinite ? SBZ_NONFINITE : SBZ_DTMIN; break; }
      h = W.ctl[0];
      const double ih = W.ctl[1], s = W.ctl[2];
      const CSet& CJ = W.cs[sJ];
      ST z1[NSL], z2[NSL], P[NSL];
      lat_factor_start(g, W, F, R, CJ, comps, n, k, h, s, dg);
      if (moved) lat_matvec<NSL, ST, true, false>(g, W, R, W.x, CJ, k34, f0, ft, false);  // f(t, y), ∂f/∂τ, beside the chain LU
      lat_factor_finish(g, W, F, S, R, M, at, z1, z2, P);
      const double tn = W.ctl[3];
      double b[NSL], Fv[NSL], Y[NSL], Ul[NSL], un[NSL];
      float isk[NSL];  // refinement stopping weights
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) isk[sl] = 1.0f / f64_to_f32(atol + rtol * fabs(y[sl]));
      int rk = A.refine;
      // the stage count opaque to the compiler: one copy of the stage body
      int nst;
      asm volatile("mov.u32 %0, %1;" : "=r"(nst) : "n"(TB::S));
#pragma unroll 1
      for (int st = 0; st < nst; ++st) {
        if (st == 0) {
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) b[sl] = fma(W.hd[0], ft[sl], f0[sl]);
        } else {
          double cu[NSL];
          const double ka = W.tA[st], kc = W.tC[st], kd = W.td[st];
          const int kq = W.tq[st], kinc = W.tinc[st];
          const double hdst = W.hd[st];
          if (st == 1) {
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) { Y[sl] = fma(ka, Ul[sl], y[sl]); cu[sl] = kc * Ul[sl]; }
          } else {
            // the companions' sums and the last stage's term; stages 7 and 8 add the previous stage
            bar_sync(LB_SUM, kLatThreads);
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) {
              if (kinc) Y[sl] = Y[sl] + Ul[sl];
              else Y[sl] = fma(ka, Ul[sl], W.PA[R.i[sl]]);
              cu[sl] = fma(kc, Ul[sl], W.PC[R.i[sl]]);
            }
          }
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n) W.x[R.i[sl]] = Y[sl];
          if (st == 1) bar_sync(LB_COEF, kSolvers + 96);
          bar_sync(LB_MAIN, kSolvers);
          lat_matvec<NSL, ST, false, false>(g, W, R, W.x, W.cs[kq < TB::NTIME ? kq : sE], k34, Fv, un, false);
          const bool hd = (dkey(kd) & 0x7fffffffffffffffll) != 0;
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) {
            b[sl] = fma(ih, cu[sl], Fv[sl]);
            if (hd) b[sl] = fma(hdst, ft[sl], b[sl]);
          }
        }
        // U = W⁻¹ b with FP64 iterative refinement (see stage_solve); the later stages are refined only
        // when stage 1's first correction is at or above refine_skip (error-weight units)
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n) W.r[R.i[sl]] = to_st<ST>(b[sl]);
        float c1 = 1e30f;
        for (int it = 0;; ++it) {
          if (it == 0 && st >= 1 && st < TB::S - 1) bar_sync(LB_RHS, kLatThreads);
          else bar_sync(LB_MAIN, kSolvers);
          lat_solve_M<1, NSL, ST>(g, S, F, W.r, W.r);
          ST psi, ph, u[NSL];
          lat_functionals_st(g, F, W.r, psi, ph);
          const ST t0 = fma(F.S01, psi, F.S00 * ph), t1 = fma(F.S11, psi, F.S10 * ph);
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) {
            const int ic = R.i[sl] < n ? R.i[sl] : 0, a = at[sl];
            const ST ri = W.r[ic], ra = W.r[a >= 0 ? a : ic];
            const ST rh = a >= 0 ? ri + P[sl] * ra : ri;
            u[sl] = R.i[sl] < n ? rh + z1[sl] * t0 + z2[sl] * t1 : ST(0);
          }
          if (it == 0) {
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) Ul[sl] = from_st(u[sl]);
          } else {
            float c = 0.0f;
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl)
              if (R.i[sl] < n) { Ul[sl] += from_st(u[sl]); c = fmaxf(c, fabsf((float)u[sl]) * isk[sl]); }
            const int r = it - 1;
            const bool first = r == 0 && st == 0;
            if (r + 1 < rk || first) {
              const float cm = lat_max(g, W, c);
              if (first) c1 = cm;
              if (r + 1 < rk && cm < 1e-3f) break;
            }
          }
          if (it >= rk) break;
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n) W.x[R.i[sl]] = Ul[sl];
          bar_sync(LB_MAIN, kSolvers);
          double JU[NSL];
          lat_matvec<NSL, ST, false, false>(g, W, R, W.x, CJ, k34, JU, un, false);
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl)
            if (R.i[sl] < n) W.r[R.i[sl]] = to_st<ST>(b[sl] - fma(s, Ul[sl], -JU[sl]));  // s U - J U ≈ b first: rounding of order ε|b|
        }
        if (st == 0) rk = (A.refine > 0 && c1 < A.refine_skip) ? 0 : A.refine;
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) W.Us[st][R.i[sl]] = Ul[sl];
      }
      // new state (stiffly accurate: y1 = last stage input + last stage); the companions form the error
      // norm and the next step while the factorisation's inputs are formed as if it were accepted (the
      // FP64 pipes are left to them: f(t1, y1) waits for the chain LU)
      double y1[NSL];
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) { y1[sl] = Y[sl] + Ul[sl]; if (R.i[sl] < n) W.x[R.i[sl]] = y1[sl]; }
      bar_sync(LB_STEP, kLatThreads);
      lat_factor_inputs(g, W, F, R, W.cs[sE], n, dg);
      bar_sync(LB_CTL, kSolvers + 32);
      const int acc = W.accept;
      if (acc == 1) {
        { const int tsw = sJ; sJ = sE; sE = tsw; }
        if (taus && jout < A.ntau && dkey(taus[jout]) <= dkey(tn)) {
          // continuous extension y(t + θh) = (1-θ) y + θ (y1 + (1-θ)(K0 + θ K1 + θ² K2))
          double K[TB::NDENSE][NSL];
#pragma unroll
          for (int r = 0; r < TB::NDENSE; ++r)
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) {
              double v = 0;
#pragma unroll
              for (int j = 0; j < TB::S; ++j) {
                if (TB::dense(r, j) == 0.0) continue;
                v += TB::dense(r, j) * W.Us[j][R.i[sl]];
              }
              K[r][sl] = v;
            }
          while (jout < A.ntau && dkey(taus[jout]) <= dkey(tn)) {
            const double tau = taus[jout];
            const double th = (tau - t) / (tn - t), th1 = 1.0 - th;
            double yo[NSL];
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) yo[sl] = th1 * y[sl] + th * (y1[sl] + th1 * (K[0][sl] + th * (K[1][sl] + th * K[2][sl])));
            lat_emit(g, W, R, A, cd, tab, M, mk, tau, yo, item, jout);
            ++jout;
          }
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n) W.x[R.i[sl]] = y1[sl];  // operator input of f(t1, y1)
          bar_sync(LB_MAIN, kSolvers);
        }
        t = tn;
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) y[sl] = y1[sl];
        ++nacc;
        nonfinite = false;
        moved = true;
      } else {
        ++nrej;
        nonfinite = acc == 2;
        moved = false;
        // J's coefficients (at t), f and ∂f/∂τ stay valid; the companions now may refill the step-end set
        bar_sync(LB_REJ, kLatThreads);
        lat_factor_inputs(g, W, F, R, W.cs[sJ], n, dg);
      }
    }
  }
  // saved times never reached (failed mode): zero
  if (taus) for (; jout < A.ntau; ++jout) zero_output(A, gt, kSolvers, n, item, jout);
  bool finite = true;
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n && !isfinite(y[sl])) finite = false;
  bar_sync(LB_MAIN, kSolvers);
  finite = lat_sum(g, W.red, LB_MAIN, finite ? 0.0 : 1.0) == 0.0;
  if (status == SBZ_OK && !finite) status = SBZ_NONFINITE;
  if (A.output == SBZ_OUT_DELTA_M) {
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) if (R.i[sl] < n) W.x[R.i[sl]] = y[sl];
    lat_coef1(g, W, W.cs[kNSets - 1], tend, false, false, cd, tab, M, mk);
    if (g.wq == 0) {
      const double d = delta_m(g.lane, M, cd, W.Bo, W.x, mk);
      if (gt == 0) A.out[item] = d;
    }
  }
  if (gt == 0) {
    if (A.status) A.status[item] = status;
    if (A.steps) { A.steps[2 * item] = nacc; A.steps[2 * item + 1] = nrej; }
  }
}

// ---- companion warps -----------------------------------------------------------------------------------
// The 8x8 head inverse by one warp (as ptk::factorize): Gauss-Jordan with partial pivoting on [H | I],
// one column per lane.
template <int NSL, typename ST>
__device__ __forceinline__ void lat_head_inverse(int lane, LatMem<NSL, ST>& W) {
  const int q = lane & 15;
  ST col[8];
#pragma unroll
  for (int r = 0; r < 8; ++r) col[r] = q < 8 ? W.H[r * 8 + q] : ST(r == q - 8 ? 1 : 0);
  if (q == 4) col[4] -= W.hcorr[0];  // F2 (Schur complement of the F tail)
  if (q == 7) col[7] -= W.hcorr[1];  // G2 (G tail)
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    int p = kk;
    auto best = mag_key(col[kk]);
#pragma unroll
    for (int r = kk + 1; r < 8; ++r) { const auto v = mag_key(col[r]); if (v > best) { best = v; p = r; } }
    p = __shfl_sync(FULL, p, kk);
    ST vp = col[kk];
#pragma unroll
    for (int r = kk + 1; r < 8; ++r) if (r == p) { vp = col[r]; col[r] = col[kk]; }
    col[kk] = vp;
    ST m[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) m[r] = __shfl_sync(FULL, col[r], kk);
    const ST ip = lat_rcp<ST>(m[kk]);
    col[kk] *= ip;
#pragma unroll
    for (int r = 0; r < 8; ++r) if (r != kk) col[r] -= m[r] * col[kk];
  }
  if (lane >= 8 && lane < 16) {
#pragma unroll
    for (int r = 0; r < 8; ++r) W.Hinv[r * 8 + (lane - 8)] = col[r];
  }
}

// Coefficients at the five later stage times, by the first three companion warps: base scalars of two
// times per warp, then the expressions, the derivative ones (the step end's) on warps 0 and 1, one per
// lane, the value-only ones mostly on warp 2 (a derivative costs about three values of FP64 work).
template <int NSL, typename ST>
__device__ __forceinline__ void lat_coefs(const LGrp& g, LatMem<NSL, ST>& W, int sE, const CosmoDesc* cd, const double* __restrict__ tab,
                                          const ModelDesc& M, const ModeK& mk) {
  constexpr int nt = TB::NTIME;
  {
    const int q = 2 * g.wq + (g.lane >> 4);
    const bool live = q < nt;
    coef_base(g.lane, live, live && q == nt - 1, false, live ? W.ctl[4 + q] : 1.0, cd, tab, M.nx, mk, W.B[live ? q : 0], W.dB[live ? q : 0], W.src);
  }
  bar_sync(LB_CO3, 96);
  const int ne = M.nexpr_t, nval = (nt - 1) * ne;
  if (g.wq < 2)
    for (int e = g.wq * 32 + g.lane; e < ne; e += 64) coef_expr(cd->expr[e], W.B[nt - 1], W.dB[nt - 1], true, W.cs[sE]);
  for (int r = 0; r * 32 < nval; ++r) {
    const int m = r % 7;
    if (g.wq != (m < 5 ? 2 : m - 5)) continue;
    const int p = r * 32 + g.lane;
    if (p < nval) { const int q = p / ne; coef_expr(cd->expr[p - q * ne], W.B[q], W.dB[q], false, W.cs[1 + q]); }
  }
}

template <int NSL, typename ST>
__device__ void lat_companion(const PtArgs& A, const ModelDesc& M, LatMem<NSL, ST>& W, const LGrp& g, const double* tab, int item, const ModeK& mk) {
  const int gt = g.gt, n = M.n;
  const CosmoDesc* cd = &W.cdesc;
  const double rtol = A.rtol, atol = A.atol, inv_n = 1.0 / n;
  const double tend = cd->tau0;
  double t = fmin(fmax(A.item_tau_ini[item], cd->tau_start), tend);
  if (!(t < tend)) return;
  constexpr double kLogErrFloor = -9.210340371976184;  // log(1e-4): the controller's floor on errold
  double lerrold = kLogErrFloor;  // log of the previous accepted error norm
  bool rejected = false, nonfinite = false, first = true;
  double tn = t;
  int sJ = 0, sE = TB::NTIME;
  int64_t iters = 0;
  // rows in the error norm (its sum's order) and in the stage sums: slot 1 on warp 3, and with two warps of rows
  // those of warp 0 on warp 2, whose sub-partition's solver warp has none (warp 0's has the head rows)
  int ci[NSL], si[NSL];
  double y[NSL], y1[NSL], ys[NSL], ys1[NSL];  // state rows of ci and si
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) { ci[sl] = comp_of<4>(gt, sl); si[sl] = sl * kSolvers + ((gt + 32 * sl) & (kSolvers - 1)); }
  if (n <= 64 && (g.wq & 1) == 0) si[0] = gt ^ 64;
  const int nw = n > 96 ? 4 : (n + 31) / 32;  // warps with rows in the error norm
  bool act[NSL];
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) act[sl] = __any_sync(FULL, si[sl] < n);
  bar_sync(LB_STEP, kLatThreads);
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) { y[sl] = ci[sl] < n ? W.x[ci[sl]] : 0.0; ys[sl] = si[sl] < n ? W.x[si[sl]] : 0.0; }
  for (;;) {
    if (first && g.wq == 3) bar_arrive(LB_CTL, kSolvers + 32);  // the first step's control is the solvers'
    bar_sync(LB_COMP, kSolvers);  // control seen by every companion warp
    if (!first) {
      rejected = W.accept != 1;
      if (rejected) {
        bar_sync(LB_REJ, kLatThreads);
      } else {
        t = tn;
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) { y[sl] = y1[sl]; ys[sl] = ys1[sl]; }
        const int tsw = sJ; sJ = sE; sE = tsw;
      }
    }
    first = false;
    const int fl = W.ctlf;  // the solver warps leave the loop on the same tests, in the same order
    if (fl & 1) break;
    if (++iters > A.maxiters) break;
    if (fl & 2) break;
    const double h = W.ctl[0];
    tn = W.ctl[3];
    if (g.wq < 3) {
      lat_coefs(g, W, sE, cd, tab, M, mk);
      bar_arrive(LB_COEF, kSolvers + 96);
    } else {
      bar_sync(LB_DD, kSolvers + 32);
      lat_chain_lu(g.lane, W, M);
      __syncwarp();
      bar_arrive(LB_LU, kSolvers + 32);
      bar_sync(LB_HROW, 64);
      lat_head_inverse(g.lane, W);
      __syncwarp();
      bar_arrive(LB_HEAD, kSolvers + 32);
    }
    // stage sums: after stage j's solution add its term to every later stage's sums, the next one's first
    double a[4][NSL], c[6][NSL];  // stages 2..5 (inputs) and 2..7 (right-hand sides)
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) {
#pragma unroll
      for (int q = 0; q < 4; ++q) a[q][sl] = ys[sl];
#pragma unroll
      for (int q = 0; q < 6; ++q) c[q][sl] = 0;
    }
#pragma unroll
    for (int j = 0; j < TB::S - 2; ++j) {
      bar_sync(LB_RHS, kLatThreads);
      double u[NSL];
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) {
        u[sl] = si[sl] < n ? W.Us[j][si[sl]] : 0.0;
        if (act[sl]) {
          if (j + 2 < 6) { a[j < 4 ? j : 0][sl] = fma(TB::A(j + 2, j), u[sl], a[j < 4 ? j : 0][sl]); W.PA[si[sl]] = a[j < 4 ? j : 0][sl]; }
          c[j][sl] = fma(TB::C(j + 2, j), u[sl], c[j][sl]);
          W.PC[si[sl]] = c[j][sl];
        }
      }
      bar_arrive(LB_SUM, kLatThreads);
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl)
        if (act[sl]) {
#pragma unroll
          for (int i = j + 3; i < TB::S; ++i) {
            if (i < 6) a[i - 2][sl] = fma(TB::A(i, j), u[sl], a[i - 2][sl]);
            c[i - 2][sl] = fma(TB::C(i, j), u[sl], c[i - 2][sl]);
          }
        }
    }
    // FP64 error norm of the last stage
    bar_sync(LB_STEP, kLatThreads);
    double e2 = 0;
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) {
      const int i = ci[sl];
      ys1[sl] = si[sl] < n ? W.x[si[sl]] : 0.0;
      if (i < n) {
        y1[sl] = W.x[i];
        const double ul = W.Us[TB::S - 1][i];
        const double sk = atol + rtol * __longlong_as_double(max(dkey(fabs(y[sl])), dkey(fabs(y1[sl]))));
        const double q = ul / sk;
        e2 += q * q;
      }
    }
    e2 = warp_sum(e2);
    if (g.lane == 0) W.rede[g.wq] = e2;
    __syncwarp();
    if (g.wq < 3) {
      bar_arrive(LB_ERR, kSolvers);
    } else {  // step control
      double left = tend - tn, tmin = 1e-14 * tn;  // of an accepted step, before the wait
      bar_sync(LB_ERR, kSolvers);
      double err2 = W.rede[0];
      for (int w = 1; w < nw; ++w) err2 += W.rede[w];  // the others are zero
      err2 *= inv_n;  // squared RMS error norm
      // err2 >= 0: accepted when finite and at most 1, by its bit pattern (inf, NaN and any sign-bit
      // pattern compare above 1 as unsigned)
      const bool ok = (unsigned long long)dkey(err2) <= (unsigned long long)dkey(1.0);
      if (ok) nonfinite = false;
      else if ((dkey(err2) & 0x7ff0000000000000ll) == 0x7ff0000000000000ll) nonfinite = true;  // inf or NaN, kept until a step is accepted
      double hp;
      if (ok) {
        // PI controller fac = 0.9 err^-beta1 errold^beta2 (OrdinaryDiffEq's defaults for the method's order)
        const double lerr = 0.5 * log(dmax(err2, 1e-20));
        double fac = 0.9 * exp(-TB::beta1 * lerr + TB::beta2 * lerrold);
        fac = dmin(10.0, dmax(0.2, fac));
        if (rejected) fac = dmin(fac, 1.0);
        lerrold = dmax(lerr, kLogErrFloor);
        hp = h * fac;
      } else {
        hp = nonfinite ? 0.2 * h : h * dmax(0.2, 0.9 * exp(-0.5 * TB::rej * log(err2)));
      }
      if (g.lane == 0) W.accept = ok ? 1 : nonfinite ? 2 : 0;
      const double tc = ok ? tn : t;
      if (!ok) { left = tend - t; tmin = 1e-14 * t; }
      const double te = lat_publish(g.lane, W, hp, tc, tend, left, tmin);
      __syncwarp();
      bar_arrive(LB_CTL, kSolvers + 32);
      lat_publish_times(g.lane, W, hp, tc, te);
    }
  }
}

template <int NSL, typename ST>
__global__ void __launch_bounds__(kLatThreads, 1) pt_lat_kernel(PtArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ModelDesc& M = *reinterpret_cast<ModelDesc*>(smem_raw);
  constexpr size_t mb = (sizeof(ModelDesc) + 15) & ~size_t(15);
  CompDesc* comps = reinterpret_cast<CompDesc*>(smem_raw + mb);
  LatMem<NSL, ST>& W = *reinterpret_cast<LatMem<NSL, ST>*>(smem_raw + mb + (((size_t)A.model_n * sizeof(CompDesc) + 15) & ~size_t(15)));
  const int tid = threadIdx.x;
  for (int i = tid; i < (int)sizeof(ModelDesc) / 4; i += kLatThreads) reinterpret_cast<int*>(&M)[i] = reinterpret_cast<const int*>(A.model)[i];
  for (int i = tid; i < A.model_n * (int)sizeof(CompDesc) / 4; i += kLatThreads) reinterpret_cast<int*>(comps)[i] = reinterpret_cast<const int*>(A.comps)[i];
  for (int i = tid; i < kNSets * (int)(sizeof(CSet) / sizeof(double)); i += kLatThreads) reinterpret_cast<double*>(W.cs)[i] = 0;
  for (int i = tid; i <= kSolvers * NSL; i += kLatThreads) { W.x[i] = 0; W.f[i] = 0; W.r[i] = 0; W.Z1[i] = 0; W.Z2[i] = 0; }
  if (tid < TB::S) {
    W.tA[tid] = tid ? kRos.A[tid][tid - 1] : 0.0; W.tC[tid] = tid ? kRos.C[tid][tid - 1] : 0.0; W.td[tid] = kRos.d[tid];
    W.tq[tid] = kRos.tslot[tid]; W.tinc[tid] = kRos.incr[tid];
  }
  for (int i = tid; i < kSolvers * NSL; i += kLatThreads) { W.PA[i] = 0; W.PC[i] = 0; W.bP[i] = 0; }
  __syncthreads();
  const bool solver = tid < kSolvers;
  const int n = M.n;
  LGrp g;
  g.gt = tid & (kSolvers - 1); g.lane = tid & 31; g.wq = g.gt >> 5; g.rp = 0;
  g.fc = g.lane < M.npsi ? M.psiComp[g.lane] : (g.lane >= kMaxFun && g.lane - kMaxFun < M.nrho) ? M.rhoComp[g.lane - kMaxFun] : n;
  const int nf = M.npsi > M.nrho ? M.npsi : M.nrho;
  g.ftop = nf > 8 ? 8 : nf > 4 ? 4 : nf > 2 ? 2 : 1;
  // functionals: a warp without rows if there is one, else warp 1 (no head rows, one slot)
  g.fw = n <= 96 ? 3 : 1;
  g.pp = 0; g.act = 0;
  int at[NSL];
#pragma unroll
  for (int s = 0; s < NSL; ++s) {
    const int i = solver ? lat_comp(g.gt, s) : comp_of<4>(g.gt, s);
    if (__any_sync(FULL, i < n)) g.act |= 1u << s;
    if (__any_sync(FULL, i < n && (comps[i < n ? i : 0].phid != CV_ZERO || comps[i < n ? i : 0].psid != CV_ZERO))) g.pp |= 1u << s;
    at[s] = -1;
    for (int c = 0; c < 2; ++c) if (i >= M.chFirst[c] && i <= M.chLast[c]) at[s] = M.chAttach[c];
  }
  const Rows<NSL> R = load_rows<NSL>(g, M, comps);
  LatScan<ST> S;
  {
    const int c0 = 2 * g.wq, c1 = c0 + 1;
    S.pair = c0 < M.nchain;
    const int f0 = S.pair ? M.chFirst[c0] : 0, l0 = S.pair ? M.chLast[c0] : -1;
    const int f1 = c1 < M.nchain ? M.chFirst[c1] : 0, l1 = c1 < M.nchain ? M.chLast[c1] : -1;
    S.n0 = l0 - f0 + 1; S.n1 = l1 - f1 + 1;
    S.i0 = l0 - g.lane; S.i1 = l1 - g.lane;
    S.on0 = S.i0 >= f0; S.on1 = S.i1 >= f1;
    S.j0 = S.on0 ? S.i0 : 0; S.j1 = S.on1 ? S.i1 : 0;
    const int L = S.n0 > S.n1 ? S.n0 : S.n1;
    S.more = L > 8;
#pragma unroll
    for (int q = 0; q < 5; ++q) { S.f0[q] = S.f1[q] = S.b0[q] = S.b1[q] = ST(0); }
    S.d0 = S.d1 = ST(0);
  }
  for (;;) {
    if (tid == 0) W.item = (int)atomicAdd(A.counter, 1u);
    __syncthreads();
    const int slot = W.item;
    __syncthreads();  // every thread has read the slot before the next mode overwrites it
    if (slot >= A.nitems) break;
    const int item = A.order ? A.order[slot] : slot;
    const int c = A.item_cosmo ? A.item_cosmo[item] : 0;
    {
      const int* src = reinterpret_cast<const int*>(A.cosmos + c);
      int* dst = reinterpret_cast<int*>(&W.cdesc);
      for (int q = tid; q < (int)(sizeof(CosmoDesc) / 4); q += kLatThreads) dst[q] = src[q];
    }
    ModeK mk;
    mk.k = A.item_k[item]; mk.k2 = mk.k * mk.k; mk.ik = 1.0 / mk.k; mk.ik2 = mk.ik * mk.ik;
    __syncthreads();
    coef_mode(tid, kLatThreads, W.cs, &W.cdesc, M, mk);
    __syncthreads();
    const double* tab = A.tables + (size_t)c * A.table_stride;
    if (solver) lat_solver<NSL, ST>(A, M, comps, W, g, R, S, at, tab, A.taus ? A.taus + (size_t)c * A.ntau : nullptr, item, mk);
    else lat_companion<NSL, ST>(A, M, W, g, tab, item, mk);
  }
}

template <int NSL, typename ST>
int launch_lat(const PtArgs& A, int num_sms, cudaStream_t stream) {
  const size_t smem = ((sizeof(ModelDesc) + 15) & ~size_t(15)) + (((size_t)A.model_n * sizeof(CompDesc) + 15) & ~size_t(15)) + sizeof(LatMem<NSL, ST>);
  auto kern = pt_lat_kernel<NSL, ST>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return SBZ_ERR_CUDA;
  const int grid = A.nitems < num_sms ? A.nitems : num_sms;
  kern<<<grid > 0 ? grid : 1, kLatThreads, smem, stream>>>(A);
  return cudaGetLastError() == cudaSuccess ? SBZ_OK : SBZ_ERR_CUDA;
}

}  // namespace ptk
}  // namespace sbz
