#pragma once
// Throughput kernel: two to four modes of four warps or eight modes of two warps per SM, for launches of
// many modes per SM.
//
// Such launches are bound by the FP64 pipes (a step of the n = 133 model at the default tolerances is
// about 1,700 FP64 warp instructions, 27k cycles on the four pipes of an SM) if enough modes share an
// SM to hide each other's latency.  The generic kernel's shapes did not: one warp per mode keeps 41 KB
// of shared memory per mode (four modes per SM) and an unrolled step that streams through the
// instruction cache (187k cycles of an SM per step), four warps per mode two modes per SM (64k).  Here
// a mode takes 25 KB at n = 133: arrays have the model's length, what only one phase of the step uses
// shares memory with what only another uses (the stage solutions with the factorisation's inputs, the
// base scalars and the output pass), intermediate coefficient sets have no derivatives, row descriptors
// sit in registers and the cosmology is read through L1.  The step is rolled (one copy of each phase);
// the metric functionals of an operator product are formed by one of a mode's warps.
// Sums keep the order of the generic kernel (the error norm that of the launch shape it stands in for,
// PtArgs::norm_warps), so the results are the same bit for bit in mixed precision.
//
// Modes per SM: the more, the better the FP64 pipes are used and the slower each mode, so a launch takes as
// many as its longest modes allow (thr_modes_per_sm in sbz_pt.cu).  16 cosmologies, k to 0.2 h/Mpc, default
// tolerances, ms (the generic kernel's shape for the launch / 2 / 3 / 4 / 8 modes per SM here):
//   n = 47   1,328 modes 69.5 / 56.8 / 61.7   2,400 122 / - / 72.0 / 77.4   4,800 237 / - / - / 136 / 115
//   n = 133  1,328 modes 79.5 / 78.3 / 85.3   2,400 140 / - / 103 / 104     4,800 276 / - / - / 187 / 183
//   n = 133, k to 0.05: 1,328 45.4 / 44.8 / 34.3   2,400 79.1 / - / 60.4 / 56.3   5,000 491 / - / - / - / 104
#include "sbz_pt_lat.cuh"

namespace sbz {
namespace ptk {


// Shared memory of one mode (pointers into its slice).
template <typename ST>
struct ThrMem {
  double *x, *Us, *csJE, *csM, *B, *dB;  // B, dB inside Us
  ST *r, *Z1, *Z2, *dinv, *sub, *bP, *fA, *bA, *H, *Hinv;
  ST *dd, *sup, *mfw;                    // inside Us
  double *f;                             // inside Us
  struct Small {
    double src[4], fun[4], red[4], ctl[4 + kMaxT], tau1;  // tau1: time of a single-set evaluation
    ST hmul[2], hcorr[2], wS[kWF], fS[4];
    float redf[2][4];
    int ctlf, item;
  }* s;
  int st;  // array stride
};
__host__ __device__ inline int thr_stride(int n) { return (n + 1 + 3) & ~3; }  // one zero entry at n
template <typename ST>
__host__ __device__ inline size_t thr_mode_bytes(int n) {
  const size_t st = thr_stride(n);
  // x, Us | J and E sets, four value sets | r, Z1, Z2, dinv, sub, bP, fA, bA | H, Hinv | small
  size_t us = 8 * st * TB::S;
  const size_t ub = 8 * (kMaxT + 1) * B_COUNT + 3 * st * sizeof(ST);  // what Us also holds (small models)
  if (us < ub) us = ub;
  size_t b = 8 * st + us + 2 * sizeof(CSet) + 4 * 8 * (kNCV + kWF) + 16 * st * sizeof(ST) + 128 * sizeof(ST) + sizeof(typename ThrMem<ST>::Small);
  return (b + 15) & ~size_t(15);
}
template <typename ST>
__device__ inline ThrMem<ST> thr_mem(unsigned char* p, int n) {
  ThrMem<ST> W;
  const size_t st = thr_stride(n);
  W.st = (int)st;
  W.x = reinterpret_cast<double*>(p); p += 8 * st;
  W.Us = reinterpret_cast<double*>(p);
  W.B = W.Us; W.dB = W.Us + kMaxT * B_COUNT;
  W.f = W.Us;
  W.dd = reinterpret_cast<ST*>(W.Us + (kMaxT + 1) * B_COUNT); W.sup = W.dd + st; W.mfw = W.sup + st;
  size_t us = 8 * st * TB::S;
  const size_t ub = 8 * (kMaxT + 1) * B_COUNT + 3 * st * sizeof(ST);
  if (us < ub) us = ub;
  p += us;
  W.csJE = reinterpret_cast<double*>(p); p += 2 * sizeof(CSet);
  W.csM = reinterpret_cast<double*>(p); p += 4 * 8 * (kNCV + kWF);
  ST* q = reinterpret_cast<ST*>(p);
  W.r = q; W.Z1 = q + st; W.Z2 = q + 2 * st; W.dinv = q + 3 * st; W.sub = q + 4 * st; W.bP = q + 5 * st;
  W.fA = q + 6 * st; W.bA = q + 11 * st;
  q += 16 * st;
  W.H = q; W.Hinv = q + 64; q += 128;
  W.s = reinterpret_cast<typename ThrMem<ST>::Small*>(q);
  return W;
}
// A coefficient set: operator coefficients and functional weights with (J, E, output) or without
// (intermediate stage times) τ-derivatives.
struct TSet { const double *cv, *w, *cvd, *wd; };
__device__ __forceinline__ TSet thr_set_je(const double* base, int k) {
  const CSet* c = reinterpret_cast<const CSet*>(base) + k;
  return TSet{c->cv, c->w, c->cvd, c->wd};
}
__device__ __forceinline__ TSet thr_set_mid(const double* csM, int q) {
  const double* p = csM + q * (kNCV + kWF);
  return TSet{p, p + kNCV, nullptr, nullptr};
}

template <int G>
struct TGrp {
  static constexpr int NT = 32 * G;
  int gt, lane, wq, bar, fc, ftop, rp;
  int fw;  // warp that forms the metric functionals
  unsigned pp, act;
};
template <int G>
__device__ __forceinline__ void tsync(const TGrp<G>& g) { bar_sync(g.bar, 32 * G); }
// Slot s starts s warps on, so a partial last slot falls on a warp without the head rows.
template <int G>
__device__ __forceinline__ int thr_comp(int gt, int s) { return s * 32 * G + ((gt + (G == 2 ? 32 : 64) * s) & (32 * G - 1)); }

template <int NSL>
struct TRows {  // indices packed: ip | in << 8 | sp << 16 | dg << 24, coupling to the metric functionals (coefficient | (0: Ψ, 1: Φ̇) << 8) | at << 16
  double A[NSL], C[NSL];
  unsigned a[NSL], b[NSL];
  unsigned ea, eb;  // head rows' extra terms: e0 | e0c << 8 | e1 << 16 | e1c << 24, e3 | e3a << 8 | e3b << 16
};

// Ψ, Φ̇ of x by one warp, published; see lat_matvec for the order of a row's terms.
template <int G, int NSL, typename ST, bool DT, bool DSRC>
__device__ __forceinline__ Fun thr_matvec(const TGrp<G>& g, const ThrMem<ST>& W, const TRows<NSL>& R, const double* x, const TSet& C, int n, double k34,
                                          double (&out)[NSL], double (&dout)[NSL], bool want) {
  const double *cv = C.cv, *cvd = C.cvd;
  Fun F{0, 0, 0, 0};
  const bool uses = g.pp != 0 || (want && g.wq == 0);
  if (g.wq == g.fw) {
    auto sum = [&](const double* w, double& psi, double& rho) {
      double t = w[g.lane] * x[g.fc];
#pragma unroll
      for (int o = 8; o; o >>= 1)
        if (o <= g.ftop) t += __shfl_xor_sync(FULL, t, o);
      psi = t;  // valid on lane 0
      rho = __shfl_down_sync(FULL, t, 16);
    };
    double rho, drho = 0;
    sum(C.w, F.psi, rho);
    if (DT) sum(C.wd, F.dpsi, drho);
    F.phd = phidot(cv, rho, x[0], F.psi);
    if (DT) F.dphd = cvd[CV_PA] * rho + cv[CV_PA] * drho + cvd[CV_PB] * x[0] + cvd[CV_MH] * F.psi + cv[CV_MH] * F.dpsi;
    if (g.lane == 0) {
      W.s->fun[0] = F.psi; W.s->fun[1] = F.phd;
      if (DT) { W.s->fun[2] = F.dpsi; W.s->fun[3] = F.dphd; }
    }
    __syncwarp();
    bar_arrive(g.bar + 1, 32 * G);
  } else if (!uses) {
    bar_arrive(g.bar + 1, 32 * G);
  }
#pragma unroll
  for (int s = 0; s < NSL; ++s) {
    double o = 0, d = 0;
    if ((g.act >> s) & 1u) {
      const unsigned a = R.a[s];
      const int i = thr_comp<G>(g.gt, s);
      const double ax = R.A[s] * x[a & 255] + R.C[s] * x[(a >> 8) & 255], xi = x[i < n ? i : n];
      o = cv[(a >> 16) & 255] * ax + cv[a >> 24] * xi;
      if (DT) d = cvd[(a >> 16) & 255] * ax + cvd[a >> 24] * xi;
      if (s == 0 && g.wq == 0) {
        const unsigned ea = R.ea, eb = R.eb;
        const double x0 = x[(ea >> 8) & 255], x1 = x[ea >> 24], x3 = x[(eb >> 8) & 255] - k34 * x[(eb >> 16) & 255];
        o += cv[ea & 255] * x0 + cv[(ea >> 16) & 255] * x1 + cv[eb & 255] * x3;
        if (DT && !DSRC) d += cvd[ea & 255] * x0 + cvd[(ea >> 16) & 255] * x1 + cvd[eb & 255] * x3;
      }
    }
    out[s] = o;
    if (DT) dout[s] = d;
  }
  if (uses && g.wq != g.fw) bar_sync(g.bar + 1, 32 * G);
  if (want && g.wq == 0) {
    F.psi = W.s->fun[0]; F.phd = W.s->fun[1];
    if (DT) { F.dpsi = W.s->fun[2]; F.dphd = W.s->fun[3]; }
  }
#pragma unroll
  for (int s = 0; s < NSL; ++s)
    if ((g.pp >> s) & 1u) {  // see lat_matvec
      const int fd = R.b[s] & 255, fx = (R.b[s] >> 8) & 1;
      const double v = W.s->fun[fx], c = cv[fd];
      out[s] = __dadd_rn(out[s], __dmul_rn(c, v));
      if (DT) dout[s] = __dadd_rn(dout[s], fma(c, W.s->fun[2 + fx], __dmul_rn(cvd[fd], v)));
    }
  if (DT && DSRC && g.wq == 0) {
    const unsigned ea = R.ea, eb = R.eb;
    const double x0 = x[(ea >> 8) & 255], x1 = x[ea >> 24], x3 = x[(eb >> 8) & 255] - k34 * x[(eb >> 16) & 255];
    dout[0] += cvd[ea & 255] * x0 + cvd[(ea >> 16) & 255] * x1 + cvd[eb & 255] * x3;
  }
  return F;
}

// Coefficients at nt times into sets: the q-th by `put(q)`, derivatives for the last one when dlast.
template <int G, typename ST, typename Put>
__device__ __forceinline__ void thr_coefs(const TGrp<G>& g, const ThrMem<ST>& W, const double* taus, int nt, bool dlast, bool source, const CosmoDesc* cd,
                                          const double* __restrict__ tab, const ModelDesc& M, const ModeK& mk, Put put) {
#pragma unroll 1
  for (int pass = g.wq; 2 * pass < nt; pass += G) {
    const int q = 2 * pass + (g.lane >> 4);
    const bool live = q < nt;
    coef_base(g.lane, live, live && dlast && q == nt - 1, source, live ? taus[q] : 1.0, cd, tab, M.nx, mk, W.B + (live ? q : 0) * B_COUNT, W.dB,
              W.s->src);
  }
  tsync(g);
  const int ne = M.nexpr_t;
  auto one = [&](int q, int e, bool deriv) {
    const CoefExpr& X = cd->expr[e];
    const double *Bq = W.B + q * B_COUNT, *dBq = W.dB;
    const double p0 = Bq[X.b[0]], p1 = Bq[X.b[1]], p2 = Bq[X.b[2]];
    const double q0 = Bq[X.b[3]], q1 = Bq[X.b[4]], q2 = Bq[X.b[5]];
    const double p12 = p1 * p2, q12 = q1 * q2;
    const double val = fma(X.K1, p0 * p12, X.K2 * (q0 * q12));
    const TSet C = put(q);
    const int d = X.dest;
    const_cast<double*>(d < kNCV ? C.cv : C.w - kNCV)[d] = val;
    if (C.cvd) {
      double dval = 0;
      if (deriv) {
        const double dp0 = dBq[X.b[0]], dp1 = dBq[X.b[1]], dp2 = dBq[X.b[2]];
        const double dq0 = dBq[X.b[3]], dq1 = dBq[X.b[4]], dq2 = dBq[X.b[5]];
        const double dP = fma(dp0, p12, p0 * fma(dp1, p2, p1 * dp2));
        const double dQ = fma(dq0, q12, q0 * fma(dq1, q2, q1 * dq2));
        dval = fma(X.K1, dP, X.K2 * dQ);
      }
      const_cast<double*>(d < kNCV ? C.cvd : C.wd - kNCV)[d] = dval;
    }
  };
#pragma unroll 1
  for (int p = g.gt; p < nt * ne; p += (32 * G)) { const int q = p / ne; one(q, p - q * ne, dlast && q == nt - 1); }
  tsync(g);
}

// M⁻¹ on NV vectors in place (r complete on entry, a group barrier at the end): warp w eliminates the chain
// pairs w, w + G, ...; warp 0 solves the head after its first pair (the photon tails).
template <int NV, int G, typename ST>
__device__ __forceinline__ void thr_solve_M(const TGrp<G>& g, const ThrMem<ST>& W, const ModelDesc& M, ST is, ST ihc, ST* v0, ST* v1) {
  const int lane = g.lane, st = W.st;
  if (g.wq == G - 1) {
    const ST a2 = v0[2] * ihc, a1 = (v0[1] - a2) * is, a0 = v0[0] * is;
    ST c0 = 0, c1 = 0, c2 = 0;
    if (NV > 1) { c2 = v1[2] * ihc; c1 = (v1[1] - c2) * is; c0 = v1[0] * is; }
    __syncwarp();
    if (lane == 0) {
      v0[0] = a0; v0[1] = a1; v0[2] = a2;
      if (NV > 1) { v1[0] = c0; v1[1] = c1; v1[2] = c2; }
    }
  }
#pragma unroll 1
  for (int p = g.wq; 2 * p < M.nchain; p += G) {
    const ChainPair c = chain_pair(M, p);
    const int i0 = c.l0 - lane, i1 = c.l1 - lane;
    const bool on0 = i0 >= c.f0, on1 = i1 >= c.f1;
    const int j0 = on0 ? i0 : 11, j1 = on1 ? i1 : 11;  // off-chain lanes read a chain row and select zero
    const ST r0 = v0[j0], r1 = v0[j1];
    ST x0 = on0 ? r0 : ST(0), x1 = on1 ? r1 : ST(0), y0 = ST(0), y1 = ST(0);
    if (NV > 1) { const ST s0 = v1[j0], s1 = v1[j1]; y0 = on0 ? s0 : ST(0); y1 = on1 ? s1 : ST(0); }
    auto fwd = [&](int q) {
      const int d = 1 << q;
      const ST a0 = W.fA[q * st + j0], a1 = W.fA[q * st + j1];
      const ST m0 = on0 ? a0 : ST(0), m1 = on1 ? a1 : ST(0);
      const ST px0 = shfl_up_(x0, d), px1 = shfl_up_(x1, d);
      x0 += m0 * px0; x1 += m1 * px1;
      if (NV > 1) { const ST py0 = shfl_up_(y0, d), py1 = shfl_up_(y1, d); y0 += m0 * py0; y1 += m1 * py1; }
    };
    auto bwd = [&](int q) {
      const int d = 1 << q;
      const ST a0 = W.bA[q * st + j0], a1 = W.bA[q * st + j1];
      const ST m0 = on0 ? a0 : ST(0), m1 = on1 ? a1 : ST(0);
      const ST px0 = __shfl_down_sync(FULL, x0, d), px1 = __shfl_down_sync(FULL, x1, d);
      x0 += m0 * px0; x1 += m1 * px1;
      if (NV > 1) { const ST py0 = __shfl_down_sync(FULL, y0, d), py1 = __shfl_down_sync(FULL, y1, d); y0 += m0 * py0; y1 += m1 * py1; }
    };
    const bool more = c.l0 - c.f0 >= 8 || c.l1 - c.f1 >= 8;
    fwd(0); fwd(1); fwd(2);
    if (more) { fwd(3); fwd(4); }
    if (p == 0) {
      ST hb0 = v0[3 + (lane & 7)], hb1 = NV > 1 ? v1[3 + (lane & 7)] : ST(0);
      const ST hm = lane == 4 ? W.s->hmul[0] : lane == 7 ? W.s->hmul[1] : ST(0);
      const ST c0 = __shfl_sync(FULL, x0, c.l0 - c.f0), c1 = __shfl_sync(FULL, x1, c.l1 - c.f1);
      hb0 -= hm * (lane == 4 ? c0 : c1);
      if (NV > 1) {
        const ST e0 = __shfl_sync(FULL, y0, c.l0 - c.f0), e1 = __shfl_sync(FULL, y1, c.l1 - c.f1);
        hb1 -= hm * (lane == 4 ? e0 : e1);
      }
      ST o0 = 0, o1 = 0;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const ST hq = W.Hinv[(lane & 7) * 8 + q];
        o0 += hq * __shfl_sync(FULL, hb0, q);
        if (NV > 1) o1 += hq * __shfl_sync(FULL, hb1, q);
      }
      if (lane < 8) { v0[3 + lane] = o0; if (NV > 1) v1[3 + lane] = o1; }
    }
    const ST e0 = W.dinv[j0], e1 = W.dinv[j1];
    const ST d0 = on0 ? e0 : ST(0), d1 = on1 ? e1 : ST(0);
    x0 *= d0; x1 *= d1;
    if (NV > 1) { y0 *= d0; y1 *= d1; }
    bwd(0); bwd(1); bwd(2);
    if (more) { bwd(3); bwd(4); }
    if (on0) { v0[i0] = x0; if (NV > 1) v1[i0] = y0; }
    if (on1) { v0[i1] = x1; if (NV > 1) v1[i1] = y1; }
  }
  tsync(g);
}

template <int G, typename ST>
__device__ __forceinline__ void thr_functionals_st(const TGrp<G>& g, const ThrMem<ST>& W, const ST* v, ST& psi, ST& phd) {
  ST t = W.s->wS[g.lane] * v[g.fc];
#pragma unroll
  for (int o = 8; o; o >>= 1)
    if (o <= g.ftop) t += __shfl_xor_sync(FULL, t, o);
  psi = __shfl_sync(FULL, t, 0);
  const ST rho = __shfl_sync(FULL, t, 16);
  phd = W.s->fS[0] * rho + W.s->fS[1] * v[0] + W.s->fS[2] * psi;
}

// Factorisation of M = s I - B for the Jacobian set C: see ptk::factorize.
template <int G, int NSL, typename ST>
__device__ __forceinline__ void thr_factorize(const TGrp<G>& g, const ThrMem<ST>& W, const TRows<NSL>& R, const TSet& C, const CompDesc* __restrict__ comps,
                                              const ModelDesc& M, double k, double h, double s, ST& is, ST& ihc, ST (&S4)[4]) {
  const int lane = g.lane, n = M.n, st = W.st;
  const double* cv = C.cv;
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) {
    const int i = thr_comp<G>(g.gt, sl);
    if (i < n) {
      const unsigned a = R.a[sl], b = R.b[sl];
      const double spv = cv[(a >> 16) & 255];
      W.dd[i] = to_st<ST>(s - cv[a >> 24]);
      W.sup[i] = to_st<ST>(-spv * R.C[sl]);
      W.sub[i] = to_st<ST>(-spv * R.A[sl]);
      const ST c = to_st<ST>(cv[b & 255]);
      W.Z1[i] = (b >> 8) & 1 ? c : ST(0);
      W.Z2[i] = (b >> 8) & 1 ? ST(0) : c;
    }
  }
  if (g.wq == 0) W.s->wS[lane] = to_st<ST>(C.w[lane]);
  else if (g.wq == 1 && lane < 3) W.s->fS[lane] = to_st<ST>(cv[lane == 0 ? CV_PA : lane == 1 ? CV_PB : CV_MH]);
  tsync(g);
  if (g.wq == 0) {
    if (lane < M.nchain) {
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
      if (lane < 2) {
        const ST hm = W.sup[M.chAttach[lane]] * dn;
        W.s->hmul[lane] = hm;
        W.s->hcorr[lane] = hm * W.sub[first];
      }
    }
  } else if (g.wq == G - 1 && lane >= 16 && lane < 24) {  // assemble head row 3 + j
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
  is = to_st<ST>(h * TB::gam);
  ihc = lat_rcp<ST>(to_st<ST>(s - cv[CV_MH]));
  tsync(g);
  // Kogge-Stone multipliers of the chains, one per warp and pass; the head inverse on warp 0
#pragma unroll 1
  for (int ch = g.wq > 0 ? g.wq - 1 : M.nchain; ch < M.nchain; ch += G - 1) {
    const int first = M.chFirst[ch], last = M.chLast[ch], L = last - first + 1, i = last - lane;
    const bool on = i >= first;
    const int j = on ? i : 11;
    const ST e = W.dinv[j], m = W.mfw[j], u = W.sub[j];
    ST a = (on && lane > 0) ? -m : ST(0), c = on ? -e * u : ST(0);
#pragma unroll
    for (int q = 0; q < 5; ++q) {
      const int d = 1 << q;
      const ST p = shfl_up_(a, d), z = __shfl_down_sync(FULL, c, d);
      const bool up = lane >= d, in = lane + d < L;
      if (on) { W.fA[q * st + i] = up ? a : ST(0); W.bA[q * st + i] = in ? c : ST(0); }
      if (up) a *= p;
      if (in) c *= z;
    }
    if (on) W.bP[i] = c;
  }
  if (g.wq == 0) {
    const int q = lane & 15;
    ST col[8];
#pragma unroll
    for (int r = 0; r < 8; ++r) col[r] = q < 8 ? W.H[r * 8 + q] : ST(r == q - 8 ? 1 : 0);
    if (q == 4) col[4] -= W.s->hcorr[0];
    if (q == 7) col[7] -= W.s->hcorr[1];
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
  tsync(g);
  thr_solve_M<2, G, ST>(g, W, M, is, ihc, W.Z1, W.Z2);
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) {  // head-value terms of the chain back substitutions (own rows)
    const int i = thr_comp<G>(g.gt, sl);
    const int at = (int)((R.b[sl] >> 16) & 255);
    if (i < n && at) { const ST P = W.bP[i]; W.Z1[i] += P * W.Z1[at]; W.Z2[i] += P * W.Z2[at]; }
  }
  ST psi1, p1, psi2, p2;
  thr_functionals_st(g, W, W.Z1, psi1, p1);
  thr_functionals_st(g, W, W.Z2, psi2, p2);
  const ST a = 1 - p1, b = -p2, c = -psi1, d = 1 - psi2;
  const ST idet = sizeof(ST) == 8 ? lat_rcp<ST>(a * d - b * c) : ST(1) / (a * d - b * c);
  S4[0] = d * idet; S4[1] = -b * idet; S4[2] = -c * idet; S4[3] = a * idet;
}

// Σ over the rows of v² in the order of the generic kernel with `nw` warps per mode: there warp w keeps, per
// lane, the squares of its 32-row blocks in slot order, sums its lanes by a butterfly, and the warps' sums
// are added in order.  v in shared memory (q), complete; every thread gets the sum.
template <int G>
__device__ __forceinline__ double thr_norm2(const TGrp<G>& g, double* red, const double* q, int n, int nw) {
  auto add = [&](double& e, int block) {
    const int i = 32 * block + g.lane;
    if (i < n) { const double v = q[i]; e = fma(v, v, e); }
  };
  if (nw == 1) {
    double e = 0;
#pragma unroll 1
    for (int b = 0; 32 * b < n; ++b) add(e, b);
    return warp_sum(e);
  }
#pragma unroll 1
  for (int w = g.wq; w < nw; w += G) {
    double e = 0;
    if (nw == 2) { add(e, w); add(e, 2 + (w ^ 1)); add(e, 4 + w); }
    else { add(e, w); add(e, 4 + ((w + 3) & 3)); }
    e = warp_sum(e);
    if (g.lane == 0) red[w] = e;
  }
  tsync(g);
  double s = 0;
  for (int w = 0; w < nw; ++w) s += red[w];
  return s;
}

template <int G, int NSL, typename ST>
__device__ void thr_emit(const TGrp<G>& g, const ThrMem<ST>& W, const TRows<NSL>& R, const PtArgs& A, const CosmoDesc* cd, const double* tab,
                         const ModelDesc& M, const ModeK& mk, double tau, const double (&y)[NSL], int item, int j) {
  const int n = M.n;
  if (A.output == SBZ_OUT_STATE) {
    double* o = A.out + ((size_t)item * A.ntau + j) * n;
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(g.gt, sl); if (i < n) o[i] = y[sl]; }
    return;
  }
  if (A.output != SBZ_OUT_SOURCES && A.output != SBZ_OUT_SOURCES4 && A.output != SBZ_OUT_FACTORS) return;
  const TSet C = thr_set_je(W.csM, 0);  // the intermediate sets are free between steps
  const double k34 = 0.75 * mk.k;
  for (int i = g.gt; i < (int)(sizeof(CSet) / 8); i += (32 * G)) W.csM[i] = 0;
  tsync(g);
  coef_mode_set(g.gt, (32 * G), const_cast<double*>(C.cv), const_cast<double*>(C.w), cd, M, mk);
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(g.gt, sl); if (i < n) W.x[i] = y[sl]; }
  if (g.gt == 0) W.s->tau1 = tau;
  tsync(g);
  thr_coefs(g, W, &W.s->tau1, 1, true, true, cd, tab, M, mk, [&](int) { return C; });
  const double kd = W.B[B_KD];
  double fy[NSL], dJy[NSL], Jf[NSL], un[NSL];
  const Fun F = thr_matvec<G, NSL, ST, true, true>(g, W, R, W.x, C, n, k34, fy, dJy, true);
  tsync(g);  // the base scalars share memory with f
#pragma unroll
  for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(g.gt, sl); if (i < n) W.f[i] = fy[sl]; }
  if (g.gt == 0) W.f[n] = 0;
  tsync(g);
  const Fun Ff = thr_matvec<G, NSL, ST, false, false>(g, W, R, W.f, C, n, k34, Jf, un, true);
  if (g.wq == 0) {
    const double gv = dJy[0] + Jf[0];
    const double g7 = __shfl_sync(FULL, gv, 7), g8 = __shfl_sync(FULL, gv, 8), g10 = __shfl_sync(FULL, gv, 10);
    if (g.gt == 0) write_output(A, cd, mk, tau, W.x, W.f, W.s->src, kd, F.psi, F.phd, F.dpsi + Ff.psi, (g8 + g10) + g7, item, j);
  }
  tsync(g);
}

template <int G, int NSL, typename ST>
__device__ void thr_body(const PtArgs& A, const ModelDesc& M, const CompDesc* __restrict__ comps, const ThrMem<ST>& W, TGrp<G>& g, const TRows<NSL>& R) {
  const int gt = g.gt, n = M.n;
  const double rtol = A.rtol, atol = A.atol, inv_n = 1.0 / n;
  const int nw = A.norm_warps;
  for (int i = gt; i < (int)(2 * sizeof(CSet) / 8); i += (32 * G)) W.csJE[i] = 0;
  if (gt == 0) { W.x[n] = 0; W.r[n] = 0; W.Z1[n] = 0; W.Z2[n] = 0; }
  for (;;) {
    tsync(g);
    if (gt == 0) W.s->item = (int)atomicAdd(A.counter, 1u);
    tsync(g);
    const int slot = W.s->item;
    if (slot >= A.nitems) break;
    const int item = A.order ? A.order[slot] : slot;
    const int c = A.item_cosmo ? A.item_cosmo[item] : 0;
    const CosmoDesc* cd = A.cosmos + c;
    const double* tab = A.tables + (size_t)c * A.table_stride;
    const double* taus = A.taus ? A.taus + (size_t)c * A.ntau : nullptr;
    ModeK mk;
    mk.k = A.item_k[item]; mk.k2 = mk.k * mk.k; mk.ik = 1.0 / mk.k; mk.ik2 = mk.ik * mk.ik;
    const double k = mk.k, k34 = 0.75 * k;
    const double tend = cd->tau0;
    double t = fmin(fmax(A.item_tau_ini[item], cd->tau_start), tend);
    int status = SBZ_OK;
    int64_t nacc = 0, nrej = 0;
    double y[NSL], f0[NSL], ft[NSL];
    int sJ = 0;  // index of the Jacobian set in csJE; the step-end set is the other
    // the mode's constant coefficients into the intermediate sets (again after an output pass, which uses
    // their memory)
    auto mid_sets = [&]() {
      for (int i = gt; i < 4 * (kNCV + kWF); i += (32 * G)) W.csM[i] = 0;
      tsync(g);
      for (int q = 0; q < 4; ++q) { const TSet C = thr_set_mid(W.csM, q); coef_mode_set(gt, (32 * G), const_cast<double*>(C.cv), const_cast<double*>(C.w), cd, M, mk); }
    };
    for (int q = 0; q < 2; ++q) { const TSet C = thr_set_je(W.csJE, q); coef_mode_set(gt, (32 * G), const_cast<double*>(C.cv), const_cast<double*>(C.w), cd, M, mk); }
    auto one_set = [&](double tau, int set, bool deriv) {  // one time into J/E set `set`
      if (gt == 0) W.s->tau1 = tau;
      tsync(g);
      const TSet C = thr_set_je(W.csJE, set);
      thr_coefs(g, W, &W.s->tau1, 1, deriv, false, cd, tab, M, mk, [&](int) { return C; });
    };
    one_set(t, 1, false);
    {
      const IcScal ic = ic_scalars(g.lane, M, cd, W.B, k, t);
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) {
        const int i = thr_comp<G>(gt, sl);
        const double v = i < n ? ic_value(i, M, cd, W.B, ic, k) : 0.0;
        y[sl] = v;
        if (i < n) W.x[i] = v;
      }
      tsync(g);
      // Φ from k²(Φ - Ψ) = 12πa²Π with the initial shears: Ψ(y) is linear with unit weight on Φ
      double psi0;
      {
        double tt = thr_set_je(W.csJE, 1).w[g.lane] * W.x[g.fc];
#pragma unroll
        for (int o = 8; o; o >>= 1) tt += __shfl_xor_sync(FULL, tt, o);
        psi0 = __shfl_sync(FULL, tt, 0);
      }
      tsync(g);
      if (gt == 0) { y[0] = ic.Psi - psi0; W.x[0] = y[0]; }
      tsync(g);
    }
    int jout = 0;
    if (taus) {
      while (jout < A.ntau && taus[jout] <= t) {
        if (taus[jout] < t) zero_output(A, gt, (32 * G), n, item, jout);
        else thr_emit(g, W, R, A, cd, tab, M, mk, t, y, item, jout);
        ++jout;
      }
    }
    if (t < tend) {
      mid_sets();
      one_set(t, sJ, true);
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.x[i] = y[sl]; }
      tsync(g);
      thr_matvec<G, NSL, ST, true, false>(g, W, R, W.x, thr_set_je(W.csJE, sJ), n, k34, f0, ft, false);
      double h;
      {
        auto norm = [&](const double (&v)[NSL]) {
          tsync(g);
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.Us[i] = v[sl]; }
          tsync(g);
          return thr_norm2(g, W.s->red, W.Us, n, nw);
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
        tsync(g);
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.x[i] = y[sl] + h0 * f0[sl]; }
        one_set(t + h0, sJ ^ 1, false);
        double f1[NSL], un[NSL];
        thr_matvec<G, NSL, ST, false, false>(g, W, R, W.x, thr_set_je(W.csJE, sJ ^ 1), n, k34, f1, un, false);
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) { const double sk = atol + fabs(y[sl]) * rtol; q0[sl] = (f1[sl] - f0[sl]) / (h0 * sk); }
        const double d2 = sqrt(norm(q0) * inv_n);
        const double mx = fmax(d1, d2);
        const double h1 = (mx <= 1e-15 || !isfinite(mx)) ? fmax(1e-6, 1e-3 * h0) : pow(0.01 / mx, 0.2);
        h = fmin(100 * h0, h1);
        if (!isfinite(h) || h <= 0) h = 1e-6 * fmax(1.0, t);
      }
      constexpr double kLogErrFloor = -9.210340371976184;  // log(1e-4): the controller's floor on errold
      double lerrold = kLogErrFloor;
      bool rejected = false, nonfinite = false;
      int64_t iters = 0;
      auto publish = [&](double hp, double tc) {  // warp 1
        double inv = 1.0 / (g.lane == 1 ? hp * TB::gam : hp);
        const bool done = !(tc < tend);
        const double left = tend - tc;
        if (tc + 1.01 * hp >= tend) { hp = left; inv = 1.0 / (g.lane == 1 ? hp * TB::gam : hp); }
        const bool tiny = !(hp > 1e-14 * tc);
        const double te = (hp == left) ? tend : tc + hp;
        double cs = 0;
#pragma unroll
        for (int q = 1; q < TB::NTIME; ++q) {
          int st = 1;
#pragma unroll
          for (int i = 1; i < TB::S; ++i) if (TB::tslot(i) == q) st = i;
          if (g.lane == 3 + q) cs = TB::c(st);
        }
        const double ts = tc + cs * hp;
        double* ctl = W.s->ctl;
        if (g.lane == 0) { W.s->ctlf = (done ? 1 : 0) | (tiny ? 2 : 0); ctl[0] = hp; ctl[1] = inv; ctl[3] = te; ctl[4 + TB::NTIME - 1] = te; }
        if (g.lane == 1) ctl[2] = inv;
        if (g.lane >= 4 && g.lane < 4 + TB::NTIME - 1) ctl[g.lane] = ts;
      };
      tsync(g);
      if (g.wq == 1) publish(h, t);
      for (;;) {
        tsync(g);
        const int fl = W.s->ctlf;
        if (fl & 1) break;
        if (++iters > A.maxiters) { status = SBZ_MAXITERS; break; }
        if (fl & 2) { status = nonfinite ? SBZ_NONFINITE : SBZ_DTMIN; break; }
        h = W.s->ctl[0];
        const double ih = W.s->ctl[1], s = W.s->ctl[2], tn = W.s->ctl[3];
        const TSet CJ = thr_set_je(W.csJE, sJ);
        thr_coefs(g, W, W.s->ctl + 4, TB::NTIME, true, false, cd, tab, M, mk,
                  [&](int q) { return q == TB::NTIME - 1 ? thr_set_je(W.csJE, sJ ^ 1) : thr_set_mid(W.csM, q); });
        ST is, ihc, S4[4];
        thr_factorize(g, W, R, CJ, comps, M, k, h, s, is, ihc, S4);
        double b[NSL], Y[NSL], Ul[NSL], un[NSL];
        float isk[NSL];
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) isk[sl] = 1.0f / f64_to_f32(atol + rtol * fabs(y[sl]));
        int rk = A.refine;
        int nst;
        asm volatile("mov.u32 %0, %1;" : "=r"(nst) : "n"(TB::S));
#pragma unroll 1
        for (int stg = 0; stg < nst; ++stg) {
          if (stg == 0) {
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) b[sl] = fma(h * TB::d(0), ft[sl], f0[sl]);
          } else {
            const bool inc = kRos.incr[stg] != 0;
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) {
              const int i = thr_comp<G>(gt, sl);
              if ((g.act >> sl) & 1u) {
                const double* u = W.Us + (i < n ? i : 0);
                double v;
                if (inc) {
                  v = Y[sl] + Ul[sl];
                } else {
                  v = y[sl];
#pragma unroll 2
                  for (int j = 0; j < stg; ++j) v = fma(kRos.A[stg][j], u[j * W.st], v);
                }
                Y[sl] = v;
                if (i < n) W.x[i] = v;
              }
            }
            tsync(g);
            const int q = kRos.tslot[stg];
            double Fv[NSL];
            thr_matvec<G, NSL, ST, false, false>(g, W, R, W.x, q < TB::NTIME ? thr_set_mid(W.csM, q - 1) : thr_set_je(W.csJE, sJ ^ 1), n, k34, Fv, un, false);
            const bool hd = kRos.hasd[stg] != 0;
            const double hdst = h * kRos.d[stg];
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) {
              if (!((g.act >> sl) & 1u)) { b[sl] = 0; continue; }
              const int i = thr_comp<G>(gt, sl);
              const double* u = W.Us + (i < n ? i : 0);
              double cu = 0;
#pragma unroll 2
              for (int j = 0; j < stg; ++j) cu = fma(kRos.C[stg][j], u[j * W.st], cu);
              b[sl] = fma(ih, cu, Fv[sl]);
              if (hd) b[sl] = fma(hdst, ft[sl], b[sl]);
            }
          }
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.r[i] = to_st<ST>(b[sl]); }
          float c1 = 1e30f;
          for (int it = 0;; ++it) {
            tsync(g);
            thr_solve_M<1, G, ST>(g, W, M, is, ihc, W.r, W.r);
            ST psi, ph;
            thr_functionals_st(g, W, W.r, psi, ph);
            const ST t0 = fma(S4[1], psi, S4[0] * ph), t1 = fma(S4[3], psi, S4[2] * ph);
            float cm = 0.0f;
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) {
              const int i = thr_comp<G>(gt, sl), ic = i < n ? i : 0, at = (int)((R.b[sl] >> 16) & 255);
              const ST ri = W.r[ic];
              ST rh = ri;
              if (at) rh = fma(W.bP[ic], W.r[at], ri);
              const ST u = i < n ? fma(W.Z2[ic], t1, fma(W.Z1[ic], t0, rh)) : ST(0);
              if (it == 0) Ul[sl] = from_st(u);
              else if (i < n) { Ul[sl] += from_st(u); cm = fmaxf(cm, fabsf((float)u) * isk[sl]); }
            }
            if (it > 0) {
              const int r = it - 1;
              const bool first = r == 0 && stg == 0;
              if (r + 1 < rk || first) {
                const unsigned m = __reduce_max_sync(FULL, __float_as_uint(cm));
                if (g.lane == 0) W.s->redf[g.rp][g.wq] = __uint_as_float(m);
                tsync(g);
                float mx = 0;
#pragma unroll
                for (int w = 0; w < G; ++w) mx = fmaxf(mx, W.s->redf[g.rp][w]);
                g.rp ^= 1;
                if (first) c1 = mx;
                if (r + 1 < rk && mx < 1e-3f) break;
              }
            }
            if (it >= rk) break;
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.x[i] = Ul[sl]; }
            tsync(g);
            double JU[NSL];
            thr_matvec<G, NSL, ST, false, false>(g, W, R, W.x, CJ, n, k34, JU, un, false);
#pragma unroll
            for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.r[i] = to_st<ST>(b[sl] - fma(s, Ul[sl], -JU[sl])); }
          }
          if (stg == 0) rk = (A.refine > 0 && c1 < A.refine_skip) ? 0 : A.refine;
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.Us[stg * W.st + i] = Ul[sl]; }
        }
        // new state and the FP64 error norm of the last stage; its weighted rows go through r's place in x
        double y1[NSL];
#pragma unroll
        for (int sl = 0; sl < NSL; ++sl) {
          const int i = thr_comp<G>(gt, sl);
          y1[sl] = Y[sl] + Ul[sl];
          if (i < n) {
            const double sk = atol + rtol * __longlong_as_double(max(dkey(fabs(y[sl])), dkey(fabs(y1[sl]))));
            W.x[i] = Ul[sl] / sk;
          }
        }
        tsync(g);
        const double err2 = thr_norm2(g, W.s->red, W.x, n, nw) * inv_n;
        if ((unsigned long long)dkey(err2) <= (unsigned long long)dkey(1.0)) {
          tsync(g);
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.x[i] = y1[sl]; }
          tsync(g);
          if (g.wq == 1) {
            const double lerr = 0.5 * log(dmax(err2, 1e-20));
            double fac = 0.9 * exp(-TB::beta1 * lerr + TB::beta2 * lerrold);
            fac = dmin(10.0, dmax(0.2, fac));
            if (rejected) fac = dmin(fac, 1.0);
            lerrold = dmax(lerr, kLogErrFloor);
            publish(h * fac, tn);
          }
          sJ ^= 1;
          thr_matvec<G, NSL, ST, true, false>(g, W, R, W.x, thr_set_je(W.csJE, sJ), n, k34, f0, ft, false);
          if (taus && jout < A.ntau && dkey(taus[jout]) <= dkey(tn)) {
            double K[TB::NDENSE][NSL];
#pragma unroll
            for (int r = 0; r < TB::NDENSE; ++r)
#pragma unroll
              for (int sl = 0; sl < NSL; ++sl) {
                const int i = thr_comp<G>(gt, sl);
                double v = 0;
#pragma unroll
                for (int j = 0; j < TB::S; ++j) {
                  if (TB::dense(r, j) == 0.0) continue;
                  v = fma(TB::dense(r, j), W.Us[j * W.st + (i < n ? i : 0)], v);
                }
                K[r][sl] = v;
              }
            tsync(g);  // x readers of the f1 product and readers of Us are done
            while (jout < A.ntau && dkey(taus[jout]) <= dkey(tn)) {
              const double tau = taus[jout];
              const double th = (tau - t) / (tn - t), th1 = 1.0 - th;
              double yo[NSL];
#pragma unroll
              for (int sl = 0; sl < NSL; ++sl) yo[sl] = th1 * y[sl] + th * (y1[sl] + th1 * (K[0][sl] + th * (K[1][sl] + th * K[2][sl])));
              thr_emit(g, W, R, A, cd, tab, M, mk, tau, yo, item, jout);
              ++jout;
            }
            mid_sets();
          }
          t = tn;
#pragma unroll
          for (int sl = 0; sl < NSL; ++sl) y[sl] = y1[sl];
          ++nacc;
          rejected = false; nonfinite = false;
        } else {
          ++nrej;
          rejected = true;
          if ((dkey(err2) & 0x7ff0000000000000ll) == 0x7ff0000000000000ll) nonfinite = true;  // inf or NaN
          if (g.wq == 1) publish(nonfinite ? 0.2 * h : h * dmax(0.2, 0.9 * exp(-0.5 * TB::rej * log(err2))), t);
        }
      }
    }
    if (taus) for (; jout < A.ntau; ++jout) zero_output(A, gt, (32 * G), n, item, jout);
    bool finite = true;
#pragma unroll
    for (int sl = 0; sl < NSL; ++sl) if (thr_comp<G>(gt, sl) < n && !isfinite(y[sl])) finite = false;
    tsync(g);
    finite = __all_sync(FULL, finite);
    if (g.lane == 0) W.s->redf[0][g.wq] = finite ? 0.0f : 1.0f;
    tsync(g);
    float bad = 0;
#pragma unroll
    for (int w = 0; w < G; ++w) bad += W.s->redf[0][w];
    finite = bad == 0.0f;
    if (status == SBZ_OK && !finite) status = SBZ_NONFINITE;
    if (A.output == SBZ_OUT_DELTA_M) {
#pragma unroll
      for (int sl = 0; sl < NSL; ++sl) { const int i = thr_comp<G>(gt, sl); if (i < n) W.x[i] = y[sl]; }
      one_set(tend, 1, false);
      if (g.wq == 0) {
        const double d = delta_m(g.lane, M, cd, W.B, W.x, mk);
        if (gt == 0) A.out[item] = d;
      }
    }
    if (gt == 0) {
      if (A.status) A.status[item] = status;
      if (A.steps) { A.steps[2 * item] = nacc; A.steps[2 * item + 1] = nrej; }
    }
  }
}

// Shared memory of a block of `modes` modes.
template <typename ST>
__host__ inline size_t thr_block_bytes(int n, int modes) { return ((sizeof(ModelDesc) + 15) & ~size_t(15)) + modes * thr_mode_bytes<ST>(n); }
// Modes of two warps that an SM holds (two blocks of four, or one: 228 KB of shared memory, 1 KB of it per block for the
// driver).  Two to four modes of four warps fit at every size.
template <typename ST>
__host__ inline int thr2_resident(int n) { return 2 * (thr_block_bytes<ST>(n, 4) + 1024) <= 228 * 1024 ? 8 : 4; }

// NT threads per block (NT / (32 G) modes), MINB blocks per SM: 128 x 3 keeps 168 registers per thread (no spills but
// 16 bytes in FP64), 256 x 2 runs 16 warps per SM on 128 (spills of 124 to 140 bytes with one row per lane, 378 (FP64
// 724) with two, 1,052 with three: two-warp modes above 128 equations).
template <int G, int NT, int MINB, int NSL, typename ST>
__global__ void __launch_bounds__(NT, MINB) pt_thr_kernel(PtArgs A) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  ModelDesc& M = *reinterpret_cast<ModelDesc*>(smem_raw);
  constexpr size_t mb = (sizeof(ModelDesc) + 15) & ~size_t(15);
  const int tid = threadIdx.x;
  for (int i = tid; i < (int)sizeof(ModelDesc) / 4; i += blockDim.x) reinterpret_cast<int*>(&M)[i] = reinterpret_cast<const int*>(A.model)[i];
  __syncthreads();
  const int grp = tid / (32 * G), n = M.n;
  const ThrMem<ST> W = thr_mem<ST>(smem_raw + mb + grp * thr_mode_bytes<ST>(n), n);
  TGrp<G> g;
  g.gt = tid & ((32 * G) - 1); g.lane = tid & 31; g.wq = g.gt >> 5; g.bar = 1 + 2 * grp; g.rp = 0;
  g.fc = g.lane < M.npsi ? M.psiComp[g.lane] : (g.lane >= kMaxFun && g.lane - kMaxFun < M.nrho) ? M.rhoComp[g.lane - kMaxFun] : n;
  const int nf = M.npsi > M.nrho ? M.npsi : M.nrho;
  g.ftop = nf > 8 ? 8 : nf > 4 ? 4 : nf > 2 ? 2 : 1;
  g.fw = G == 4 && n <= 96 ? 3 : 1;  // a warp without rows if there is one, else not the head rows' warp
  g.pp = 0; g.act = 0;
  TRows<NSL> R;
#pragma unroll
  for (int s = 0; s < NSL; ++s) {
    const int i = thr_comp<G>(g.gt, s);
    const bool on = i < n;
    const CompDesc& D = A.comps[on ? i : 0];
    R.A[s] = on ? D.A : 0.0; R.C[s] = on ? D.C : 0.0;
    int at = 0;
    for (int c = 0; c < 2; ++c) if (i >= M.chFirst[c] && i <= M.chLast[c]) at = M.chAttach[c];
    R.a[s] = on ? (unsigned)D.ip | (unsigned)D.inx << 8 | (unsigned)D.sp << 16 | (unsigned)D.dg << 24 : (unsigned)n | (unsigned)n << 8;
    const unsigned fx = D.psid != CV_ZERO ? 0u : 1u;  // no row has both couplings
    R.b[s] = on ? (unsigned)(fx ? D.phid : D.psid) | fx << 8 | (unsigned)at << 16 : 0u;
    if (__any_sync(FULL, on)) g.act |= 1u << s;
    if (__any_sync(FULL, on && (D.phid != CV_ZERO || D.psid != CV_ZERO))) g.pp |= 1u << s;
  }
  {
    const bool on = g.gt < n && g.gt < 32;
    const CompDesc& D = A.comps[on ? g.gt : 0];
    const bool drag = D.dx != CV_ZERO;
    R.ea = (unsigned)D.e0 | (unsigned)D.e0c << 8 | (unsigned)D.e1 << 16 | (unsigned)D.e1c << 24;
    R.eb = (unsigned)(drag ? D.dx : D.e2) | (unsigned)(drag ? D.dxa : D.e2c) << 8 | (unsigned)(drag ? D.dxb : n) << 16;
  }
  thr_body<G, NSL, ST>(A, M, A.comps, W, g, R);
}

template <int G, int NT, int MINB, int NSL, typename ST>
int launch_thr(const PtArgs& A, int max_blocks, int num_sms, cudaStream_t stream) {
  constexpr int modes = NT / (32 * G);
  const size_t smem = thr_block_bytes<ST>(A.model_n, modes);
  auto kern = pt_thr_kernel<G, NT, MINB, NSL, ST>;
  if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return SBZ_ERR_CUDA;
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, NT, smem) != cudaSuccess) return SBZ_ERR_CUDA;
  if (per_sm > max_blocks) per_sm = max_blocks;
  if (per_sm < 1) per_sm = 1;
  const int want = (A.nitems + modes - 1) / modes;
  const int grid = want < num_sms * per_sm ? want : num_sms * per_sm;
  kern<<<grid > 0 ? grid : 1, NT, smem, stream>>>(A);
  return cudaGetLastError() == cudaSuccess ? SBZ_OK : SBZ_ERR_CUDA;
}

}  // namespace ptk
}  // namespace sbz
