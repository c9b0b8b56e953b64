// Line-of-sight kernels.
//
//   SphericalBesselCache (src/observables/angular.jl:18-26): table of j_l(x) and j_l'(x) at the
//     requested l on x = range(0, xmax, length = trunc(xmax/dx)) (+ a duplicated end point),
//     contiguous in l.  Built here by one thread per x with recurrences in l (upward where
//     l < x, Miller's downward recurrence normalised by j_0 or j_1 elsewhere).
//   cache evaluation (angular.jl:29-48): linear or cubic Hermite in x; the Hermite slopes are
//     scaled by the requested dx, as in the reference.
//   los_integrate (angular.jl:109-185): trapezoid in τ of S(τ,k) j_l(k(τ0-τ)); threads over l (of one
//     or a few k), so every table read is a coalesced row segment; Limber branch for l >= l_limber.
//   spectrum_cmb k-integral (angular.jl:198-223): natural cubic spline through (0,0) and the
//     integrand values, integrated exactly: a weighted sum over k (weights from one tridiagonal solve on
//     the host); the allocation-free entry factorises the system once and every l runs the two sweeps.
#include <cuda_runtime.h>
#include <algorithm>
#include <cstdint>
#include <cmath>
#include "sbz_los.cuh"

namespace sbz {
namespace {

// (2 l + 1)-like integers as doubles by integer operations (the FP64 pipe, which would convert them, is
// what bounds the recurrences); n >= 1.
__device__ __forceinline__ double int_as_f64(unsigned n) {
  const int e = 31 - __clz(n);
  return __longlong_as_double((long long)(((unsigned long long)(1022 + e) << 52) + ((unsigned long long)n << (52 - e))));
}

// Table of j_l and j_l' (and their FP32 copy): one thread per x runs the recurrence in l, two FP64
// instructions per l (the coefficient's product and one FMA).  A warp collects 16 multipoles of its 32
// points in shared memory and writes them as 128-byte row pieces; stored straight from the threads,
// every value was a 32-byte sector of its own, and the Miller part rescaled its rows in place.  cf:
// l/(2l+1), (l+1)/(2l+1) per multipole (j_l' = l/(2l+1) j_{l-1} - (l+1)/(2l+1) j_{l+1}).  Bound: the FP64
// pipes, 2 l_max + 4 nl warp instructions per 32 points (1.0 ms of FP64 issue for 200 multipoles to
// 2,500 on 119k points; 12.1 ms before).
constexpr int kBesTile = 16;
__global__ void __launch_bounds__(128) bessel_table_kernel(BesselDev J, const int* __restrict__ ls, const double* __restrict__ cf, int Lmax) {
  __shared__ double ty[4][kBesTile][33], td[4][kBesTile][33];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int N = J.nx - 1;  // last row duplicates row N-1
  const int ix0 = (blockIdx.x * 4 + warp) * 32, ix = ix0 + lane;
  if (ix0 >= N) return;
  const int nl = J.nl, L = Lmax + 1;  // one above the largest l (for the derivative)
  const bool live = ix < N;
  const double xr = !live ? 1.0 : ix == N - 1 ? J.xmax : ix * J.step;
  const bool zero = xr == 0.0;
  const double x = zero ? 1.0 : xr;
  const bool up = x > L && !zero;  // upward recurrence, stable for l < x; Miller's downward one elsewhere
  const unsigned mup = __ballot_sync(0xffffffffu, live && up), mdn = __ballot_sync(0xffffffffu, live && !up);
  double s, c;
  sincos(x, &s, &c);
  const double ix1 = 1.0 / x;
  const double j0 = s * ix1, j1 = (s * ix1 - c) * ix1;
  auto flush = [&](int q0, unsigned rows) {  // multipoles q0 .. q0 + 15 of the rows in `rows`
    __syncwarp();
    const int q = lane & 15, nq = min(kBesTile, nl - q0);
    for (int r = lane >> 4; r < 32; r += 2) {
      if (!((rows >> r) & 1u) || q >= nq) continue;
      const double v = ty[warp][q][r], d = td[warp][q][r];
      for (int row = ix0 + r, last = 0; last < 2; ++last) {
        const size_t o = (size_t)row * nl + q0 + q;
        J.y[o] = v;
        if (J.hermite) J.dy[o] = d;
        J.yf2[o] = make_float2((float)v, J.hermite ? (float)d : 0.0f);
        if (row != N - 1) break;
        row = N;  // the duplicated end point
      }
    }
    __syncwarp();
  };
  auto put = [&](int q, int l, double v, double d) {
    if (zero) { v = l == 0 ? 1.0 : 0.0; d = l == 1 ? 1.0 / 3.0 : 0.0; }
    ty[warp][q & 15][lane] = v;
    td[warp][q & 15][lane] = d;
  };
  if (mup) {
    double jm = c * ix1, jc = j0, jn = j1;  // j_{l-1}, j_l, j_{l+1} at l = 0
    int q = 0, lq = ls[0];
    for (int l = 0; l <= Lmax; ++l) {
      if (l == lq) {
        put(q, l, jc, l == 0 ? -jn : fma(cf[2 * q], jm, -(cf[2 * q + 1] * jn)));
        if ((q & 15) == 15 || q == nl - 1) flush(q & ~15, mup);
        lq = ++q < nl ? ls[q] : -1;
      }
      const double jnn = fma(int_as_f64(2 * l + 3) * ix1, jn, -jc);
      jm = jc; jc = jn; jn = jnn;
    }
  }
  if (mdn) {
    // downward from well above max(l, x), normalised by j_0 or j_1; rescaled by 2^-600 (exact) when it grows
    // past 2^600.  The first run finds the normalisation and the number of rescalings, the second stores.
    const int Ls = L + 30 + (int)sqrt(40.0 * (L + 1));
    const double down = ldexp(1.0, -600);
    double tp = 0.0, tc = 1e-300;  // t_{l+1}, t_l at l = Ls
    int K = 0;
    auto step = [&](int l) {
      const double tm = fma(int_as_f64(2 * l + 1) * ix1, tc, -tp);  // t_{l-1}
      return tm;
    };
    auto advance = [&](double tm, int& k) {
      tp = tc; tc = tm;
      if ((__double2hiint(tc) & 0x7fffffff) >= (1023 + 600) << 20) { tp *= down; tc *= down; ++k; }
    };
#pragma unroll 4
    for (int l = Ls; l >= 1; --l) advance(step(l), K);
    const double norm = (fabs(j0) >= fabs(j1)) ? j0 / tc : j1 / tp;
    auto scaled = [&](double v, int m) {
      v *= norm;
      for (int i = 0; i < min(m, 4); ++i) v *= down;
      return v;
    };
    tp = 0.0; tc = 1e-300;
    int k = 0, q = nl - 1, lq = ls[q];
    for (int l = Ls; l >= 0; --l) {
      const double tm = l > 0 ? step(l) : 0.0;
      if (l == lq) {
        put(q, l, scaled(tc, K - k), l == 0 ? scaled(-tp, K - k) : scaled(fma(cf[2 * q], tm, -(cf[2 * q + 1] * tp)), K - k));
        if ((q & 15) == 0) flush(q & ~15, mdn);
        lq = --q >= 0 ? ls[q] : -1;
      }
      if (l > 0) advance(tm, k);
    }
  }
}

__device__ __forceinline__ double jl_interp(const BesselDev& J, int il, double x) {
  double w = x * J.invdx;
  const int i = (int)w;
  w -= i;
  const double ym = J.y[(size_t)i * J.nl + il], yp = J.y[(size_t)(i + 1) * J.nl + il];
  if (!J.hermite) return fma(w, yp - ym, ym);
  const double dym = J.dy[(size_t)i * J.nl + il], dyp = J.dy[(size_t)(i + 1) * J.nl + il];
  const double wm1 = w - 1.0;
  return (1 + 2 * w) * wm1 * wm1 * ym + w * w * (3 - 2 * w) * yp + w * wm1 * (wm1 * dym + w * dyp) * J.dx;
}

__global__ void bessel_eval_kernel(BesselDev J, int il, int n, const double* __restrict__ x, double* __restrict__ out) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = jl_interp(J, il, x[i]);
}

// Line of sight in FP64 over the flattened (k, l < il_limber): what depends on (k, τ) only — table row,
// interpolation weights, w_τ S — is formed once per k and time in shared memory by the block (256
// consecutive (k, l), so a few k), and a thread spends 4 FP64 instructions on j_l and one per source
// (one source: the weights carry it) instead of about 22.  Bound: the FP64 pipes; 777 k x 401 τ x 97 l x
// 2 sources 1.71 ms before.
// S: [it * st_t + ik * st_k + s].
template <int NSRC, bool HERM>
__global__ void __launch_bounds__(256) los_kernel(BesselDev J, const double* __restrict__ S, int64_t st_t, int64_t st_k,
                                                  const double* __restrict__ chi, const double* __restrict__ wts, int ntau, int nk,
                                                  const double* __restrict__ ks, int il_limber, int chunk, double* __restrict__ out) {
  extern __shared__ double sm[];
  constexpr int NC = HERM ? 4 : 2, NW = NSRC == 1 ? NC : NC + NSRC;  // doubles per (k, time)
  const int64_t f0 = (int64_t)blockIdx.x * 256, ftot = (int64_t)nk * il_limber;
  const int k0 = (int)(f0 / il_limber), k1 = (int)((min(f0 + 256, ftot) - 1) / il_limber), nkb = k1 - k0 + 1;
  int* rows = reinterpret_cast<int*>(sm + (size_t)nkb * chunk * NW);
  const int64_t fi = f0 + threadIdx.x;
  const bool live = fi < ftot;
  const int ik = live ? (int)(fi / il_limber) : k0, il = live ? (int)(fi - (int64_t)ik * il_limber) : 0;
  const int nl = J.nl, kb = ik - k0;
  double acc[NSRC];
#pragma unroll
  for (int s = 0; s < NSRC; ++s) acc[s] = 0;
  for (int t0 = 0; t0 < ntau; t0 += chunk) {
    const int nt = min(chunk, ntau - t0);
    __syncthreads();
    for (int e = threadIdx.x; e < nkb * nt; e += 256) {
      const int b = e / nt, t = e - b * nt, it = t0 + t;
      const double wpos = ks[k0 + b] * chi[it] * J.invdx;
      const int i = (int)wpos;
      const double w = wpos - i, v = w - 1.0;
      double* p = sm + ((size_t)b * chunk + t) * NW;
      double c[4];
      if (HERM) { c[0] = (1 + 2 * w) * v * v; c[1] = w * w * (3 - 2 * w); c[2] = w * v * v * J.dx; c[3] = w * w * v * J.dx; }
      else { c[0] = 1 - w; c[1] = w; }
      const double* Sp = S + it * st_t + (k0 + b) * st_k;
      if (NSRC == 1) {
        const double ws = wts[it] * Sp[0];
#pragma unroll
        for (int q = 0; q < NC; ++q) p[q] = ws * c[q];
      } else {
#pragma unroll
        for (int q = 0; q < NC; ++q) p[q] = c[q];
#pragma unroll
        for (int s = 0; s < NSRC; ++s) p[NC + s] = wts[it] * Sp[s];
      }
      rows[b * chunk + t] = i;
    }
    __syncthreads();
    const double* p = sm + (size_t)kb * chunk * NW;
    const int* r = rows + kb * chunk;
#pragma unroll 4
    for (int t = 0; t < nt; ++t, p += NW) {
      const size_t o = (size_t)r[t] * nl + il;
      const double y0 = __ldg(J.y + o), y1 = __ldg(J.y + o + nl);
      double j = NSRC == 1 ? acc[0] : 0.0;
      if (HERM) j = fma(p[2], __ldg(J.dy + o), fma(p[3], __ldg(J.dy + o + nl), j));
      j = fma(p[0], y0, fma(p[1], y1, j));
      if (NSRC == 1) {
        acc[0] = j;
      } else {
#pragma unroll
        for (int s = 0; s < NSRC; ++s) acc[s] = fma(p[NC + s], j, acc[s]);
      }
    }
  }
  if (live)
#pragma unroll
    for (int s = 0; s < NSRC; ++s) out[((size_t)ik * nl + il) * NSRC + s] = acc[s];
}

// Mixed-precision line of sight: one block per k, 256 threads over l (up to 4 l per thread).
// Per chunk of 256 times the block tabulates, in FP64, what depends on (k, τ) only: the table row
// of x = k χ, the interpolation weights and w_τ S(τ, k); the l-threads then interpolate the FP32
// table and accumulate in FP32 over the chunk, adding chunk totals in FP64.
constexpr int kLosChunk = 256, kLosMaxL = 4;
template <int NSRC>
__global__ void __launch_bounds__(256) los_f32_kernel(const float2* __restrict__ tab, int nl, double invdx, double dx, int hermite,
                                                      const double* __restrict__ S, int64_t st_t, int64_t st_k, const double* __restrict__ chi,
                                                      const double* __restrict__ wts, int ntau, int nk, const double* __restrict__ ks,
                                                      int il_limber, double* __restrict__ out) {
  __shared__ int s_i[kLosChunk];
  __shared__ float4 s_w[kLosChunk];
  __shared__ float s_S[kLosChunk][NSRC];
  const int ik = blockIdx.x;
  const double k = ks[ik];
  double acc[kLosMaxL][NSRC];
#pragma unroll
  for (int m = 0; m < kLosMaxL; ++m)
#pragma unroll
    for (int s = 0; s < NSRC; ++s) acc[m][s] = 0;
  for (int t0 = 0; t0 < ntau; t0 += kLosChunk) {
    const int nt = min(kLosChunk, ntau - t0);
    __syncthreads();
    for (int t = threadIdx.x; t < nt; t += blockDim.x) {
      const int it = t0 + t;
      const double wpos = k * chi[it] * invdx;
      const int i = (int)wpos;
      const float w = (float)(wpos - i), wm1 = w - 1.0f;
      float4 ww;
      if (hermite) {
        ww.x = (1.0f + 2.0f * w) * wm1 * wm1; ww.y = w * w * (3.0f - 2.0f * w);
        ww.z = (float)(w * wm1 * wm1 * dx); ww.w = (float)(w * w * wm1 * dx);
      } else {
        ww.x = 1.0f - w; ww.y = w; ww.z = 0.0f; ww.w = 0.0f;
      }
      s_i[t] = i; s_w[t] = ww;
      const double wt = wts[it];
#pragma unroll
      for (int s = 0; s < NSRC; ++s) s_S[t][s] = (float)(wt * S[it * st_t + ik * st_k + s]);
    }
    __syncthreads();
#pragma unroll
    for (int m = 0; m < kLosMaxL; ++m) {
      const int il = threadIdx.x + blockDim.x * m;
      if (il < il_limber) {
        float p[NSRC];
#pragma unroll
        for (int s = 0; s < NSRC; ++s) p[s] = 0.0f;
#pragma unroll 4
        for (int t = 0; t < nt; ++t) {
          const int i = s_i[t];
          const float4 ww = s_w[t];
          const float2 a = __ldg(tab + (size_t)i * nl + il), b = __ldg(tab + (size_t)(i + 1) * nl + il);
          const float j = fmaf(ww.x, a.x, fmaf(ww.y, b.x, fmaf(ww.z, a.y, ww.w * b.y)));
#pragma unroll
          for (int s = 0; s < NSRC; ++s) p[s] = fmaf(s_S[t][s], j, p[s]);
        }
#pragma unroll
        for (int s = 0; s < NSRC; ++s) acc[m][s] += (double)p[s];
      }
    }
  }
#pragma unroll
  for (int m = 0; m < kLosMaxL; ++m) {
    const int il = threadIdx.x + blockDim.x * m;
    if (il < il_limber)
#pragma unroll
      for (int s = 0; s < NSRC; ++s) out[((size_t)ik * nl + il) * NSRC + s] = acc[m][s];
  }
}

// C_l = Σ_i a_i (Y_i + Y_{i+1}) - e_i (Y_{i+1} - Y_i) over the intervals between the points (0, 0) and
// (k, Y = g A B), ae: (a_i, e_i): trapezoid and the spline's correction on the differences (one weight per point,
// trapezoid and corrections of both sides added up, would cancel between close points: 1e-8 of C_l where two are 1e-9
// apart).  8 l by 32 runs of intervals per block: an FP64 instruction costs the same for any number of lanes, so a warp
// takes four runs.
__global__ void __launch_bounds__(256) cl_pair_kernel(int nk, const double* __restrict__ g, const double2* __restrict__ ae, int nl,
                                                      const double* __restrict__ A, const double* __restrict__ B, double* __restrict__ Cl) {
  __shared__ double red[32][9];
  const int lx = threadIdx.x & 7, run = threadIdx.x >> 3, il = blockIdx.x * 8 + lx;
  const int i0 = (int)((long long)nk * run / 32), i1 = (int)((long long)nk * (run + 1) / 32);
  auto Y = [&](int i) { return g[i] * A[(size_t)i * nl + il] * B[(size_t)i * nl + il]; };
  double sum = 0;
  if (il < nl) {
    double y0 = i0 > 0 && i0 < i1 ? Y(i0 - 1) : 0.0;
#pragma unroll 4
    for (int i = i0; i < i1; ++i) {
      const double y1 = Y(i);
      const double2 w = ae[i];
      sum = fma(w.x, y0 + y1, fma(-w.y, y1 - y0, sum));
      y0 = y1;
    }
  }
  red[run][lx] = sum;
  __syncthreads();
  if (run == 0 && il < nl) {
    double t = 0;
    for (int q = 0; q < 32; ++q) t += red[q][lx];
    Cl[il] = t;
  }
}

// C_l as a weighted sum over k: one block per (pair, l), FP64 throughout.
__global__ void __launch_bounds__(256) cl_dot_kernel(int nk, const double* __restrict__ g, int nl, int ns,
                                                     const double* __restrict__ Th, const int* __restrict__ pa,
                                                     const int* __restrict__ pb, double* __restrict__ Cl) {
  const int il = blockIdx.x % nl, q = blockIdx.x / nl;
  const int A = pa[q], B = pb[q];
  double sum = 0;
  for (int i = threadIdx.x; i < nk; i += blockDim.x) {
    const size_t o = ((size_t)i * nl + il) * ns;
    sum = fma(g[i] * Th[o + A], Th[o + B], sum);
  }
  __shared__ double red[8];
#pragma unroll
  for (int o = 16; o; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = sum;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
    Cl[blockIdx.x] = tot;
  }
}

// Limber approximation (src/observables/angular.jl:154-178); one thread per (k, l >= l_limber).
__global__ void limber_kernel(const int* __restrict__ ls, int nl, int il_limber, int nsrc, const double* __restrict__ S,
                              int64_t st_t, int64_t st_k, const double* __restrict__ taus, const double* __restrict__ chi, int ntau, int nk,
                              const double* __restrict__ ks, double* __restrict__ out) {
  const int nlim = nl - il_limber;
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= nk * nlim) return;
  const int ik = t / nlim, il = il_limber + t % nlim;
  const double k = ks[ik], l = ls[il];
  const double x = (l + 0.5) / k;
  const double tau0 = taus[ntau - 1];
  for (int s = 0; s < nsrc; ++s) out[((size_t)ik * nl + il) * nsrc + s] = 0;
  if (!(x <= chi[0])) return;
  // first index with taus[i] >= tau0 - x
  int lo = 0, hi = ntau;
  const double target = tau0 - x;
  while (lo < hi) { const int mid = (lo + hi) >> 1; if (taus[mid] < target) lo = mid + 1; else hi = mid; }
  const int im = lo;
  if (im == 0) return;
  const int ip = im - 1;
  const double chim = chi[im], chip = chi[ip], dchi = chip - chim;
  for (int s = 0; s < nsrc; ++s) {
    auto Sv = [&](int i) { return S[i * st_t + ik * st_k + s]; };
    const double Sm = Sv(im), Sp = Sv(ip);
    const double dSm = (im <= ntau - 2) ? (Sv(im + 1) - Sp) / (chi[im + 1] - chip) : (Sp - Sm) / dchi;
    const double dSp = (ip >= 1) ? (Sm - Sv(im - 2)) / (chim - chi[im - 2]) : (Sp - Sm) / dchi;
    const double u = (x - chim) / dchi, u2 = u * u, u3 = u2 * u;
    const double Sx = (2 * u3 - 3 * u2 + 1) * Sm + (u3 - 2 * u2 + u) * dchi * dSm + (-2 * u3 + 3 * u2) * Sp + (u3 - u2) * dchi * dSp;
    out[((size_t)ik * nl + il) * nsrc + s] = sqrt(M_PI / (2 * l + 1)) * Sx / k;
  }
}

// C_l: natural cubic spline (z0 = zN = 0) through (0,0),(k_i, y_i); factors of the interior
// tridiagonal system (shared by all l) are precomputed: cprime[i], inv_den[i].
__global__ void cl_kernel(int nk, const double* __restrict__ ks, const double* __restrict__ P0, int nl,
                          const double* __restrict__ ThA, const double* __restrict__ ThB,
                          const double* __restrict__ cprime, const double* __restrict__ invden,
                          double* __restrict__ zbuf, double* __restrict__ Cl) {
  const int il = blockIdx.x * blockDim.x + threadIdx.x;
  if (il >= nl) return;
  const int np = nk + 1;  // points incl. (0, 0)
  auto X = [&](int i) { return i == 0 ? 0.0 : ks[i - 1]; };
  auto Y = [&](int i) { return i == 0 ? 0.0 : (2.0 / M_PI) * ks[i - 1] * ks[i - 1] * P0[i - 1] * ThA[(size_t)(i - 1) * nl + il] * ThB[(size_t)(i - 1) * nl + il]; };
  double* z = zbuf + (size_t)il;  // strided by nl: z[i * nl]
  // forward sweep on interior rows i = 1..np-2 (Thomas), d' stored in z
  double yprev = Y(0), ycur = Y(1);
  double dprev = 0;
  for (int i = 1; i <= np - 2; ++i) {
    const double ynext = Y(i + 1);
    const double h0 = X(i) - X(i - 1), h1 = X(i + 1) - X(i);
    const double rhs = 6 * ((ynext - ycur) / h1 - (ycur - yprev) / h0);
    const double d = (rhs - h0 * dprev) * invden[i];
    z[(size_t)i * nl] = d;
    dprev = d;
    yprev = ycur; ycur = ynext;
  }
  // back substitution; integrate on the fly
  double znext = 0, sum = 0;  // z_{np-1} = 0
  double ynext = Y(np - 1);
  for (int i = np - 2; i >= 0; --i) {
    const double zi = (i >= 1) ? z[(size_t)i * nl] - cprime[i] * znext : 0.0;
    const double yi = Y(i);
    const double h = X(i + 1) - X(i);
    sum += h * (yi + ynext) * 0.5 - h * h * h * (zi + znext) / 24.0;
    znext = zi; ynext = yi;
  }
  Cl[il] = sum;
}

// ---- source k-interpolation (src/observables/fourier.jl:227-247, 464-547) --------------------
// Coarse sources Sc[(i*ntau + j)*3 + src[s]] (perturbation-kernel layout) -> fine
// Sf[(f*ntau + j)*ns + s] (a fine k's times are contiguous, as the line of sight reads them), the last time
// (χ = 0, angular.jl:296) zero.  Columns c = j*ns + s; every access runs along the columns.
// Natural cubic spline in y = f(k): the tridiagonal factors depend only on the coarse y grid.
// Right-hand sides, scaled for the sweep: z <- rhs_i invden_i.
__global__ void __launch_bounds__(256) kinterp_spline_rhs(int ntau, int ns, const int* __restrict__ src, const double* __restrict__ Sc,
                                                          const double* __restrict__ y, const double* __restrict__ invden, double* __restrict__ z, int nc) {
  const int col = blockIdx.x * 256 + threadIdx.x, ncol = ntau * ns;
  if (col >= ncol) return;
  const int j = col / ns, s = src[col - j * ns];
  auto V = [&](int q) { return Sc[((size_t)q * ntau + j) * 3 + s]; };
  for (int i = blockIdx.y + 1; i <= nc - 2; i += gridDim.y) {
    const double v = V(i);
    const double c = 6 * invden[i], a1 = c / (y[i + 1] - y[i]), a0 = c / (y[i] - y[i - 1]);
    z[(size_t)i * ncol + col] = a1 * (V(i + 1) - v) - a0 * (v - V(i - 1));
  }
}

// Thomas sweeps, one thread per column: one FMA per row and direction (the divisions and differences are in
// kinterp_spline_rhs), the next eight rows' values loaded ahead of the chain.  Bound: the serial chain,
// 2 (nc - 2) FMAs.  With the right-hand side inside the sweep (two FP64 divisions per row) 400 rows x
// 1,000 columns took 586 µs.
__global__ void __launch_bounds__(32) kinterp_spline_sweep(int nc, int ncol, const double* __restrict__ y, const double* __restrict__ cprime,
                                                           const double* __restrict__ invden, double* __restrict__ z) {
  const int col = blockIdx.x * 32 + threadIdx.x;
  if (col >= ncol) return;
  constexpr int U = 8;
  double* zc = z + col;
  zc[0] = 0;
  zc[(size_t)(nc - 1) * ncol] = 0;
  double d = 0, e[U], g[U];
  auto loadf = [&](int i) {
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const int r = min(i + q, nc - 2);
      e[q] = zc[(size_t)r * ncol];
      g[q] = (y[r] - y[r - 1]) * invden[r];
    }
  };
  auto loadb = [&](int i) {
#pragma unroll
    for (int q = 0; q < U; ++q) {
      const int r = max(i - q, 1);
      e[q] = zc[(size_t)r * ncol];
      g[q] = cprime[r];
    }
  };
  loadf(1);
  for (int i = 1; i <= nc - 2; i += U) {
    double ce[U], cg[U];
#pragma unroll
    for (int q = 0; q < U; ++q) { ce[q] = e[q]; cg[q] = g[q]; }
    if (i + U <= nc - 2) loadf(i + U);
#pragma unroll
    for (int q = 0; q < U; ++q)
      if (i + q <= nc - 2) { d = fma(-cg[q], d, ce[q]); zc[(size_t)(i + q) * ncol] = d; }
  }
  d = 0;
  loadb(nc - 2);
  for (int i = nc - 2; i >= 1; i -= U) {
    double ce[U], cg[U];
#pragma unroll
    for (int q = 0; q < U; ++q) { ce[q] = e[q]; cg[q] = g[q]; }
    if (i - U >= 1) loadb(i - U);
#pragma unroll
    for (int q = 0; q < U; ++q)
      if (i - q >= 1) { d = fma(-cg[q], d, ce[q]); zc[(size_t)(i - q) * ncol] = d; }
  }
}

// Interpolation at fine point f: weights of (z_i, z_{i+1}, v_i, v_{i+1}) once per block (blockIdx.y: 8 fine
// points, one per warp and pass), four FP64 instructions per value (five divisions each before).
__global__ void __launch_bounds__(256) kinterp_spline_eval(int ntau, int ns, int nf, const int* __restrict__ src, const double* __restrict__ Sc,
                                                           const double* __restrict__ y, const double* __restrict__ yf, const int* __restrict__ iv,
                                                           const double* __restrict__ z, double* __restrict__ Sf) {
  __shared__ double w[8][4];
  const int ncol = ntau * ns, col = blockIdx.x * 256 + threadIdx.x;
  const int j = col / ns, s = col < ncol ? src[col - j * ns] : 0;
  const bool last = j == ntau - 1;
  for (int f0 = blockIdx.y * 8; f0 < nf; f0 += gridDim.y * 8) {
    __syncthreads();
    if (threadIdx.x < 8 && f0 + threadIdx.x < nf) {
      const int f = f0 + threadIdx.x, i = iv[f];
      const double h = y[i + 1] - y[i], a = y[i + 1] - yf[f], b = yf[f] - y[i];
      double* p = w[threadIdx.x];
      p[0] = a * a * a / (6 * h) - h * a / 6; p[1] = b * b * b / (6 * h) - h * b / 6; p[2] = a / h; p[3] = b / h;
    }
    __syncthreads();
    if (col < ncol) {
#pragma unroll 4
      for (int q = 0; q < 8; ++q) {
        const int f = f0 + q;
        if (f >= nf) break;
        const int i = iv[f];
        const double v0 = Sc[((size_t)i * ntau + j) * 3 + s], v1 = Sc[((size_t)(i + 1) * ntau + j) * 3 + s];
        const double z0 = z[(size_t)i * ncol + col], z1 = z[(size_t)(i + 1) * ncol + col];
        Sf[(size_t)f * ncol + col] = last ? 0.0 : fma(z0, w[q][0], fma(z1, w[q][1], fma(v0, w[q][2], v1 * w[q][3])));
      }
    }
  }
}

// Barycentric interpolation (Chebyshev points): Sf = Σ_c M[f][c] Sc[c], M built on the host; four fine
// points per thread share a coarse value's load.
__global__ void __launch_bounds__(256) kinterp_bary(int nc, int ntau, int ns, int nf, const int* __restrict__ src, const double* __restrict__ Sc,
                                                    const double* __restrict__ Mw, double* __restrict__ Sf) {
  const int col = blockIdx.x * 256 + threadIdx.x, ncol = ntau * ns;
  if (col >= ncol) return;
  const int j = col / ns, s = src[col - j * ns];
  for (int f0 = blockIdx.y * 4; f0 < nf; f0 += gridDim.y * 4) {
    const double* m[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) m[q] = Mw + (size_t)min(f0 + q, nf - 1) * nc;
    double acc[4] = {0, 0, 0, 0};
#pragma unroll 2
    for (int c = 0; c < nc; ++c) {
      const double v = Sc[((size_t)c * ntau + j) * 3 + s];
#pragma unroll
      for (int q = 0; q < 4; ++q) acc[q] = fma(__ldg(m[q] + c), v, acc[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q)
      if (f0 + q < nf) Sf[(size_t)(f0 + q) * ncol + col] = j == ntau - 1 ? 0.0 : acc[q];
  }
}

// Θ scaling after the line-of-sight integral (angular.jl:301-306): T /= k; E *= √((l+2)!/(l-2)!)/k².
__global__ void theta_scale(int nk, int nl, int ns, const double* __restrict__ ks, const int* __restrict__ ls,
                            int sT, int sE, double* __restrict__ Th) {
  const size_t t = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= (size_t)nk * nl) return;
  const int ik = (int)(t / nl), il = (int)(t % nl);
  const double k = ks[ik], l = ls[il];
  if (sT >= 0) Th[t * ns + sT] /= k;
  if (sE >= 0) Th[t * ns + sE] *= sqrt((l + 2) * (l + 1) * l * (l - 1)) / (k * k);
}

}  // namespace

int kinterp_spline_launch(int nc, int ntau, int ns, int nf, const int* d_src, const double* d_Sc, const double* d_y,
                          const double* d_yf, const int* d_iv, const double* d_cprime, const double* d_invden, double* d_z,
                          double* d_Sf, cudaStream_t st) {
  const int ncol = ntau * ns, cb = (ncol + 255) / 256;
  kinterp_spline_rhs<<<dim3(cb, std::min(nc - 2, 65535)), 256, 0, st>>>(ntau, ns, d_src, d_Sc, d_y, d_invden, d_z, nc);
  kinterp_spline_sweep<<<(ncol + 31) / 32, 32, 0, st>>>(nc, ncol, d_y, d_cprime, d_invden, d_z);
  kinterp_spline_eval<<<dim3(cb, std::min((nf + 7) / 8, 65535)), 256, 0, st>>>(ntau, ns, nf, d_src, d_Sc, d_y, d_yf, d_iv, d_z, d_Sf);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int kinterp_bary_launch(int nc, int ntau, int ns, int nf, const int* d_src, const double* d_Sc, const double* d_M, double* d_Sf,
                        cudaStream_t st) {
  kinterp_bary<<<dim3((ntau * ns + 255) / 256, std::min((nf + 3) / 4, 65535)), 256, 0, st>>>(nc, ntau, ns, nf, d_src, d_Sc, d_M, d_Sf);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int theta_scale_launch(int nk, int nl, int ns, const double* d_ks, const int* d_ls, int sT, int sE, double* d_Th, cudaStream_t st) {
  const size_t total = (size_t)nk * nl;
  theta_scale<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(nk, nl, ns, d_ks, d_ls, sT, sE, d_Th);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int bessel_build(BesselDev& J, const int* d_ls, const double* d_cf, int Lmax, cudaStream_t st) {
  const int N = J.nx - 1;
  bessel_table_kernel<<<(N + 127) / 128, 128, 0, st>>>(J, d_ls, d_cf, Lmax);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int los_f32_launch(const BesselDev& J, const int* d_ls, int nsrc, const double* d_S, long long st_t, long long st_k, const double* d_taus, const double* d_chi,
                   const double* d_w, int ntau, int nk, const double* d_ks, int il_limber, double* d_out, cudaStream_t st) {
  if (!J.yf2 || il_limber > 256 * kLosMaxL || nk <= 0) return -1;
  switch (nsrc) {
    case 1: los_f32_kernel<1><<<nk, 256, 0, st>>>(J.yf2, J.nl, J.invdx, J.dx, J.hermite, d_S, st_t, st_k, d_chi, d_w, ntau, nk, d_ks, il_limber, d_out); break;
    case 2: los_f32_kernel<2><<<nk, 256, 0, st>>>(J.yf2, J.nl, J.invdx, J.dx, J.hermite, d_S, st_t, st_k, d_chi, d_w, ntau, nk, d_ks, il_limber, d_out); break;
    case 3: los_f32_kernel<3><<<nk, 256, 0, st>>>(J.yf2, J.nl, J.invdx, J.dx, J.hermite, d_S, st_t, st_k, d_chi, d_w, ntau, nk, d_ks, il_limber, d_out); break;
    default: return -1;
  }
  const int nlim = J.nl - il_limber;
  if (nlim > 0) {
    const int tot = nk * nlim;
    limber_kernel<<<(tot + 127) / 128, 128, 0, st>>>(d_ls, J.nl, il_limber, nsrc, d_S, st_t, st_k, d_taus, d_chi, ntau, nk, d_ks, d_out);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int cl_dot_launch(int nk, const double* d_g, int nl, int ns, const double* d_Th, int npair, const int* d_pa, const int* d_pb,
                  double* d_Cl, cudaStream_t st) {
  cl_dot_kernel<<<nl * npair, 256, 0, st>>>(nk, d_g, nl, ns, d_Th, d_pa, d_pb, d_Cl);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int bessel_eval(const BesselDev& J, int il, int n, const double* d_x, double* d_out, cudaStream_t st) {
  bessel_eval_kernel<<<(n + 255) / 256, 256, 0, st>>>(J, il, n, d_x, d_out);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

template <int NSRC>
static int los_launch_n(const BesselDev& J, const double* d_S, long long st_t, long long st_k, const double* d_chi, const double* d_w, int ntau,
                        int nk, const double* d_ks, int il_limber, double* d_out, cudaStream_t st) {
  const long long tot = (long long)nk * il_limber;
  const int nkb = 256 / il_limber + 2;  // k values a block can touch
  const int nw = (J.hermite ? 4 : 2) + (NSRC == 1 ? 0 : NSRC);
  const int chunk = std::max(1, std::min(64, (int)(40 * 1024 / (nkb * (nw * sizeof(double) + sizeof(int))))));
  const size_t smem = (size_t)nkb * chunk * (nw * sizeof(double) + sizeof(int));
  const unsigned grid = (unsigned)((tot + 255) / 256);
  if (J.hermite) los_kernel<NSRC, true><<<grid, 256, smem, st>>>(J, d_S, st_t, st_k, d_chi, d_w, ntau, nk, d_ks, il_limber, chunk, d_out);
  else los_kernel<NSRC, false><<<grid, 256, smem, st>>>(J, d_S, st_t, st_k, d_chi, d_w, ntau, nk, d_ks, il_limber, chunk, d_out);
  return 0;
}

int los_launch(const BesselDev& J, const int* d_ls, int nsrc, const double* d_S, long long st_t, long long st_k, const double* d_taus,
               const double* d_chi, const double* d_w, int ntau, int nk, const double* d_ks, int il_limber,
               double* d_out, cudaStream_t st) {
  if (nk > 0 && il_limber > 0) {
    switch (nsrc) {
      case 1: los_launch_n<1>(J, d_S, st_t, st_k, d_chi, d_w, ntau, nk, d_ks, il_limber, d_out, st); break;
      case 2: los_launch_n<2>(J, d_S, st_t, st_k, d_chi, d_w, ntau, nk, d_ks, il_limber, d_out, st); break;
      case 3: los_launch_n<3>(J, d_S, st_t, st_k, d_chi, d_w, ntau, nk, d_ks, il_limber, d_out, st); break;
      default: return -1;
    }
  }
  const int nlim = J.nl - il_limber;
  if (nlim > 0 && nk > 0) {
    const int tot = nk * nlim;
    limber_kernel<<<(tot + 127) / 128, 128, 0, st>>>(d_ls, J.nl, il_limber, nsrc, d_S, st_t, st_k, d_taus, d_chi, ntau, nk, d_ks, d_out);
  }
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int cl_pair_launch(int nk, const double* d_g, const double2* d_ae, int nl, const double* d_A, const double* d_B, double* d_Cl, cudaStream_t st) {
  cl_pair_kernel<<<(nl + 7) / 8, 256, 0, st>>>(nk, d_g, d_ae, nl, d_A, d_B, d_Cl);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

int cl_launch(int nk, const double* d_ks, const double* d_P0, int nl, const double* d_ThA, const double* d_ThB,
              const double* d_cprime, const double* d_invden, double* d_zbuf, double* d_Cl, cudaStream_t st) {
  cl_kernel<<<(nl + 127) / 128, 128, 0, st>>>(nk, d_ks, d_P0, nl, d_ThA, d_ThB, d_cprime, d_invden, d_zbuf, d_Cl);
  return cudaGetLastError() == cudaSuccess ? 0 : -2;
}

}  // namespace sbz
