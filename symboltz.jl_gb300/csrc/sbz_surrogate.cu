// Source surrogate: an MLP (nin → nhidden × width, SiLU → nout) trained and evaluated with the
// project's BF16 tensor-core GEMM (sbz_mlp_gemm.cuh) and FP32 accumulation.
//
// Layout: layer l maps kin_l → nrow_l features; the input is padded to 64 columns and the output
// to 64 rows (TMA/UMMA granularity), padding weights stay zero (their gradients are zero).  Master
// weights, Adam moments and gradients are FP32 [nrow][kin]; the GEMMs read BF16 copies W [nrow][kin]
// (forward) and Wt [kin][nrow] (backward).  Activations are BF16 [batch][features] (the weight-gradient
// GEMMs read them with the batch as their K dimension); the last layer writes FP32 so the loss is not
// quantised.  A training step:
//   gather    X_0, targets T of the step's random batch
//   forward   X_l = SiLU(X_{l-1} W_lᵀ + b_l)          (EPI_ACT, pre-activations Z_l kept)
//   loss      Y = X_L W_Lᵀ + b_L (FP32), dY = 2 (Y - T) / (batch · nout), db_L = Σ_batch dY
//   backward  dZ_{l-1} = (dZ_l W_l) ⊙ SiLU'(Z_{l-1})  (EPI_DACT, db_{l-1} = Σ_batch dZ_{l-1})
//             dW_l = dZ_lᵀ X_{l-1} (EPI_F32 with rows along K, split K)
//   Adam      one launch over every parameter: gradient summed, FP32 update, BF16 W and Wt refreshed.
// Sums over the batch leave the kernels as partial sums (a split of K, 32 or 256 rows) that the Adam launch adds
// in their order, so equal trainings give equal bits.
// The step (about 20 launches) is captured once in a CUDA graph and replayed; the step counter
// and the learning rate live in device memory so the replayed graph needs no new parameters.
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <string>
#include <vector>
#include "../../include/symboltz_gb300.h"
#include "sbz_mlp_gemm.cuh"

namespace sbz {
int capi_fail(int code, const char* msg);
namespace mlp {
int gemm(const GemmArgs& g, const void* A, const void* B, cudaStream_t st);
int gemm_splits(int M, int N, int K);
}
}  // namespace sbz

using bf16 = __nv_bfloat16;

namespace {

constexpr int kPadIn = 64, kPadOut = 64;

struct Layer {
  int kin, nrow;      // padded sizes (GEMM K and N)
  int nin, nout;      // logical sizes
  float *W, *b, *mW, *vW, *mb, *vb;  // FP32 [nrow][kin], [nrow]
  float *gW, *gb;     // gradients of sbz_surrogate_gradients, same shapes
  float *pW, *pb;     // partial sums of the gradients: [splits][nrow][kin], [row blocks][nrow]
  bf16 *Wh, *Wt;      // BF16 [nrow][kin], [kin][nrow]
  bool gT;            // a partial sum in pW is transposed ([kin][nrow])
};

template <class T>
cudaError_t dalloc(T** p, size_t n) { return cudaMalloc(p, sizeof(T) * (n ? n : 1)); }

}  // namespace

struct sbz_surrogate {
  int nin = 0, width = 0, nhidden = 0, nout = 0, batch = 0;
  std::vector<Layer> L;
  // activations (batch rows): X[0] input, X[l] output of hidden layer l; Z[l] pre-activations
  std::vector<bf16*> X, Z, dZ;
  float* Yf = nullptr;        // [batch][64] last-layer product (before bias)
  bf16* dY = nullptr;
  float* T = nullptr;         // [batch][nout] targets of the step
  double *loss = nullptr, *ploss = nullptr;  // loss and its partial sums (row blocks)
  unsigned char* grads = nullptr;  // loss, every layer's gW and gb, then the partial sums
  unsigned* err = nullptr;
  float *dataX = nullptr, *dataY = nullptr;
  long long ndata = 0;
  long long step = 0;
  unsigned long long seed = 0;
  cudaStream_t stream = nullptr;
  long long* dstep = nullptr;  // device step counter (incremented at the start of each step)
  float* dlr = nullptr;        // device learning rate
  void* segs = nullptr;        // device tables of Adam segments: of the training batch, and of the last gradients call
  int nseg = 0;
  int nadam = 0;               // blocks of the Adam launch
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t graph_exec = nullptr;
};

namespace {

// ---- kernels ---------------------------------------------------------------------------------

// Batch assembly: sample i takes data row idx = hash(step, i) mod n (uniform with replacement).
__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {
  z += 0x9E3779B97F4A7C15ull;
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

// dstep (if not null): the step is *dstep + 1 (the graph-captured training step reads the device counter,
// which loss_grad advances).  X0 rows are written whole (padding zero).  A warp assembles 32 rows: one hash per
// lane, row pieces along the row (one thread per row wrote 2-byte pieces of 64 rows: 47 µs for 65,536 rows).
__global__ void __launch_bounds__(128) gather_batch(int batch, int nin, int nout, const float* __restrict__ dX, const float* __restrict__ dY,
                                                    long long n, const long long* __restrict__ dstep, unsigned long long seed, int random,
                                                    bf16* __restrict__ X0, float* __restrict__ T) {
  __shared__ long long rows[4][32];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, i0 = (blockIdx.x * 4 + warp) * 32;
  if (i0 >= batch) return;  // batch is a multiple of 32
  {
    const int i = i0 + lane;
    long long r = i;
    if (random) {
      const unsigned long long step = (unsigned long long)(dstep ? *dstep + 1 : 0);
      r = (long long)(mix64(seed ^ mix64(step * 0x100000001B3ull + (unsigned long long)i)) % (unsigned long long)n);
    }
    rows[warp][lane] = r < n ? r : -1;
  }
  __syncwarp();
#pragma unroll 8
  for (int q = 0; q < 32; ++q) {
    const long long r = rows[warp][q];
    const float* x = dX + (r < 0 ? 0 : r) * nin;
    const int j = 2 * lane;
    const float a = r >= 0 && j < nin ? x[j] : 0.0f, b = r >= 0 && j + 1 < nin ? x[j + 1] : 0.0f;
    reinterpret_cast<__nv_bfloat162*>(X0 + (size_t)(i0 + q) * kPadIn)[lane] = __floats2bfloat162_rn(a, b);
  }
  if (T)
    for (int e = lane; e < 32 * nout; e += 32) {
      const int q = e / nout;
      const long long rq = rows[warp][q];
      T[(size_t)i0 * nout + e] = rq >= 0 ? dY[rq * nout + (e - q * nout)] : 0.0f;
    }
}

__global__ void set_value(float* dst, float v) { *dst = v; }

// loss and output gradient: y = Yf + b (FP32), r = y - t, dY = 2 r / (batch · nout) (BF16; padding columns
// stay zero), and a block's part of the loss and of the bias gradient Σ_rows dY[.][j] (as rounded; [block][kPadOut]).
// 256 threads per block.  Advances the device step counter (if not null; nothing else here reads it).
constexpr int kLossThreads = 256;
__global__ void __launch_bounds__(kLossThreads) loss_grad(int batch, int nout, const float* __restrict__ Yf, const float* __restrict__ b,
                                                           const float* __restrict__ T, bf16* __restrict__ dY, float* __restrict__ pb,
                                                           double* __restrict__ ploss, long long* __restrict__ dstep) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  __shared__ float cs[kLossThreads / 32][kPadOut];
  double l = 0;
  const float sc = 2.0f / ((float)batch * nout);
  for (int j = 0; j < nout; ++j) {
    float g = 0.0f;
    if (i < batch) {
      const float r = Yf[(size_t)i * kPadOut + j] + b[j] - T[(size_t)i * nout + j];
      l += (double)r * r;
      g = sc * r;
    }
    const bf16 gh = __float2bfloat16(g);
    if (i < batch) dY[(size_t)i * kPadOut + j] = gh;
    float w = __bfloat162float(gh);
    for (int o = 16; o; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if ((threadIdx.x & 31) == 0) cs[threadIdx.x >> 5][j] = w;
  }
  __shared__ double red[kLossThreads / 32];
  for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = l;
  __syncthreads();
  if (threadIdx.x == 0) {
    double s = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += red[w];
    ploss[blockIdx.x] = s / ((double)batch * nout);
    if (dstep && blockIdx.x == 0) ++*dstep;
  }
  if (threadIdx.x < nout) {
    float s = 0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += cs[w][threadIdx.x];
    pb[(size_t)blockIdx.x * kPadOut + threadIdx.x] = s;
  }
}

// Sum in the order of the additions, compensated (their rounding errors are summed beside): the result is the terms'
// sum but for about one rounding.
struct Sum {
  float s = 0.0f, c = 0.0f;
  __device__ void add(float x) {
    const float t = s + x, y = t - s;
    c += (s - (t - y)) + (x - y);
    s = t;
  }
  __device__ float value() const { return isfinite(c) ? s + c : s; }  // an infinite term makes c NaN
};

// The gradients from their partial sums, and with ADAM the update of every parameter, in one launch: 1,024 weights of
// a layer (with BF16 copies [nrow][kin] and [kin][nrow]) or 32 biases per block, the last block the loss.  `start` is
// the segment's first block; the biases come first (up to 2,048 parts behind each other, weights at most 76).  The bias
// corrections use the device step counter.  Bound: reading the parts from HBM (151 MB for 4 x 512 wide layers and 65,536
// rows: 40 µs).  A warp reads 512 (input and output layer: 256) consecutive bytes of eight parts at a time (83 µs by
// 32 x 32 tiles, 128 bytes).
struct Seg {
  float *p, *m, *v, *g;
  const float* part;
  long long stride;  // between partial sums
  bf16 *ph, *pt;
  int parts, start, gT, nrow, kin;
};

template <bool ADAM>
__global__ void __launch_bounds__(256, 3) apply_grads(const Seg* __restrict__ segs, int nseg, const double* __restrict__ ploss, int nloss,
                                                      double* __restrict__ loss, const long long* __restrict__ step,
                                                      const float* __restrict__ lr, float b1, float b2, float eps) {
  __shared__ float tile[16 * 68];
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  if (blockIdx.x == gridDim.x - 1) {  // the loss: lane sums of every 32nd part, then a butterfly
    if (ty > 0) return;
    double l = 0;
    for (int i = tx; i < nloss; i += 32) l += ploss[i];
    for (int o = 16; o; o >>= 1) l += __shfl_xor_sync(0xffffffffu, l, o);
    if (tx == 0) *loss = l;
    return;
  }
  int q = 0;
  while (q + 1 < nseg && segs[q + 1].start <= (int)blockIdx.x) ++q;
  const Seg S = segs[q];
  const int blk = blockIdx.x - S.start;
  const float t = ADAM ? (float)*step : 0.0f, rate = ADAM ? *lr : 0.0f;
  const float c1 = 1.0f / (1.0f - exp2f(t * log2f(b1))), c2 = 1.0f / (1.0f - exp2f(t * log2f(b2)));
  auto adam = [&](float& p, float& m, float& v, float g) {
    m = b1 * m + (1 - b1) * g;
    v = b2 * v + (1 - b2) * g * g;
    p = p - rate * (m * c1) / (sqrtf(v * c2) + eps);
  };
  auto update = [&](size_t i, float g) {
    if (!ADAM) { S.g[i] = g; return 0.0f; }
    float p = S.p[i], m = S.m[i], v = S.v[i];
    adam(p, m, v, g);
    S.p[i] = p; S.m[i] = m; S.v[i] = v;
    return p;
  };
  if (!S.ph) {  // 32 biases: an eighth of the parts per warp, then the eighths
    const int i = blk * 32 + tx, q0 = (int)((long long)S.parts * ty / 8), q1 = (int)((long long)S.parts * (ty + 1) / 8);
    Sum a;
    for (int r = q0; r < q1; r += 32) {
      float x[32];
#pragma unroll
      for (int u = 0; u < 32; ++u) x[u] = r + u < q1 ? __ldg(S.part + (r + u) * S.stride + i) : 0.0f;
#pragma unroll
      for (int u = 0; u < 32; ++u) a.add(x[u]);
    }
    tile[ty * 32 + tx] = a.s;
    tile[256 + ty * 32 + tx] = a.c;
    __syncthreads();
    if (ty > 0) return;
    Sum b;
    for (int w = 0; w < 8; ++w) { b.add(tile[w * 32 + tx]); b.c += tile[256 + w * 32 + tx]; }
    update(i, b.value());
    return;
  }
  // 8 x 128 or 16 x 64 values of a part (its columns are the outputs when transposed), four in a row per thread
  const int pc = S.gT ? S.nrow : S.kin, tc = pc % 128 == 0 ? 128 : 64, tr = 1024 / tc, l4 = tc / 4;
  const int row0 = blk / (pc / tc) * tr, col0 = blk % (pc / tc) * tc, x4 = tid % l4 * 4, y = tid / l4;
  const size_t at = (size_t)(row0 + y) * pc + col0 + x4;
  Sum a[4];
  for (int r = 0; r < S.parts; r += 8) {
    float4 x[8];
#pragma unroll
    for (int u = 0; u < 8; ++u)
      x[u] = r + u < S.parts ? __ldg(reinterpret_cast<const float4*>(S.part + (r + u) * S.stride + at)) : make_float4(0.0f, 0.0f, 0.0f, 0.0f);
#pragma unroll
    for (int u = 0; u < 8; ++u) { a[0].add(x[u].x); a[1].add(x[u].y); a[2].add(x[u].z); a[3].add(x[u].w); }
  }
  const float4 g = make_float4(a[0].value(), a[1].value(), a[2].value(), a[3].value());
  if (S.gT) {  // one column of the part (an output) per 16 threads
    *reinterpret_cast<float4*>(tile + y * 68 + x4) = g;
    __syncthreads();
    const int k = tid % 16;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const int r = tid / 16 + 16 * j;
      const size_t i = (size_t)(col0 + r) * S.kin + row0 + k;
      const float p = update(i, tile[k * 68 + r]);
      if (ADAM) { S.ph[i] = __float2bfloat16(p); S.pt[(size_t)(row0 + k) * S.nrow + col0 + r] = __float2bfloat16(p); }
    }
    return;
  }
  if (!ADAM) { *reinterpret_cast<float4*>(S.g + at) = g; return; }
  float4 p = *reinterpret_cast<const float4*>(S.p + at), m = *reinterpret_cast<const float4*>(S.m + at), v = *reinterpret_cast<const float4*>(S.v + at);
  adam(p.x, m.x, v.x, g.x); adam(p.y, m.y, v.y, g.y); adam(p.z, m.z, v.z, g.z); adam(p.w, m.w, v.w, g.w);
  *reinterpret_cast<float4*>(S.p + at) = p; *reinterpret_cast<float4*>(S.m + at) = m; *reinterpret_cast<float4*>(S.v + at) = v;
  *reinterpret_cast<uint2*>(S.ph + at) = make_uint2(sbz::mlp::pack_bf16(p.x, p.y), sbz::mlp::pack_bf16(p.z, p.w));
  *reinterpret_cast<float4*>(tile + y * tc + x4) = p;
  __syncthreads();
  // a column's 8 rows are 16 bytes of the transposed copy
  if (tid < tc * tr / 8) {
    const int k = tid % tc, r = tid / tc * 8;
    unsigned w[4];
#pragma unroll
    for (int j = 0; j < 4; ++j) w[j] = sbz::mlp::pack_bf16(tile[(r + 2 * j) * tc + k], tile[(r + 2 * j + 1) * tc + k]);
    *reinterpret_cast<uint4*>(S.pt + (size_t)(col0 + k) * S.nrow + row0 + r) = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

__global__ void to_bf16(int n, const float* __restrict__ p, int nrow, int kin, bf16* __restrict__ ph, bf16* __restrict__ pt) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int r = i / kin, k = i - r * kin;
  ph[i] = __float2bfloat16(p[i]);
  pt[(size_t)k * nrow + r] = __float2bfloat16(p[i]);
}

__global__ void add_bias_out(int rows, int nout, const float* __restrict__ Yf, const float* __restrict__ b, float* __restrict__ out) {
  const int t = blockIdx.x * blockDim.x + threadIdx.x;
  if (t >= rows * nout) return;
  const int i = t / nout, j = t - i * nout;
  out[t] = Yf[(size_t)i * kPadOut + j] + b[j];
}

// ---- host helpers ----------------------------------------------------------------------------

int F(int code, const std::string& m) { return sbz::capi_fail(code, m.c_str()); }
#define SCU(x)                                                                        \
  do {                                                                                \
    cudaError_t e_ = (x);                                                             \
    if (e_ != cudaSuccess) return F(SBZ_ERR_CUDA, std::string(#x ": ") + cudaGetErrorString(e_)); \
  } while (0)

unsigned long long splitmix(unsigned long long& s) {
  unsigned long long z = (s += 0x9E3779B97F4A7C15ull);
  z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
  z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
  return z ^ (z >> 31);
}

void free_all(sbz_surrogate* s) {
  for (auto& l : s->L)
    for (void* p : {(void*)l.W, (void*)l.b, (void*)l.mW, (void*)l.vW, (void*)l.mb, (void*)l.vb, (void*)l.Wh, (void*)l.Wt})
      if (p) cudaFree(p);
  for (auto* v : {&s->X, &s->Z, &s->dZ})
    for (bf16* p : *v) if (p) cudaFree(p);
  for (void* p : {(void*)s->Yf, (void*)s->dY, (void*)s->T, (void*)s->grads, (void*)s->err, (void*)s->dataX, (void*)s->dataY,
                  (void*)s->dstep, (void*)s->dlr, s->segs})
    if (p) cudaFree(p);
  if (s->graph_exec) cudaGraphExecDestroy(s->graph_exec);
  if (s->graph) cudaGraphDestroy(s->graph);
  if (s->stream) cudaStreamDestroy(s->stream);
}

int refresh_bf16(sbz_surrogate* s) {
  for (auto& l : s->L) {
    const int n = l.nrow * l.kin;
    to_bf16<<<(n + 255) / 256, 256, 0, s->stream>>>(n, l.W, l.nrow, l.kin, l.Wh, l.Wt);
  }
  return cudaGetLastError() == cudaSuccess ? SBZ_OK : F(SBZ_ERR_CUDA, "surrogate: weight copy");
}

int gemm(sbz_surrogate* s, sbz::mlp::GemmArgs g, const bf16* A, const bf16* B) {
  g.err = s->err;
  const int r = sbz::mlp::gemm(g, A, B, s->stream);
  return r == SBZ_OK ? SBZ_OK : F(r, "surrogate: GEMM launch");
}

// out = act(A Bᵀ + bias) or, with z_in, (A Bᵀ) ⊙ act'(z_in) of an N-wide layer
int layer(sbz_surrogate* s, int M, int N, int K, const bf16* A, const bf16* B, const float* bias, bf16* out, bf16* z_out, const bf16* z_in,
          float* colpart) {
  sbz::mlp::GemmArgs g{};
  g.M = M; g.N = N; g.K = K; g.epi = z_in ? sbz::mlp::EPI_DACT : sbz::mlp::EPI_ACT; g.act = sbz::mlp::ACT_SILU; g.bias = bias;
  g.out_bf16 = out; g.ldo = N; g.n_valid = N; g.z_out = z_out; g.z_in = z_in; g.colpart = colpart;
  return gemm(s, g, A, B);
}

// partial sums of AᵀB over the batch, A [batch][M] and B [batch][N]
int weight_gradient(sbz_surrogate* s, int M, int N, const bf16* A, const bf16* B, float* part) {
  sbz::mlp::GemmArgs g{};
  g.M = M; g.N = N; g.K = s->batch; g.epi = sbz::mlp::EPI_F32; g.ldo = N; g.n_valid = N; g.part = part; g.rows_k = 1;
  return gemm(s, g, A, B);
}

// forward pass of `rows` (multiple of 128, ≤ batch) rows already in X[0]; result in Yf.  With
// `train`, the pre-activations are written for the backward pass.
int forward(sbz_surrogate* s, int rows, bool train) {
  const int nl = (int)s->L.size();
  for (int l = 0; l < nl - 1; ++l) {
    const Layer& y = s->L[l];
    const int r = layer(s, rows, y.nrow, y.kin, s->X[l], y.Wh, y.b, s->X[l + 1], train ? s->Z[l + 1] : nullptr, nullptr, nullptr);
    if (r) return r;
  }
  const Layer& o = s->L[nl - 1];
  sbz::mlp::GemmArgs g{};
  g.M = rows; g.N = o.nrow; g.K = o.kin; g.epi = sbz::mlp::EPI_F32; g.out_f32 = s->Yf; g.ldo = kPadOut; g.n_valid = s->nout;
  g.max_splits = 2;  // two parts added to zero give the same bits in either order
  return gemm(s, g, s->X[nl - 1], o.Wh);
}

// backward pass after forward(train) + loss_grad (dY and the output layer's pb set): partial sums of the weight
// gradients into pW, of the bias gradients into pb by the EPI_DACT epilogues
int backward(sbz_surrogate* s) {
  const int B = s->batch, nl = (int)s->L.size();
  // output layer: dW_Lᵀ = X_{L-1}ᵀ dY ([kin][64]); dZ_{L-1} = (dY W_L) ⊙ SiLU'(Z_{L-1})
  const Layer& o = s->L[nl - 1];
  int r = weight_gradient(s, o.kin, kPadOut, s->X[nl - 1], s->dY, o.pW);
  if (r) return r;
  r = layer(s, B, o.kin, kPadOut, s->dY, o.Wt, nullptr, s->dZ[nl - 1], nullptr, s->Z[nl - 1], s->L[nl - 2].pb);
  if (r) return r;
  // hidden layers l = nl-2 .. 0: input X[l], output gradient dZ[l+1]
  for (int l = nl - 2; l >= 0; --l) {
    const Layer& y = s->L[l];
    r = weight_gradient(s, y.nrow, y.kin, s->dZ[l + 1], s->X[l], y.pW);
    if (r) return r;
    if (l > 0) {
      r = layer(s, B, y.kin, y.nrow, s->dZ[l + 1], y.Wt, nullptr, s->dZ[l], nullptr, s->Z[l], s->L[l - 1].pb);
      if (r) return r;
    }
  }
  return cudaGetLastError() == cudaSuccess ? SBZ_OK : F(SBZ_ERR_CUDA, "surrogate: backward");
}

int loss_blocks(int rows) { return (rows + kLossThreads - 1) / kLossThreads; }

// forward + loss + backward of the `rows` rows in X[0] with targets T; advances dstep (if given)
int forward_backward(sbz_surrogate* s, int rows, long long* dstep) {
  int r = forward(s, rows, true);
  if (r) return r;
  loss_grad<<<loss_blocks(rows), kLossThreads, 0, s->stream>>>(rows, s->nout, s->Yf, s->L.back().b, s->T, s->dY, s->L.back().pb, s->ploss, dstep);
  return backward(s);
}

// splits of the batch in a layer's weight gradient, and row blocks in its bias gradient
int weight_parts(const Layer& y, int rows) { return y.gT ? sbz::mlp::gemm_splits(y.kin, y.nrow, rows) : sbz::mlp::gemm_splits(y.nrow, y.kin, rows); }
int bias_parts(const Layer& y, int rows) { return y.gT ? loss_blocks(rows) : rows / 32; }

std::vector<Seg> make_segs(const sbz_surrogate* s, int rows, int& blocks) {
  std::vector<Seg> segs;
  blocks = 0;
  for (auto& l : s->L) {
    segs.push_back(Seg{l.b, l.mb, l.vb, l.gb, l.pb, l.nrow, nullptr, nullptr, bias_parts(l, rows), blocks, 0, l.nrow, 1});
    blocks += l.nrow / 32;
  }
  for (auto& l : s->L) {
    segs.push_back(Seg{l.W, l.mW, l.vW, l.gW, l.pW, (long long)l.nrow * l.kin, l.Wh, l.Wt, weight_parts(l, rows), blocks, l.gT ? 1 : 0, l.nrow, l.kin});
    blocks += l.nrow * l.kin / 1024;
  }
  return segs;
}

// one training step on the stream (captured into the step graph)
int train_step(sbz_surrogate* s) {
  const int B = s->batch;
  gather_batch<<<(B + 127) / 128, 128, 0, s->stream>>>(B, s->nin, s->nout, s->dataX, s->dataY, s->ndata, s->dstep, s->seed, 1, s->X[0], s->T);
  int r = forward_backward(s, B, s->dstep);
  if (r) return r;
  apply_grads<true><<<s->nadam + 1, 256, 0, s->stream>>>(static_cast<const Seg*>(s->segs), s->nseg, s->ploss, loss_blocks(B), s->loss, s->dstep, s->dlr,
                                                         0.9f, 0.999f, 1e-8f);
  return cudaGetLastError() == cudaSuccess ? SBZ_OK : F(SBZ_ERR_CUDA, "surrogate: training step");
}

int check_err(sbz_surrogate* s) {
  unsigned e = 0;
  SCU(cudaMemcpyAsync(&e, s->err, sizeof e, cudaMemcpyDeviceToHost, s->stream));
  SCU(cudaStreamSynchronize(s->stream));
  return e ? F(SBZ_ERR_CUDA, "surrogate: GEMM pipeline wait ran out") : SBZ_OK;
}

// flat parameter order: per layer W [nout][nin] (logical, row-major) then b [nout]
long long nparams(const sbz_surrogate* s) {
  long long n = 0;
  for (auto& l : s->L) n += (long long)l.nout * l.nin + l.nout;
  return n;
}

}  // namespace

extern "C" {

int sbz_surrogate_create(int nin, int width, int nhidden, int nout, int batch, unsigned long long seed, sbz_surrogate** out) {
  if (!out || nin < 1 || nin > kPadIn || nout < 1 || nout > kPadOut || width < 128 || width % 128 || nhidden < 1 || batch < 128 ||
      batch % 128)
    return F(SBZ_ERR_ARG, "sbz_surrogate_create: need 1 <= nin, nout <= 64, width % 128 == 0, nhidden >= 1, batch % 128 == 0");
  auto* s = new sbz_surrogate();
  s->nin = nin; s->width = width; s->nhidden = nhidden; s->nout = nout; s->batch = batch; s->seed = seed;
  auto bail = [&](const char* m) { free_all(s); delete s; return F(SBZ_ERR_CUDA, m); };
  if (cudaStreamCreateWithFlags(&s->stream, cudaStreamNonBlocking) != cudaSuccess) return bail("surrogate: stream");
  const int nl = nhidden + 1;
  s->L.resize(nl);
  unsigned long long rs = seed * 0x2545F4914F6CDD1Dull + 1;
  for (int l = 0; l < nl; ++l) {
    Layer& y = s->L[l];
    y = Layer{};
    y.nin = l == 0 ? nin : width;
    y.kin = l == 0 ? kPadIn : width;
    y.nout = l == nl - 1 ? nout : width;
    y.nrow = l == nl - 1 ? kPadOut : width;
    y.gT = l == nl - 1;
    const size_t nw = (size_t)y.nrow * y.kin;
    if (dalloc(&y.W, nw) || dalloc(&y.mW, nw) || dalloc(&y.vW, nw) || dalloc(&y.b, y.nrow) || dalloc(&y.mb, y.nrow) ||
        dalloc(&y.vb, y.nrow) || dalloc(&y.Wh, nw) || dalloc(&y.Wt, nw))
      return bail("surrogate: weight allocation");
    // Glorot-uniform weights on the logical block, zero padding and biases
    std::vector<float> w(nw, 0.0f);
    const float a = std::sqrt(6.0f / (float)(y.nin + y.nout));
    for (int r = 0; r < y.nout; ++r)
      for (int k = 0; k < y.nin; ++k) w[(size_t)r * y.kin + k] = a * (2.0f * (float)((splitmix(rs) >> 11) * 0x1.0p-53) - 1.0f);
    cudaMemcpy(y.W, w.data(), sizeof(float) * nw, cudaMemcpyHostToDevice);
    cudaMemset(y.b, 0, sizeof(float) * y.nrow);
    for (float* p : {y.mW, y.vW}) cudaMemset(p, 0, sizeof(float) * nw);
    for (float* p : {y.mb, y.vb}) cudaMemset(p, 0, sizeof(float) * y.nrow);
  }
  {
    size_t off = 256;  // the loss, then gW and gb per layer and the partial sums, on 256-byte boundaries
    auto take = [&](size_t bytes) { const size_t o = off; off += (bytes + 255) & ~size_t(255); return o; };
    std::vector<size_t> o;
    for (auto& y : s->L) {
      const size_t nw = sizeof(float) * (size_t)y.nrow * y.kin, nb = sizeof(float) * (size_t)y.nrow;
      for (size_t n : {nw, nb, nb * bias_parts(y, batch), nw * weight_parts(y, batch)}) o.push_back(take(n));
    }
    const size_t ol = take(sizeof(double) * loss_blocks(batch));
    if (dalloc(&s->grads, off)) return bail("surrogate: gradient allocation");
    s->loss = reinterpret_cast<double*>(s->grads);
    s->ploss = reinterpret_cast<double*>(s->grads + ol);
    auto at = [&](int i) { return reinterpret_cast<float*>(s->grads + o[i]); };
    for (int l = 0; l < nl; ++l) { s->L[l].gW = at(4 * l); s->L[l].gb = at(4 * l + 1); s->L[l].pb = at(4 * l + 2); s->L[l].pW = at(4 * l + 3); }
    cudaMemset(s->loss, 0, sizeof(double));
    cudaMemset(s->L[nl - 1].pb, 0, sizeof(float) * kPadOut * loss_blocks(batch));  // padding columns that no kernel writes
  }
  s->X.assign(nl, nullptr); s->Z.assign(nl, nullptr); s->dZ.assign(nl, nullptr);
  for (int l = 0; l < nl; ++l) {
    const int w = l == 0 ? kPadIn : width;
    if (dalloc(&s->X[l], (size_t)batch * w)) return bail("surrogate: activation allocation");
    if (l > 0 && (dalloc(&s->Z[l], (size_t)batch * w) || dalloc(&s->dZ[l], (size_t)batch * w)))
      return bail("surrogate: activation allocation");
  }
  if (dalloc(&s->Yf, (size_t)batch * kPadOut) || dalloc(&s->dY, (size_t)batch * kPadOut) ||
      dalloc(&s->T, (size_t)batch * nout) || dalloc(&s->err, 1))
    return bail("surrogate: buffer allocation");
  cudaMemset(s->err, 0, sizeof(unsigned));
  // padding columns that no kernel writes
  cudaMemset(s->dY, 0, sizeof(bf16) * (size_t)batch * kPadOut);
  {
    const std::vector<Seg> segs = make_segs(s, batch, s->nadam);
    s->nseg = (int)segs.size();
    if (dalloc(&s->dstep, 1) || dalloc(&s->dlr, 1) || cudaMalloc(&s->segs, 2 * sizeof(Seg) * segs.size()) != cudaSuccess)
      return bail("surrogate: buffer allocation");
    cudaMemcpy(s->segs, segs.data(), sizeof(Seg) * segs.size(), cudaMemcpyHostToDevice);
    cudaMemset(s->dstep, 0, sizeof(long long));
  }
  if (refresh_bf16(s) != SBZ_OK) { free_all(s); delete s; return SBZ_ERR_CUDA; }
  if (cudaStreamSynchronize(s->stream) != cudaSuccess) return bail("surrogate: initialisation");
  *out = s;
  return SBZ_OK;
}

void sbz_surrogate_destroy(sbz_surrogate* s) {
  if (!s) return;
  if (s->stream) cudaStreamSynchronize(s->stream);
  free_all(s);
  delete s;
}

long long sbz_surrogate_nparams(const sbz_surrogate* s) { return s ? nparams(s) : 0; }

int sbz_surrogate_get_params(const sbz_surrogate* s, float* params) {
  if (!s || !params) return F(SBZ_ERR_ARG, "null argument");
  long long o = 0;
  for (auto& l : s->L) {
    std::vector<float> w((size_t)l.nrow * l.kin), b(l.nrow);
    SCU(cudaMemcpy(w.data(), l.W, sizeof(float) * w.size(), cudaMemcpyDeviceToHost));
    SCU(cudaMemcpy(b.data(), l.b, sizeof(float) * b.size(), cudaMemcpyDeviceToHost));
    for (int r = 0; r < l.nout; ++r)
      for (int k = 0; k < l.nin; ++k) params[o++] = w[(size_t)r * l.kin + k];
    for (int r = 0; r < l.nout; ++r) params[o++] = b[r];
  }
  return SBZ_OK;
}

int sbz_surrogate_set_params(sbz_surrogate* s, const float* params) {
  if (!s || !params) return F(SBZ_ERR_ARG, "null argument");
  long long o = 0;
  for (auto& l : s->L) {
    std::vector<float> w((size_t)l.nrow * l.kin, 0.0f), b(l.nrow, 0.0f);
    for (int r = 0; r < l.nout; ++r)
      for (int k = 0; k < l.nin; ++k) w[(size_t)r * l.kin + k] = params[o++];
    for (int r = 0; r < l.nout; ++r) b[r] = params[o++];
    SCU(cudaMemcpy(l.W, w.data(), sizeof(float) * w.size(), cudaMemcpyHostToDevice));
    SCU(cudaMemcpy(l.b, b.data(), sizeof(float) * b.size(), cudaMemcpyHostToDevice));
  }
  int r = refresh_bf16(s);
  if (r) return r;
  SCU(cudaStreamSynchronize(s->stream));
  return SBZ_OK;
}

int sbz_surrogate_set_data(sbz_surrogate* s, long long n, const float* X, const float* Y) {
  if (!s || n < 1 || !X || !Y) return F(SBZ_ERR_ARG, "sbz_surrogate_set_data: bad arguments");
  if (s->stream) cudaStreamSynchronize(s->stream);
  if (s->graph_exec) { cudaGraphExecDestroy(s->graph_exec); s->graph_exec = nullptr; }
  if (s->graph) { cudaGraphDestroy(s->graph); s->graph = nullptr; }
  if (s->dataX) cudaFree(s->dataX);
  if (s->dataY) cudaFree(s->dataY);
  s->dataX = s->dataY = nullptr;
  SCU(dalloc(&s->dataX, (size_t)n * s->nin));
  SCU(dalloc(&s->dataY, (size_t)n * s->nout));
  SCU(cudaMemcpy(s->dataX, X, sizeof(float) * n * s->nin, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(s->dataY, Y, sizeof(float) * n * s->nout, cudaMemcpyHostToDevice));
  s->ndata = n;
  return SBZ_OK;
}

int sbz_surrogate_train(sbz_surrogate* s, int nsteps, double lr, double* loss_out) {
  if (!s || nsteps < 0 || !(lr > 0)) return F(SBZ_ERR_ARG, "sbz_surrogate_train: bad arguments");
  if (!s->dataX) return F(SBZ_ERR_STATE, "sbz_surrogate_train: no training data (sbz_surrogate_set_data)");
  set_value<<<1, 1, 0, s->stream>>>(s->dlr, (float)lr);
  int r = SBZ_OK;
  if (!s->graph_exec && nsteps > 0) {
    // the first step runs eagerly (kernel attributes, tensor-map encoder), the next is captured
    if ((r = train_step(s))) return r;
    ++s->step;
    --nsteps;
    SCU(cudaStreamSynchronize(s->stream));
    SCU(cudaStreamBeginCapture(s->stream, cudaStreamCaptureModeThreadLocal));
    r = train_step(s);
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(s->stream, &g);
    if (r || e != cudaSuccess) {
      if (g) cudaGraphDestroy(g);
      return r ? r : F(SBZ_ERR_CUDA, std::string("surrogate: step capture: ") + cudaGetErrorString(e));
    }
    s->graph = g;
    SCU(cudaGraphInstantiate(&s->graph_exec, s->graph, 0));
  }
  for (int it = 0; it < nsteps; ++it) SCU(cudaGraphLaunch(s->graph_exec, s->stream));
  s->step += nsteps;
  if (loss_out) SCU(cudaMemcpyAsync(loss_out, s->loss, sizeof(double), cudaMemcpyDeviceToHost, s->stream));
  return check_err(s);
}

int sbz_surrogate_gradients(sbz_surrogate* s, int n, const float* X, const float* Y, double* loss, float* grads) {
  if (!s || n < 1 || n > s->batch || n % 128 || !X || !Y) return F(SBZ_ERR_ARG, "sbz_surrogate_gradients: n % 128 == 0, n <= batch");
  // run one forward/backward on exactly these n rows (batch rows beyond n are zero inputs with zero
  // targets and do not contribute: their loss terms are excluded by using batch = n below)
  const int keepB = s->batch;
  s->batch = n;
  float *dx = nullptr, *dy = nullptr;
  SCU(dalloc(&dx, (size_t)n * s->nin));
  SCU(dalloc(&dy, (size_t)n * s->nout));
  SCU(cudaMemcpy(dx, X, sizeof(float) * n * s->nin, cudaMemcpyHostToDevice));
  SCU(cudaMemcpy(dy, Y, sizeof(float) * n * s->nout, cudaMemcpyHostToDevice));
  gather_batch<<<(n + 127) / 128, 128, 0, s->stream>>>(n, s->nin, s->nout, dx, dy, n, nullptr, 0, 0, s->X[0], s->T);
  int r = forward_backward(s, n, nullptr);
  s->batch = keepB;
  if (!r) {
    int blocks = 0;
    const std::vector<Seg> segs = make_segs(s, n, blocks);
    Seg* d = static_cast<Seg*>(s->segs) + s->nseg;
    if (cudaMemcpyAsync(d, segs.data(), sizeof(Seg) * segs.size(), cudaMemcpyHostToDevice, s->stream) != cudaSuccess) r = F(SBZ_ERR_CUDA, "surrogate: gradients");
    else apply_grads<false><<<blocks + 1, 256, 0, s->stream>>>(d, s->nseg, s->ploss, loss_blocks(n), s->loss, nullptr, nullptr, 0.9f, 0.999f, 1e-8f);
  }
  cudaFree(dx); cudaFree(dy);
  if (r) return r;
  if ((r = check_err(s))) return r;
  if (loss) SCU(cudaMemcpy(loss, s->loss, sizeof(double), cudaMemcpyDeviceToHost));
  if (grads) {
    long long o = 0;
    for (auto& l : s->L) {
      std::vector<float> g((size_t)l.nrow * l.kin), b(l.nrow);
      SCU(cudaMemcpy(g.data(), l.gW, sizeof(float) * g.size(), cudaMemcpyDeviceToHost));
      SCU(cudaMemcpy(b.data(), l.gb, sizeof(float) * b.size(), cudaMemcpyDeviceToHost));
      for (int rr = 0; rr < l.nout; ++rr)
        for (int k = 0; k < l.nin; ++k) grads[o++] = g[(size_t)rr * l.kin + k];
      for (int rr = 0; rr < l.nout; ++rr) grads[o++] = b[rr];
    }
  }
  return SBZ_OK;
}

int sbz_surrogate_infer(sbz_surrogate* s, long long n, const float* X, float* Y) {
  if (!s || n < 0 || (n && (!X || !Y))) return F(SBZ_ERR_ARG, "sbz_surrogate_infer: bad arguments");
  if (n == 0) return SBZ_OK;
  const int B = s->batch;
  float *dx = nullptr, *dyo = nullptr;
  const long long chunk = std::min<long long>(n, 1ll << 22);
  SCU(dalloc(&dx, (size_t)chunk * s->nin));
  SCU(dalloc(&dyo, (size_t)B * s->nout));
  int r = SBZ_OK;
  for (long long c0 = 0; c0 < n && !r; c0 += chunk) {
    const long long cn = std::min(chunk, n - c0);
    if (cudaMemcpyAsync(dx, X + c0 * s->nin, sizeof(float) * cn * s->nin, cudaMemcpyHostToDevice, s->stream) != cudaSuccess) { r = SBZ_ERR_CUDA; break; }
    for (long long b0 = 0; b0 < cn && !r; b0 += B) {
      const int rows = (int)std::min<long long>(B, cn - b0);
      const int prow = (rows + 127) / 128 * 128;
      gather_batch<<<(prow + 127) / 128, 128, 0, s->stream>>>(prow, s->nin, s->nout, dx + b0 * s->nin, nullptr, rows, nullptr, 0, 0, s->X[0], nullptr);
      if ((r = forward(s, prow, false))) break;
      add_bias_out<<<(rows * s->nout + 255) / 256, 256, 0, s->stream>>>(rows, s->nout, s->Yf, s->L.back().b, dyo);
      if (cudaMemcpyAsync(Y + (c0 + b0) * s->nout, dyo, sizeof(float) * rows * s->nout, cudaMemcpyDeviceToHost, s->stream) != cudaSuccess)
        r = SBZ_ERR_CUDA;
    }
  }
  cudaStreamSynchronize(s->stream);
  cudaFree(dx); cudaFree(dyo);
  if (r) return r == SBZ_ERR_CUDA ? F(r, "sbz_surrogate_infer: copy") : r;
  return check_err(s);
}

// flat binary: "SBZMLP01", int32 nin, width, nhidden, nout, then the FP32 parameters in
// sbz_surrogate_get_params order (little-endian)
int sbz_surrogate_save(const sbz_surrogate* s, const char* path) {
  if (!s || !path) return F(SBZ_ERR_ARG, "null argument");
  std::vector<float> p((size_t)nparams(s));
  int r = sbz_surrogate_get_params(s, p.data());
  if (r) return r;
  FILE* f = std::fopen(path, "wb");
  if (!f) return F(SBZ_ERR_ARG, std::string("cannot write ") + path);
  const int hdr[4] = {s->nin, s->width, s->nhidden, s->nout};
  bool ok = std::fwrite("SBZMLP01", 1, 8, f) == 8 && std::fwrite(hdr, sizeof(int), 4, f) == 4 &&
            std::fwrite(p.data(), sizeof(float), p.size(), f) == p.size();
  ok = (std::fclose(f) == 0) && ok;
  return ok ? SBZ_OK : F(SBZ_ERR_ARG, std::string("write failed: ") + path);
}

int sbz_surrogate_load(const char* path, int batch, sbz_surrogate** out) {
  if (!path || !out) return F(SBZ_ERR_ARG, "null argument");
  FILE* f = std::fopen(path, "rb");
  if (!f) return F(SBZ_ERR_ARG, std::string("cannot read ") + path);
  char magic[8];
  int hdr[4];
  if (std::fread(magic, 1, 8, f) != 8 || std::memcmp(magic, "SBZMLP01", 8) || std::fread(hdr, sizeof(int), 4, f) != 4) {
    std::fclose(f);
    return F(SBZ_ERR_ARG, "not a surrogate weight file");
  }
  sbz_surrogate* s = nullptr;
  int r = sbz_surrogate_create(hdr[0], hdr[1], hdr[2], hdr[3], batch, 0, &s);
  if (r) { std::fclose(f); return r; }
  std::vector<float> p((size_t)nparams(s));
  const bool ok = std::fread(p.data(), sizeof(float), p.size(), f) == p.size();
  std::fclose(f);
  if (!ok) { sbz_surrogate_destroy(s); return F(SBZ_ERR_ARG, "truncated surrogate weight file"); }
  if ((r = sbz_surrogate_set_params(s, p.data()))) { sbz_surrogate_destroy(s); return r; }
  *out = s;
  return SBZ_OK;
}

}  // extern "C"
