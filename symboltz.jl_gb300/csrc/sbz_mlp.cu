// Source surrogate: dense-layer GEMM launcher (tensor maps, tile choice) and C-ABI test entry.
#include <cudaTypedefs.h>
#include <algorithm>
#include <cstdio>
#include <mutex>
#include "../../include/symboltz_gb300.h"
#include "sbz_mlp_gemm.cuh"

namespace sbz {
int capi_fail(int code, const char* msg);

namespace mlp {
int gemm_splits(int M, int N, int K);

namespace {

PFN_cuTensorMapEncodeTiled_v12000 g_encode = nullptr;
std::mutex g_mu;

bool get_encode() {
  std::lock_guard<std::mutex> lock(g_mu);
  if (g_encode) return true;
  void* fn = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &fn, 12000, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess || !fn)
    return false;
  g_encode = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(fn);
  return true;
}

// 2-D tensor map of a bf16 (or FP32) [rows][cols] row-major matrix (row stride ld elements), box box_cols x box_rows,
// 128-byte swizzle
bool tmap(CUtensorMap* tm, const void* ptr, int rows, int cols, int ld, int box_cols, int box_rows, bool f32 = false) {
  const cuuint64_t dims[2] = {(cuuint64_t)cols, (cuuint64_t)rows};
  const cuuint64_t strides[1] = {(cuuint64_t)ld * (f32 ? 4 : 2)};
  const cuuint32_t box[2] = {(cuuint32_t)box_cols, (cuuint32_t)box_rows};
  const cuuint32_t es[2] = {1, 1};
  return g_encode(tm, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(ptr), dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) == CUDA_SUCCESS;
}
// operand [rows][cols] without padding, box 64 x box_rows
bool tmap_operand(CUtensorMap* tm, const void* ptr, int rows, int cols, int box_rows) {
  return tmap(tm, ptr, rows, cols, cols, BK, box_rows);
}

int num_sms() {
  static int n = 0;
  if (!n) {
    int dev = 0;
    cudaGetDevice(&dev);
    if (cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess || n < 1) n = 1;
  }
  return n;
}

bool aligned16(const void* p) { return ((uintptr_t)p & 15) == 0; }

// Shapes of gemm_act_kernel: whole 128-column tiles, 16-byte row strides and bases.  65,536 x 512
// x 512 forward and backward: 45 and 46 µs, where one tile per CTA and two CTAs per SM with the same epilogue took
// 55 and 57 (64 inputs: 30 and 33).
bool act_tiles(const GemmArgs& g, int bn) {
  if (g.epi == EPI_F32 || bn < 128 || g.n_valid != g.N || g.ldo % 8 || !aligned16(g.out_bf16) || !aligned16(g.bias)) return false;
  if (g.epi == EPI_DACT && !aligned16(g.z_in)) return false;
  return g.epi != EPI_ACT || !g.z_out || aligned16(g.z_out);
}

template <int BN>
int launch_act(const GemmArgs& g, const void* A, const void* B, cudaStream_t st) {
  CUtensorMap ta, tb, to, tz;
  const void* z = g.epi == EPI_DACT ? static_cast<const void*>(g.z_in) : g.z_out;
  if (!tmap_operand(&ta, A, g.M, g.K, BM) || !tmap_operand(&tb, B, g.N, g.K, BN) || !tmap(&to, g.out_bf16, g.M, g.N, g.ldo, 64, 32))
    return SBZ_ERR_CUDA;
  tz = to;
  if (z && !tmap(&tz, z, g.M, g.N, g.ldo, 64, 32)) return SBZ_ERR_CUDA;
  constexpr size_t smem = gemm_act_smem_bytes<BN>();
  static_assert(smem <= 227 * 1024, "shared memory of an SM");
  static bool attr_set = false;  // set once, outside any stream capture of a later call
  if (!attr_set) {
    if (cudaFuncSetAttribute(gemm_act_kernel<BN>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return SBZ_ERR_CUDA;
    attr_set = true;
  }
  const int tiles = (g.N / BN) * (g.M / BM);
  gemm_act_kernel<BN><<<std::min(tiles, num_sms()), kActThreads, smem, st>>>(ta, tb, to, tz, g);
  return cudaGetLastError() == cudaSuccess ? SBZ_OK : SBZ_ERR_CUDA;
}

template <int BN>
int launch(const GemmArgs& g, const void* A, const void* B, cudaStream_t st) {
  if constexpr (BN >= 128)
    if (act_tiles(g, BN)) return launch_act<BN>(g, A, B, st);
  if (g.colpart) return SBZ_ERR_ARG;  // only gemm_act_kernel forms column sums
  int splits = g.epi == EPI_F32 ? gemm_splits(g.M, g.N, g.K) : 1;
  if (!g.part && g.max_splits > 0) splits = std::min(splits, g.max_splits);
  // partial tiles are added atomically into a zeroed output: one 2-D fill of its region (its rows may be longer than n_valid)
  if (splits > 1 && !g.part && !g.accumulate &&
      cudaMemset2DAsync(g.out_f32, sizeof(float) * (size_t)g.ldo, 0, sizeof(float) * (size_t)g.n_valid, (size_t)g.M, st) != cudaSuccess)
    return SBZ_ERR_CUDA;
  CUtensorMap ta, tb, td;
  if (g.rows_k) {  // [K][M], [K][N] in pieces of 64 x 64
    if (!tmap_operand(&ta, A, g.K, g.M, BK) || !tmap_operand(&tb, B, g.K, g.N, BK)) return SBZ_ERR_CUDA;
  } else if (!tmap_operand(&ta, A, g.M, g.K, BM) || !tmap_operand(&tb, B, g.N, g.K, BN)) {
    return SBZ_ERR_CUDA;
  }
  td = ta;
  if (g.part && !tmap(&td, g.part, splits * g.M, g.N, g.N, 32, 32, true)) return SBZ_ERR_CUDA;
  const size_t smem = gemm_smem_bytes<BN>();
  auto k = gemm_tn_kernel<BN>;
  static bool attr_set = false;  // set once, outside any stream capture of a later call
  if (!attr_set) {
    if (cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return SBZ_ERR_CUDA;
    attr_set = true;
  }
  k<<<dim3(g.N / BN, g.M / BM, splits), kThreads, smem, st>>>(ta, tb, td, g);
  return cudaGetLastError() == cudaSuccess ? SBZ_OK : SBZ_ERR_CUDA;
}

}  // namespace

// Splits of K of an FP32 product.  Weight gradients have few output tiles and a long K (the batch): about two CTAs per
// SM, at least 4 K-steps each.
int gemm_splits(int M, int N, int K) {
  const int bn = N % 256 == 0 ? 256 : N % 128 == 0 ? 128 : 64;
  const int tiles = (N / bn) * (M / BM), KT = K / BK;
  return tiles < 2 * num_sms() ? std::max(1, std::min(KT / 4, 2 * num_sms() / tiles)) : 1;
}

// D = A Bᵀ (AᵀB of [K][M] and [K][N] operands with rows_k) with the fused epilogue of g; M % 128 == 0, N % 64 == 0, K % 64 == 0, A and B 16-byte
// aligned (TMA).  The widest tile that divides N is used.
int gemm(const GemmArgs& g, const void* A, const void* B, cudaStream_t st) {
  if (g.M <= 0 || g.M % BM || g.N <= 0 || g.N % 64 || g.K <= 0 || g.K % BK) return SBZ_ERR_ARG;
  if (((uintptr_t)A | (uintptr_t)B) & 15 || (g.rows_k && g.epi != EPI_F32)) return SBZ_ERR_ARG;
  if (!get_encode()) return SBZ_ERR_CUDA;
  if (g.N % 256 == 0) return launch<256>(g, A, B, st);
  if (g.N % 128 == 0) return launch<128>(g, A, B, st);
  return launch<64>(g, A, B, st);
}

}  // namespace mlp
}  // namespace sbz

namespace {
unsigned* g_flag = nullptr;  // pipeline-timeout flag of the test entry (one per process)
}

extern "C" int sbz_mlp_gemm(int M, int N, int K, const void* A, const void* B, int epi, int act, const float* bias, void* out,
                            int ldo, int n_valid, int accumulate, void* z_out, const void* z_in, void* stream) {
  using namespace sbz::mlp;
  if (!A || !B || !out || epi < EPI_F32 || epi > EPI_DACT || (epi == EPI_DACT && !z_in))
    return sbz::capi_fail(SBZ_ERR_ARG, "sbz_mlp_gemm: bad arguments");
  if (!g_flag && cudaMalloc(&g_flag, sizeof(unsigned)) != cudaSuccess) return sbz::capi_fail(SBZ_ERR_CUDA, "sbz_mlp_gemm: flag");
  cudaStream_t st = static_cast<cudaStream_t>(stream);
  if (cudaMemsetAsync(g_flag, 0, sizeof(unsigned), st) != cudaSuccess) return sbz::capi_fail(SBZ_ERR_CUDA, "sbz_mlp_gemm: flag");
  GemmArgs g{};
  g.M = M; g.N = N; g.K = K; g.epi = epi; g.act = act; g.bias = bias;
  g.out_bf16 = static_cast<__nv_bfloat16*>(out); g.out_f32 = static_cast<float*>(out);
  g.ldo = ldo; g.n_valid = n_valid > 0 ? n_valid : N; g.accumulate = accumulate;
  g.z_out = static_cast<__nv_bfloat16*>(z_out); g.z_in = static_cast<const __nv_bfloat16*>(z_in); g.err = g_flag;
  const int r = gemm(g, A, B, st);
  if (r == SBZ_ERR_ARG) return sbz::capi_fail(r, "sbz_mlp_gemm: sizes must satisfy M%128, N%64, K%64 == 0 and 16-byte aligned operands");
  if (r != SBZ_OK) return sbz::capi_fail(r, "sbz_mlp_gemm: launch or tensor-map failure");
  unsigned flag = 0;
  if (cudaMemcpyAsync(&flag, g_flag, sizeof flag, cudaMemcpyDeviceToHost, st) != cudaSuccess || cudaStreamSynchronize(st) != cudaSuccess)
    return sbz::capi_fail(SBZ_ERR_CUDA, "sbz_mlp_gemm: kernel failed");
  if (flag) return sbz::capi_fail(SBZ_ERR_CUDA, "sbz_mlp_gemm: pipeline wait ran out");
  return SBZ_OK;
}
