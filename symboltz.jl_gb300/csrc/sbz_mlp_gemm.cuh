// BF16 tensor-core GEMM for the source surrogate's dense layers (sm_103a: TMA + tcgen05 + TMEM).
//
//   D[M x N] = A[M x K] · B[N x K]ᵀ   (A, B bf16 row-major with K contiguous, FP32 accumulation)
//   D[M x N] = A[K x M]ᵀ · B[K x N]   (the same with rows along K: the weight gradients, whose K is the batch)
//
// Warp 0 lane 0 streams 128 x 64 and BN x 64 K-slices into a shared-memory ring of stages_for<BN>() slots with
// TMA (128-byte swizzle); warp 1 lane 0 issues tcgen05.mma (kind::f16, M = 128, N = BN, K = 16) into a TMEM
// accumulator and releases ring slots with tcgen05.commit; the epilogue warps read the accumulator with
// tcgen05.ld (warp w owns TMEM lanes 32(w mod 4).. = tile rows) and apply the fused epilogue:
//   EPI_F32   out_f32 = D (+ out_f32 when accumulate; split-K CTAs add with atomics), or split-K partial tiles
//             stored side by side for an ordered sum
//   EPI_ACT   z = D + bias; out = bf16(act(z)); optional z_out = bf16(z)    forward layers
//   EPI_DACT  out = bf16(D · act'(z_in))                                   backward layers
// Two kernels: gemm_act_kernel (whole tiles of the activation epilogues) is persistent, and its epilogue runs
// beside the next tile's product; gemm_tn_kernel (one 128 x BN tile per CTA, two CTAs per SM) does EPI_F32 and
// activation outputs that TMA cannot store.
// Every mbarrier wait is bounded: a wait that runs out sets *err and the CTA skips ahead to its
// TMEM release, so a fault in the pipeline cannot hang the GPU.
#pragma once
#include <cuda.h>
#include <cuda_bf16.h>
#include <cuda_runtime.h>
#include <cstdint>

namespace sbz {
namespace mlp {

constexpr int BM = 128, BK = 64, kThreads = 256;
template <int BN>
__host__ __device__ constexpr int stages_for() { return BN >= 256 ? 2 : BN >= 128 ? 3 : 4; }  // (BM + BN) · BK · 2 B · stages ≤ 96 KB
constexpr unsigned kWaitLimit = 1u << 24;
enum { EPI_F32 = 0, EPI_ACT = 1, EPI_DACT = 2 };
enum { ACT_NONE = 0, ACT_SILU = 1 };

struct GemmArgs {
  int M, N, K;
  int epi, act;
  const float* bias;            // [N] (EPI_ACT), may be null
  __nv_bfloat16* out_bf16;      // EPI_ACT / EPI_DACT
  float* out_f32;               // EPI_F32
  int ldo;                      // output row stride (elements)
  int n_valid;                  // columns < n_valid are stored
  int accumulate;               // EPI_F32: add to the output
  float* part;                  // EPI_F32: if not null, split z stores its tile at rows z M .. of [splits M][N] instead
  int max_splits;               // EPI_F32 without part: most splits of K (0: as many as gemm_splits gives)
  __nv_bfloat16* z_out;         // EPI_ACT: pre-activation (ldo stride), may be null
  const __nv_bfloat16* z_in;    // EPI_DACT: pre-activation of this layer (ldo stride)
  int rows_k;                   // operands are [K][M] and [K][N] (EPI_F32)
  float* colpart;               // EPI_DACT: [M / 32][N] sums of out over 32 rows (as stored, bf16-rounded; 8-byte aligned); may be null
  unsigned* err;                // set to 1 by a CTA whose pipeline wait ran out
};

template <int BN>
constexpr size_t gemm_smem_bytes() {
  constexpr int STAGES = stages_for<BN>();
  return 1024 /* alignment slack */ + (size_t)STAGES * (BM + BN) * BK * 2 + (2 * STAGES + 1) * 8 + 16 + BN * 4 /* bias */;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* b, unsigned count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* b, unsigned bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_wait(uint64_t* b, uint32_t parity) {
  const uint32_t a = smem_u32(b);
  for (unsigned i = 0; i < kWaitLimit; ++i) {
    uint32_t ready;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ready)
        : "r"(a), "r"(parity)
        : "memory");
    if (ready) return true;
  }
  return false;
}
__device__ __forceinline__ void mbar_arrive(uint64_t* b) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(b)) : "memory");
}
__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* tm, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
          smem_u32(dst)),
      "l"(reinterpret_cast<uint64_t>(tm)), "r"(x), "r"(y), "r"(smem_u32(bar))
      : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// shared-memory matrix descriptor: K-major tile written by TMA with 128-byte swizzle
// (rows of 128 B, 8-row groups 1024 B apart), start address in 16-byte units
__device__ __forceinline__ uint64_t desc_sw128(const void* p) {
  uint64_t d = (uint64_t)((smem_u32(p) & 0x3FFFFu) >> 4);
  d |= (uint64_t)1 << 16;            // leading-dimension offset (unused by swizzled K-major)
  d |= (uint64_t)(1024 >> 4) << 32;  // stride-dimension offset: next 8-row group
  d |= (uint64_t)1 << 46;            // descriptor version
  d |= (uint64_t)2 << 61;            // 128-byte swizzle
  return d;
}

// the same for a tile with rows along K ([64 K-rows][64 columns] pieces of 8 KB as TMA writes them): 128-byte rows
// of 64 columns, 8-row groups 1024 B apart, the next 64 columns one piece further
__device__ __forceinline__ uint64_t desc_sw128_rows_k(const void* p) {
  uint64_t d = (uint64_t)((smem_u32(p) & 0x3FFFFu) >> 4);
  d |= (uint64_t)(8192 >> 4) << 16;  // leading-dimension offset: next 64 columns
  d |= (uint64_t)(1024 >> 4) << 32;  // stride-dimension offset: next 8 K-rows
  d |= (uint64_t)1 << 46;
  d |= (uint64_t)2 << 61;
  return d;
}

template <int BN>
__device__ __forceinline__ uint32_t idesc_bf16(bool rows_k) {
  return (rows_k ? (1u << 15) | (1u << 16) : 0u)  // A, B: M (N) contiguous
         | (1u << 4)                  // D: FP32
         | (1u << 7) | (1u << 10)     // A, B: BF16
         | ((uint32_t)(BN >> 3) << 17) // N
         | ((uint32_t)(BM >> 4) << 24); // M
}

__device__ __forceinline__ void mma_f16(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc, bool accumulate) {
  asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}" ::"r"(d), "l"(a),
               "l"(b), "r"(idesc), "r"((uint32_t)accumulate)
               : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {  // arrives when the products issued so far are done
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// SiLU and its derivative with the hardware's exponential and reciprocal.  Their flush-to-zero forms: e^{-z} below
// 2^-126 vanishes beside 1, and above 2^126 the reciprocal is 0 as it is from __fdividef (the limits 0 and 1 are
// right); the plain forms' range scaling was about a quarter of the epilogue's instructions.
__device__ __forceinline__ float sigmoid_fast(float z) {
  float e, s;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(e) : "f"(z * -1.4426950408889634f));
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(s) : "f"(1.0f + e));
  return s;
}
__device__ __forceinline__ float silu(float z) { return z * sigmoid_fast(z); }
__device__ __forceinline__ float dsilu(float z) {
  const float s = sigmoid_fast(z);
  return s * (1.0f + z * (1.0f - s));
}

__device__ __forceinline__ unsigned pack_bf16(float a, float b) {
  const __nv_bfloat162 p = __floats2bfloat162_rn(a, b);
  return *reinterpret_cast<const unsigned*>(&p);
}
__device__ __forceinline__ float bf16_lo(unsigned u) { return __uint_as_float(u << 16); }
__device__ __forceinline__ float bf16_hi(unsigned u) { return __uint_as_float(u & 0xFFFF0000u); }

__device__ __forceinline__ void tma_store_2d(const CUtensorMap* tm, int x, int y, const void* src) {
  asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(reinterpret_cast<uint64_t>(tm)),
               "r"(x), "r"(y), "r"(smem_u32(src))
               : "memory");
}
__device__ __forceinline__ void tma_store_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
__device__ __forceinline__ void tma_store_wait_read() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void proxy_fence() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }

// 32 accumulator columns of the warp's 32 rows (lane = row)
__device__ __forceinline__ void tmem_load32(uint32_t taddr, uint32_t (&v)[32]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x32.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%"
      "22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
      : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]), "=r"(v[9]),
        "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]), "=r"(v[17]), "=r"(v[18]),
        "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]), "=r"(v[25]), "=r"(v[26]), "=r"(v[27]),
        "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
      : "r"(taddr));
  asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

// Activation layers (EPI_ACT, EPI_DACT) of whole 128 x BN tiles: one CTA per SM takes every gridDim-th tile, and
// the accumulator is double-buffered in TMEM, so the epilogue of a tile (about 25 µs per 65,536 x 512 layer, bound
// by instruction issue) runs beside the loads and the product of the next one: 45 µs at 512 inputs with three ring slots
// of 48 KB, 55 with two.  HBM takes 30 of them at the copy rate (67 MB read, 134 written); the 402 MB from L2 are not the
// bound (a third less of them, weight tiles shared by two CTAs, took as long).  Warp 0 loads, warp 1 issues the products,
// 16 epilogue warps take 32 rows x 64 columns each (BN = 128: eight of them per tile, in turn).  A warp stages its tiles in 4 KB of
// shared memory and one lane stores them with TMA: every global sector is written whole, where 16-byte stores
// from 32 rows at a stride of 1 KB wrote halves.  128-byte rows, 128-byte swizzle (16-byte piece p of row r at
// p ^ (r mod 8): conflict-free by rows and by columns).  EPI_DACT loads its pre-activations by TMA one tile ahead
// and overwrites them; its column sums are read back down the columns, two per lane.
constexpr int kActWarps = 16, kActThreads = 64 + 32 * kActWarps, kStage = 4096;
template <int BN>
__host__ __device__ constexpr int act_stages() { return BN >= 256 ? 3 : 5; }  // what the staging leaves of 227 KB
template <int BN>
constexpr size_t gemm_act_smem_bytes() {
  return 1024 /* alignment slack */ + (size_t)act_stages<BN>() * (BM + BN) * BK * 2 + kActWarps * kStage +
         (2 * act_stages<BN>() + 4 + kActWarps) * 8 + 16;
}

// Σ over rows r, r + D, r + 2D, .. < 32 of the bf16 pairs at(row), as a tree (a row with the one 16 below it first):
// five roundings deep, where a chain has 31.
template <int D, class At>
__device__ __forceinline__ float2 row_tree(const At& at, int r) {
  if constexpr (D == 32) {
    const unsigned u = at(r);
    return make_float2(bf16_lo(u), bf16_hi(u));
  } else {
    const float2 a = row_tree<2 * D>(at, r), b = row_tree<2 * D>(at, r + D);
    return make_float2(a.x + b.x, a.y + b.y);
  }
}

template <int BN>
__global__ void __launch_bounds__(kActThreads, 1) gemm_act_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB,
                                                                  const __grid_constant__ CUtensorMap tmO, const __grid_constant__ CUtensorMap tmZ,
                                                                  GemmArgs g) {
  constexpr int STAGES = act_stages<BN>(), SETS = 256 / BN;  // warp sets that take tiles in turn
  extern __shared__ unsigned char smem_raw[];
  unsigned char* sA = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sB = sA + (size_t)STAGES * BM * BK * 2;
  unsigned char* stage = sB + (size_t)STAGES * BN * BK * 2;
  uint64_t* full = (uint64_t*)(stage + kActWarps * kStage);
  uint64_t* empty = full + STAGES;
  uint64_t* tfull = empty + STAGES;   // accumulator ready / read, per TMEM buffer
  uint64_t* tempty = tfull + 2;
  uint64_t* zbar = tempty + 2;        // one per epilogue warp (pre-activation tiles)
  uint32_t* tmem_slot = (uint32_t*)(zbar + kActWarps);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int nt = g.N / BN, ntiles = nt * (g.M / BM), KT = g.K / BK;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    for (int b = 0; b < 2; ++b) { mbar_init(&tfull[b], 1); mbar_init(&tempty[b], kActWarps / SETS); }
    for (int w = 0; w < kActWarps; ++w) mbar_init(&zbar[w], 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(2 * BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool ok = true;
  if (warp == 0) {
    if (lane == 0) {  // TMA producer
      int c = 0;
      for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x)
        for (int kt = 0; kt < KT; ++kt, ++c) {
          const int s = c % STAGES;
          if (!mbar_wait(&empty[s], ((uint32_t)(c / STAGES) & 1u) ^ 1u)) { ok = false; break; }
          mbar_expect_tx(&full[s], (unsigned)((BM + BN) * BK * 2));
          tma_load_2d(sA + (size_t)s * BM * BK * 2, &tmA, kt * BK, t / nt * BM, &full[s]);
          tma_load_2d(sB + (size_t)s * BN * BK * 2, &tmB, kt * BK, t % nt * BN, &full[s]);
        }
    }
  } else if (warp == 1) {
    if (lane == 0) {  // MMA issuer
      const uint32_t idesc = idesc_bf16<BN>(false);
      int c = 0, it = 0;
      for (int t = blockIdx.x; ok && t < ntiles; t += gridDim.x, ++it) {
        const uint32_t acc_addr = tmem + (uint32_t)(it & 1) * BN;
        if (!mbar_wait(&tempty[it & 1], ((uint32_t)(it >> 1) & 1u) ^ 1u)) { ok = false; break; }
        tc_fence_after();
        for (int kt = 0; kt < KT; ++kt, ++c) {
          const int s = c % STAGES;
          if (!mbar_wait(&full[s], (uint32_t)(c / STAGES) & 1u)) { ok = false; break; }
          tc_fence_after();
          const uint64_t ad = desc_sw128(sA + (size_t)s * BM * BK * 2), bd = desc_sw128(sB + (size_t)s * BN * BK * 2);
#pragma unroll
          for (int kk = 0; kk < BK / 16; ++kk) mma_f16(acc_addr, ad + 2 * kk, bd + 2 * kk, idesc, (kt | kk) != 0);
          mma_commit(&empty[s]);
        }
        mma_commit(&tfull[it & 1]);
      }
    }
  } else {
    const int e = warp - 2, set = e / (kActWarps / SETS), group = (e >> 2) % (BN / 64), quarter = warp & 3;
    unsigned char* buf = stage + e * kStage;
    uint64_t* zb = zbar + e;
    const bool dact = g.epi == EPI_DACT;
    auto load_z = [&](int t) {
      mbar_expect_tx(zb, kStage);
      tma_load_2d(buf, &tmZ, t % nt * BN + group * 64, t / nt * BM + quarter * 32, zb);
    };
    const int step = SETS * gridDim.x, t0 = blockIdx.x + set * gridDim.x;
    if (dact && lane == 0 && t0 < ntiles) load_z(t0);
    int h = 0;  // tiles of this warp
    for (int t = t0; t < ntiles; t += step, ++h) {
      const int it = h * SETS + set, col = t % nt * BN + group * 64, row0 = t / nt * BM + quarter * 32;
      ok = mbar_wait(&tfull[it & 1], (uint32_t)(it >> 1) & 1u) && (!dact || mbar_wait(zb, (uint32_t)h & 1u));
      ok = __all_sync(0xffffffffu, ok) != 0;  // the TMEM loads below are warp-collective
      if (!ok) break;
      tc_fence_after();
      uint4 zp[8];  // EPI_ACT: pre-activations, staged after the outputs
      if (!dact) {  // the last tile's stores have read the buffer (EPI_DACT: before its pre-activations were loaded)
        if (lane == 0) tma_store_wait_read();
        __syncwarp();
      }
#pragma unroll
      for (int hc = 0; hc < 2; ++hc) {
        uint32_t v[32];
        tmem_load32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)((it & 1) * BN + group * 64 + hc * 32), v);
        if (hc == 1) {  // the accumulator is in registers
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(&tempty[it & 1]);
        }
#pragma unroll
        for (int p = 0; p < 4; ++p) {  // 16-byte pieces of the lane's row
          const int off = lane * 128 + (((hc * 4 + p) ^ (lane & 7)) << 4);
          uint4 out, zz;
          unsigned* o = reinterpret_cast<unsigned*>(&out);
          unsigned* z = reinterpret_cast<unsigned*>(&zz);
          float4 b[2] = {};
          if (dact) {
            zz = *reinterpret_cast<const uint4*>(buf + off);
          } else if (g.bias) {
            b[0] = __ldg(reinterpret_cast<const float4*>(g.bias + col + hc * 32) + 2 * p);
            b[1] = __ldg(reinterpret_cast<const float4*>(g.bias + col + hc * 32) + 2 * p + 1);
          }
          const float* bias = reinterpret_cast<const float*>(b);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int j = 8 * p + 2 * q;
            if (dact) {
              const float d0 = __uint_as_float(v[j]), d1 = __uint_as_float(v[j + 1]);
              o[q] = g.act == ACT_SILU ? pack_bf16(d0 * dsilu(bf16_lo(z[q])), d1 * dsilu(bf16_hi(z[q]))) : pack_bf16(d0, d1);
            } else {
              const float z0 = __uint_as_float(v[j]) + bias[2 * q], z1 = __uint_as_float(v[j + 1]) + bias[2 * q + 1];
              z[q] = pack_bf16(z0, z1);
              o[q] = g.act == ACT_SILU ? pack_bf16(silu(z0), silu(z1)) : z[q];
            }
          }
          *reinterpret_cast<uint4*>(buf + off) = out;
          zp[hc * 4 + p] = zz;
        }
      }
      proxy_fence();
      __syncwarp();
      if (lane == 0) {
        tma_store_2d(&tmO, col, row0, buf);
        tma_store_commit();
      }
      if (!dact && g.z_out) {
        if (lane == 0) tma_store_wait_read();
        __syncwarp();
#pragma unroll
        for (int p = 0; p < 8; ++p) *reinterpret_cast<uint4*>(buf + lane * 128 + ((p ^ (lane & 7)) << 4)) = zp[p];
        proxy_fence();
        __syncwarp();
        if (lane == 0) {
          tma_store_2d(&tmZ, col, row0, buf);
          tma_store_commit();
        }
      }
      if (dact && g.colpart) {  // columns col + 2 lane, + 1 (the store above only reads the tile)
        auto at = [&](int r) { return *reinterpret_cast<const unsigned*>(buf + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + (lane & 3) * 4); };
        reinterpret_cast<float2*>(g.colpart + (size_t)(row0 / 32) * g.N + col)[lane] = row_tree<1>(at, 0);
      }
      if (dact && t + step < ntiles) {  // the next tile's pre-activations, once this tile is read
        __syncwarp();
        if (lane == 0) { tma_store_wait_read(); load_z(t + step); }
      }
    }
    if (lane == 0) tma_store_wait_read();  // shared memory is read; the writes are complete when the kernel is
  }
  __syncwarp();
  tc_fence_before();
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * BN) : "memory");
  if (!ok) atomicExch(g.err, 1u);
}

template <int BN>
__global__ void __launch_bounds__(kThreads, 2) gemm_tn_kernel(const __grid_constant__ CUtensorMap tmA,
                                                         const __grid_constant__ CUtensorMap tmB, const __grid_constant__ CUtensorMap tmD,
                                                         GemmArgs g) {
  constexpr int STAGES = stages_for<BN>();
  extern __shared__ unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* sA = base;
  unsigned char* sB = sA + (size_t)STAGES * BM * BK * 2;
  uint64_t* full = (uint64_t*)(sB + (size_t)STAGES * BN * BK * 2);
  uint64_t* empty = full + STAGES;
  uint64_t* done = empty + STAGES;
  uint32_t* tmem_slot = (uint32_t*)(done + 1);
  float* sbias = (float*)(tmem_slot + 4);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int n0 = blockIdx.x * BN, m0 = blockIdx.y * BM;
  // split-K (EPI_F32 only): CTA z owns K-steps [kt0, kt0 + KT) of the g.K / BK
  const int KTall = g.K / BK;
  const int kt0 = (int)((long long)KTall * blockIdx.z / gridDim.z);
  const int KT = (int)((long long)KTall * (blockIdx.z + 1) / gridDim.z) - kt0;
  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) { mbar_init(&full[s], 1); mbar_init(&empty[s], 1); }
    mbar_init(done, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int j = threadIdx.x; j < BN; j += kThreads) sbias[j] = (g.bias && n0 + j < g.n_valid) ? g.bias[n0 + j] : 0.0f;
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(BN) : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  bool ok = true;
  if (warp == 0 && lane == 0) {  // TMA producer
    for (int kt = 0; kt < KT; ++kt) {
      const int s = kt % STAGES;
      const uint32_t ph = (uint32_t)(kt / STAGES) & 1u;
      if (!mbar_wait(&empty[s], ph ^ 1u)) { ok = false; break; }
      mbar_expect_tx(&full[s], (unsigned)((BM + BN) * BK * 2));
      unsigned char* a = sA + (size_t)s * BM * BK * 2;
      unsigned char* b = sB + (size_t)s * BN * BK * 2;
      const int k0 = (kt0 + kt) * BK;
      if (g.rows_k) {
        for (int i = 0; i < BM / 64; ++i) tma_load_2d(a + i * 8192, &tmA, m0 + i * 64, k0, &full[s]);
        for (int i = 0; i < BN / 64; ++i) tma_load_2d(b + i * 8192, &tmB, n0 + i * 64, k0, &full[s]);
      } else {
        tma_load_2d(a, &tmA, k0, m0, &full[s]);
        tma_load_2d(b, &tmB, k0, n0, &full[s]);
      }
    }
  } else if (warp == 1 && lane == 0) {  // MMA issuer
    const bool rows_k = g.rows_k;
    const uint32_t idesc = idesc_bf16<BN>(rows_k);
    const uint64_t kstep = rows_k ? 2048 >> 4 : 32 >> 4;  // 16 elements of K: 16 rows, or 32 B inside the swizzled row
    for (int kt = 0; kt < KT; ++kt) {
      const int s = kt % STAGES;
      const uint32_t ph = (uint32_t)(kt / STAGES) & 1u;
      if (!mbar_wait(&full[s], ph)) { ok = false; break; }
      tc_fence_after();
      const unsigned char* a = sA + (size_t)s * BM * BK * 2;
      const unsigned char* b = sB + (size_t)s * BN * BK * 2;
      const uint64_t ad = rows_k ? desc_sw128_rows_k(a) : desc_sw128(a), bd = rows_k ? desc_sw128_rows_k(b) : desc_sw128(b);
#pragma unroll
      for (int kk = 0; kk < BK / 16; ++kk) {
        mma_f16(tmem, ad + kstep * kk, bd + kstep * kk, idesc, (kt | kk) != 0);
      }
      mma_commit(&empty[s]);
    }
    mma_commit(done);
  }
  __syncwarp();
  // epilogue: thread = tile row m0 + 32 (warp mod 4) + lane, columns of half warp / 4
  if (!mbar_wait(done, 0)) ok = false;
  ok = __syncthreads_and(ok) != 0;  // CTA-uniform: the TMEM loads below are warp-collective
  tc_fence_after();
  const int quarter = warp & 3, half = warp >> 2;
  const int row = m0 + quarter * 32 + lane;
  // 16-byte accesses along the rows of whatever the epilogue touches
  const uintptr_t bases = g.epi == EPI_F32 ? (uintptr_t)g.out_f32 : (uintptr_t)g.out_bf16 | (uintptr_t)(g.epi == EPI_ACT ? g.z_out : g.z_in);
  const bool vec_rows = g.ldo % 8 == 0 && (bases & 15) == 0;
  if (ok && g.part) {
    // split K: 32 x 32 tiles staged in the operand ring (12 KB per warp, three buffers; rows of 128 bytes,
    // 128-byte swizzle) and stored by TMA, each split in its own rows; whoever reads them adds them in the splits'
    // order.  Added here (by TMA or atomics, in the order of arrival) a gradient differed in its last bits from run
    // to run, which BF16 weights and Adam's quotient grew to 1e-5 of the weights in 16 steps
    unsigned char* buf = base + warp * 12288;
    int q = 0;
#pragma unroll 1
    for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32, ++q) {
      uint32_t v[32];
      tmem_load32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
      unsigned char* b = buf + q % 3 * 4096;
      if (q >= 3) {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 2;" ::: "memory");
        __syncwarp();
      }
#pragma unroll
      for (int p = 0; p < 8; ++p) *reinterpret_cast<uint4*>(b + lane * 128 + ((p ^ (lane & 7)) << 4)) = make_uint4(v[4 * p], v[4 * p + 1], v[4 * p + 2], v[4 * p + 3]);
      proxy_fence();
      __syncwarp();
      if (lane == 0) { tma_store_2d(&tmD, n0 + c0, blockIdx.z * g.M + m0 + quarter * 32, b); tma_store_commit(); }
    }
    if (lane == 0) tma_store_wait_read();
    __syncwarp();
  } else if (ok) {
#pragma unroll 1
    for (int c0 = half * (BN / 2); c0 < (half + 1) * (BN / 2); c0 += 32) {
      uint32_t v[32];
      tmem_load32(tmem + ((uint32_t)(quarter * 32) << 16) + (uint32_t)c0, v);
      const int col = n0 + c0;
      if (col >= g.n_valid) continue;  // warp-uniform
      const bool live = row < g.M;
      const size_t o = (size_t)row * g.ldo + col;
      const int nv = min(32, g.n_valid - col);
      const bool vec = nv == 32 && vec_rows;
      if (g.epi == EPI_F32) {
        if (!live) continue;
        float* out = g.out_f32 + o;
        if (gridDim.z > 1) {
          if (vec) {
#pragma unroll
            for (int q = 0; q < 8; ++q)
              atomicAdd(reinterpret_cast<float4*>(out) + q, make_float4(__uint_as_float(v[4 * q]), __uint_as_float(v[4 * q + 1]),
                                                                         __uint_as_float(v[4 * q + 2]), __uint_as_float(v[4 * q + 3])));
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) if (j < nv) atomicAdd(out + j, __uint_as_float(v[j]));
          }
        } else {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            if (j >= nv) continue;
            const float d = __uint_as_float(v[j]);
            out[j] = g.accumulate ? out[j] + d : d;
          }
        }
        continue;
      }
      unsigned yp[16];  // bf16 pairs of the stored row
      if (g.epi == EPI_ACT) {
        unsigned zp[16];
#pragma unroll
        for (int p = 0; p < 16; ++p) {
          const float z0 = __uint_as_float(v[2 * p]) + sbias[c0 + 2 * p], z1 = __uint_as_float(v[2 * p + 1]) + sbias[c0 + 2 * p + 1];
          zp[p] = pack_bf16(z0, z1);
          yp[p] = g.act == ACT_SILU ? pack_bf16(silu(z0), silu(z1)) : zp[p];
        }
        if (live) {
          if (vec) {
            uint4* dst = reinterpret_cast<uint4*>(g.out_bf16 + o);
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[q] = make_uint4(yp[4 * q], yp[4 * q + 1], yp[4 * q + 2], yp[4 * q + 3]);
            if (g.z_out) {
              uint4* dz = reinterpret_cast<uint4*>(g.z_out + o);
#pragma unroll
              for (int q = 0; q < 4; ++q) dz[q] = make_uint4(zp[4 * q], zp[4 * q + 1], zp[4 * q + 2], zp[4 * q + 3]);
            }
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j) {
              if (j >= nv) continue;
              const unsigned short yj = (unsigned short)((j & 1) ? yp[j >> 1] >> 16 : yp[j >> 1] & 0xFFFFu);
              const unsigned short zj = (unsigned short)((j & 1) ? zp[j >> 1] >> 16 : zp[j >> 1] & 0xFFFFu);
              g.out_bf16[o + j] = __ushort_as_bfloat16(yj);
              if (g.z_out) g.z_out[o + j] = __ushort_as_bfloat16(zj);
            }
          }
        }
      } else {  // EPI_DACT
        unsigned zp[16];
        if (live && vec) {
          const uint4* src = reinterpret_cast<const uint4*>(g.z_in + o);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const uint4 t = src[q];
            zp[4 * q] = t.x; zp[4 * q + 1] = t.y; zp[4 * q + 2] = t.z; zp[4 * q + 3] = t.w;
          }
        } else {
#pragma unroll
          for (int p = 0; p < 16; ++p) {
            const unsigned a = (live && 2 * p < nv) ? (unsigned)__bfloat16_as_ushort(g.z_in[o + 2 * p]) : 0u;
            const unsigned b = (live && 2 * p + 1 < nv) ? (unsigned)__bfloat16_as_ushort(g.z_in[o + 2 * p + 1]) : 0u;
            zp[p] = a | (b << 16);
          }
        }
#pragma unroll
        for (int p = 0; p < 16; ++p) {
          const float d0 = (live && 2 * p < nv) ? __uint_as_float(v[2 * p]) : 0.0f;
          const float d1 = (live && 2 * p + 1 < nv) ? __uint_as_float(v[2 * p + 1]) : 0.0f;
          yp[p] = g.act == ACT_SILU ? pack_bf16(d0 * dsilu(bf16_lo(zp[p])), d1 * dsilu(bf16_hi(zp[p]))) : pack_bf16(d0, d1);
        }
        if (live) {
          if (vec) {
            uint4* dst = reinterpret_cast<uint4*>(g.out_bf16 + o);
#pragma unroll
            for (int q = 0; q < 4; ++q) dst[q] = make_uint4(yp[4 * q], yp[4 * q + 1], yp[4 * q + 2], yp[4 * q + 3]);
          } else {
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < nv) g.out_bf16[o + j] = __ushort_as_bfloat16((unsigned short)((j & 1) ? yp[j >> 1] >> 16 : yp[j >> 1] & 0xFFFFu));
          }
        }
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (warp == 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(BN) : "memory");
  if (!ok && lane == 0) atomicExch(g.err, 1u);
}

}  // namespace mlp
}  // namespace sbz
