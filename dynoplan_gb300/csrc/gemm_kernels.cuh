// gemm_kernels.cuh -- BF16 GEMM on the 5th-generation tensor cores (sm_103a).
//
//   C[M x N] = A[M x K] * B[N x K]^T      A, B bf16 row-major (K contiguous),
//                                          FP32 accumulation in tensor memory
//
// One CTA of 128 threads computes a 128-row tile with every N column (N a
// multiple of 16, <= 256) in one tcgen05.mma chain of M=128 x N x K=16
// instructions; gridDim.y splits K.  K is consumed in chunks of 64 (one
// 128-byte swizzle atom) staged into two shared-memory buffers: threads
// stage chunk i+1 while the tensor cores run chunk i; an mbarrier that the
// MMA commit arrives on tells the stagers when a buffer is free again.
// Every wait is bounded: on expiry the kernel sets *err, drains, frees its
// tensor memory and returns.  The epilogue reads one accumulator row per
// thread (tcgen05.ld 32x32b) and hands 16 columns at a time to `Epi`.
#pragma once

#include <cuda.h>
#include <cuda_bf16.h>

#include "f32x2.cuh"
#include "umma.cuh"

namespace dpg {

constexpr int kGemmThreads = 128;
constexpr int kGemmKChunk = 64;

__host__ __device__ constexpr int tmem_cols_for(int n) {
  return n <= 32 ? 32 : (n <= 64 ? 64 : (n <= 128 ? 128 : 256));
}
__host__ __device__ constexpr size_t gemm_smem_bytes(int N) {
  // two stages of (A 128x64 + B Nx64) bf16, 1024-aligned, + barriers + slack
  return 2 * (size_t)(128 * 128 + N * 128) + 1024 + 64;
}

template <int N, class Epi>
__global__ void __launch_bounds__(kGemmThreads) gemm_bf16_tn(const __nv_bfloat16 *__restrict__ A,
                                                              const __nv_bfloat16 *__restrict__ B, int M,
                                                              int K, int k_per_split, Epi epi, int *err) {
  static_assert(N % 16 == 0 && N >= 16 && N <= 256, "N");
  extern __shared__ unsigned char smem_raw[];
  // 1024-byte aligned stage buffers
  const uint32_t raw = umma::smem_u32(smem_raw);
  unsigned char *base = smem_raw + ((1024 - (raw & 1023)) & 1023);
  constexpr int kA = 128 * 128, kB = N * 128;
  unsigned char *tileA[2] = {base, base + kA + kB};
  unsigned char *tileB[2] = {base + kA, base + 2 * kA + kB};
  uint64_t *mbar = reinterpret_cast<uint64_t *>(base + 2 * (kA + kB));
  uint32_t *tslot = reinterpret_cast<uint32_t *>(mbar + 2);
  __shared__ int s_bad;

  const int m0 = blockIdx.x * 128;
  const int kbeg = blockIdx.y * k_per_split;
  const int kend = min(K, kbeg + k_per_split);
  const int nchunks = (kend - kbeg) / kGemmKChunk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t kCols = tmem_cols_for(N);
  constexpr uint32_t idesc = umma::idesc_bf16_f32(128, N);

  if (threadIdx.x == 0) {
    umma::mbar_init(&mbar[0], 1);
    umma::mbar_init(&mbar[1], 1);
    umma::mbar_fence_init();
    s_bad = 0;
  }
  if (warp == 0) {
    umma::tmem_alloc(tslot, kCols);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot;
  const int rows_valid = min(128, M - m0);

  bool bad = false;
  int issued = 0;  // chunks whose MMAs were issued (identical in every thread)
  for (int i = 0; i < nchunks && !bad; i++) {
    const int s = i & 1;
    if (i >= 2) {  // buffer s is free once the MMAs of chunk i-2 are done
      bool ok = umma::mbar_wait(&mbar[s], ((i - 2) >> 1) & 1);
      if (__syncthreads_or(!ok)) { bad = true; break; }
    }
    const int k0 = kbeg + i * kGemmKChunk;
    umma::stage_kmajor(tileA[s], A + (int64_t)m0 * K, K, 128, rows_valid, k0, 1);
    umma::stage_kmajor(tileB[s], B, K, N, N, k0, 1);
    umma::fence_proxy_async_smem();
    __syncthreads();
    if (threadIdx.x == 0) {
      umma::fence_after_sync();
      const uint32_t a0 = umma::smem_u32(tileA[s]), b0 = umma::smem_u32(tileB[s]);
#pragma unroll
      for (int kk = 0; kk < kGemmKChunk / 16; kk++)
        umma::mma_bf16(tmem, umma::sdesc_kmajor_sw128(a0 + kk * 32), umma::sdesc_kmajor_sw128(b0 + kk * 32),
                       idesc, (i > 0 || kk > 0) ? 1u : 0u);
      umma::commit(&mbar[s]);
    }
    issued = i + 1;
  }
  if (!bad && nchunks > 0) {  // all MMAs done
    const int last = nchunks - 1;
    bool ok = umma::mbar_wait(&mbar[last & 1], (last >> 1) & 1);
    bad = __syncthreads_or(!ok);
  }
  if (bad) {
    if (threadIdx.x == 0) atomicExch(err, 1);
    // let in-flight MMAs finish before the tensor memory is released
    if (issued > 0) umma::mbar_wait(&mbar[(issued - 1) & 1], ((issued - 1) >> 1) & 1, 1u << 20);
  } else if (nchunks > 0) {
    umma::fence_after_sync();
    const int row = 32 * warp + lane;
    const uint32_t lane_addr = tmem + ((uint32_t)(32 * warp) << 16);
#pragma unroll 1
    for (int c0 = 0; c0 < N; c0 += 16) {
      float v[16];
      umma::tmem_ld16(lane_addr + c0, v);
      if (m0 + row < M) epi(m0 + row, c0, v);
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, kCols);
}

// ---- TMA-fed, warp-specialised form ------------------------------------------
//
// Same contract and tile (128 rows x all N columns in TMEM, K in 64-wide
// SW128 k-blocks), but the operands arrive by TMA (cp.async.bulk.tensor,
// 128-byte swizzle written by the copy engine) into a ring of S stages:
// thread 0 of warp 0 issues the loads, thread 0 of warp 1 the MMAs; a stage
// is refilled once the MMAs that read it have committed to its `empty`
// barrier.  All four warps run the epilogue.  Rows beyond M load as zeros.
// Every wait is bounded; on expiry the kernel sets *err, waits (bounded)
// for its copies and MMAs in flight, frees its tensor memory and returns.
__host__ __device__ constexpr int tma_stages(int N) {
  return (110 * 1024) / (128 * 128 + N * 128) < 2 ? 2
         : ((110 * 1024) / (128 * 128 + N * 128) > 4 ? 4 : (110 * 1024) / (128 * 128 + N * 128));
}
// deeper ring for long K (one CTA per SM): up to 200 KB of stages
__host__ __device__ constexpr int tma_stages_deep(int N) {
  return (200 * 1024) / (128 * 128 + N * 128) < 2 ? 2
         : ((200 * 1024) / (128 * 128 + N * 128) > 6 ? 6 : (200 * 1024) / (128 * 128 + N * 128));
}
__host__ __device__ constexpr size_t gemm_tma_smem_bytes(int N, int S) {
  return (size_t)S * (128 * 128 + N * 128) + 1024 + 256;
}

constexpr int kTmaThreads = 256;  // 8 warps: all of them drain the accumulator

template <int N, class Epi, int S = tma_stages(N)>
__global__ void __launch_bounds__(kTmaThreads) gemm_bf16_tma(const __grid_constant__ CUtensorMap tmA,
                                                               const __grid_constant__ CUtensorMap tmB, int M,
                                                               int K, int k_per_split, Epi epi, int *err) {
  static_assert(N % 16 == 0 && N >= 16 && N <= 256, "N");
  static_assert(S >= 2, "stages");
  constexpr uint32_t kA = 128 * 128, kB = N * 128, kStage = kA + kB;
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = umma::smem_u32(smem_raw);
  unsigned char *base = smem_raw + ((1024 - (raw & 1023)) & 1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(base + S * kStage);
  uint64_t *empty = full + S;
  uint64_t *done = empty + S;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
  __shared__ int s_bad;

  const int m0 = blockIdx.x * 128;
  const int kbeg = blockIdx.y * k_per_split;
  const int kend = min(K, kbeg + k_per_split);
  const int nchunks = (kend - kbeg) / kGemmKChunk;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  constexpr uint32_t kCols = tmem_cols_for(N);
  constexpr uint32_t idesc = umma::idesc_bf16_f32(128, N);

  if (threadIdx.x == 0) {
    for (int s = 0; s < S; s++) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], 1);
    }
    umma::mbar_init(done, 1);
    umma::mbar_fence_init();
    s_bad = 0;
  }
  if (warp == 0) {
    umma::tmem_alloc(tslot, kCols);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot;

  int loads = 0;  // (thread 0) chunks whose loads were issued
  if (threadIdx.x == 0) {
    // producer
    for (int i = 0; i < nchunks; i++) {
      const int s = i % S;
      if (i >= S && !umma::mbar_wait(&empty[s], ((i / S) - 1) & 1)) {
        s_bad = 1;
        break;
      }
      if (*(volatile int *)&s_bad) break;
      unsigned char *a = base + s * kStage;
      umma::mbar_arrive_expect_tx(&full[s], kStage);
      umma::tma_load_2d(a, &tmA, kbeg + i * kGemmKChunk, m0, &full[s]);
      umma::tma_load_2d(a + kA, &tmB, kbeg + i * kGemmKChunk, 0, &full[s]);
      loads = i + 1;
    }
  } else if (threadIdx.x == 32) {
    // MMA issuer
    for (int i = 0; i < nchunks; i++) {
      const int s = i % S;
      if (!umma::mbar_wait(&full[s], (i / S) & 1)) {
        s_bad = 1;
        break;
      }
      umma::fence_after_sync();
      const uint32_t a0 = umma::smem_u32(base + s * kStage), b0 = a0 + kA;
#pragma unroll
      for (int kk = 0; kk < kGemmKChunk / 16; kk++)
        umma::mma_bf16(tmem, umma::sdesc_kmajor_sw128(a0 + kk * 32), umma::sdesc_kmajor_sw128(b0 + kk * 32),
                       idesc, (i > 0 || kk > 0) ? 1u : 0u);
      umma::commit(&empty[s]);
    }
    umma::commit(done);  // arrives once every MMA issued above is complete
  }
  // warp w reads accumulator lanes 32 (w % 4) ...; warps 0-3 and 4-7 split
  // the columns in halves (all columns in warps 0-3 when N / 2 is not a
  // multiple of 16)
  constexpr int kHalves = (N % 32 == 0) ? 2 : 1, kNC = N / kHalves;
  const int h = warp >> 2, row = 32 * (warp & 3) + lane;
  const bool mine = h < kHalves && m0 + row < M && nchunks > 0;
  constexpr int kPre = Epi::kPrefetch ? kNC / 2 : 1;
  uint32_t pre[kPre];  // the epilogue's operands, in flight during the wait
  if constexpr (Epi::kPrefetch) {
    __syncwarp();
    if (mine) {
#pragma unroll
      for (int c = 0; c < kNC; c += 16) epi.load(m0 + row, h * kNC + c, pre + c / 2);
    }
  }
  // everyone: the accumulator is final once `done` completes
  const bool ok = nchunks > 0 && umma::mbar_wait(done, 0);
  const bool bad = __syncthreads_or(!ok || s_bad) && nchunks > 0;
  if (bad) {
    if (threadIdx.x == 0) {
      atomicExch(err, 1);
      // copies still in flight land before the block's shared memory goes
      for (int i = max(0, loads - S); i < loads; i++) umma::mbar_wait(&full[i % S], (i / S) & 1, 1u << 20);
    }
  } else if (nchunks > 0 && h < kHalves) {
    umma::fence_after_sync();
    const uint32_t lane_addr = tmem + ((uint32_t)(32 * (warp & 3)) << 16);
    if constexpr (Epi::kPrefetch) {
#pragma unroll
      for (int c = 0; c < kNC; c += 16) {
        float v[16];
        umma::tmem_ld16(lane_addr + h * kNC + c, v);
        if (mine) epi(m0 + row, h * kNC + c, v, pre + c / 2);
      }
    } else {
#pragma unroll 2
      for (int c0 = h * kNC; c0 < (h + 1) * kNC; c0 += 16) {
        float v[16];
        umma::tmem_ld16(lane_addr + c0, v);
        if (mine) epi(m0 + row, c0, v);
      }
    }
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, kCols);
}

// ---- epilogues ---------------------------------------------------------------
// 16 consecutive FP32 values as four 16-byte stores (dst 16-byte aligned)
__device__ __forceinline__ void store16(float *dst, const float *v) {
#pragma unroll
  for (int j = 0; j < 4; j++)
    reinterpret_cast<float4 *>(dst)[j] = make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]);
}

struct EpiStoreF32 {  // C = acc (ldc = row stride, only columns < n_valid)
  static constexpr bool kPrefetch = false;
  float *C;
  int ldc, n_valid;
  __device__ void operator()(int row, int c0, const float *v) const {
    float *dst = C + (int64_t)row * ldc + c0;
    if (c0 + 16 <= n_valid && (ldc & 3) == 0) {
      store16(dst, v);
      return;
    }
#pragma unroll
    for (int j = 0; j < 16; j++)
      if (c0 + j < n_valid) dst[j] = v[j];
  }
};
struct EpiAtomicF32 {  // C += acc (split-K partial sums)
  static constexpr bool kPrefetch = false;
  float *C;
  int ldc, n_valid;
  __device__ void operator()(int row, int c0, const float *v) const {
    float *dst = C + (int64_t)row * ldc + c0;
    if (c0 + 16 <= n_valid && (ldc & 3) == 0) {  // 16-byte vector atomics
#pragma unroll
      for (int j = 0; j < 4; j++)
        atomicAdd(reinterpret_cast<float4 *>(dst) + j, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
      return;
    }
#pragma unroll
    for (int j = 0; j < 16; j++)
      if (c0 + j < n_valid) atomicAdd(dst + j, v[j]);
  }
};

// GELU in its tanh form (Hendrycks & Gimpel, "Gaussian Error Linear Units",
// 2016): gelu(z) = z/2 (1 + tanh(u)), u = sqrt(2/pi) (z + 0.044715 z^3), with
// the hardware tanh (tanh.approx.f32, max relative error about 2^-11, below
// the bf16 rounding the activations get).
__device__ __forceinline__ float tanh_fast(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
constexpr float kGeluA = 0.7978845608028654f, kGeluB = 0.044715f;
__device__ __forceinline__ float gelu(float z) {
  const float t = tanh_fast(kGeluA * z * fmaf(kGeluB * z, z, 1.0f));
  return 0.5f * z * (1.0f + t);
}

// gelu and its derivative, (1 + t) / 2 + z / 2 (1 - t^2) u', of two values, with
// the roundings of the form above
__device__ __forceinline__ uint64_t gelu2_tanh(uint64_t z, uint64_t f) {
  float u0, u1;
  unpack2(mul2(mul2(pack2(kGeluA, kGeluA), z), f), u0, u1);
  return pack2(tanh_fast(u0), tanh_fast(u1));
}
__device__ __forceinline__ uint64_t gelu2_poly(uint64_t z) {
  return fma2(mul2(pack2(kGeluB, kGeluB), z), z, pack2(1.f, 1.f));
}
__device__ __forceinline__ uint64_t gelu2(uint64_t z) {
  const uint64_t t = gelu2_tanh(z, gelu2_poly(z));
  return mul2(mul2(pack2(0.5f, 0.5f), z), add2(pack2(1.f, 1.f), t));
}
__device__ __forceinline__ void gelu2_both(uint64_t z, uint64_t &h, uint64_t &d) {
  const uint64_t one = pack2(1.f, 1.f), half = pack2(0.5f, 0.5f);
  const uint64_t t = gelu2_tanh(z, gelu2_poly(z)), t1 = add2(one, t), hz = mul2(half, z);
  h = mul2(hz, t1);
  const uint64_t du = mul2(pack2(kGeluA, kGeluA), fma2(mul2(pack2(3.0f * kGeluB, 3.0f * kGeluB), z), z, one));
  const uint64_t e = fma2(t ^ 0x8000000080000000ull, t, one);  // 1 - t^2
  d = fma2(half, t1, mul2(mul2(hz, e), du));
}
// two values rounded to bf16 (the first in the low half)
__device__ __forceinline__ uint32_t to_bf16x2(uint64_t v) {
  float x, y;
  unpack2(v, x, y);
  const __nv_bfloat162 p = __floats2bfloat162_rn(x, y);
  return *reinterpret_cast<const uint32_t *>(&p);
}
__device__ __forceinline__ uint64_t from_bf16x2(uint32_t w) {
  return pack2(__uint_as_float(w << 16), __uint_as_float(w & 0xffff0000u));
}
// 32 bytes of one thread, a whole sector (p 32-byte aligned)
__device__ __forceinline__ void store32(void *p, const uint32_t *w) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(w[0]), "r"(w[1]), "r"(w[2]),
               "r"(w[3]), "r"(w[4]), "r"(w[5]), "r"(w[6]), "r"(w[7])
               : "memory");
}
__device__ __forceinline__ void load32(const void *p, uint32_t *w) {
  asm volatile("ld.global.v8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
               : "=r"(w[0]), "=r"(w[1]), "=r"(w[2]), "=r"(w[3]), "=r"(w[4]), "=r"(w[5]), "=r"(w[6]), "=r"(w[7])
               : "l"(p));
}

// z = acc + bias; writes gelu(z) in bf16, and gelu'(z) in bf16 for the backward
// pass when dgelu != nullptr.  Bound by the epilogue's issue and its two stores
// of a row's 32-byte pieces; packed arithmetic and whole-sector stores, two
// groups of columns in flight: 48.6 -> 38.5 us for 65,536 rows, K = 256.
struct EpiBiasGelu {
  static constexpr bool kPrefetch = false;
  const float *bias;
  __nv_bfloat16 *dgelu;
  __nv_bfloat16 *act;
  int ld;  // a multiple of 16
  __device__ void operator()(int row, int c0, const float *v) const {
    uint32_t h[8], d[8];
#pragma unroll
    for (int j = 0; j < 8; j++) {
      const float2 b = __ldg(reinterpret_cast<const float2 *>(bias + c0) + j);
      const uint64_t z = add2(pack2(b.x, b.y), pack2(v[2 * j], v[2 * j + 1]));
      uint64_t hh, dd;
      gelu2_both(z, hh, dd);
      h[j] = to_bf16x2(hh);
      d[j] = to_bf16x2(dd);
    }
    if (dgelu) store32(dgelu + (int64_t)row * ld + c0, d);
    store32(act + (int64_t)row * ld + c0, h);
  }
};
// dZ = dH * gelu'(Z) (gelu' kept in bf16 by the forward epilogue): the epilogue
// of dH = dZnext * W.  A thread's gelu' values are loaded before it waits for
// the accumulator (46 -> 25.5 us for 65,536 rows: the loads' latency was paid
// for every 16 columns).
struct EpiGeluGrad {
  static constexpr bool kPrefetch = true;
  const __nv_bfloat16 *dgelu;
  __nv_bfloat16 *dz;
  int ld;  // a multiple of 16
  __device__ void load(int row, int c0, uint32_t *d) const { load32(dgelu + (int64_t)row * ld + c0, d); }
  __device__ void operator()(int row, int c0, const float *v, const uint32_t *d) const {
    uint32_t h[8];
#pragma unroll
    for (int j = 0; j < 8; j++) h[j] = to_bf16x2(mul2(pack2(v[2 * j], v[2 * j + 1]), from_bf16x2(d[j])));
    store32(dz + (int64_t)row * ld + c0, h);
  }
  __device__ void operator()(int row, int c0, const float *v) const {
    uint32_t d[8];
    load(row, c0, d);
    (*this)(row, c0, v, d);
  }
};
// out = acc + bias (FP32), first n_valid columns of the first `rows` rows (the
// GEMM's row count is padded to its tile; out holds no more than these)
struct EpiBias {
  static constexpr bool kPrefetch = false;
  const float *bias;
  float *out;
  int ld, n_valid;
  int64_t rows;
  __device__ void operator()(int row, int c0, const float *v) const {
    if (row >= rows) return;
#pragma unroll
    for (int j = 0; j < 16; j++)
      if (c0 + j < n_valid) out[(int64_t)row * ld + c0 + j] = v[j] + bias[c0 + j];
  }
};

// ---- SIMT reference (CUDA cores, FP32 accumulation) ---------------------------
static __global__ void gemm_bf16_ref(const __nv_bfloat16 *A, const __nv_bfloat16 *B, float *C, int M, int N, int K) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= (int64_t)M * N) return;
  const int m = (int)(i / N), n = (int)(i % N);
  float s = 0.f;
  for (int k = 0; k < K; k++) s += __bfloat162float(A[(int64_t)m * K + k]) * __bfloat162float(B[(int64_t)n * K + k]);
  C[i] = s;
}

}  // namespace dpg
