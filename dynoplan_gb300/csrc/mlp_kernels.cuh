// mlp_kernels.cuh -- element-wise and data-movement kernels of the surrogate
// MLP (the GEMMs are gemm_kernels.cuh).
//
// Input row of a (node, primitive) pair, 128 bf16 (K of the first GEMM is a
// multiple of 64; columns 96..127 are zero):
//   [0, 16)   node state, normalised (position to [-1, 1] over the
//             environment box, angles / pi, velocities / 4), zero padded
//   [16, 80)  8 x 8 occupancy patch around the node: cell (i, j) is 1 when its
//             box overlaps an obstacle (0.75 m cells, patch centred on the
//             node, world-aligned)
//   [80, 96)  the primitive's learned 16-D embedding
// Outputs per pair: [collision logit, cost-to-go].
#pragma once

#include <cuda_bf16.h>

#include "expand_kernels.cuh"
#include "gemm_kernels.cuh"

namespace dpg {

constexpr int kMlpIn = 128, kMlpNodeFeat = 80, kMlpEmb = 16, kMlpHidden = 256, kMlpOutPad = 16;
constexpr int kOccSide = 8;
constexpr float kOccCell = 0.75f;

// goal the cost-to-go refers to: slots 13.. of the state block hold
// (goal - position), normalised like the position
struct GoalView {
  int has;
  double g[3];
};

// The environment box as the features use it.
struct FeatureScale {
  double lo[3], ext[3], inv[3];  // lower bound, extent, 1 / extent
  int ok[3];  // the extent is not zero
};

// eight bf16 values to dst, at once when it is 16-byte aligned (vec)
__device__ __forceinline__ void store8(__nv_bfloat16 *dst, uint4 v, bool vec) {
  if (vec) {
    *reinterpret_cast<uint4 *>(dst) = v;
    return;
  }
  const __nv_bfloat16 *h = reinterpret_cast<const __nv_bfloat16 *>(&v);
#pragma unroll
  for (int i = 0; i < 8; i++) dst[i] = h[i];
}

// a / b from inv = 1 / b as rounded: the product corrected by its remainder,
// which gives the rounded quotient (P. Markstein, "Computation of elementary
// functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990).
// Three FP64 operations; a division each took 100,000 quadrotor nodes with a goal
// from 43.7 to 54.4 us.  An infinite product (exponent bits all ones) has no
// remainder.
__device__ __forceinline__ double divide_by(double a, double b, double inv) {
  const double q = a * inv, r = fma(fma(-q, b, a), inv, q);
  return (__double2hiint(q) & 0x7ff00000) == 0x7ff00000 ? q : r;
}

// normalised state of one node (16 values)
template <int KIND>
__device__ __forceinline__ void node_state_features(const double *x, const FeatureScale &fs, const GoalView &gv, float *s) {
  using R = Robot<KIND>;
#pragma unroll
  for (int i = 0; i < 16; i++) s[i] = 0.f;
#pragma unroll
  for (int i = 0; i < R::POSD; i++) s[i] = fs.ok[i] ? (float)fma(2.0, divide_by(x[i] - fs.lo[i], fs.ext[i], fs.inv[i]), -1.0) : 0.f;
#pragma unroll
  for (int i = R::POSD; i < R::NX; i++) {
    const bool raw = KIND == DPG_ROBOT_QUAD3D && i < 7;
    const bool angle = KIND != DPG_ROBOT_QUAD3D && (i == 2 || (KIND == DPG_ROBOT_CAR1 && i == 3));
    s[i] = angle ? wrap_pi_f64(x[i]) * 0.31830988618f : (float)(raw ? x[i] : x[i] * 0.25);
  }
  if (gv.has) {
#pragma unroll
    for (int i = 0; i < R::POSD; i++) s[13 + i] = fs.ok[i] ? (float)(2.0 * divide_by(gv.g[i] - x[i], fs.ext[i], fs.inv[i])) : 0.f;
  }
}

// Per node: normalised state + occupancy patch (80 bf16).  A block of 256
// threads takes 32 nodes, eight lanes a node.  The patch is separable: an
// obstacle covers the cells (i, j) whose column i overlaps it in x and whose
// row j does in y, so it costs 8 + 8 tests and one outer product of two bytes
// instead of 64 cell tests; lane t of a node takes the obstacles t, t + 8, ..,
// the eight 64-bit masks are combined by shuffles and each lane writes the
// eight cells of a row as 16 bytes.  Warp 0 also writes the states, a lane a
// node (FP64, which runs at 1/64 of the FP32 rate: all lanes busy, and
// multiplications by the host's 2 / extent for divisions).
// Bound by instruction issue; 100,000 car1 nodes, 80 obstacles: 27 us,
// against 405 us for a thread per node testing 64 cells one after the other.
constexpr int kFeatNodes = 32;
template <int KIND>
__global__ void __launch_bounds__(8 * kFeatNodes) mlp_node_features(NodeView nv, EnvView ev, FeatureScale fs, GoalView gv,
                                                                    __nv_bfloat16 *feat) {
  using R = Robot<KIND>;
  static_assert(kOccSide == 8 && kMlpNodeFeat == 16 + 64, "a byte a row, eight rows");
  const int64_t n0 = (int64_t)blockIdx.x * kFeatNodes;
  const bool vec = (reinterpret_cast<uintptr_t>(feat) & 15) == 0;  // 16-byte stores
  if (threadIdx.x < kFeatNodes && n0 + threadIdx.x < nv.N) {
    const int64_t n = n0 + threadIdx.x;
    float s[16];
    node_state_features<KIND>(nv.x64 + n * R::NX, fs, gv, s);
    __align__(16) __nv_bfloat16 h[16];
#pragma unroll
    for (int i = 0; i < 16; i++) h[i] = __float2bfloat16_rn(s[i]);
    __nv_bfloat16 *f = feat + n * kMlpNodeFeat;  // rows of 160 bytes
    store8(f, reinterpret_cast<const uint4 *>(h)[0], vec);
    store8(f + 8, reinterpret_cast<const uint4 *>(h)[1], vec);
  }
  const int t = threadIdx.x & 7;
  const int64_t n = n0 + (threadIdx.x >> 3);
  const double *x = nv.x64 + min(n, nv.N - 1) * R::NX;
  const float px = (float)x[0], py = (float)x[1], pz = R::POSD == 3 ? (float)x[2] : 0.f;
  const float h = 0.5f * kOccCell;
  float cx[8], cy[8];  // cell centres
#pragma unroll
  for (int i = 0; i < 8; i++) {
    cx[i] = px + (i - 3.5f) * kOccCell;
    cy[i] = py + (i - 3.5f) * kOccCell;
  }
  uint32_t lo = 0u, hi = 0u;  // rows 0-3, 4-7: a byte a row, bit i = column i
  using Ob = std::conditional_t<R::POSD == 3, Obs3<float>, Obs2<float>>;
  const Ob *obs = (const Ob *)ev.obs32;
  for (int o = t; o < ev.n_obs; o += 8) {
    const Ob ob = obs[o];
    if constexpr (R::POSD == 3) {
      if (!(fabsf(pz - ob.cz) <= h + ob.hz)) continue;
    }
    uint32_t mx = 0u, my = 0u;
#pragma unroll
    for (int i = 0; i < 8; i++) {
      if (fabsf(cx[i] - ob.cx) <= h + ob.hx) mx |= 1u << i;
      if (fabsf(cy[i] - ob.cy) <= h + ob.hy) my |= 1u << i;
    }
    // four bits to the low bits of four bytes, times the byte of columns
    lo |= (((my & 15u) * 0x00204081u) & 0x01010101u) * mx;
    hi |= (((my >> 4) * 0x00204081u) & 0x01010101u) * mx;
  }
#pragma unroll
  for (int d = 1; d < 8; d <<= 1) {
    lo |= __shfl_xor_sync(0xffffffffu, lo, d);
    hi |= __shfl_xor_sync(0xffffffffu, hi, d);
  }
  if (n >= nv.N) return;
  const uint32_t row = ((t < 4 ? lo : hi) >> (8 * (t & 3))) & 0xffu;
  uint32_t w[4];  // 1.0 in bf16 is 0x3f80
#pragma unroll
  for (int i = 0; i < 4; i++) w[i] = ((row >> (2 * i)) & 1u) * 0x3f80u | ((row >> (2 * i + 1)) & 1u) * 0x3f800000u;
  store8(feat + n * kMlpNodeFeat + 16 + 8 * t, make_uint4(w[0], w[1], w[2], w[3]), vec);
}

// X[b] = [node_feat[node[b]] | emb[prim[b]] | 0], one thread per 16-byte chunk
static __global__ void mlp_assemble(const __nv_bfloat16 *node_feat, const __nv_bfloat16 *emb, const uint32_t *node,
                                    const uint32_t *prim, int64_t B, int64_t B_pad, __nv_bfloat16 *X) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int64_t b = i / (kMlpIn / 8);
  const int c = (int)(i % (kMlpIn / 8));
  if (b >= B_pad) return;
  uint4 v = make_uint4(0, 0, 0, 0);
  if (b < B) {
    if (c < kMlpNodeFeat / 8)
      v = reinterpret_cast<const uint4 *>(node_feat + (int64_t)node[b] * kMlpNodeFeat)[c];
    else if (c < (kMlpNodeFeat + kMlpEmb) / 8)
      v = reinterpret_cast<const uint4 *>(emb + (int64_t)prim[b] * kMlpEmb)[c - kMlpNodeFeat / 8];
  }
  reinterpret_cast<uint4 *>(X)[i] = v;
}

__device__ __forceinline__ float softplus(float x) { return x > 20.f ? x : log1pf(__expf(x)); }
__device__ __forceinline__ float sigmoid(float x) { return 1.f / (1.f + __expf(-x)); }

// The training step's head: [l, c] = acc + bias, then
//   loss = mean_b [softplus(l) - y l  +  0.5 w (c - t)^2]
// (a NaN target leaves its head out of the loss).  Writes dY = d loss / d [l, c]
// (bf16, rows of 64; columns 0-15 of every row, the others are zero from the
// start) and adds the loss to *loss_sum and the column sums of dY, the head's
// bias gradient, to db.  The step's hyper-parameters [lr, w, ..] live in device
// memory, so that a captured step can be replayed with new values.  (A launch
// of its own for the loss took 10.7 us at 65,536 rows, the head's GEMM 11.9.)
struct EpiHeadLoss {
  static constexpr bool kPrefetch = false;
  const float *bias, *target, *hp;
  int64_t B;
  __nv_bfloat16 *dY;
  double *loss_sum;
  float *db;
  __device__ void operator()(int row, int c0, const float *v) const {  // c0 = 0, whole warps
    const float w = hp[1];
    float l = 0.f, g0 = 0.f, g1 = 0.f;
    uint32_t d[8] = {};
    if (row < B) {
      const float lg = v[0] + bias[0], ct = v[1] + bias[1];
      const float2 yt = reinterpret_cast<const float2 *>(target)[row];
      const float inv = 1.f / (float)B;
      __nv_bfloat162 g = __floats2bfloat162_rn(0.f, 0.f);
      if (!isnan(yt.x)) {
        l += softplus(lg) - yt.x * lg;
        g.x = __float2bfloat16_rn((sigmoid(lg) - yt.x) * inv);
      }
      if (!isnan(yt.y)) {
        l += 0.5f * w * (ct - yt.y) * (ct - yt.y);
        g.y = __float2bfloat16_rn(w * (ct - yt.y) * inv);
      }
      d[0] = *reinterpret_cast<const uint32_t *>(&g);
      g0 = __bfloat162float(g.x);
      g1 = __bfloat162float(g.y);
    }
    store32(dY + (int64_t)row * 64, d);
    for (int o = 16; o > 0; o >>= 1) {
      l += __shfl_down_sync(0xffffffffu, l, o);
      g0 += __shfl_down_sync(0xffffffffu, g0, o);
      g1 += __shfl_down_sync(0xffffffffu, g1, o);
    }
    if ((threadIdx.x & 31) == 0) {
      if (l != 0.f) atomicAdd(loss_sum, (double)l);
      if (g0 != 0.f) atomicAdd(db, g0);
      if (g1 != 0.f) atomicAdd(db + 1, g1);
    }
  }
};

// dE[prim[b]] += dX[b, 80:96]: the epilogue of the 16-column product
// dZ1 * W1[:, 80:96] (the embedding part of the layer-1 input gradient)
struct EpiEmbGrad {
  static constexpr bool kPrefetch = false;
  const uint32_t *prim;
  float *demb;
  int64_t B;
  __device__ void operator()(int row, int c0, const float *v) const {
    if (row >= B) return;
    float4 *dst = reinterpret_cast<float4 *>(demb + (int64_t)prim[row] * kMlpEmb);
#pragma unroll
    for (int j = 0; j < 4; j++) atomicAdd(dst + j, make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
  }
};

// out[C x R] = in[R x C]^T (bf16), 32x32 tiles
static __global__ void transpose_bf16(const __nv_bfloat16 *in, __nv_bfloat16 *out, int64_t R, int64_t C) {
  __shared__ __nv_bfloat16 t[32][33];
  const int64_t r0 = blockIdx.x * (int64_t)32, c0 = blockIdx.y * 32;
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int64_t r = r0 + i, c = c0 + threadIdx.x;
    t[i][threadIdx.x] = (r < R && c < C) ? in[r * C + c] : __float2bfloat16_rn(0.f);
  }
  __syncthreads();
  for (int i = threadIdx.y; i < 32; i += blockDim.y) {
    const int64_t c = c0 + i, r = r0 + threadIdx.x;
    if (c < C && r < R) out[c * R + r] = t[threadIdx.x][i];
  }
}

// out[c] += sum_r in[r x 256 + c]: a thread a column over 512 rows a block, 32 at a time
static __global__ void __launch_bounds__(kMlpHidden) column_sums(const __nv_bfloat16 *in, int64_t rows, float *out) {
  float s = 0.f;
  const int64_t end = min(rows, (blockIdx.x + (int64_t)1) * 512);
  for (int64_t r0 = blockIdx.x * (int64_t)512; r0 < end; r0 += 32) {
    float p = 0.f;
    for (int64_t r = r0; r < min(end, r0 + 32); r++) p += __bfloat162float(in[r * kMlpHidden + threadIdx.x]);
    s += p;
  }
  atomicAdd(out + threadIdx.x, s);
}

// ---------------------------------------------------------------------------
// Weight and bias gradients of all four layers in one launch:
//   g[m][n] += sum_b a[b][m] b[b][n]      a, b bf16 row-major, a row per pair
// (layers 1-3: a = dZ, b = the layer's input; layer 4: a = H3, b = dY, stored
// transposed).  The contraction runs over the rows, so both operands are read
// MN-major straight from the row-major activations (boxes of 64 rows x 64
// columns by TMA): no transposed copies are written.  A layer's CTAs take
// ranges of 64-row chunks; a CTA holds the whole gradient, two M = 128 tiles of
// up to 256 columns, in TMEM, so each operand is read once, and adds it to g
// (float4 atomics) at the end or after every kWgRun chunks an accumulator: longer
// runs' error against 64 bits exceeds that of sums over 900 rows (rms of dW3 at
// 65,536 rows of one sign 2.3e-6, 1.2e-6 with 900 rows, 0.95e-6 with these).  Warps 4-7 sum the columns of a (the bias
// gradients) from the staged tiles while the tensor cores use them.
// Bound by reading the operands (2 x 33.5 MB a hidden layer at 65,536 rows):
// all four layers 49 us; as transposed copies written by the layers'
// epilogues (another 230 MB) and a split-K launch per layer 155 us, without the
// writes.  Every wait is bounded, as above.
struct alignas(128) WgradJob {
  CUtensorMap a, b;  // boxes of 64 columns x 64 rows
  float *g, *db;     // db: column sums of a (may be null)
  int ld, n;         // row stride of g; columns of b used (multiple of 16)
  int transposed;    // g[n][m] (the two non-zero columns of dY) instead of g[m][n]
  int cta0, ctas;    // the layer's CTAs
};
struct alignas(128) WgradArgs {
  WgradJob job[4];
};
constexpr int kWgThreads = 256, kWgStages = 3, kWgRun = 14;
constexpr uint32_t kWgBlock = 64 * 128;        // 64 rows x 64 columns
constexpr uint32_t kWgStage = 8 * kWgBlock;    // a: 256 columns, b: up to 256
constexpr size_t kWgSmem = 1024 + kWgStages * kWgStage + 256;

static __global__ void __launch_bounds__(kWgThreads, 1) mlp_wgrad(const __grid_constant__ WgradArgs A, int64_t n_chunks,
                                                                  int *err) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = umma::smem_u32(smem_raw);
  unsigned char *base = smem_raw + ((1024 - (raw & 1023)) & 1023);
  uint64_t *full = reinterpret_cast<uint64_t *>(base + kWgStages * kWgStage);
  uint64_t *empty = full + kWgStages, *done = empty + kWgStages;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
  volatile int *bad = reinterpret_cast<volatile int *>(tslot + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  int ji = 0;
  while (ji < 3 && (int)blockIdx.x >= A.job[ji].cta0 + A.job[ji].ctas) ji++;
  const WgradJob &J = A.job[ji];
  const int64_t rel = (int)blockIdx.x - J.cta0;
  const int64_t c0 = n_chunks * rel / J.ctas, c1 = n_chunks * (rel + 1) / J.ctas;
  const int n = (int)(c1 - c0), b_blocks = (J.n + 63) / 64;
  const uint32_t bytes = (4 + b_blocks) * kWgBlock;
  if (tid == 0) {
    for (int s = 0; s < kWgStages; s++) {
      umma::mbar_init(&full[s], 1);
      umma::mbar_init(&empty[s], J.db ? 5 : 1);  // the MMAs, and the four summing warps
    }
    umma::mbar_init(done, 1);
    umma::mbar_fence_init();
    *bad = 0;
  }
  if (warp == 0) {
    umma::tmem_alloc(tslot, 512);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot;

  // Accumulators: the tensor cores cut a sum's low bits at every step of 16 rows,
  // so one takes at most kWgRun chunks.  Chunk i goes to accumulator i % sets
  // (256 columns of TMEM hold several of a narrow layer's); a CTA with more than
  // sets * kWgRun chunks adds its accumulators to g several times.
  const int stride = J.n <= 32 ? 32 : J.n <= 128 ? 128 : 256, sets = 256 / stride;
  const int runs = (n + sets * kWgRun - 1) / (sets * kWgRun);
  int loads = 0;  // (thread 0) chunks whose loads were issued
  uint32_t ms = 0, mparity = 0;  // (warp 1) the next stage, parity of its next completion
  float s0 = 0.f, s1 = 0.f;      // (warps 4-7) column sums
  bool failed = false;
  for (int run = 0; run < runs && !failed; run++) {
    const int i0 = (int)((int64_t)n * run / runs), i1 = (int)((int64_t)n * (run + 1) / runs);
    if (tid == 0) {
      for (; loads < min(n, i1 + kWgStages); loads++) {  // and the next run's first ones
        const int s = loads % kWgStages;
        if ((loads >= kWgStages && !umma::mbar_wait(&empty[s], ((loads / kWgStages) - 1) & 1)) || *bad) {
          *bad = 1;
          break;
        }
        unsigned char *st = base + s * kWgStage;
        const int row = (int)(64 * (c0 + loads));
        umma::mbar_arrive_expect_tx(&full[s], bytes);
        for (int k = 0; k < 4; k++) umma::tma_load_2d(st + k * kWgBlock, &J.a, 64 * k, row, &full[s]);
        for (int k = 0; k < b_blocks; k++) umma::tma_load_2d(st + (4 + k) * kWgBlock, &J.b, 64 * k, row, &full[s]);
      }
    } else if (warp == 1) {
      const uint32_t idesc = umma::idesc_bf16_f32(128, J.n) | umma::kIdescMnMajorAB;
      const uint64_t ad = umma::sdesc_mnmajor_sw128(umma::smem_u32(base), kWgBlock);
      const uint64_t bd = ad + (4 * kWgBlock >> 4);
      bool ok = true;
      umma::fence_after_sync();
      for (int i = i0; i < i1; i++) {
        if (!umma::mbar_wait_warp(&full[ms], mparity)) {
          ok = false;
          break;
        }
        umma::fence_after_sync();
        const uint64_t so = ms * (kWgStage >> 4);
        const uint32_t acc = tmem + (uint32_t)((i - i0) % sets * stride);
        if (umma::elect_one()) {
#pragma unroll
          for (int mt = 0; mt < 2; mt++)
#pragma unroll
            for (int kk = 0; kk < 4; kk++)  // 16 rows a step
              umma::mma_bf16(acc + 256u * mt, ad + so + mt * (2 * kWgBlock >> 4) + kk * (2048 >> 4),
                             bd + so + kk * (2048 >> 4), idesc, (i - i0 >= sets || kk > 0) ? 1u : 0u);
          umma::commit(&empty[ms]);
        }
        __syncwarp();
        if (++ms == kWgStages) {
          ms = 0;
          mparity ^= 1u;
        }
      }
      if (!ok && lane == 0) *bad = 1;
      if (umma::elect_one()) umma::commit(done);  // once every MMA issued above is complete
      __syncwarp();
    } else if (warp >= 4 && J.db) {
      // column sums of a: a thread two columns (word w of block k), over the rows,
      // 32 at a time (a running sum over a CTA's 1,500 rows loses small ones)
      const int k = warp - 4;
      for (int i = i0; i < i1; i++) {
        const int s = i % kWgStages;
        if (!umma::mbar_wait_warp(&full[s], (i / kWgStages) & 1)) {
          if (lane == 0) *bad = 1;
          break;
        }
        const unsigned char *t = base + s * kWgStage + k * kWgBlock;
#pragma unroll
        for (int r0 = 0; r0 < 64; r0 += 32) {
          float p0 = 0.f, p1 = 0.f;
#pragma unroll 16
          for (int r = r0; r < r0 + 32; r++) {
            const uint32_t v = *reinterpret_cast<const uint32_t *>(t + r * 128 + (((lane >> 2) ^ (r & 7)) << 4) + 4 * (lane & 3));
            p0 += __uint_as_float(v << 16);
            p1 += __uint_as_float(v & 0xffff0000u);
          }
          s0 += p0;
          s1 += p1;
        }
        __syncwarp();
        if (lane == 0) umma::mbar_arrive(&empty[s]);
      }
    }
    __syncwarp();
    const bool fin = umma::mbar_wait(done, run & 1);
    failed = __syncthreads_or(!fin || *bad);
    if (failed) break;
    umma::fence_after_sync();
    const int q = warp & 3, mt = warp >> 2, m = 128 * mt + 32 * q + lane;
    const uint32_t src = tmem + ((uint32_t)(32 * q) << 16) + 256u * (uint32_t)mt;
    for (int c = 0; c < J.n; c += 16) {
      const int k = (c + 16 * (int)rel) % J.n;  // (the layer's CTAs start at different columns)
      float v[16];
      umma::tmem_ld16(src + k, v);
      for (int a = 1; a < min(sets, i1 - i0); a++) {
        float u[16];
        umma::tmem_ld16(src + a * stride + k, u);
#pragma unroll
        for (int e = 0; e < 16; e++) v[e] += u[e];
      }
      if (J.transposed) {
        atomicAdd(J.g + m, v[0]);
        atomicAdd(J.g + J.ld + m, v[1]);
      } else {
        // four lanes exchange their rows' 16-byte pieces, so that an instruction adds
        // 64 bytes of a row (a piece of each row is half of a sector: the atomics of
        // two runs took 6 us more of a step)
#pragma unroll
        for (int d = 1; d < 4; d <<= 1)
#pragma unroll
          for (int j = 0; j < 4; j++) {
            if (j & d) continue;
#pragma unroll
            for (int e = 0; e < 4; e++) {
              const float a = v[4 * j + e], b = v[4 * (j + d) + e];
              const float o = __shfl_xor_sync(0xffffffffu, lane & d ? a : b, d);
              v[4 * j + e] = lane & d ? o : a;
              v[4 * (j + d) + e] = lane & d ? b : o;
            }
          }
#pragma unroll
        for (int j = 0; j < 4; j++)
          atomicAdd(reinterpret_cast<float4 *>(J.g + (int64_t)((m & ~3) + j) * J.ld + k) + (lane & 3),
                    make_float4(v[4 * j], v[4 * j + 1], v[4 * j + 2], v[4 * j + 3]));
      }
    }
    umma::fence_before_sync();
    __syncthreads();  // the next run's MMAs write the accumulators
  }
  if (failed) {
    if (tid == 0) {
      atomicExch(err, 1);
      // copies still in flight land before the block's shared memory goes
      for (int i = max(0, loads - kWgStages); i < loads; i++)
        umma::mbar_wait(&full[i % kWgStages], (i / kWgStages) & 1, 1u << 20);
    }
  } else if (warp >= 4 && J.db && n > 0) {
    atomicAdd(J.db + 64 * (warp - 4) + 2 * lane, s0);
    atomicAdd(J.db + 64 * (warp - 4) + 2 * lane + 1, s1);
  }
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

// Adam over every parameter in one launch: segment s is elements
// [start[s], start[s + 1]) of the concatenation; the bf16 copy (w16) and the
// transposed bf16 copy (wT[(k % cols) * ldT + k / cols]) are written when set.
struct AdamSeg {
  float *w, *m, *v;
  const float *g;
  __nv_bfloat16 *w16, *wT;
  int cols, ldT;
};
constexpr int kAdamSegs = 9;
struct AdamArgs {
  AdamSeg seg[kAdamSegs];
  int64_t start[kAdamSegs + 1];
};
static __global__ void adam_all(AdamArgs a, const float *hp, float b1, float b2, float eps) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= a.start[kAdamSegs]) return;
  int s = 0;
  while (s + 1 < kAdamSegs && i >= a.start[s + 1]) s++;
  const AdamSeg &q = a.seg[s];
  const int64_t k = i - a.start[s];
  const float lr = hp[0], bc1 = hp[2], bc2 = hp[3];
  const float gi = q.g[k];
  const float mi = b1 * q.m[k] + (1.f - b1) * gi;
  const float vi = b2 * q.v[k] + (1.f - b2) * gi * gi;
  q.m[k] = mi;
  q.v[k] = vi;
  const float wi = q.w[k] - lr * (mi / bc1) / (sqrtf(vi / bc2) + eps);
  q.w[k] = wi;
  if (q.w16) q.w16[k] = __float2bfloat16_rn(wi);
  if (q.wT) q.wT[(k % q.cols) * q.ldT + k / q.cols] = __float2bfloat16_rn(wi);
}

static __global__ void f32_to_bf16(const float *in, __nv_bfloat16 *out, int64_t n) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i < n) out[i] = __float2bfloat16_rn(in[i]);
}

// ---------------------------------------------------------------------------
// Fused forward: the whole MLP for 128-row tiles in one persistent kernel.
//
// One CTA per SM (512 threads) walks tiles m0 = 128 * (blockIdx.x + k *
// gridDim.x).  A tile's activations live in one 64 KB shared-memory buffer
// (128 rows x 256 bf16, SW128 K-major): the gathered input [node features |
// embedding | 0] first, then H1, H2, H3, each written over the previous
// one once the layer's MMAs have read it.  Accumulators (128 x 256 FP32)
// sit in TMEM; the epilogue adds the bias, applies GELU and writes bf16
// back into the buffer.  W1..W3 stream by TMA in 64-column chunks (32 KB)
// into four stages -- a whole layer -- while the previous epilogue runs;
// W4 (16 x 256) stays resident.  Thread 0 issues every TMA and MMA.
// Every wait is bounded: on expiry the kernel sets *err, drains its copies
// and MMAs (bounded), frees TMEM and returns.
struct FusedArgs {
  const __nv_bfloat16 *node_feat, *emb;
  const uint32_t *node, *prim;
  const float *b1, *b2, *b3, *b4;
  float *out;  // [B x 2]
  int64_t B;
  int *err;
};
constexpr int kFusedThreads = 512;  // 16 warps: 4 per accumulator lane quarter
constexpr uint32_t kActBytes = 128 * kMlpHidden * 2;        // 64 KB
constexpr uint32_t kWChunk = kMlpHidden * 128;              // 256 rows x 64 bf16 = 32 KB
constexpr uint32_t kW4Bytes = kMlpOutPad * kMlpHidden * 2;  // 8 KB
constexpr size_t kFusedSmem = 1024 + kActBytes + 4 * kWChunk + kW4Bytes + 256;

static __global__ void __launch_bounds__(kFusedThreads, 1)
    mlp_forward_fused(const __grid_constant__ CUtensorMap tw1, const __grid_constant__ CUtensorMap tw2,
                      const __grid_constant__ CUtensorMap tw3, const __grid_constant__ CUtensorMap tw4, FusedArgs a) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = umma::smem_u32(smem_raw);
  unsigned char *act = smem_raw + ((1024 - (raw & 1023)) & 1023);
  unsigned char *wst = act + kActBytes;           // 4 weight stages
  unsigned char *w4 = wst + 4 * kWChunk;          // resident W4, 4 k-blocks of 16 rows
  uint64_t *wfull = reinterpret_cast<uint64_t *>(w4 + kW4Bytes);  // [4]
  uint64_t *w4full = wfull + 4;
  uint64_t *done = w4full + 1;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(done + 1);
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t n_tiles = (a.B + 127) / 128;
  __shared__ __align__(16) float sbias[3][kMlpHidden];  // b1..b3, read by the epilogues
  for (int i = tid; i < 3 * kMlpHidden; i += kFusedThreads)
    sbias[i / kMlpHidden][i % kMlpHidden] = (i < kMlpHidden ? a.b1 : (i < 2 * kMlpHidden ? a.b2 : a.b3))[i % kMlpHidden];
  const void *wmap[3] = {&tw1, &tw2, &tw3};
  constexpr uint32_t kIdesc = umma::idesc_bf16_f32(128, kMlpHidden);
  constexpr uint32_t kIdesc4 = umma::idesc_bf16_f32(128, kMlpOutPad);

  if (tid == 0) {
    for (int s = 0; s < 4; s++) umma::mbar_init(&wfull[s], 1);
    umma::mbar_init(w4full, 1);
    umma::mbar_init(done, 1);
    umma::mbar_fence_init();
  }
  if (warp == 0) {
    umma::tmem_alloc(tslot, 256);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot;

  // thread 0's bookkeeping: phase of each weight stage, loads in flight
  uint32_t wphase = 0;      // bit s: parity of the next completion of stage s
  uint32_t inflight = 0;    // bit s: a load into stage s not yet waited for
  uint32_t done_phase = 0;  // parity of the next `done` completion
  bool w4_inflight = false;
  auto load_layer = [&](int l) {  // all chunks of W(l+1), l = 0..2
    const int chunks = (l == 0 ? kMlpIn : kMlpHidden) / 64;
    for (int j = 0; j < chunks; j++) {
      umma::mbar_arrive_expect_tx(&wfull[j], kWChunk);
      umma::tma_load_2d(wst + j * kWChunk, wmap[l], 64 * j, 0, &wfull[j]);
      inflight |= 1u << j;
    }
  };
  if (tid == 0 && blockIdx.x < n_tiles) {
    umma::mbar_arrive_expect_tx(w4full, kW4Bytes);
    for (int j = 0; j < 4; j++) umma::tma_load_2d(w4 + j * (kMlpOutPad * 128), &tw4, 64 * j, 0, w4full);
    w4_inflight = true;
    load_layer(0);
  }
  bool w4_ready = false;
  bool bad = false;  // this thread saw a wait expire; block-wide decisions use __syncthreads_or

  for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
    const int64_t m0 = t * 128;
    // ---- gather the input rows into the buffer (k-blocks 0 and 1)
    for (int i = tid; i < 128 * (kMlpIn / 8); i += kFusedThreads) {
      const int r = i / (kMlpIn / 8), c = i % (kMlpIn / 8);
      const int64_t b = m0 + r;
      uint4 v = make_uint4(0, 0, 0, 0);
      if (b < a.B) {
        if (c < kMlpNodeFeat / 8)
          v = reinterpret_cast<const uint4 *>(a.node_feat + (int64_t)a.node[b] * kMlpNodeFeat)[c];
        else if (c < (kMlpNodeFeat + kMlpEmb) / 8)
          v = reinterpret_cast<const uint4 *>(a.emb + (int64_t)a.prim[b] * kMlpEmb)[c - kMlpNodeFeat / 8];
      }
      *reinterpret_cast<uint4 *>(act + umma::kmajor_offset(128, r, c)) = v;
    }
    umma::fence_proxy_async_smem();
    umma::fence_before_sync();
    __syncthreads();

    for (int l = 0; l < 4; l++) {
      // ---- MMAs of layer l (thread 0)
      if (tid == 0) {
        umma::fence_after_sync();
        const uint32_t a0 = umma::smem_u32(act);
        if (l < 3) {
          const int chunks = (l == 0 ? kMlpIn : kMlpHidden) / 64;
          for (int j = 0; j < chunks && !bad; j++) {
            if (!umma::mbar_wait(&wfull[j], (wphase >> j) & 1)) { bad = true; break; }
            wphase ^= 1u << j;
            inflight &= ~(1u << j);
            umma::fence_after_sync();
            const uint32_t b0 = umma::smem_u32(wst + j * kWChunk), ak = a0 + j * (128 * 128);
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
              umma::mma_bf16(tmem, umma::sdesc_kmajor_sw128(ak + kk * 32), umma::sdesc_kmajor_sw128(b0 + kk * 32),
                             kIdesc, (j > 0 || kk > 0) ? 1u : 0u);
          }
        } else {
          if (!w4_ready) {
            if (umma::mbar_wait(w4full, 0)) {
              w4_ready = true;
              w4_inflight = false;
            } else {
              bad = true;
            }
          }
          for (int j = 0; j < 4 && !bad; j++) {
            const uint32_t b0 = umma::smem_u32(w4 + j * (kMlpOutPad * 128)), ak = a0 + j * (128 * 128);
#pragma unroll
            for (int kk = 0; kk < 4; kk++)
              umma::mma_bf16(tmem, umma::sdesc_kmajor_sw128(ak + kk * 32), umma::sdesc_kmajor_sw128(b0 + kk * 32),
                             kIdesc4, (j > 0 || kk > 0) ? 1u : 0u);
          }
        }
        umma::commit(done);  // also after an expired wait: arrives once the issued MMAs are done
      }
      // ---- wait for the accumulator; refill the weight stages
      if (umma::mbar_wait(done, done_phase)) done_phase ^= 1u;
      else bad = true;
      if (tid == 0 && !bad) {
        if (l == 0) load_layer(1);
        else if (l == 1) load_layer(2);
        else if (l == 2 && t + gridDim.x < n_tiles) load_layer(0);  // the next tile's W1
      }
      umma::fence_after_sync();
      // ---- epilogue: warps w, w + 4, w + 8, w + 12 share accumulator lanes
      // 32 (w % 4), 64 columns each
      const int q = warp & 3, h = warp >> 2, row = 32 * q + lane;
      const uint32_t lane_addr = tmem + ((uint32_t)(32 * q) << 16);
      if (l < 3 && !bad) {
        const float *bias = sbias[l];
#pragma unroll 1
        for (int c0 = 64 * h; c0 < 64 * (h + 1); c0 += 32) {
          float v[32];
          umma::tmem_ld32(lane_addr + c0, v);
          __align__(16) __nv_bfloat162 hb[16];
#pragma unroll
          for (int j = 0; j < 16; j++)
            hb[j] = __floats2bfloat162_rn(gelu(v[2 * j] + bias[c0 + 2 * j]), gelu(v[2 * j + 1] + bias[c0 + 2 * j + 1]));
#pragma unroll
          for (int k = 0; k < 4; k++)
            *reinterpret_cast<uint4 *>(act + umma::kmajor_offset(128, row, c0 / 8 + k)) =
                reinterpret_cast<const uint4 *>(hb)[k];
        }
        umma::fence_proxy_async_smem();
      } else if (l == 3 && !bad && h == 0) {
        float v[16];
        umma::tmem_ld16(lane_addr, v);
        const int64_t b = m0 + row;
        if (b < a.B) {
          a.out[b * 2] = v[0] + a.b4[0];
          a.out[b * 2 + 1] = v[1] + a.b4[1];
        }
      }
      umma::fence_before_sync();
      bad = __syncthreads_or(bad);  // the same decision in every thread
      if (bad) break;
    }
    if (bad) break;
  }
  if (bad && tid == 0) {
    atomicExch(a.err, 1);
    // copies still in flight land, and MMAs finish, before the memory goes
    for (int s = 0; s < 4; s++)
      if (inflight & (1u << s)) umma::mbar_wait(&wfull[s], (wphase >> s) & 1, 1u << 20);
    if (w4_inflight) umma::mbar_wait(w4full, 0, 1u << 20);
    umma::mbar_wait(done, done_phase, 1u << 20);
  }
  if (!bad && tid == 0 && w4_inflight) umma::mbar_wait(w4full, 0, 1u << 20);  // no tile: W4 never used
  umma::fence_before_sync();
  __syncthreads();
  if (warp == 0) umma::tmem_dealloc(tmem, 256);
}


// ---------------------------------------------------------------------------
// The same forward, warp-specialised, with two tiles in flight per CTA: while
// the epilogue warps turn one tile's accumulator into its next activations,
// the tensor cores run the other tile's layer.  Each of the two tile slots has
// 64 KB of shared memory (128 rows x 256 bf16, SW128 K-major) for the input
// rows and the activations, each written over the last, and 256 columns of
// TMEM.  Warps 0-15 run the epilogues, warp 16 (one lane) streams W1..W3 by TMA
// through a ring of 32-column K-chunks, warp 17 issues the MMAs, warps 18-21
// gather input rows, a thread a row, and write the outputs.  Order of the work,
// for the MMAs and the epilogues alike: layer 1 of slots 0 and 1, layer 2 of
// both, layer 3 of both, then the next two tiles.
//
// Layer l + 1 of a slot starts once the epilogue has read layer l's accumulator
// and written its activations (hready), layer 1 of the next tile once layer 3's
// accumulator was read (accfree) and the slot refilled (xready), which starts
// once the layer-3 MMAs have read the activations (xfree).  H3 stays in
// registers: the two outputs are dot products with the two rows of W4, summed
// over the four column groups by the gather warps before they refill the slot.
// Biases and W4 are in shared memory (read through L1, a layer's epilogue took
// 5,800 clocks instead of 3,350): with chunks of 32 columns (64-byte swizzle)
// the ring needs 80 KB, which leaves the room, and N = 256 keeps the input
// operand's reads at one a k-step.
// The epilogue's FP32 arithmetic is packed two columns an instruction
// (fma.rn.f32x2); with 16 tanh a clock an SM it needs 2,048 clocks a layer
// (measured 2,600 to 3,000 with its hand-over), the MMAs 2,048 (768 for layer
// 1, whose columns past 96 are zero and left out; measured 3,000 to 4,000 while
// both slots' weights stream from L2, which bounds the kernel now).
// 1,048,576 pairs: 0.39 ms, a call 0.405 ms, 0.42 of the measured bf16 peak (one tile in
// flight, two accumulators alternating by layer: 0.596 ms, 0.29); 65,536 pairs
// 36 us (53), one tile 17 us (19).  Measured beside it: eight epilogue warps a
// slot 5 % slower; chunks of 128 rows x 64 columns (N = 128) 20 % slower.
// Every wait is bounded: on expiry the kernel sets *err, waits (bounded) for its
// copies and MMAs in flight, frees TMEM and returns.
constexpr int kFwdThreads = 704;  // 16 epilogue warps + TMA warp + MMA warp + 4 gather warps
constexpr int kFwdEpiWarps = 16;
constexpr int kFwdGatherThreads = 128;
constexpr int kFwdStages = 5;
constexpr int kFwdK = 32;                              // columns of a weight chunk
constexpr uint32_t kFwdChunk = kMlpHidden * kFwdK * 2;  // 256 rows x 32 bf16 = 16 KB
// biases of layers 1-3, W4's two rows (FP32), partial outputs [slot][column group][row]
constexpr uint32_t kFwdConst = (3 + 2) * kMlpHidden * 4, kFwdPart = 2 * 4 * 128 * 8;
constexpr size_t kFwdSmem = 1024 + 2 * kActBytes + kFwdStages * kFwdChunk + kFwdConst + kFwdPart + 256;

static __global__ void __launch_bounds__(kFwdThreads, 1)
    mlp_forward_pair(const __grid_constant__ CUtensorMap tw1, const __grid_constant__ CUtensorMap tw2,
                     const __grid_constant__ CUtensorMap tw3, const __nv_bfloat16 *__restrict__ w4, FusedArgs a) {
  extern __shared__ unsigned char smem_raw[];
  const uint32_t raw = umma::smem_u32(smem_raw);
  unsigned char *act = smem_raw + ((1024 - (raw & 1023)) & 1023);  // two slots
  unsigned char *wst = act + 2 * kActBytes;                        // weight stages
  float *sbias = reinterpret_cast<float *>(wst + kFwdStages * kFwdChunk);       // [3][256]
  float *sw4 = sbias + 3 * kMlpHidden;                                          // [2][256]
  float2 *spart = reinterpret_cast<float2 *>(sw4 + 2 * kMlpHidden);             // [slot][group][128]
  uint64_t *wfull = reinterpret_cast<uint64_t *>(spart + 2 * 4 * 128);          // [stages]
  uint64_t *wempty = wfull + kFwdStages;                                       // [stages]
  uint64_t *hready = wempty + kFwdStages;                                      // [2]
  uint64_t *xready = hready + 2;                                               // [2]
  uint64_t *xfree = xready + 2;                                                // [2]
  uint64_t *accfull = xfree + 2;                                               // [2]
  uint64_t *accfree = accfull + 2;                                             // [2]
  uint64_t *pready = accfree + 2;                                              // [2]
  uint64_t *drain = pready + 2;
  uint32_t *tslot = reinterpret_cast<uint32_t *>(drain + 1);
  volatile int *bad = reinterpret_cast<volatile int *>(tslot + 1), *consumed = bad + 1, *mma_done = bad + 2;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int64_t n_tiles = (a.B + 127) / 128;
  // tile of slot s in iteration i
  auto tile_at = [&](int i, int s) { return blockIdx.x + (int64_t)(2 * i + s) * gridDim.x; };
  constexpr uint32_t kIdesc = umma::idesc_bf16_f32(128, kMlpHidden);
  for (int i = tid; i < 5 * kMlpHidden; i += kFwdThreads) {
    const int l = i / kMlpHidden, c = i % kMlpHidden;
    sbias[i] = l < 3 ? (l == 0 ? a.b1 : l == 1 ? a.b2 : a.b3)[c] : __bfloat162float(w4[(l - 3) * kMlpHidden + c]);
  }
  if (tid == 0) {
    for (int s = 0; s < kFwdStages; s++) {
      umma::mbar_init(&wfull[s], 1);
      umma::mbar_init(&wempty[s], 1);
    }
    for (int s = 0; s < 2; s++) {
      umma::mbar_init(&hready[s], kFwdEpiWarps);
      umma::mbar_init(&pready[s], kFwdEpiWarps);
      umma::mbar_init(&xready[s], kFwdGatherThreads / 32);
      umma::mbar_init(&xfree[s], 1);
      umma::mbar_init(&accfull[s], 1);
      umma::mbar_init(&accfree[s], kFwdEpiWarps);
    }
    umma::mbar_init(drain, 1);
    umma::mbar_fence_init();
    *bad = 0;
    *consumed = 0;
    *mma_done = 0;
  }
  if (warp == 0) {
    umma::tmem_alloc(tslot, 512);
    umma::tmem_relinquish();
  }
  umma::fence_before_sync();
  __syncthreads();
  umma::fence_after_sync();
  const uint32_t tmem = *tslot;

  if (warp == 16) {
    // ---- TMA producer: W1 (3 chunks: the used columns), W2, W3 (8 each), for each slot's tile
    if (lane == 0 && blockIdx.x < n_tiles) {
      const void *wmap[3] = {&tw1, &tw2, &tw3};
      int cnt = 0;
      bool ok = true;
      for (int i = 0; tile_at(i, 0) < n_tiles && ok; i++)
        for (int l = 0; l < 3 && ok; l++)
          for (int s = 0; s < 2 && ok; s++) {
            if (tile_at(i, s) >= n_tiles) continue;
            for (int j = 0; j < (l == 0 ? kMlpNodeFeat + kMlpEmb : kMlpHidden) / kFwdK; j++, cnt++) {
              const int st = cnt % kFwdStages;
              if ((cnt >= kFwdStages && !umma::mbar_wait(&wempty[st], ((cnt / kFwdStages) - 1) & 1)) || *bad) {
                *bad = 1;
                ok = false;
                break;
              }
              umma::mbar_arrive_expect_tx(&wfull[st], kFwdChunk);
              umma::tma_load_2d(wst + st * kFwdChunk, wmap[l], kFwdK * j, 0, &wfull[st]);
            }
          }
      // Copies still in flight land before the block's memory goes: once the
      // MMA thread has stopped (it publishes mma_done; waited for at most
      // ~2 s of SM clock, far beyond any batch), the loads it did not consume
      // are waited for, bounded.
      const long long t0 = clock64();
      while (*mma_done == 0 && clock64() - t0 < 4000000000ll) {
      }
      if (*bad)
        for (int i = *consumed; i < cnt; i++) umma::mbar_wait(&wfull[i % kFwdStages], (i / kFwdStages) & 1, 1u << 20);
    }
  } else if (warp == 17) {
    // ---- MMA issuer: the whole warp walks the schedule, so that the
    // descriptors are warp-uniform, and an elected lane issues (a wait and four
    // MMAs: 360 clocks of issue this way, 510 from one lane's branch)
    bool ok = true, issued_any = false;
    uint32_t st = 0, parity = 0;  // the next weight stage, parity of its next completion
    int cnt = 0;
    const uint64_t a_desc = umma::sdesc_kmajor_sw128(umma::smem_u32(act));
    const uint64_t b_desc = umma::sdesc_kmajor_sw64(umma::smem_u32(wst));
    auto layer = [&](auto first, int s) -> bool {
      constexpr bool kFirst = decltype(first)::value;
      const uint64_t ad = a_desc + s * (kActBytes >> 4);
      const uint32_t acc = tmem + 256u * (uint32_t)s;
#pragma unroll
      for (int j = 0; j < (kFirst ? kMlpNodeFeat + kMlpEmb : kMlpHidden) / kFwdK; j++) {
        if (!umma::mbar_wait_warp(&wfull[st], parity)) return false;
        umma::fence_after_sync();
        const uint64_t bd = b_desc + st * (kFwdChunk >> 4);
        if (umma::elect_one()) {
#pragma unroll
          for (int kk = 0; kk < kFwdK / 16; kk++)  // the input's k-blocks of 64 columns hold two chunks
            umma::mma_bf16(acc, ad + (j >> 1) * (128 * 128 >> 4) + 4 * (j & 1) + 2 * kk, bd + 2 * kk, kIdesc,
                           (j > 0 || kk > 0) ? 1u : 0u);
          umma::commit(&wempty[st]);
        }
        __syncwarp();
        cnt++;
        if (++st == kFwdStages) {
          st = 0;
          parity ^= 1u;
        }
      }
      return true;
    };
    for (int i = 0; tile_at(i, 0) < n_tiles && ok; i++)
      for (int l = 0; l < 3 && ok; l++)
        for (int s = 0; s < 2 && ok; s++) {
          if (tile_at(i, s) >= n_tiles) continue;
          if (__any_sync(0xffffffffu, *bad) ||
              (l == 0 ? !umma::mbar_wait_warp(&xready[s], i & 1) || (i > 0 && !umma::mbar_wait_warp(&accfree[s], (i - 1) & 1))
                      : !umma::mbar_wait_warp(&hready[s], (2 * i + l - 1) & 1))) {
            ok = false;
            break;
          }
          issued_any = true;
          ok = l == 0 ? layer(std::true_type{}, s) : layer(std::false_type{}, s);
          if (!ok) break;
          if (umma::elect_one()) {
            if (l == 2) umma::commit(&xfree[s]);  // the slot may be refilled once these MMAs are done
            umma::commit(&accfull[s]);
          }
          __syncwarp();
        }
    if (!ok && lane == 0) *bad = 1;
    if (issued_any) {  // the MMAs issued are complete before the memory goes
      if (umma::elect_one()) umma::commit(drain);
      __syncwarp();
      umma::mbar_wait_warp(drain, 0, 1u << 20);
    }
    if (lane == 0) {
      *consumed = cnt;
      __threadfence_block();
      *mma_done = 1;
    }
  } else if (warp >= 18) {
    // ---- gather warps, a thread a row: the outputs of the slot's last tile,
    // then the input row of its next one (node features and embedding, 16-byte
    // chunks 0-9 and 10-11, loaded before the waits)
    static_assert(kFwdGatherThreads == 128 && kMlpNodeFeat == 80 && kMlpEmb == 16, "a gather thread a row, 12 chunks");
    const int r = tid - 18 * 32;
    const float b40 = __ldg(a.b4), b41 = __ldg(a.b4 + 1);
    // (decisions to stop are the same for a whole warp)
    for (int i = 0; tile_at(i - 1, 0) < n_tiles && !__any_sync(0xffffffffu, *bad); i++)  // (i = 0: always)
      for (int s = 0; s < 2; s++) {
        const bool more = tile_at(i, s) < n_tiles;
        const int64_t b = tile_at(i, s) * 128 + r;
        uint4 v[12];
#pragma unroll
        for (int k = 0; k < 12; k++) v[k] = make_uint4(0, 0, 0, 0);
        if (more && b < a.B) {
          const uint4 *nf = reinterpret_cast<const uint4 *>(a.node_feat + (int64_t)a.node[b] * kMlpNodeFeat);
          const uint4 *em = reinterpret_cast<const uint4 *>(a.emb + (int64_t)a.prim[b] * kMlpEmb);
#pragma unroll
          for (int k = 0; k < 12; k++) v[k] = k < 10 ? nf[k] : em[k - 10];
        }
        if (i > 0 && tile_at(i - 1, s) < n_tiles) {
          if (!__all_sync(0xffffffffu, umma::mbar_wait(&pready[s], (i - 1) & 1))) {
            *bad = 1;
            break;
          }
          float2 o = make_float2(b40, b41);
#pragma unroll
          for (int g = 0; g < 4; g++) {
            const float2 p = spart[512 * s + 128 * g + r];
            o.x += p.x;
            o.y += p.y;
          }
          const int64_t ob = tile_at(i - 1, s) * 128 + r;
          if (ob < a.B) {
            a.out[ob * 2] = o.x;
            a.out[ob * 2 + 1] = o.y;
          }
        }
        if (!more) continue;
        // (pready follows accfull of layer 3, so the slot's MMAs are done: xfree is there too)
        if (!__all_sync(0xffffffffu, i == 0 || umma::mbar_wait(&xfree[s], (i - 1) & 1))) {
          *bad = 1;
          break;
        }
#pragma unroll
        for (int k = 0; k < 12; k++)
          *reinterpret_cast<uint4 *>(act + s * kActBytes + umma::kmajor_offset(128, r, k)) = v[k];
        umma::fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) umma::mbar_arrive(&xready[s]);
      }
  } else {
    // ---- epilogue warps: H1, H2, then the partial outputs.  Warp w:
    // accumulator lanes 32 (w % 4) .., columns 64 (w / 4) ..
    const int q = warp & 3, cg = warp >> 2, row = 32 * q + lane;
    bool ok = true;
    for (int i = 0; tile_at(i, 0) < n_tiles && ok && !__any_sync(0xffffffffu, *bad); i++)
      for (int l = 0; l < 3 && ok; l++)
        for (int s = 0; s < 2; s++) {
          if (tile_at(i, s) >= n_tiles) continue;
          if (!__all_sync(0xffffffffu, umma::mbar_wait(&accfull[s], (3 * i + l) & 1))) {
            ok = false;
            break;
          }
          const uint32_t src = tmem + ((uint32_t)(32 * q) << 16) + 256u * (uint32_t)s + 64u * (uint32_t)cg;
          unsigned char *slot = act + s * kActBytes;
          umma::fence_after_sync();
          const float4 *bias = reinterpret_cast<const float4 *>(sbias + kMlpHidden * l + 64 * cg);
          uint64_t a0 = pack2(0.f, 0.f), a1 = a0;
          uint32_t r[2][16];  // this block's values and the next one's, in flight
          umma::tmem_ld16_async(src, r[0]);
#pragma unroll
          for (int j = 0; j < 4; j++) {
            const int c0 = 64 * cg + 16 * j;
            float4 bv[4];
#pragma unroll
            for (int k = 0; k < 4; k++) bv[k] = bias[4 * j + k];
            uint32_t *v = r[j & 1];
            umma::tmem_wait16(v);
            if (j < 3) umma::tmem_ld16_async(src + 16u * (j + 1), r[(j + 1) & 1]);
            uint64_t g[8];
#pragma unroll
            for (int k = 0; k < 4; k++) {
              auto f = [&](int e) { return __uint_as_float(v[4 * k + e]); };
              g[2 * k] = gelu2(add2(pack2(f(0), f(1)), pack2(bv[k].x, bv[k].y)));
              g[2 * k + 1] = gelu2(add2(pack2(f(2), f(3)), pack2(bv[k].z, bv[k].w)));
            }
            uint32_t hb[8];
#pragma unroll
            for (int k = 0; k < 8; k++) hb[k] = to_bf16x2(g[k]);
            if (l < 2) {
              *reinterpret_cast<uint4 *>(slot + umma::kmajor_offset(128, row, c0 / 8)) = make_uint4(hb[0], hb[1], hb[2], hb[3]);
              *reinterpret_cast<uint4 *>(slot + umma::kmajor_offset(128, row, c0 / 8 + 1)) =
                  make_uint4(hb[4], hb[5], hb[6], hb[7]);
            } else {  // the two outputs: rows 0 and 1 of W4
#pragma unroll
              for (int k = 0; k < 4; k++) {
                const float4 w0 = *reinterpret_cast<const float4 *>(sw4 + c0 + 4 * k);
                const float4 w1 = *reinterpret_cast<const float4 *>(sw4 + kMlpHidden + c0 + 4 * k);
                const uint64_t h0 = from_bf16x2(hb[2 * k]), h1 = from_bf16x2(hb[2 * k + 1]);
                a0 = fma2(h0, pack2(w0.x, w0.y), a0);
                a1 = fma2(h0, pack2(w1.x, w1.y), a1);
                a0 = fma2(h1, pack2(w0.z, w0.w), a0);
                a1 = fma2(h1, pack2(w1.z, w1.w), a1);
              }
            }
          }
          if (l < 2) {
            umma::fence_proxy_async_smem();
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) umma::mbar_arrive(&hready[s]);
          } else {
            float x0, y0, x1, y1;
            unpack2(a0, x0, y0);
            unpack2(a1, x1, y1);
            spart[512 * s + 128 * cg + row] = make_float2(x0 + y0, x1 + y1);
            umma::fence_before_sync();
            __syncwarp();
            if (lane == 0) {
              umma::mbar_arrive(&accfree[s]);
              umma::mbar_arrive(&pready[s]);
            }
          }
        }
    if (!ok) *bad = 1;
  }
  umma::fence_before_sync();
  __syncthreads();
  if (tid == 0 && *bad) atomicExch(a.err, 1);
  umma::fence_after_sync();
  if (warp == 0) umma::tmem_dealloc(tmem, 512);
}

}  // namespace dpg
