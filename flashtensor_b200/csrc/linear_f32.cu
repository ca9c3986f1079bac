// out[M, N] = x[M, K] w[N, K]^T + bias[N] in f32, for the projections around the linear-attention
// core of the reference's SimA and EA benchmark programs (bench/sima.mlir:3-5,18-22: f32, C = 128).
//
// f32 accuracy on the bf16 tensor pipe: every operand is split into three bf16 terms,
// x = h + m + l (8 significant bits each, what is left out is below 2^-26 |x|), and the six
// products h.h, h.m, m.h, m.m, h.l, l.h are accumulated in f32 in TMEM; the dropped ones are below
// 2^-26 of |x||w|, under the rounding of an f32 product.  The CUDA cores' 74 TFLOP/s would need
// 66 us for the 4.9 GFLOP of the QKV projection at B64 N784 C128; six bf16 products at the tensor
// pipe's rate need 15, and the 103 MB it moves 16.
//
// One persistent CTA per SM owns a block of 128 output columns and walks tiles of 128 rows of x.  The
// product is formed transposed, out^T = w x^T: the split weights are the A operand and stay in TMEM
// for the whole kernel, so the MMAs read only the x tile from shared memory (with both operands
// there, a 128 x 128 MMA takes all of its bandwidth and the warps that write the next tile stall:
// 38 us instead of the figure below), and an accumulator lane is an output column, so a warp's store
// is one 128-byte line of an output row.
//   warps 0-7    load x (a whole tile ahead), split it and store the three terms as swizzled K-major tiles
//   warp 8       issues tcgen05.mma into one of two accumulators
//   warps 9-12   split the weights into TMEM; then accumulator + bias to global memory
// The small products of a tile are accumulated before any h.h: the tensor pipe truncates when it adds
// to an accumulator, and forty small terms added to a large sum would each leave a bias there
// (measured at K = 128: 4.1e-7 relative error in the natural order, against 1.5e-7 of an f32 GEMM on
// the CUDA cores).
// The split is sound while its terms and products stay clear of both ends of the exponent range.  Infinities
// and values that round to one have no residual: they, like anything that overflows, leave a sum that is not
// finite.  Terms and products below 2^-126 are flushed: with weights below 2^20 that costs a sum 2^-98 at most,
// which is below the rounding of one of 2^-72 or more.  So a sum that is not finite or below 2^-72, and a
// column with a weight outside [2^-100, 2^20) that is not zero, is computed on the CUDA cores (plain_dot) by
// the warps that store it; which way a result takes depends on its own row and column.  (Folded weights hold the values
// of a batch, which may be large: there the bounds are 2^100 and, as both of the above grow with the weights, 2^-92
// of the column's largest for the sum.)  That is for the odd row
// or column: all rows at 1e-25 take 1460 us instead of 34, rows of nothing but zeros, which need a look at x only, 91.
// Measured at B64 N784 C128 (M = 50176, K = 128), calls back to back, bias included: N = 384 (QKV) 32 us,
// N = 128 (output) 14.6 us; the f32 GEMM of the BLAS library with its bias pass takes 200 and 64.  A launch is set-up
// for a third of it, so the warps that split x start while the weights are still being split (4.5 us of a
// whole SimA block of that size).  Eight epilogue warps, four to an accumulator, are slower (38 and 17 us: what they and the
// splitting warps share is the way to shared memory), and so are plain stores instead of TMA's.
#include <cuda_bf16.h>

#include "f32_keep.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"
#include "tma_host.h"

namespace asuka {
using namespace sm100;

namespace {

constexpr int kTile = 128;               // rows of x and output columns of a tile
constexpr int kMaxK = 128;
constexpr int kChunk = 64;               // reduction columns of one 128-byte swizzled row of bf16
constexpr uint32_t kTermBytes = kTile * kChunk * 2;  // one bf16 term of a [128 x 64] piece
constexpr uint32_t kPieceBytes = 3 * kTermBytes;
constexpr uint32_t kStageBytes = (kMaxK / kChunk) * kPieceBytes;  // a tile of x: 96 KB
constexpr int kSplitWarps = 8;
constexpr int kThreads = (kSplitWarps + 1 + 4) * 32;
constexpr uint32_t kOutBytes = 32 * 32 * 4;                       // one TMA store of a warp: 32 rows x 32 columns
constexpr uint32_t kSmemBytes = 2 * kStageBytes + 4 * 2 * kOutBytes + 1024;
constexpr uint32_t kTermCols = kMaxK / 2;  // TMEM columns of one term of the weights
constexpr uint32_t kAccCol = 3 * kTermCols;

// What a launch multiplies.
//   kPlain    rows of one matrix with one set of weights
//   kBatched  every batch's rows with weights of its own (N <= 128); a CTA stays within one batch
//   kSoftmax  the same, every group of 32 values of a row replaced by its softmax first (EA's queries)
enum LinMode { kPlain = 0, kBatched = 1, kSoftmax = 2 };

struct LinParams {
  const float* x;
  const float* w;
  const float* bias;
  float* out;
  int M, N, K;           // M: rows of a batch
  int64_t x_sn, x_sb;    // strides of x between rows and between batches
  int64_t w_sb;          // ... and of w between batches
  int n_tiles, chunks;
  int splits, cta_rows;  // (batched) CTAs per batch, and the rows of each, a multiple of 32
  FoldScales scales;     // (batched)
  int tma_out;  // rows of `out` can be described to TMA (N a multiple of 4)
  uint32_t* status;
};

constexpr float kWeightLow = 7.8886090522101181e-31f;                            // 2^-100
constexpr float kSumLow = 2.1175823681357508e-22f;                               // 2^-72
constexpr float kSumPerWeight = 2.0194839173657902e-28f;                         // 2^-92 (folded weights)
// (softmax) 1 / 32, which the values of a group average.  It is taken off them before they are multiplied and comes back
// as that share of the sum of the column's weights, in f32: products of values that are all positive have the signs of
// the weights, and what the tensor pipe truncates of each then adds up.  EA block, error against 64 bits with and without,
// B64 N784 C128 1.09e-7 and 1.66e-7, B4 N300 1.33e-7 and 1.94e-7 (core and projection apart 1.57e-7 and 1.76e-7); with
// queries ten times as large, which pick few features, keys five times and values about 3, B4 N300 1.82e-7 and 3.26e-7
// (1.88e-7).  What the sum of the weights is rounded by stays below 2^-24 of the largest folded weights of the column,
// also in a row that picks none but small ones.
constexpr float kShare = 0.03125f;
template <int kMode> constexpr float kWeightHighOf = kMode == kPlain ? 1048576.f : 1.2676506002282294e30f;  // 2^20, 2^100
__device__ __forceinline__ float max3_nan(float a, float b, float c) {
  float y;
  asm("max.NaN.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}
__device__ __forceinline__ float min3(float a, float b, float c) {
  float y;
  asm("min.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

// largest (NaN if there is one) and smallest magnitude of eight values
__device__ __forceinline__ void extent8(const float (&v)[8], float* big, float* small) {
  float a[8];
#pragma unroll
  for (int i = 0; i < 8; ++i) a[i] = fabsf(v[i]);
  *big = max3_nan(max3_nan(a[0], a[1], a[2]), max3_nan(a[3], a[4], a[5]), max3_nan(a[6], a[7], a[7]));
  *small = min3(min3(a[0], a[1], a[2]), min3(a[3], a[4], a[5]), min3(a[6], a[7], a[7]));
}

// e^x of a difference from the maximum (linattn32.cu)
__device__ __forceinline__ float exp_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}
// softmax over the kLanes neighbouring lanes that hold kN values each of a group
template <int kLanes, int kN>
__device__ __forceinline__ void softmax_group(float (&v)[kN]) {
  float m = v[0];
#pragma unroll
  for (int i = 1; i < kN; ++i) m = fmaxf(m, v[i]);
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
#pragma unroll
  for (int i = 0; i < kN; ++i) v[i] = exp_fast(v[i] - m);
  float sum = (v[0] + v[1]) + (v[2] + v[3]);
  if constexpr (kN == 8) sum += (v[4] + v[5]) + (v[6] + v[7]);
#pragma unroll
  for (int o = 1; o < kLanes; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
  const float inv = __frcp_rn(sum);
#pragma unroll
  for (int i = 0; i < kN; ++i) v[i] *= inv;
}

// a factor of powers of two, kept as the upper half of its bits
__device__ __forceinline__ float rescale(uint16_t upper) { return __uint_as_float(static_cast<uint32_t>(upper) << 16); }

// One row of x against the 32 columns from n_base on, by a whole warp: lane l takes reduction columns 4l to
// 4l + 3 and returns the sum for output column n_base + l.  (Batched: `rescale_rows` holds the factors of these columns.)
template <int kMode>
__device__ __noinline__ float plain_dot(const float* __restrict__ x_row, const float* __restrict__ w, const uint16_t (*rescale_rows)[4],
                                        int n_base, int N, int K) {
  const int lane = threadIdx.x & 31;
  const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
  const bool live = lane * 4 < K;
  float4 xv = live ? __ldg(reinterpret_cast<const float4*>(x_row) + lane) : zero;
  if constexpr (kMode == kSoftmax) {
    float v[4] = {xv.x, xv.y, xv.z, xv.w};
    softmax_group<8>(v);
    xv = live ? make_float4(v[0], v[1], v[2], v[3]) : zero;
  }
  float part[32];
#pragma unroll
  for (int c = 0; c < 32; ++c) {
    float4 wv = live ? __ldg(reinterpret_cast<const float4*>(w + static_cast<int64_t>(min(n_base + c, N - 1)) * K) + lane) : zero;
    if constexpr (kMode != kPlain) {
      const float f = rescale(rescale_rows[c][lane >> 3]);
      wv = make_float4(mul_keep(wv.x, f), mul_keep(wv.y, f), mul_keep(wv.z, f), mul_keep(wv.w, f));
    }
    part[c] = fma_keep(xv.x, wv.x, fma_keep(xv.y, wv.y, fma_keep(xv.z, wv.z, fma_keep(xv.w, wv.w, 0.f))));
  }
  // every exchange adds two lanes' sums and halves the columns a lane still holds
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool upper = (lane & o) != 0;
#pragma unroll
    for (int c = 0; c < o; ++c)
      part[c] = add_keep(upper ? part[c + o] : part[c], __shfl_xor_sync(0xffffffffu, upper ? part[c] : part[c + o], o));
  }
  return part[0];
}

// Which of the 32 rows from `x` on (`rows` of them there) have a value other than zero: one bit each.  (Rows
// of zeros, a batch's padding, have sums of zero that need no second look; eight loads in flight.)
__device__ __noinline__ uint32_t rows_not_zero(const float* __restrict__ x, int64_t x_sn, int rows, int K) {
  const int lane = threadIdx.x & 31;
  uint32_t mask = 0;
  for (int r0 = 0; r0 < 32; r0 += 8) {
    float4 v[8];
#pragma unroll
    for (int r = 0; r < 8; ++r)
      v[r] = r0 + r < rows && lane * 4 < K ? __ldg(reinterpret_cast<const float4*>(x + (r0 + r) * x_sn) + lane)
                                           : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const uint32_t bits = __float_as_uint(v[r].x) | __float_as_uint(v[r].y) | __float_as_uint(v[r].z) | __float_as_uint(v[r].w);
      if (__any_sync(0xffffffffu, (bits << 1) != 0u)) mask |= 1u << (r0 + r);
    }
  }
  return mask;
}

struct LinBars {
  uint64_t x_full[2], x_empty[2];
  uint64_t acc_full[2], acc_empty[2];
};

__device__ __forceinline__ uint32_t pack_bf16(float lo, float hi) {
  __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
  return *reinterpret_cast<uint32_t*>(&v);
}
// eight f32 values to their three bf16 terms, eight values in 16 bytes each
__device__ __forceinline__ void split8(const float (&v)[8], uint4 (&t)[3]) {
  uint32_t w[3][4];
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    float a = v[2 * i], b = v[2 * i + 1];
#pragma unroll
    for (int s = 0; s < 3; ++s) {
      const uint32_t p = pack_bf16(a, b);
      w[s][i] = p;
      const float ra = __uint_as_float(p << 16), rb = __uint_as_float(p & 0xffff0000u);
      a -= ra;  // (exact; an infinity leaves NaN)
      b -= rb;
    }
  }
#pragma unroll
  for (int s = 0; s < 3; ++s) t[s] = make_uint4(w[s][0], w[s][1], w[s][2], w[s][3]);
}

__device__ __forceinline__ void record_timeout(uint32_t* status, uint32_t site) {
  atomicAdd(&status[0], 1u);
  status[1] = site;
}

template <int kMode>
__global__ void __launch_bounds__(kThreads, 1) linear_f32_kernel(const __grid_constant__ CUtensorMap map_out, const LinParams p) {
  constexpr float kWeightHigh = kWeightHighOf<kMode>;
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) LinBars bars;
  __shared__ __align__(8) uint16_t rescale_s[kMode == kPlain ? 1 : kTile][4];  // (batched) by column: factors of its heads' weights
  __shared__ uint32_t tmem_base_s;
  __shared__ uint32_t abort_s;
  const uint32_t sX = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* const gX = smem_raw + (sX - smem_u32(smem_raw));

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile uint32_t* abortp = &abort_s;
  // This CTA's tiles start at rows row_first, row_first + row_step, ... of batch `batch` and end at row_end.
  // Plain: CTAs are dealt out over the column blocks; those of one block share its row tiles.
  int nb = 0, batch = 0, row_first, row_step, row_end;
  if constexpr (kMode == kPlain) {
    nb = static_cast<int>(blockIdx.x) % p.n_tiles;
    row_first = static_cast<int>(blockIdx.x) / p.n_tiles * kTile;
    row_step = (static_cast<int>(gridDim.x) - nb + p.n_tiles - 1) / p.n_tiles * kTile;  // (CTAs of this column block)
    row_end = p.M;
  } else {
    batch = static_cast<int>(blockIdx.x) / p.splits;
    row_first = static_cast<int>(blockIdx.x) % p.splits * p.cta_rows;
    row_step = kTile;
    row_end = min(p.M, row_first + p.cta_rows);
  }
  const int n0 = nb * kTile;
  const float* const x = p.x + batch * p.x_sb;
  const float* const w = p.w + batch * p.w_sb;

  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars.x_full[i]), kSplitWarps * 32);
      mbar_init(smem_u32(&bars.x_empty[i]), 1);
      mbar_init(smem_u32(&bars.acc_full[i]), 1);
      mbar_init(smem_u32(&bars.acc_empty[i]), 128);
    }
    mbar_fence_init();
  }
  if (warp == kSplitWarps) {
    __syncwarp();
    tmem_alloc(smem_u32(&tmem_base_s), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tbase = tmem_base_s;
  const int wq = warp & 3;  // (epilogue warps) TMEM lane quarter
  const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
  const int n = n0 + wq * 32 + lane;  // (epilogue warps) this thread's output column
  float w_big = 0.f, w_small = kWeightHigh;  // (epilogue warps) of that column's weights, the zeros apart
  float w_sum[4] = {0.f, 0.f, 0.f, 0.f};     // (softmax, epilogue warps) the sum of that column's weights
  uint32_t least = 127u;                     // (batched, epilogue warps) exponent of the scale of that column's weights
  // (batched: the kernel ahead, which writes the weights, reads x itself and has waited for whatever wrote it before
  // this one could start: the splitting warps need not wait; EA block 79.7 -> 76.8 us)
  if (kMode == kPlain || warp >= kSplitWarps) griddep_wait();
  griddep_launch_dependents();
  if (warp > kSplitWarps) {
    // the weights of this block of columns, split once: thread = output column = TMEM lane
    const float* src = w + static_cast<int64_t>(min(n, p.N - 1)) * p.K;
    float4 next[8];  // the next 32 weights
    auto load = [&](int k0) {
#pragma unroll
      for (int i = 0; i < 8; ++i)  // (K is a multiple of 8)
        next[i] = n < p.N && k0 + i * 4 < p.K ? __ldg(reinterpret_cast<const float4*>(src + k0) + i) : make_float4(0.f, 0.f, 0.f, 0.f);
    };
    load(0);
    if constexpr (kMode != kPlain) {
      // the exponents of the scales that the column's heads were folded with: all are brought to that of the largest,
      // by 2^-126 at most
      const uint8_t* e_ptr = reinterpret_cast<const uint8_t*>(p.scales.ptr + batch * p.scales.per_batch +
                                                              static_cast<int>(blockIdx.x) % p.splits * p.scales.per_cta);
      uint32_t e[4];
#pragma unroll
      for (int h = 0; h < 4; ++h) e[h] = n < p.N && h * 32 < p.K ? __ldcg(e_ptr + h * p.K + n) : 254u;
      least = min(min(e[0], e[1]), min(e[2], e[3]));
#pragma unroll
      for (int h = 0; h < 4; ++h) rescale_s[wq * 32 + lane][h] = static_cast<uint16_t>((127u - min(e[h] - least, 126u)) << 7);
    }
    for (int k0 = 0; k0 < p.chunks * kChunk; k0 += 32) {
      uint32_t t[3][16];
      const float f = kMode == kPlain ? 1.f : rescale(rescale_s[kMode == kPlain ? 0 : wq * 32 + lane][k0 >> 5]);
#pragma unroll
      for (int g = 0; g < 4; ++g) {
        const int k = k0 + g * 8;
        const float4 lo = next[2 * g], hi = next[2 * g + 1];
        float v[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
        if constexpr (kMode != kPlain) {
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = mul_keep(v[i], f);
        }
        if constexpr (kMode == kSoftmax) w_sum[g] += ((v[0] + v[1]) + (v[2] + v[3])) + ((v[4] + v[5]) + (v[6] + v[7]));
        float big, small;
        extent8(v, &big, &small);
        w_big = max3_nan(w_big, big, big);
        w_small = k < p.K ? fminf(w_small, small) : w_small;
        uint4 q[3];
        split8(v, q);
#pragma unroll
        for (int s = 0; s < 3; ++s) {
          t[s][g * 4 + 0] = q[s].x;
          t[s][g * 4 + 1] = q[s].y;
          t[s][g * 4 + 2] = q[s].z;
          t[s][g * 4 + 3] = q[s].w;
        }
      }
      load(k0 + 32);
#pragma unroll
      for (int s = 0; s < 3; ++s) tmem_st16(tbase + lane_base + s * kTermCols + k0 / 2, t[s]);
    }
    tmem_wait_st();
    if (w_small < kWeightLow) {  // a zero, which is no matter, or not: look again
      w_small = kWeightHigh;
      if (n < p.N)
        for (int k = 0; k < p.K; ++k) {
          float a = __ldg(src + k);
          if constexpr (kMode != kPlain) a = mul_keep(a, rescale(rescale_s[wq * 32 + lane][k >> 5]));
          if ((__float_as_uint(a) << 1) != 0u) w_small = fminf(w_small, fabsf(a));  // (a subnormal counts as 0)
        }
    }
  }
  if (warp >= kSplitWarps) {  // (the splitting warps have nothing to do with the weights and are at work already)
    tc_fence_before_sync();
    named_bar_sync(1, kThreads - kSplitWarps * 32);
    tc_fence_after_sync();
  }

  if (warp < kSplitWarps) {
    // ------------------------------------------------------------------ load and split x
    // A thread takes 8 columns (32 bytes) of four rows of every 64-column piece; eight threads cover
    // a row's 256 bytes.  The next tile's loads are in flight while this one is split.
    const int c = tid & 7, row0 = tid >> 3;  // rows row0, +32, +64, +96
    float4 v[2][4][2];
    auto fetch = [&](int row_t) {
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        const int k = ch * kChunk + c * 8;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
          const int row = row_t + row0 + i * 32;
          const bool live = row < row_end && k < p.K;
          const float4* src = reinterpret_cast<const float4*>(x + static_cast<int64_t>(row) * (kMode == kPlain ? p.K : p.x_sn) + k);
          v[ch][i][0] = live ? __ldg(src) : make_float4(0.f, 0.f, 0.f, 0.f);
          v[ch][i][1] = live ? __ldg(src + 1) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
      }
    };
    uint32_t t = 0;
    if (row_first < row_end) fetch(row_first);
    for (int row_t = row_first; row_t < row_end; row_t += row_step, ++t) {
      const int st = t & 1;
      if (t >= 2 && !mbar_wait(smem_u32(&bars.x_empty[st]), ((t >> 1) - 1) & 1, abortp)) {
        if (lane == 0) record_timeout(p.status, 81);
        break;
      }
#pragma unroll
      for (int ch = 0; ch < 2; ++ch) {
        if (ch < p.chunks) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const float4 lo = v[ch][i][0], hi = v[ch][i][1];
            float e[8] = {lo.x, lo.y, lo.z, lo.w, hi.x, hi.y, hi.z, hi.w};
            if constexpr (kMode == kSoftmax) {  // (past K the weights are zero)
              softmax_group<4>(e);
#pragma unroll
              for (int x = 0; x < 8; ++x) e[x] -= kShare;
            }
            uint4 q[3];
            split8(e, q);
#pragma unroll
            for (int s = 0; s < 3; ++s)
              *reinterpret_cast<uint4*>(gX + st * kStageBytes + ch * kPieceBytes + s * kTermBytes +
                                        sw128_offset(row0 + i * 32, c)) = q[s];
          }
        }
      }
      if (row_t + row_step < row_end) fetch(row_t + row_step);
      fence_proxy_async_smem();
      mbar_arrive(smem_u32(&bars.x_full[st]));
    }
  } else if (warp == kSplitWarps) {
    // ------------------------------------------------------------------ MMA issuer
    auto wait_all = [&](uint64_t* bar, uint32_t parity, uint32_t site) -> bool {
      const bool good = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, abortp));
      if (!good && lane == 0) record_timeout(p.status, site);
      return good;
    };
    uint32_t t = 0;
    for (int row_t = row_first; row_t < row_end; row_t += row_step, ++t) {
      const int st = t & 1;
      // (the rows of the tile are the N of the MMA: a batch's last tile of few rows costs as much as it has)
      const uint32_t idesc = umma_idesc_f16(UMMA_BF16, UMMA_K_MAJOR, UMMA_K_MAJOR, 128,
                                            kMode == kPlain ? kTile : min(kTile, (row_end - row_t + 15) & ~15));
      if (t >= 2 && !wait_all(&bars.acc_empty[st], ((t >> 1) - 1) & 1, 82)) break;
      if (!wait_all(&bars.x_full[st], (t >> 1) & 1, 83)) break;
      tc_fence_after_sync();
      if (elect_one()) {
        constexpr int kW[6] = {2, 0, 1, 1, 0, 0}, kX[6] = {0, 2, 1, 0, 1, 0};
        const uint32_t acc = tbase + kAccCol + st * 128;
#pragma unroll
        for (int pr = 0; pr < 6; ++pr) {
          for (int ch = 0; ch < p.chunks; ++ch) {
            const uint64_t xd =
                umma_smem_desc_sw128(sX + st * kStageBytes + ch * kPieceBytes + kX[pr] * kTermBytes, 16, 1024);
            const uint32_t wt = tbase + kW[pr] * kTermCols + ch * (kChunk / 2);
#pragma unroll
            for (int kk = 0; kk < 4; ++kk)
              umma_ts(acc, wt + kk * 8, xd + kk * 2, idesc, (pr > 0 || ch > 0 || kk > 0) ? 1u : 0u);
          }
        }
        umma_commit(smem_u32(&bars.x_empty[st]));
        umma_commit(smem_u32(&bars.acc_full[st]));
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------------ epilogue
    uint8_t* const stage = gX + 2 * kStageBytes + wq * 2 * kOutBytes;
    if (kMode != kPlain && p.scales.per_cta != 0) fence_proxy_async_global();  // (they lay in what this warp now stores by TMA)
    const float bias = n < p.N ? __ldg(p.bias + n) : 0.f;
    float* const out = p.out + static_cast<int64_t>(batch) * p.M * p.N;
    const float sum_low = kMode == kPlain ? kSumLow : fmaxf(kSumLow, w_big * kSumPerWeight);
    const float unscale = kMode == kPlain ? 1.f : __uint_as_float((254u - least) << 23);
    // (softmax) what the shares taken off the queries amount to, in every row alike
    const float shared = kMode != kSoftmax ? 0.f : kShare * ((w_sum[0] + w_sum[1]) + (w_sum[2] + w_sum[3]));
    auto result = [&](float sum) { return kMode == kPlain ? add_keep(sum, bias) : fma_keep(sum, unscale, bias); };
    const bool zero_col = w_big == 0.f;  // a sum of zero is right (with a subnormal weight it is a plain one)
    const bool plain_col = !(w_big < kWeightHigh) || w_small < kWeightLow;
    const bool any_plain_col = __any_sync(0xffffffffu, plain_col);
    uint32_t t = 0;
    for (int row_t = row_first; row_t < row_end; row_t += row_step, ++t) {
      const int st = t & 1;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.acc_full[st]), (t >> 1) & 1, abortp))) {
        if (lane == 0) record_timeout(p.status, 84);
        break;
      }
      tc_fence_after_sync();
      float big = 0.f, small = kWeightHigh;  // of this column's sums in the tile
      bool again = any_plain_col;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        uint32_t u[32];
        tmem_ld32(tbase + lane_base + kAccCol + st * 128 + q * 32, u);
        uint8_t* const dst = stage + (q & 1) * kOutBytes;
        if (lane == 0) tma_store_wait_read_n<1>();  // the store before last has left this half of the stage
        __syncwarp();
        tmem_wait_ld();
        if constexpr (kMode == kSoftmax) {
#pragma unroll
          for (int r = 0; r < 32; ++r) u[r] = __float_as_uint(__uint_as_float(u[r]) + shared);
        }
        if (row_t + q * 32 + 32 > row_end) {  // (rows past the end, zero as well, are not stored)
#pragma unroll
          for (int r = 0; r < 32; ++r) u[r] = row_t + q * 32 + r < row_end ? u[r] : __float_as_uint(kWeightHigh);
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {
          float b8, s8;
          extent8(reinterpret_cast<const float(&)[8]>(u[g * 8]), &b8, &s8);
          big = max3_nan(big, b8, b8);
          small = fminf(small, s8);
        }
        if (q == 3) {
          again = __any_sync(0xffffffffu, !(big < INFINITY) || (small < sum_low && !zero_col)) || again;
          if (!again) {
            tc_fence_before_sync();
            mbar_arrive(smem_u32(&bars.acc_empty[st]));
          }
        }
#pragma unroll
        for (int r = 0; r < 32; ++r)
          *reinterpret_cast<float*>(dst + sw128_offset(r, lane >> 2) + (lane & 3) * 4) = result(__uint_as_float(u[r]));
        const int row_q = row_t + q * 32;
        if (p.tma_out) {
          fence_proxy_async_smem();
          __syncwarp();
          if (lane == 0) {
            if (row_q < row_end && n < p.N) tma_store_4d(&map_out, smem_u32(dst), n, row_q, batch, 0);  // (lane 0: n is the block's first column)
            tma_store_commit();
          }
        } else if (n < p.N) {  // (a thread reads back only what it wrote)
          for (int r = 0; r < 32 && row_q + r < row_end; ++r)
            out[static_cast<int64_t>(row_q + r) * p.N + n] =
                *reinterpret_cast<const float*>(dst + sw128_offset(r, lane >> 2) + (lane & 3) * 4);
        }
      }
      if (again) {
        // results that the sum is not good enough for, over what has just been stored
        if (lane == 0) tma_store_wait_all();
        __syncwarp();
#pragma unroll 1
        for (int q = 0; q < 4; ++q) {
          const int row_q = row_t + q * 32;
          uint32_t u[32];
          tmem_ld32(tbase + lane_base + kAccCol + st * 128 + q * 32, u);
          tmem_wait_ld();
          uint32_t mine = 0;  // this column's rows
#pragma unroll
          for (int r = 0; r < 32; ++r) {
            const float a = fabsf(__uint_as_float(u[r]) + shared);
            if (!(a < INFINITY) || (a < sum_low && !zero_col)) mine |= 1u << r;
          }
          if (plain_col) mine = 0xffffffffu;
          uint32_t left = __reduce_or_sync(0xffffffffu, mine);
          if (kMode != kSoftmax && !any_plain_col && left != 0u) left &= rows_not_zero(x + row_q * p.x_sn, p.x_sn, row_end - row_q, p.K);
          for (; left != 0u; left &= left - 1u) {
            const int r = __ffs(left) - 1;
            if (row_q + r >= row_end) break;
            const float y = plain_dot<kMode>(x + (row_q + r) * p.x_sn, w, rescale_s + (kMode == kPlain ? 0 : wq * 32), n0 + wq * 32, p.N, p.K);
            if (((mine >> r) & 1u) != 0u && n < p.N) out[static_cast<int64_t>(row_q + r) * p.N + n] = result(y);
          }
        }
        tc_fence_before_sync();
        mbar_arrive(smem_u32(&bars.acc_empty[st]));
      }
    }
    if (lane == 0) tma_store_wait_all();
    __syncwarp();
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == kSplitWarps) {
    __syncwarp();
    tmem_dealloc(tbase, 512);
  }
}

}  // namespace

static cudaError_t launch(LinParams& p, int mode, int64_t batches, unsigned grid, cudaStream_t stream) {
  p.chunks = (p.K + kChunk - 1) / kChunk;
  p.status = device_status_words();
  p.tma_out = p.N % 4 == 0 ? 1 : 0;
  CUtensorMap mo = {};
  if (p.tma_out) {
    const uint64_t row_bytes = static_cast<uint64_t>(p.N) * 4, batch_bytes = row_bytes * p.M;
    const uint64_t dims[4] = {static_cast<uint64_t>(p.N), static_cast<uint64_t>(p.M), static_cast<uint64_t>(batches), 1};
    const uint64_t strides[3] = {row_bytes, batch_bytes, batch_bytes};
    const uint32_t box[4] = {32, 32, 1, 1};
    if (tma_host::make_f32_map_sw128(&mo, p.out, dims, strides, box) != 0) return cudaErrorInvalidValue;
  }
  auto kern = mode == kPlain ? linear_f32_kernel<kPlain> : mode == kBatched ? linear_f32_kernel<kBatched> : linear_f32_kernel<kSoftmax>;
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmemBytes);
  if (e != cudaSuccess) return e;
  e = launch_dependent(kern, dim3(grid), dim3(kThreads), kSmemBytes, stream, mo, p);
  count_launch();
  return e;
}

cudaError_t launch_linear_f32(const float* x, const float* w, const float* bias, float* out, int M, int N, int K,
                              int num_sms, cudaStream_t stream) {
  LinParams p = {};
  p.x = x;
  p.w = w;
  p.bias = bias;
  p.out = out;
  p.M = M;
  p.N = N;
  p.K = K;
  p.x_sn = K;
  p.n_tiles = (N + kTile - 1) / kTile;
  const int64_t tiles = static_cast<int64_t>((M + kTile - 1) / kTile) * p.n_tiles;
  const int64_t most = num_sms > p.n_tiles ? num_sms : p.n_tiles;  // (every column block needs a CTA)
  return launch(p, kPlain, 1, static_cast<unsigned>(tiles < most ? tiles : most), stream);
}

BatchSplit linear_f32_split(int B, int M, int num_sms) {
  // the split with the shortest launch, in rows of work per SM; a CTA's set-up (launch, weights to TMEM, first
  // tile) takes about as long as 160 rows
  BatchSplit out = {};
  const int pieces = (M + 31) / 32;
  int64_t best = 0;
  for (int s = 1; s <= pieces && s <= num_sms; ++s) {
    const int rows = (pieces + s - 1) / s * 32, splits = (M + rows - 1) / rows;
    const int64_t cost = (static_cast<int64_t>(B) * splits + num_sms - 1) / num_sms * (rows + 160);
    if (out.splits == 0 || cost < best) {
      best = cost;
      out.rows = rows;
      out.splits = splits;
    }
  }
  return out;
}

cudaError_t launch_linear_f32_batched(const float* x, int64_t x_sb, int64_t x_sn, const float* w, int w_rows, const float* bias, float* out,
                                      int B, int M, int N, int K, bool softmax, const BatchSplit& split, const FoldScales& scales,
                                      cudaStream_t stream) {
  LinParams p = {};
  p.x = x;
  p.w = w;
  p.bias = bias;
  p.out = out;
  p.M = M;
  p.N = N;
  p.K = K;
  p.x_sn = x_sn;
  p.x_sb = x_sb;
  p.w_sb = static_cast<int64_t>(w_rows) * K;
  p.n_tiles = 1;
  p.splits = split.splits;
  p.cta_rows = split.rows;
  p.scales = scales;
  return launch(p, softmax ? kSoftmax : kBatched, B, static_cast<unsigned>(B) * p.splits, stream);
}

}  // namespace asuka
