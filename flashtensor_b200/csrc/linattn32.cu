// Linear attention at head_dim 32 in f32: the attention core of the reference's SimA and EA
// benchmark programs at their own shapes (bench/sima.mlir:13-17, bench/ea.mlir:13-17:
// tensor<64x4x784x32xf32>), between the QKV projection and the output projection.
//
//   SimA  out = (Q / sum_n|Q|) . ((K / sum_n|K|)^T . V)      (normalisations over the sequence n)
//   EA    out = softmax_d(Q)   . (softmax_n(K)^T . V)
//
// With 32 features the two products are 2 flops per byte moved, far too few for tensor-core tiles:
// CUDA-core code, bound by how much of the [N, 32] slices (one 128-byte line per row and tensor) is
// in flight.  One CTA per (batch, head), two to an SM; every tile of 64 rows comes and goes by TMA:
//   pass A  K, V (and SimA's Q) through a ring of four stages; eight warps take eight rows of a
//           stage each.  A lane keeps an 8 x 4 block of the 32 x 32 product K'^T V in registers, so a
//           row costs it three 16-byte reads of shared memory (a whole column per lane needs eight
//           for K's row alone, and shared memory was what the kernel waited for).  The statistics are gathered on the way: SimA's
//           sums of |K| and |Q|; for EA each warp exponentiates K in place against a running
//           reference of its own per column, raised (with its partial product rescaled) only when
//           a value exceeds it by more than a factor of 2^8, so no pass over K precedes the product.
//   pass B  Q through a ring of eight tiles; the output row is written over the row of Q it came
//           from and leaves by TMA.
// Multiply-adds are the packed two-wide f32 FMAs of sm_100; every sum runs in a fixed order.
// Measured at B64 H4 N784 (SimA / EA): three passes of plain loads with sixteen rows of a warp in
// flight 58 / 67 us, this kernel 37 / 47 us.
// In a whole block (kFold) there is no pass B: the kernel multiplies the 32 x 32 matrices with the output
// projection, and linear_f32.cu applies the product to the queries (this kernel 23 us then; the block, SimA / EA,
// 87 / 95 -> 77 / 85 us with it and the projections' earlier start, on one card).  For blocks of some length only, see
// fold_from in bind.cpp.
#include "f32_keep.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"
#include "tma_host.h"

namespace asuka {
using namespace sm100;

namespace {

constexpr int kD = 32;
constexpr int kWarps = 8;
constexpr int kThreads = (kWarps + 1) * 32;  // + the producer warp
constexpr int kRows = 64;                    // rows of a tile
constexpr int kWarpRows = kRows / kWarps;
constexpr uint32_t kTileBytes = kRows * kD * 4;
constexpr int kStages = 4;                   // pass A: K, V, Q tiles
constexpr int kQStages = 8;                  // pass B: Q tiles, in the part of the ring above the partial products
constexpr uint32_t kPartBytes = kWarps * kD * kD * 4;
constexpr uint32_t kSmemBytes = kStages * 3 * kTileBytes + 1024;
constexpr int kFoldLoads = 4;                // (kFold) 16-byte pieces of a thread of a head's 128 columns at most
constexpr float kSlack = 5.5f;               // EA: by how much a key may exceed its warp's reference (e^5.5 = 2^8)
static_assert(kPartBytes + kQStages * kTileBytes <= kStages * 3 * kTileBytes, "pass B's ring");

struct Lin32Params {
  int N, H;
  const float* w_o;  // (kFold) output projection [32 H, 32 H], and where its product with every batch's M' goes
  float* w_fold;     // [B, fold_rows, 32 H], 32 H rows of it
  int fold_rows;
  FoldScales scales;
  int scale_copies;  // of a batch's words
  uint32_t* status;
};

struct Lin32Bars {
  uint64_t a_full[kStages], a_empty[kStages];
  uint64_t b_full[kQStages], b_empty[kQStages];
};

// e^x of a difference from a reference: the difference is taken first and scaled to powers of two after it.
// (Scaling the values first rounds each by 2^-24 of itself, not of the difference: with an offset of 100
// common to all keys the output was off by 1.7e-5 of itself, with -1000 by 1.3e-4; this way by 1.2e-7 with and without.)
__device__ __forceinline__ float exp_fast(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x * 1.4426950408889634f));
  return y;
}
__device__ __forceinline__ float warp_max(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x = fmaxf(x, __shfl_xor_sync(0xffffffffu, x, o));
  return x;
}
__device__ __forceinline__ float warp_sum(float x) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
  return x;
}
__device__ __forceinline__ void record_timeout(uint32_t* status, uint32_t site) {
  atomicAdd(&status[0], 1u);
  status[1] = site;
}

template <bool kEA, bool kFold>
__global__ void __launch_bounds__(kThreads, 2)
linattn32_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                 const __grid_constant__ CUtensorMap map_v, const __grid_constant__ CUtensorMap map_out,
                 const Lin32Params p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) Lin32Bars bars;
  __shared__ float m_s[kD][kD + 1];                 // M' = normalised K'^T V, [d][e]
  __shared__ __align__(16) float scale_s[kWarps][kD];  // EA: rescale factors of a warp's partial product
  __shared__ float stat_s[2][kWarps][kD];           // SimA: sum|K|, sum|Q|; EA: reference, sum of K'
  __shared__ __align__(4) uint8_t e_s[4 * kD];      // (kFold) exponents of this head's scales (f32_keep.cuh), by column
  __shared__ uint32_t abort_s;
  const uint32_t ring = (smem_u32(smem_raw) + 1023u) & ~1023u;
  float* const ring_gen = reinterpret_cast<float*>(smem_raw + (ring - smem_u32(smem_raw)));

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  volatile uint32_t* abortp = &abort_s;
  const int b = blockIdx.x / p.H, h = blockIdx.x % p.H;
  const int n_tiles = (p.N + kRows - 1) / kRows;

  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < kStages; ++i) {
      mbar_init(smem_u32(&bars.a_full[i]), 1);
      mbar_init(smem_u32(&bars.a_empty[i]), kWarps);
    }
    for (int i = 0; i < kQStages; ++i) {
      mbar_init(smem_u32(&bars.b_full[i]), 1);
      mbar_init(smem_u32(&bars.b_empty[i]), kWarps);
    }
    mbar_fence_init();
  }
  __syncthreads();
  griddep_wait();
  griddep_launch_dependents();

  // ---- pass A
  const int e0 = (lane & 7) * 4, d0 = (lane >> 3) * 8;  // this lane's block of a 32 x 32 product
  float2 acc[4][4];  // [e][pair of d]
#pragma unroll
  for (int e = 0; e < 4; ++e)
#pragma unroll
    for (int d = 0; d < 4; ++d) acc[e][d] = make_float2(0.f, 0.f);
  float s0 = kEA ? -INFINITY : 0.f, s1 = 0.f;
  if (warp == kWarps) {
    if (lane == 0) {
      int t = 0;
      for (; t < n_tiles; ++t) {
        const int st = t % kStages;
        if (t >= kStages && !mbar_wait(smem_u32(&bars.a_empty[st]), (t / kStages - 1) & 1, abortp)) {
          record_timeout(p.status, 91);
          break;
        }
        if (t >= kStages) fence_proxy_async_smem();  // (the consumers' reads, behind the wait above, before the copy)
        const uint32_t bar = smem_u32(&bars.a_full[st]), dst = ring + st * 3 * kTileBytes;
        mbar_expect_tx(bar, (kEA ? 2 : 3) * kTileBytes);
        tma_load_4d(dst, &map_k, bar, 0, h, t * kRows, b);
        tma_load_4d(dst + kTileBytes, &map_v, bar, 0, h, t * kRows, b);
        if (!kEA) tma_load_4d(dst + 2 * kTileBytes, &map_q, bar, 0, h, t * kRows, b);
      }
      if (t < n_tiles) {  // gave up: let copies in flight land
        volatile uint32_t none = 0;
        for (int x = t > kStages ? t - kStages : 0; x < t; ++x)
          mbar_wait(smem_u32(&bars.a_full[x % kStages]), (x / kStages) & 1, &none);
      }
    }
    __syncwarp();
  } else {
    for (int t = 0; t < n_tiles; ++t) {
      const int st = t % kStages;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.a_full[st]), (t / kStages) & 1, abortp))) {
        if (lane == 0) record_timeout(p.status, 92);
        break;
      }
      float* const kt = ring_gen + (st * 3 * kTileBytes) / 4 + warp * kWarpRows * kD;
      const float* const vt = kt + kTileBytes / 4;
      const float* const qt = vt + kTileBytes / 4;
      if constexpr (kEA) {
        float kv[kWarpRows];
        float mx = -INFINITY;
#pragma unroll
        for (int u = 0; u < kWarpRows; ++u) {
          const bool live = t * kRows + warp * kWarpRows + u < p.N;
          kv[u] = live ? kt[u * kD + lane] : -INFINITY;
          mx = fmaxf(mx, kv[u]);
        }
        // (a warp whose rows all lie past the end changes nothing)
        const bool raise = mx > s0 + kSlack;
        if (__any_sync(0xffffffffu, raise)) {
          const float m_new = raise ? mx : s0;
          const float f = m_new > -INFINITY ? exp_fast(s0 - m_new) : 1.f;
          s0 = m_new;
          s1 *= f;
          scale_s[warp][lane] = f;
          __syncwarp();
          const float4 f0 = *reinterpret_cast<const float4*>(&scale_s[warp][d0]);
          const float4 f1 = *reinterpret_cast<const float4*>(&scale_s[warp][d0 + 4]);
          const float2 ff[4] = {make_float2(f0.x, f0.y), make_float2(f0.z, f0.w), make_float2(f1.x, f1.y), make_float2(f1.z, f1.w)};
#pragma unroll
          for (int e = 0; e < 4; ++e)
#pragma unroll
            for (int d = 0; d < 4; ++d) acc[e][d] = __fmul2_rn(acc[e][d], ff[d]);
        }
        // (no value above -inf yet: against 0 the -infs give 0 and a NaN, which the maximum skips, stays one)
        const float ref = s0 > -INFINITY ? s0 : 0.f;
#pragma unroll
        for (int u = 0; u < kWarpRows; ++u) {
          const float e = exp_fast(kv[u] - ref);
          s1 += e;
          kt[u * kD + lane] = e;
        }
        __syncwarp();
      } else {
#pragma unroll
        for (int u = 0; u < kWarpRows; ++u) {
          s0 += fabsf(kt[u * kD + lane]);
          s1 += fabsf(qt[u * kD + lane]);
        }
      }
      // acc[e][d] += V[row][e] * K'[row][d]
#pragma unroll
      for (int u = 0; u < kWarpRows; ++u) {
        const float4 v = *reinterpret_cast<const float4*>(vt + u * kD + e0);
        const float4 k0 = *reinterpret_cast<const float4*>(kt + u * kD + d0);
        const float4 k1 = *reinterpret_cast<const float4*>(kt + u * kD + d0 + 4);
        const float ve[4] = {v.x, v.y, v.z, v.w};
        const float2 kk[4] = {make_float2(k0.x, k0.y), make_float2(k0.z, k0.w), make_float2(k1.x, k1.y), make_float2(k1.z, k1.w)};
#pragma unroll
        for (int e = 0; e < 4; ++e)
#pragma unroll
          for (int d = 0; d < 4; ++d) acc[e][d] = __ffma2_rn(kk[d], make_float2(ve[e], ve[e]), acc[e][d]);
      }
      if constexpr (kEA) fence_proxy_async_smem();  // (K' was written over a tile that TMA refills)
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&bars.a_empty[st]));
    }
    stat_s[0][warp][lane] = s0;
    stat_s[1][warp][lane] = s1;
  }
  const int C = p.H * kD;
  float4 o[kFold ? kFoldLoads : 1];  // (kFold) this thread's part of the output projection, on its way during the barrier
  if constexpr (kFold) {
#pragma unroll
    for (int x = 0; x < kFoldLoads; ++x) {
      const int i = x * kWarps * 32 + tid, c = i >> 3;
      if (warp < kWarps && c < C) o[x] = __ldg(reinterpret_cast<const float4*>(p.w_o + c * C + h * kD) + (i & 7));
    }
  }
  __syncthreads();

  // ---- the warps' partial products to M', in warp order, while the first tiles of pass B arrive
  float* const part = ring_gen;
  float* const w_s = ring_gen + kPartBytes / 4;  // (kFold) this head's columns of the output projection, [c][e]
  const uint32_t qring = ring + kPartBytes;
  if (warp < kWarps) {
    if constexpr (kFold) {  // (the ring is free: nothing is in flight after pass A)
#pragma unroll
      for (int x = 0; x < kFoldLoads; ++x) {
        const int i = x * kWarps * 32 + tid, c = i >> 3;
        if (c < C) {  // (whole warps: C is a multiple of 32)
          const uint32_t e = fold_scale_exponent(head_max_bits(o[x]));
          const float s = __uint_as_float(e << 23);
          *reinterpret_cast<float4*>(w_s + i * 4) = make_float4(mul_keep(o[x].x, s), mul_keep(o[x].y, s), mul_keep(o[x].z, s), mul_keep(o[x].w, s));
          if ((i & 7) == 0) e_s[c] = static_cast<uint8_t>(e);
        }
      }
    }
#pragma unroll
    for (int d = 0; d < 4; ++d) {
      *reinterpret_cast<float4*>(part + (warp * kD + d0 + 2 * d) * kD + e0) =
          make_float4(acc[0][d].x, acc[1][d].x, acc[2][d].x, acc[3][d].x);
      *reinterpret_cast<float4*>(part + (warp * kD + d0 + 2 * d + 1) * kD + e0) =
          make_float4(acc[0][d].y, acc[1][d].y, acc[2][d].y, acc[3][d].y);
    }
    named_bar_sync(1, kWarps * 32);
    for (int d = warp; d < kD; d += kWarps) {
      float total = 0.f, inv;
      if constexpr (kEA) {
        float m = -INFINITY, z = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) m = fmaxf(m, stat_s[0][w][d]);
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          const float f = stat_s[0][w][d] > -INFINITY ? exp_fast(stat_s[0][w][d] - m) : 0.f;
          z = fmaf(f, stat_s[1][w][d], z);
          total = fmaf(f, part[(w * kD + d) * kD + lane], total);
        }
        inv = 1.f / z;
      } else {
        float ck = 0.f, cq = 0.f;
#pragma unroll
        for (int w = 0; w < kWarps; ++w) {
          ck += stat_s[0][w][d];
          cq += stat_s[1][w][d];
          total += part[(w * kD + d) * kD + lane];
        }
        inv = 1.f / (ck * cq);
      }
      m_s[d][lane] = total * inv;
    }
    named_bar_sync(1, kWarps * 32);
  }

  if constexpr (kFold) {
    if (warp == 0 && lane * 4 < C) {
      const uint32_t e4 = *reinterpret_cast<const uint32_t*>(&e_s[lane * 4]);
      uint32_t* dst = p.scales.ptr + b * p.scales.per_batch + h * (C / 4) + lane;
      for (int y = 0; y < p.scale_copies; ++y) dst[y * p.scales.per_cta] = e4;
    }
    // ---- out = Qn . blockdiag(M') . w_o^T + b_o: what is left of it after this kernel is one product of the
    // (EA: normalised) queries with w_fold[b][c][h * 32 + d] = sum_e M'[d][e] w_o[c][h * 32 + e], times the scale of
    // (c, h) (f32_keep.cuh)
    if (warp < kWarps) {
      float m[kD];
#pragma unroll
      for (int e = 0; e < kD; ++e) m[e] = m_s[lane][e];
      float* dst = p.w_fold + static_cast<int64_t>(b) * p.fold_rows * C + h * kD + lane;
      for (int c = warp; c < C; c += kWarps) {
        float sum[kD / 4];  // (in pairs: one running sum of thirty-two rounds more)
#pragma unroll
        for (int i = 0; i < kD / 4; ++i) {
          const float4 o = *reinterpret_cast<const float4*>(w_s + c * kD + i * 4);
          sum[i] = add_keep(fma_keep(m[4 * i], o.x, mul_keep(m[4 * i + 1], o.y)),
                            fma_keep(m[4 * i + 2], o.z, mul_keep(m[4 * i + 3], o.w)));
        }
        dst[static_cast<int64_t>(c) * C] = add_keep(add_keep(add_keep(sum[0], sum[1]), add_keep(sum[2], sum[3])),
                                                    add_keep(add_keep(sum[4], sum[5]), add_keep(sum[6], sum[7])));
      }
    }
    return;
  }

  // ---- pass B: out[n][e] = sum_d Qn[n][d] M'[d][e]; a lane keeps its 8 x 4 block of M' in registers,
  // and the four lanes with the same columns e add their parts up
  if (warp == kWarps) {
    if (lane == 0) {
      int t = 0;
      for (; t < n_tiles; ++t) {
        const int st = t % kQStages;
        if (t >= kQStages && !mbar_wait(smem_u32(&bars.b_empty[st]), (t / kQStages - 1) & 1, abortp)) {
          record_timeout(p.status, 93);
          break;
        }
        const uint32_t bar = smem_u32(&bars.b_full[st]);
        mbar_expect_tx(bar, kTileBytes);
        tma_load_4d(qring + st * kTileBytes, &map_q, bar, 0, h, t * kRows, b);
      }
      if (t < n_tiles) {
        volatile uint32_t none = 0;
        for (int x = t > kQStages ? t - kQStages : 0; x < t; ++x)
          mbar_wait(smem_u32(&bars.b_full[x % kQStages]), (x / kQStages) & 1, &none);
      }
    }
    __syncwarp();
  } else {
    float2 mb[4][4];  // [e][pair of d]
#pragma unroll
    for (int e = 0; e < 4; ++e)
#pragma unroll
      for (int d = 0; d < 4; ++d) mb[e][d] = make_float2(m_s[d0 + 2 * d][e0 + e], m_s[d0 + 2 * d + 1][e0 + e]);
    const bool hi16 = (lane & 16) != 0, hi8 = (lane & 8) != 0;
    const int e_mine = e0 + (hi16 ? 2 : 0) + (hi8 ? 1 : 0);
    for (int t = 0; t < n_tiles; ++t) {
      const int st = t % kQStages;
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.b_full[st]), (t / kQStages) & 1, abortp))) {
        if (lane == 0) record_timeout(p.status, 94);
        break;
      }
      float* const qt = ring_gen + (kPartBytes + st * kTileBytes) / 4 + warp * kWarpRows * kD;
      if constexpr (kEA) {
#pragma unroll
        for (int u = 0; u < kWarpRows; ++u) {
          const float x = qt[u * kD + lane];
          const float e = exp_fast(x - warp_max(x));
          qt[u * kD + lane] = e / warp_sum(e);
        }
        __syncwarp();
      }
      float y[kWarpRows];
#pragma unroll
      for (int u = 0; u < kWarpRows; ++u) {
        const float4 q0 = *reinterpret_cast<const float4*>(qt + u * kD + d0);
        const float4 q1 = *reinterpret_cast<const float4*>(qt + u * kD + d0 + 4);
        const float2 qq[4] = {make_float2(q0.x, q0.y), make_float2(q0.z, q0.w), make_float2(q1.x, q1.y), make_float2(q1.z, q1.w)};
        float o[4];
#pragma unroll
        for (int e = 0; e < 4; ++e) {
          float2 o2 = __fmul2_rn(qq[0], mb[e][0]);
#pragma unroll
          for (int d = 1; d < 4; ++d) o2 = __ffma2_rn(qq[d], mb[e][d], o2);
          o[e] = o2.x + o2.y;
        }
        const float a0 = __shfl_xor_sync(0xffffffffu, hi16 ? o[0] : o[2], 16) + (hi16 ? o[2] : o[0]);
        const float a1 = __shfl_xor_sync(0xffffffffu, hi16 ? o[1] : o[3], 16) + (hi16 ? o[3] : o[1]);
        y[u] = __shfl_xor_sync(0xffffffffu, hi8 ? a0 : a1, 8) + (hi8 ? a1 : a0);
      }
      __syncwarp();
#pragma unroll
      for (int u = 0; u < kWarpRows; ++u) qt[u * kD + e_mine] = y[u];
      fence_proxy_async_smem();
      __syncwarp();
      if (lane == 0) {
        const int row = t * kRows + warp * kWarpRows;
        if (row < p.N)
          tma_store_4d(&map_out, qring + st * kTileBytes + warp * kWarpRows * kD * 4, 0, h, row, b);
        tma_store_commit();
        tma_store_wait_read_n<1>();  // the tile before has left: its buffer may be refilled
        if (t > 0) mbar_arrive(smem_u32(&bars.b_empty[(t - 1) % kQStages]));
      }
      __syncwarp();
    }
    if (lane == 0) tma_store_wait_all();
    __syncwarp();
  }
  __syncthreads();
}

}  // namespace

static cudaError_t launch(const LinAttn32Args& a, const Lin32Params& fold, cudaStream_t stream) {
  const float* const w_o = fold.w_o;
  Lin32Params p = fold;
  p.N = a.N;
  p.H = a.H;
  p.status = device_status_words();
  const uint64_t dims[4] = {kD, static_cast<uint64_t>(a.H), static_cast<uint64_t>(a.N), static_cast<uint64_t>(a.B)};
  auto map = [&](CUtensorMap* m, const float* base, int64_t sh, int64_t sn, int64_t sb, uint32_t rows) {
    const uint64_t strides[3] = {static_cast<uint64_t>(sh) * 4, static_cast<uint64_t>(sn) * 4, static_cast<uint64_t>(sb) * 4};
    const uint32_t box[4] = {kD, 1, rows, 1};
    return tma_host::make_f32_map(m, base, dims, strides, box, false) == 0;
  };
  CUtensorMap mq, mk, mv, mo;
  if (!map(&mq, a.q, a.q_sh, a.q_sn, a.q_sb, kRows) || !map(&mk, a.k, a.k_sh, a.k_sn, a.k_sb, kRows) ||
      !map(&mv, a.v, a.v_sh, a.v_sn, a.v_sb, kRows))
    return cudaErrorInvalidValue;
  if (w_o != nullptr) {
    mo = mq;  // (not used)
  } else if (!map(&mo, a.out, a.o_sh, a.o_sn, a.o_sb, kWarpRows)) {
    return cudaErrorInvalidValue;
  }
  auto kern = w_o != nullptr ? (a.ea ? linattn32_kernel<true, true> : linattn32_kernel<false, true>)
                             : (a.ea ? linattn32_kernel<true, false> : linattn32_kernel<false, false>);
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmemBytes);
  if (e != cudaSuccess) return e;
  e = launch_dependent(kern, dim3(static_cast<unsigned>(a.B) * a.H), dim3(kThreads), kSmemBytes, stream, mq, mk, mv, mo, p);
  count_launch();
  return e;
}

cudaError_t launch_linattn32(const LinAttn32Args& a, cudaStream_t stream) { return launch(a, {}, stream); }

cudaError_t launch_linattn32_proj(const LinAttn32Args& a, const float* w_o, const float* b_o, float* w_fold, int fold_rows,
                                  int num_sms, cudaStream_t stream) {
  const int C = a.H * kD;
  const BatchSplit split = linear_f32_split(a.B, a.N, num_sms);
  Lin32Params fold = {};
  fold.w_o = w_o;
  fold.w_fold = w_fold;
  fold.fold_rows = fold_rows;
  if (fold_rows > C) {  // room for the scales behind the folded weights
    fold.scales = {reinterpret_cast<uint32_t*>(w_fold) + static_cast<int64_t>(C) * C, static_cast<int64_t>(fold_rows) * C, 0};
    fold.scale_copies = 1;
  } else {  // in the first row of the output that each CTA of the projection writes, before it does
    fold.scales = {reinterpret_cast<uint32_t*>(a.out), static_cast<int64_t>(a.N) * C, static_cast<int64_t>(split.rows) * C};
    fold.scale_copies = split.splits;
  }
  const cudaError_t e = launch(a, fold, stream);
  if (e != cudaSuccess) return e;
  return launch_linear_f32_batched(a.q, a.q_sb, a.q_sn, w_fold, fold_rows, b_o, a.out, a.B, a.N, C, C, a.ea != 0, split, fold.scales, stream);
}

}  // namespace asuka
