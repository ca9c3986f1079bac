// Attention forward for a handful of query rows per key/value head: the decode step of a generation
// (q_len 1, or a few speculated tokens), with or without grouped query heads.
//
// Same program as attn_fwd.cu (cases/kernels/attn.py:18-34, gemma2.py:30-33 with soft-capping): f32
// exp2 softmax, P rounded to the input type for P.V, f32 accumulation, division last.  What bounds
// it is different: every K and V row is used by the `Sq x group` query rows of its head only, so the
// work is a stream of the whole cache and the floor is its bytes over the HBM bandwidth.  The
// 256-row items of attn_fwd.cu spend the tensor pipe and the MUFU on 128-row tiles with one or a
// few live rows, fetch a head's K and V once per query head of its group, and leave the split of a
// long cache to a second launch.  Here
//   - the query rows of a group (all heads that share the K/V head, all q_len positions) form ONE
//     16-row tile, so K and V are read once;
//   - a (batch, K/V head) unit's keys are cut into up to eight parts, one CTA each, and the CTAs of
//     a unit form a cluster: partial results are merged through distributed shared memory, in rank
//     order, in the same launch and without a workspace;
//   - a CTA streams stages of 64 keys (K and V, 32 KB) by TMA through a ring deep enough to cover
//     the latency of DRAM; four warps take 16 keys of every stage each, with warp-level 16x8x16
//     matrix instructions (a tcgen05 tile would be 128 rows for at most 16) and a running maximum
//     and sum of their own, so nothing is exchanged until the end.
// Measured (bf16, q_len 1, against the 256-row items): B16, 32 query heads on 8 K/V heads, 4001 keys
// (262 MB) 210 -> 45.2 us = 5.8 TB/s; B16, 32 K/V heads, 4001 keys (1.05 GB) 213 -> 150 us = 7.0 TB/s;
// B1, 8 K/V heads, 4096 keys (17 MB) 80 -> 8.9 us; B1, 8 K/V heads, 300 keys 24.5 -> 6.5 us.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include "kernels.h"
#include "sm100_ptx.cuh"

namespace asuka {
using namespace sm100;

namespace {

constexpr int kRows = 16;         // query rows of a CTA (Sq x group of them live)
constexpr int kKeys = 64;         // keys per stage
constexpr int kWarps = 4;         // compute warps, 16 keys of a stage each
constexpr int kThreads = (kWarps + 1) * 32;
constexpr uint32_t kHalf = kKeys * 128;        // one 64-column half of a [64 x 128] 16-bit tile
constexpr uint32_t kStageBytes = 4 * kHalf;    // K and V
constexpr int kMaxStages = 6;
constexpr int kMaxCluster = 8;
constexpr uint32_t kMergeBytes = (kWarps + 1) * kRows * 128 * 4;  // O partials of the warps and of the CTA (over the stages)

struct DecParams {
  int H, Sq, Skv, group, rows;  // rows = Sq * group
  int n_tiles, stages;
  int causal;
  float scale_log2, cap_in, cap_out;
  const uint16_t* q;
  int64_t q_sb, q_ss, q_sh;
  uint16_t* out;
  int64_t o_sb, o_ss, o_sh;
  float* lse2;
  uint32_t* status;
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
template <bool kBF16>
__device__ __forceinline__ uint32_t pack2(float lo, float hi) {
  if constexpr (kBF16) {
    __nv_bfloat162 v = __floats2bfloat162_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  } else {
    __half2 v = __floats2half2_rn(lo, hi);
    return *reinterpret_cast<uint32_t*>(&v);
  }
}
__device__ __forceinline__ void ldsm4(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
__device__ __forceinline__ void ldsm4_t(uint32_t addr, uint32_t (&r)[4]) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0, %1, %2, %3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"(addr)
               : "memory");
}
template <bool kBF16>
__device__ __forceinline__ void mma16816(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  if constexpr (kBF16)
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
  else
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ uint32_t cluster_rank() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ uint32_t cluster_size() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}
__device__ __forceinline__ void cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ float ld_cluster(uint32_t smem_addr, uint32_t rank) {
  uint32_t remote;
  float v;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(remote) : "r"(smem_addr), "r"(rank));
  asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(remote) : "memory");
  return v;
}

// Grid: units x parts, the parts of a unit a cluster.
template <bool kBF16, bool kCap>
__global__ void __launch_bounds__(kThreads, 2)
attn_decode_kernel(const __grid_constant__ CUtensorMap map_k, const __grid_constant__ CUtensorMap map_v,
                   const DecParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) uint64_t full[kMaxStages], empty[kMaxStages];
  __shared__ uint32_t abort_s;
  __shared__ float warp_ml[kWarps][2][kRows];  // running maximum (log2 units) and sum of every warp's rows
  __shared__ float cta_ml[2][kRows];           // the CTA's, read by the whole cluster

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  float* merge = reinterpret_cast<float*>(smem_raw + (smem_base - smem_u32(smem_raw)));
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile uint32_t* abortp = &abort_s;
  const int parts = static_cast<int>(cluster_size()), part = static_cast<int>(cluster_rank());
  const int Hkv = p.H / p.group;
  const int unit = static_cast<int>(blockIdx.x) / parts;
  const int b = unit / Hkv, hk = unit % Hkv;
  // this CTA's stages of 64 keys
  const int t_lo = static_cast<int>(static_cast<int64_t>(p.n_tiles) * part / parts);
  const int t_hi = static_cast<int>(static_cast<int64_t>(p.n_tiles) * (part + 1) / parts);

  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < p.stages; ++i) {
      mbar_init(smem_u32(&full[i]), 1);
      mbar_init(smem_u32(&empty[i]), kWarps);
    }
    mbar_fence_init();
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  // What the ring takes first is on its way from DRAM to L2 while the kernel ahead still runs: two stages (six are slower
  // again).  Without and with, us: caches that are not in L2, as in a program with other work between two steps, B4 H16, 2000
  // keys, 14.2 and 13.7, B8 H32/8, 1000 keys, 10.3 and 9.8, B1 H128/32, 6000 keys, 20.1 and 19.3, B16 H32/8, 4001 keys, 44.2 and
  // 43.7; caches that are, 9.7 and 10.1, 7.7 and 8.0, 14.6 and 14.5, 44.0 and 43.2.
  if (warp == kWarps && lane == 0) {
    for (int t = t_lo; t < min(t_hi, t_lo + 2); ++t) {
      tma_prefetch_4d(&map_k, 0, hk, t * kKeys, b);
      tma_prefetch_4d(&map_k, 64, hk, t * kKeys, b);
      tma_prefetch_4d(&map_v, 0, hk, t * kKeys, b);
      tma_prefetch_4d(&map_v, 64, hk, t * kKeys, b);
    }
  }
  __syncthreads();
  griddep_wait();
  griddep_launch_dependents();

  if (warp == kWarps) {
    if (lane == 0) {
      int c = 0;
      bool ok = true;
      for (int t = t_lo; t < t_hi; ++t, ++c) {
        const int st = c % p.stages, use = c / p.stages;
        if (use > 0 && !mbar_wait(smem_u32(&empty[st]), (use - 1) & 1, abortp)) {
          atomicAdd(&p.status[0], 1u);
          p.status[1] = 71;
          ok = false;
          break;
        }
        if (use > 0) fence_proxy_async_smem();  // (the consumers' reads, behind the wait above, before the copy)
        const uint32_t bar = smem_u32(&full[st]), dst = smem_base + st * kStageBytes;
        mbar_expect_tx(bar, kStageBytes);
        tma_load_4d(dst, &map_k, bar, 0, hk, t * kKeys, b);
        tma_load_4d(dst + kHalf, &map_k, bar, 64, hk, t * kKeys, b);
        tma_load_4d(dst + 2 * kHalf, &map_v, bar, 0, hk, t * kKeys, b);
        tma_load_4d(dst + 3 * kHalf, &map_v, bar, 64, hk, t * kKeys, b);
      }
      if (!ok) {
        // give copies already in flight a bounded chance to land before the CTA retires
        volatile uint32_t none = 0;
        for (int x = c > p.stages ? c - p.stages : 0; x < c; ++x)
          mbar_wait(smem_u32(&full[x % p.stages]), (x / p.stages) & 1, &none);
      }
    }
    __syncwarp();
  } else {
    // Query rows of this thread: r and r + 8 of the tile; row = position * group + head in group.
    const int r0 = lane >> 2;
    uint32_t qf[8][4];  // the whole [16 x 128] query tile as matrix fragments
    int lim[2];         // last visible key of either row
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      const int r = r0 + 8 * x;
      const int pos = r / p.group, g = r % p.group;
      lim[x] = p.causal ? min(p.Skv - 1, pos + p.Skv - p.Sq) : p.Skv - 1;
      const uint32_t* src = reinterpret_cast<const uint32_t*>(
          p.q + static_cast<int64_t>(b) * p.q_sb + static_cast<int64_t>(pos) * p.q_ss +
          static_cast<int64_t>(hk * p.group + g) * p.q_sh) + (lane & 3);
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        qf[kk][x] = r < p.rows ? __ldg(src + kk * 8) : 0u;
        qf[kk][2 + x] = r < p.rows ? __ldg(src + kk * 8 + 4) : 0u;
      }
    }
    const int min_lim = p.causal ? p.Skv - p.Sq : p.Skv - 1;  // (row 0's)

    float o[16][4];
#pragma unroll
    for (int i = 0; i < 16; ++i)
#pragma unroll
      for (int e = 0; e < 4; ++e) o[i][e] = 0.f;
    float m[2] = {-INFINITY, -INFINITY}, l[2] = {0.f, 0.f};  // l: this thread's columns only
    bool ok = true;

    // addresses of this lane's rows for the 8x8 blocks: keys of the warp's 16, 16-byte chunk of a row
    const int k_row = warp * 16 + ((lane >> 4) << 3) + (lane & 7), k_chunk = (lane >> 3) & 1;
    const int v_row = warp * 16 + (((lane >> 3) & 1) << 3) + (lane & 7), v_chunk = lane >> 4;

    int c = 0;
    for (int t = t_lo; t < t_hi; ++t, ++c) {
      const int st = c % p.stages;
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&full[st]), (c / p.stages) & 1, abortp));
      if (!ok) {
        if (lane == 0) {
          atomicAdd(&p.status[0], 1u);
          p.status[1] = 72;
        }
        break;
      }
      const uint32_t sK = smem_base + st * kStageBytes, sV = sK + 2 * kHalf;
      float s[2][4] = {{0.f, 0.f, 0.f, 0.f}, {0.f, 0.f, 0.f, 0.f}};
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        uint32_t kf[4];  // keys 0-7: k 0-7, 8-15; keys 8-15: k 0-7, 8-15
        ldsm4(sK + (kk >> 2) * kHalf + sw128_offset(k_row, (kk & 3) * 2 + k_chunk), kf);
        mma16816<kBF16>(s[0], qf[kk], kf[0], kf[1]);
        mma16816<kBF16>(s[1], qf[kk], kf[2], kf[3]);
      }
      // logits in log2 units: s[j][e] is row r0 (e < 2) or r0 + 8, key 8j + 2(lane & 3) + (e & 1)
      const int key0 = t * kKeys + warp * 16;
#pragma unroll
      for (int j = 0; j < 2; ++j)
#pragma unroll
        for (int e = 0; e < 4; ++e)
          s[j][e] = kCap ? tanh_approx(s[j][e] * p.cap_in) * p.cap_out : s[j][e] * p.scale_log2;
      if (key0 + 15 > min_lim) {
#pragma unroll
        for (int j = 0; j < 2; ++j)
#pragma unroll
          for (int e = 0; e < 4; ++e)
            if (key0 + 8 * j + 2 * (lane & 3) + (e & 1) > lim[e >> 1]) s[j][e] = -INFINITY;
      }
      float mx[2], w[2];
#pragma unroll
      for (int x = 0; x < 2; ++x) {
        mx[x] = fmaxf(fmaxf(s[0][2 * x], s[0][2 * x + 1]), fmaxf(s[1][2 * x], s[1][2 * x + 1]));
        mx[x] = fmaxf(mx[x], __shfl_xor_sync(0xffffffffu, mx[x], 1));
        mx[x] = fmaxf(mx[x], __shfl_xor_sync(0xffffffffu, mx[x], 2));
        mx[x] = fmaxf(mx[x], m[x]);
        const float ref = mx[x] > -INFINITY ? mx[x] : 0.f;
        w[x] = ex2(m[x] - ref);
        m[x] = mx[x];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
          s[j][2 * x] = ex2(s[j][2 * x] - ref);
          s[j][2 * x + 1] = ex2(s[j][2 * x + 1] - ref);
        }
        l[x] = l[x] * w[x] + ((s[0][2 * x] + s[0][2 * x + 1]) + (s[1][2 * x] + s[1][2 * x + 1]));
      }
      if (__any_sync(0xffffffffu, w[0] != 1.f || w[1] != 1.f)) {
#pragma unroll
        for (int i = 0; i < 16; ++i) {
          o[i][0] *= w[0];
          o[i][1] *= w[0];
          o[i][2] *= w[1];
          o[i][3] *= w[1];
        }
      }
      const uint32_t pf[4] = {pack2<kBF16>(s[0][0], s[0][1]), pack2<kBF16>(s[0][2], s[0][3]),
                              pack2<kBF16>(s[1][0], s[1][1]), pack2<kBF16>(s[1][2], s[1][3])};
#pragma unroll
      for (int d = 0; d < 8; ++d) {
        uint32_t vf[4];  // columns 16d + 0-7: keys 0-7, 8-15; columns 16d + 8-15: keys 0-7, 8-15
        ldsm4_t(sV + (d >> 2) * kHalf + sw128_offset(v_row, (d & 3) * 2 + v_chunk), vf);
        mma16816<kBF16>(o[2 * d], pf, vf[0], vf[1]);
        mma16816<kBF16>(o[2 * d + 1], pf, vf[2], vf[3]);
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&empty[st]));
    }
    if (!ok) *abortp = 1u;
    // row sums over the four threads of a row
#pragma unroll
    for (int x = 0; x < 2; ++x) {
      l[x] += __shfl_xor_sync(0xffffffffu, l[x], 1);
      l[x] += __shfl_xor_sync(0xffffffffu, l[x], 2);
      if ((lane & 3) == 0) {
        warp_ml[warp][0][r0 + 8 * x] = m[x];
        warp_ml[warp][1][r0 + 8 * x] = l[x];
      }
    }
    // every warp has consumed every stage (and so every copy has landed): the ring becomes the
    // merge buffer
    named_bar_sync(1, kWarps * 32);
    float* mine = merge + warp * (kRows * 128);
#pragma unroll
    for (int i = 0; i < 16; ++i) {
      *reinterpret_cast<float2*>(mine + r0 * 128 + i * 8 + 2 * (lane & 3)) = make_float2(o[i][0], o[i][1]);
      *reinterpret_cast<float2*>(mine + (r0 + 8) * 128 + i * 8 + 2 * (lane & 3)) = make_float2(o[i][2], o[i][3]);
    }
    named_bar_sync(1, kWarps * 32);
    // the four warps' partial results to one per CTA, in warp order; thread = output column
    float* cta = merge + kWarps * (kRows * 128);
    for (int r = 0; r < p.rows; ++r) {
      float mm = -INFINITY;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) mm = fmaxf(mm, warp_ml[w][0][r]);
      float acc = 0.f, ll = 0.f;
#pragma unroll
      for (int w = 0; w < kWarps; ++w) {
        const float wt = warp_ml[w][0][r] > -INFINITY ? ex2(warp_ml[w][0][r] - mm) : 0.f;
        acc = fmaf(wt, merge[w * (kRows * 128) + r * 128 + tid], acc);
        ll = fmaf(wt, warp_ml[w][1][r], ll);
      }
      cta[r * 128 + tid] = acc;
      if (tid == 0) {
        cta_ml[0][r] = mm;
        cta_ml[1][r] = ll;
      }
    }
  }

  // ---- merge over the cluster, in rank order; row r is finished by the CTA of rank r mod parts
  cluster_sync();
  if (warp < kWarps) {
    const uint32_t cta_addr = smem_base + kWarps * (kRows * 128) * 4;
    for (int r = part; r < p.rows; r += parts) {
      float pm[kMaxCluster], pl[kMaxCluster], po[kMaxCluster];
#pragma unroll
      for (int x = 0; x < kMaxCluster; ++x) {
        if (x < parts) {
          pm[x] = ld_cluster(smem_u32(&cta_ml[0][r]), x);
          pl[x] = ld_cluster(smem_u32(&cta_ml[1][r]), x);
          po[x] = ld_cluster(cta_addr + (r * 128 + tid) * 4, x);
        }
      }
      float mm = -INFINITY, ll = 0.f, acc = 0.f;
#pragma unroll
      for (int x = 0; x < kMaxCluster; ++x)
        if (x < parts) mm = fmaxf(mm, pm[x]);
#pragma unroll
      for (int x = 0; x < kMaxCluster; ++x) {
        if (x < parts) {
          const float wt = pm[x] > -INFINITY ? ex2(pm[x] - mm) : 0.f;
          ll = fmaf(wt, pl[x], ll);
          acc = fmaf(wt, po[x], acc);
        }
      }
      const float y = acc / ll;
      const int pos = r / p.group, h = hk * p.group + r % p.group;
      const float hi = __shfl_down_sync(0xffffffffu, y, 1);
      if ((tid & 1) == 0)
        *reinterpret_cast<uint32_t*>(p.out + static_cast<int64_t>(b) * p.o_sb + static_cast<int64_t>(pos) * p.o_ss +
                                     static_cast<int64_t>(h) * p.o_sh + tid) = pack2<kBF16>(y, hi);
      if (p.lse2 != nullptr && tid == 0)
        p.lse2[(static_cast<size_t>(b) * p.H + h) * p.Sq + pos] = mm + log2f(ll);
    }
  }
  cluster_sync();  // no CTA leaves while another still reads its shared memory
}

}  // namespace

// The query rows of a K/V head fit one 16-row tile: up to here a 128-row tile would be at least
// seven eighths padding, and the warp-level tile keeps up with the stream (above it the tensor work
// of this kernel would grow with every further 16 rows while the 256-row items' would not).
bool attn_decode_applies(const AttnShape& s) { return static_cast<int64_t>(s.Sq) * s.group <= kRows; }

// mk, mv: boxes of 64 keys.  q and out: strides in elements.
cudaError_t launch_attn_decode(const CUtensorMap& mk, const CUtensorMap& mv, const void* q, int64_t q_sb, int64_t q_ss,
                               int64_t q_sh, void* out, int64_t o_sb, int64_t o_ss, int64_t o_sh, float* lse2,
                               const AttnShape& s, int num_sms, cudaStream_t stream) {
  DecParams p;
  p.H = s.H;
  p.Sq = s.Sq;
  p.Skv = s.Skv;
  p.group = s.group;
  p.rows = s.Sq * s.group;
  p.n_tiles = (s.Skv + kKeys - 1) / kKeys;
  p.causal = s.causal;
  p.scale_log2 = s.softmax_scale * 1.4426950408889634f;
  p.cap_in = s.softcap > 0.f ? s.softmax_scale / s.softcap : 0.f;
  p.cap_out = s.softcap * 1.4426950408889634f;
  p.q = static_cast<const uint16_t*>(q);
  p.q_sb = q_sb;
  p.q_ss = q_ss;
  p.q_sh = q_sh;
  p.out = static_cast<uint16_t*>(out);
  p.o_sb = o_sb;
  p.o_ss = o_ss;
  p.o_sh = o_sh;
  p.lse2 = lse2;
  p.status = device_status_words();
  // Parts: as many as bring the launch to two CTAs per SM (what fits side by side), at least two
  // stages each.
  const long long units = static_cast<long long>(s.B) * (s.H / s.group);
  int parts = 1;
  while (parts < kMaxCluster && units * parts * 2 <= 2LL * num_sms && p.n_tiles >= parts * 4) parts *= 2;
  // Two CTAs per SM share its memory; a launch that gives every SM one at most takes the whole of it.
  p.stages = units * parts > num_sms ? 3 : kMaxStages;
  const uint32_t smem = (p.stages * kStageBytes > kMergeBytes ? p.stages * kStageBytes : kMergeBytes) + 1024;
  void (*kern)(CUtensorMap, CUtensorMap, DecParams);
  if (s.softcap > 0.f) kern = s.bf16 ? attn_decode_kernel<true, true> : attn_decode_kernel<false, true>;
  else kern = s.bf16 ? attn_decode_kernel<true, false> : attn_decode_kernel<false, false>;
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kMaxStages * kStageBytes + 1024);
  if (e != cudaSuccess) return e;
  e = launch_dependent_cluster(kern, dim3(static_cast<unsigned>(units * parts)), dim3(kThreads), smem,
                               static_cast<unsigned>(parts), stream, mk, mv, p);
  count_launch();
  return e;
}

}  // namespace asuka
