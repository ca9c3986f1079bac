// Attention forward for sm_100a: O = softmax(Q K^T * scale + causal mask) V, plus the per-row
// base-2 log-sum-exp that the column-score pass consumes.
//
// Replaces the kernel the Asuka pipeline generates for Attn.forward (cases/kernels/attn.py:18-34):
// f32 exp2-based softmax with the division deferred until after P.V, P rounded to the input type
// for the second product, f32 accumulation, fully masked tiles skipped (the numerics fixed by
// LowerComplexReduce / RecoverTypeInKernel / ReplaceExpAndLog / EquivalentTransform / DynamicFor).
//
// The kernel is persistent: one CTA per SM walks a list of work items (256 query rows of one
// (batch, head), heaviest first, dealt out in a zigzag so that every CTA gets the same amount of
// work).  The two 128-row tiles of an item ping-pong through the tensor pipe so that the softmax of
// one overlaps the MMAs of the other, and the K/V/Q loads and the first QK^T of the next item run
// under the tail and the epilogue of the current one.
//   warp 0        TMA producer: Q once, then K tiles of 128 keys through a 3-stage ring
//   warp 2        TMA producer: V tiles through a 2-stage ring
//   warp 1        issues the tcgen05.mma of S = Q_t K^T (SMEM x SMEM)
//   warp 3        issues the tcgen05.mma of O_t += P_t V (TMEM x SMEM)
//   warps 4-7     softmax of tile 0: one thread per query row, whole row of S in registers
//   warps 8-11    softmax of tile 1
// TMEM (512 columns): S | P_0 | P_1 | O_0 | O_1.  A softmax warp takes a whole row of S into registers at
// once, so ONE S (128 f32 columns) serves both tiles in turn: it is free again 70 clocks after its QK^T,
// and the next QK^T -- the other tile's -- is issued while this tile is still being exponentiated.  P_t
// (16-bit, 64 columns each) has columns of its own.  A tile's next S is thus waiting when its softmax
// comes for it, and P.V is off the chain from one step to the next.  (With P_t over the front of S_t a
// tile's chain was softmax, P.V, QK^T: of 3180 clk per pair of steps the softmax warps waited 1360.)
// The exponent reference of a row is only taken from the first tile's true row maximum and moved when a
// later tile's maximum exceeds it by more than 2^6, so O is rescaled (a TMEM round trip) almost never.
// The epilogue writes O_t / l from registers straight to global memory.
#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cstdlib>
#include <type_traits>

#include "fast_div.cuh"
#include "kernels.h"
#include "sm100_ptx.cuh"

namespace asuka {
using namespace sm100;

namespace {

constexpr int kTile = 128;
constexpr uint32_t kTileBytes = 128 * 128 * 2;  // one [128 x 128] 16-bit tile = two swizzled halves
constexpr uint32_t kHalfBytes = kTileBytes / 2;
// How the query tiles and keys of a launch are cut into work items (each its own instantiation: what
// one mode needs per item costs the softmax warps of another registers they do not have).
//   kPair   two query tiles, each over all its keys; a K/V tile serves both
//   kSplit  two query tiles over a part of their keys; attn_merge_kernel combines the parts
//   kSolo   ONE query tile, its even key tiles on the first softmax slot and its odd ones on the second,
//           merged in the epilogue
enum FwdMode { kPair = 0, kSplit = 1, kSolo = 2 };
template <int kMode> struct Rings {
  static constexpr int kQTiles = kMode == kSolo ? 1 : 2;  // of an item
  static constexpr int kK = 3;  // K(j) is needed one iteration before V(j): give it the deeper ring
  static constexpr int kV = 2;
};
constexpr int kThreads = 384;
// Registers of the utility and of the softmax warps; what a block asks for must fit its 384 * 168 = 64512.
// The soft-capped one-tile mode has both ways of the tanh beside what its merge keeps: at 200 it spills 464
// bytes, at 216 156, at 224 112 (S4000, 8 heads 53.6 -> 51.9 us from 216 to 224, 52.5 at 232).  The others at 200 or 208:
// B1 H32 S1024 18.6 and 17.9; with split keys 128 rows over 16000, 16/4 heads, 44.3 and 45.1, soft-capped 1000 over 8000, 8/2
// heads, 50.7 and 51.4.
template <bool kCap, int kMode> struct Regs {
  static constexpr int kUtil = kCap && kMode == kSolo ? 56 : kMode == kSplit ? 96 : 88;
  static constexpr int kSoftmax = kCap && kMode == kSolo ? 224 : kMode == kSplit ? 200 : 208;
  static constexpr int kBlock = 128 * kUtil + 256 * kSoftmax;
  static_assert(kBlock <= kThreads * 168, "setmaxnreg would wait for ever");
};
constexpr uint32_t kSmemBytes = 7 * kTileBytes + 1024;
constexpr float kRescaleLimit = 6.0f;  // log2 of the largest exponential tolerated under a stale reference:
                                       // keeps a tile's row sum below 2^13, far from fp16's 65504

struct FwdParams {
  int B, H, Sq, Skv;
  int causal, diag_off;
  int nq_blocks, n_items;
  FastDiv by_units, by_heads, by_blocks, by_split;  // B * H, H, nq_blocks, B * H * parts: an item is decoded by every role
  int pair_far, nq_tiles;    // pair_far: an item is the query tiles i and nq_tiles - 1 - i (see decode_item)
  int unit_major;            // items are numbered unit by unit instead of heaviest block first
  int group;                 // query heads per key/value head (grouped-query attention)
  float scale_log2;          // softmax_scale * log2(e)
  float cap_in, cap_out;     // soft-capping: softmax_scale / cap and cap * log2(e)
  float* lse2;
  void* out;                 // [B, Sq, H, 128], 16-bit, strides in elements
  int64_t o_sb, o_ss, o_sh;
  int out_vec32;             // every output row starts on a 32-byte boundary: 256-bit stores
  uint32_t* status;
  // Key-range split, for launches with fewer work items than SMs can share evenly: the keys of
  // every item are dealt out to `parts` items of `ceil(n / parts)` key tiles each.  A query tile
  // served by more than one part leaves, per part, its unnormalised O (f32), its exponent
  // reference and its row sum in the workspace; attn_merge_kernel combines them in part order.
  int parts;
  float* part_o;             // [B*H, Sq, parts, 128]
  float* part_ml;            // [B*H, Sq, parts, 2]
};

struct Bars {
  uint64_t q_full[2], q_empty[2];
  uint64_t k_full[3], k_empty[3];
  uint64_t v_full[3], v_empty[3];
  uint64_t s_full[2], s_free, p_ready[2], pv_done[2], o_free[2];
};

__device__ __forceinline__ float ex2(float x) {
  float y;
  asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// 256-bit store: one instruction per 32-byte sector instead of two (the epilogue's stores go to 32
// different rows per warp instruction, so the number of instructions is what the LSU pays for)
__device__ __forceinline__ void st_global_v8(void* ptr, const uint32_t (&r)[8]) {
  asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(ptr), "r"(r[0]), "r"(r[1]),
               "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
               : "memory");
}

__device__ __forceinline__ float max3(float a, float b, float c) {
  float y;
  asm("max.f32 %0, %1, %2, %3;" : "=f"(y) : "f"(a), "f"(b), "f"(c));
  return y;
}

__device__ __forceinline__ float tanh_approx(float x) {
  float y;
  asm("tanh.approx.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// tanh(z / 2) for |z| < 2 on the FMA pipe, two at a time: z times a polynomial in z^2, fitted to the smallest
// relative error on that range (8.2e-5; tanh.approx has 4.9e-4).  The MUFU bounds the soft-capped kernel
// when it has both the tanh and the exponential of a logit: 8 clk each per warp and scheduler, against 6 of
// the FMA pipe for this.  Logits beyond the cap keep tanh.approx; a warp's tile that has one pays for both.
// bf16, 16/8 heads, calls back to back on a cool card: B1 S8192 367 us with tanh.approx for all, 294 with this
// for all, 417 with both; S1024 (two tiles per item, one, one) 25, 17.6, 22.  In the middle of other work, where
// the clock is lower, S8192 takes 366 and 340.
__device__ __forceinline__ float2 tanh_half2(float2 z) {
  const float2 y = __fmul2_rn(z, z);
  float2 p = make_float2(-0.000208044279133901f, -0.000208044279133901f);
  p = __ffma2_rn(p, y, make_float2(0.0037155484315007925f, 0.0037155484315007925f));
  p = __ffma2_rn(p, y, make_float2(-0.04133179038763046f, -0.04133179038763046f));
  p = __ffma2_rn(p, y, make_float2(0.4999592900276184f, 0.4999592900276184f));
  return __fmul2_rn(p, z);
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

template <bool kBF16>
__device__ __forceinline__ float2 unpack2(uint32_t w) {
  if constexpr (kBF16) {
    return __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&w));
  } else {
    return __half22float2(*reinterpret_cast<const __half2*>(&w));
  }
}

__device__ __forceinline__ void record_timeout(uint32_t* status, uint32_t site) {
  atomicAdd(&status[0], 1u);
  status[1] = site;
}

// number of 128-key tiles query tile [q0, q0+128) has to visit
__host__ __device__ __forceinline__ int kv_tiles_for(int q0, const FwdParams& p) {
  if (q0 >= p.Sq) return 0;
  int last = p.Skv - 1;
  if (p.causal) {
    const int qlast = q0 + kTile - 1 < p.Sq - 1 ? q0 + kTile - 1 : p.Sq - 1;
    last = last < qlast + p.diag_off ? last : qlast + p.diag_off;
  }
  return last / kTile + 1;
}


// One work item: 256 query rows of one (batch, head).
struct Item {
  int b, h;
  int q0[2];      // first row of each 128-row tile
  int j0;         // first key tile of this item (0 unless the keys are split)
  int n_kv[2];    // 128-key tiles each tile visits from j0 on (0: nothing for this tile in this item)
  int n_max;
  int part;       // which part of the key range this item is
  int nparts[2];  // parts that serve each tile (1: this item writes the tile's final result)
};

// Item `idx` of the launch; items are numbered heaviest first.
template <int kMode>
__device__ __forceinline__ void decode_item(int idx, const FwdParams& p, Item* item) {
  const int bh_count = p.B * p.H;
  if constexpr (kMode == kSolo) {
    const int i = p.by_units.div(idx), bh = idx - i * bh_count, b = p.by_heads.div(bh);
    const int q0 = (p.nq_tiles - 1 - i) * kTile, n = kv_tiles_for(q0, p);
    item->b = b;
    item->h = bh - b * p.H;
    item->q0[0] = item->q0[1] = q0;
    item->j0 = 0;
    item->n_kv[0] = (n + 1) / 2;
    item->n_kv[1] = n / 2;
    item->n_max = item->n_kv[0];
    item->part = 0;
    item->nparts[0] = item->nparts[1] = 1;
    return;
  }
  if constexpr (kMode == kPair) {
    // unit_major: the blocks of one (batch, head) follow each other, latest first, so that they
    // run at about the same time and K/V are in L2 for all but the first of them.  It is used
    // when K and V of the whole launch do not fit L2 (otherwise every wave of blocks would fetch
    // them from DRAM again).
    const int i = p.unit_major ? p.by_blocks.div(idx) : p.by_units.div(idx);
    const int bh = p.unit_major ? i : idx - i * bh_count;
    item->b = p.by_heads.div(bh);
    item->h = bh - item->b * p.H;
    if (p.unit_major) {
      const int qb = p.nq_blocks - 1 - (idx - i * p.nq_blocks);
      item->q0[0] = qb * 2 * kTile;
      item->q0[1] = qb * 2 * kTile + kTile;
    } else if (p.pair_far) {
      // A causal launch that fills at most one wave ends with its heaviest item, and items of
      // adjacent tiles grow with the block index.  Pairing tile i with tile nq_tiles - 1 - i makes
      // every item nq_tiles + 1 tile steps: the early tile shares the first key tiles with the
      // late one, which then runs on alone.
      const int far = p.nq_tiles - 1 - i;
      item->q0[0] = i * kTile;
      item->q0[1] = far > i ? far * kTile : p.Sq;  // (an odd count leaves the middle tile alone)
    } else {
      const int qb = p.nq_blocks - 1 - i;
      item->q0[0] = qb * 2 * kTile;
      item->q0[1] = qb * 2 * kTile + kTile;
    }
    item->j0 = 0;
    item->n_kv[0] = kv_tiles_for(item->q0[0], p);
    item->n_kv[1] = kv_tiles_for(item->q0[1], p);
    item->n_max = max(item->n_kv[0], item->n_kv[1]);
    item->part = 0;
    item->nparts[0] = item->nparts[1] = 1;
    return;
  }
  const int block = p.by_split.div(idx), rem = idx - block * bh_count * p.parts;
  const int qb = p.nq_blocks - 1 - block;
  item->part = p.by_units.div(rem);
  const int bh = rem - item->part * bh_count;
  item->b = p.by_heads.div(bh);
  item->h = bh - item->b * p.H;
  item->q0[0] = qb * 2 * kTile;
  item->q0[1] = qb * 2 * kTile + kTile;
  const int full0 = kv_tiles_for(item->q0[0], p), full1 = kv_tiles_for(item->q0[1], p);
  const int full = full0 > full1 ? full0 : full1;
  const int len = (full + p.parts - 1) / p.parts;  // key tiles per part (>= 1)
  item->j0 = item->part * len;
  const int r0 = full0 - item->j0 < len ? full0 - item->j0 : len;
  const int r1 = full1 - item->j0 < len ? full1 - item->j0 : len;
  item->n_kv[0] = r0 > 0 ? r0 : 0;
  item->n_kv[1] = r1 > 0 ? r1 : 0;
  item->n_max = item->n_kv[0] > item->n_kv[1] ? item->n_kv[0] : item->n_kv[1];
  item->nparts[0] = (full0 + len - 1) / len;
  item->nparts[1] = (full1 + len - 1) / len;
}

// The it-th item of this CTA: wave w of gridDim.x items is dealt out forwards when w is even and
// backwards when it is odd, which evens out the totals (at 32 heads and S = 4096 the busiest CTA
// gets 3 % more than the mean; assigning longest-first to the least-loaded CTA on the host would
// get within 2.5 %, the items being as coarse as they are, and was not worth a table).
template <int kMode>
__device__ __forceinline__ bool get_item(int it, const FwdParams& p, Item* item) {
  const int G = static_cast<int>(gridDim.x);
  const int r = static_cast<int>(blockIdx.x);
  const int idx = it * G + ((it & 1) ? G - 1 - r : r);
  if (idx >= p.n_items) return false;
  decode_item<kMode>(idx, p, item);
  return true;
}
// with an odd number of waves the last, backwards-dealt wave can skip a CTA that still has none
__device__ __forceinline__ int item_waves(const FwdParams& p) {
  return (p.n_items + static_cast<int>(gridDim.x) - 1) / static_cast<int>(gridDim.x);
}

// kCap: Gemma-2 style soft-capping, logits -> cap * tanh(logits / cap) before the mask
// (cases/kernels/gemma2.py:30-33; the reference emits tanh.approx.f32, to_triton.cpp:351-369, and so does
// this kernel for logits beyond the cap).
template <bool kBF16, bool kCap, int kMode>
__global__ void __launch_bounds__(kThreads, 1)
attn_fwd_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_v, const FwdParams p) {
  extern __shared__ uint8_t smem_raw[];
  constexpr int kKStages = Rings<kMode>::kK, kVStages = Rings<kMode>::kV;
  constexpr bool kOne = kMode == kSolo;  // one query tile, the two slots share its keys
  // Which roles take their first item as decoded during the set-up: kept over the fork into roles, an item makes some of
  // them spill it and reload its fields in their loops, and then decoding it again is cheaper; for the softmax warps that
  // is not in the way of the first loads.  All roles / issuers only / none, us: split keys, B1 H2 S4096 23.2 / 23.3 / 24.0, 128
  // rows over 16000 keys, 16/4 heads, 46.3 / 45.1 / 44.8; one tile per item, Keyformer B1 H4 S300 18.6 / 18.7 / 18.4 (where the
  // other kernels of a build lie moves such a figure by 0.1 to 0.4); two tiles, B1 H32 S1024 16.7 / - / 17.2.
  constexpr bool kKeepSoftmax = kMode == kPair;
  constexpr bool kKeepUtil = kMode == kPair || (kMode == kSplit && !kCap);
  __shared__ __align__(8) Bars bars;
  __shared__ float2 row_s[kOne ? kTile : 1];  // (kSolo) second slot's reference and row sum; then both slots' factors
  __shared__ uint32_t tmem_base_s;
  __shared__ uint32_t abort_s;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  const uint32_t sQ = smem_base;                          // an item's two tiles, or one tile each of two items
  const uint32_t sK = smem_base + 2 * kTileBytes;         // kKStages tiles
  const uint32_t sV = sK + kKStages * kTileBytes;         // kVStages tiles

  const int tid = threadIdx.x;
  const int warp = tid >> 5;
  const int lane = tid & 31;
  volatile uint32_t* abortp = &abort_s;
  const int n_waves = item_waves(p);

  if (tid == 0) {
    abort_s = 0;
    for (int i = 0; i < 2; ++i) {
      mbar_init(smem_u32(&bars.q_full[i]), 1);
      mbar_init(smem_u32(&bars.q_empty[i]), 1);
      mbar_init(smem_u32(&bars.s_full[i]), 1);
      mbar_init(smem_u32(&bars.p_ready[i]), 128);
      mbar_init(smem_u32(&bars.pv_done[i]), 1);
      mbar_init(smem_u32(&bars.o_free[i]), kOne ? 256 : 128);
    }
    mbar_init(smem_u32(&bars.s_free), 128);
    for (int i = 0; i < kKStages; ++i) {
      mbar_init(smem_u32(&bars.k_full[i]), 1);
      mbar_init(smem_u32(&bars.k_empty[i]), 1);
    }
    for (int i = 0; i < kVStages; ++i) {
      mbar_init(smem_u32(&bars.v_full[i]), 1);
      mbar_init(smem_u32(&bars.v_empty[i]), 1);
    }
    mbar_fence_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    tma_prefetch_desc(&map_v);
  }
  if (warp == 1) {
    __syncwarp();
    tmem_alloc(smem_u32(&tmem_base_s), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tbase = tmem_base_s;
  // The first item belongs to the set-up too, and so do its first tiles, on their way from DRAM to L2, in launches of 64
  // CTAs and more.  Without them and with them, us, inputs that are not in L2 / that are: 16 CTAs (B1 H4 S512) 9.00 and
  // 9.01 / 8.90 and 9.05, 48 (H6 S1024) 12.03 and 12.03 / 11.90 and 12.03, 64 (H8) 12.29 and 12.19 / 12.04 and 12.10, 96 (H12)
  // 12.79 and 12.60 / 12.26 and 12.28, 148 (H32) 18.01 and 17.52 / 16.95 and 16.95.  More tiles get in the way of the loads
  // behind (H2O B1 H4 S512, all of the first ring, 18.9 -> 19.2).
  Item it_;
  const bool has_first = get_item<kMode>(0, p, &it_);
  if (warp == 4 && lane == 0 && has_first && gridDim.x >= 64) {
    const int hk = it_.h / p.group, kv0 = (kMode == kSplit ? it_.j0 : 0) * kTile;
    for (int half = 0; half < 128; half += 64) {
      for (int t = 0; t < Rings<kMode>::kQTiles; ++t)
        if (it_.n_kv[t] > 0) tma_prefetch_4d(&map_q, half, it_.h, it_.q0[t], it_.b);
      tma_prefetch_4d(&map_k, half, hk, kv0, it_.b);
    }
  }
  // The set-up above may have run while the kernel ahead in the stream was still draining; q, k and
  // v may be that kernel's outputs and out / lse its inputs, so nothing is read or written before
  // it has finished.  The kernel behind this one (the column pass) may be scheduled from now on:
  // its CTAs come up on SMs whose forward CTA has retired and wait there for this grid's end.
  griddep_wait();
  griddep_launch_dependents();

  // Every role walks the same item list and keeps running counts (K tiles, V tiles, tile steps,
  // items per tile) from which ring stages and barrier parities follow; nothing is reset
  // between items.
  // 384 threads x 168 registers: the four utility warps hand most of theirs to the softmax warps
  if (warp == 0) {
    // ------------------------------------------------------------------ TMA producer: Q and K
    reg_dealloc<Regs<kCap, kMode>::kUtil>();
    if (lane == 0) {
      bool ok = true;
      uint32_t kc = 0;            // K tiles issued so far
      uint32_t qn[2] = {0, 0};    // items in which tile t was loaded so far (kSolo: loads of either buffer)
      uint32_t items = 0;
      for (int it = 0; it < n_waves && ok; ++it) {
        if (it == 0 && kKeepUtil ? !has_first : !get_item<kMode>(it, p, &it_)) continue;
        for (int x = 0; x < Rings<kMode>::kQTiles && ok; ++x) {
          if (it_.n_kv[x] == 0) continue;
          const int t = kOne ? static_cast<int>(items++ & 1) : x;
          if (qn[t] > 0) {  // the previous item's last QK^T of this tile must have read Q_t
            ok = mbar_wait(smem_u32(&bars.q_empty[t]), (qn[t] - 1) & 1, abortp);
            if (!ok) { record_timeout(p.status, 11); break; }
          }
          const uint32_t bar = smem_u32(&bars.q_full[t]);
          mbar_expect_tx(bar, kTileBytes);
          tma_load_4d(sQ + t * kTileBytes, &map_q, bar, 0, it_.h, it_.q0[x], it_.b);
          tma_load_4d(sQ + t * kTileBytes + kHalfBytes, &map_q, bar, 64, it_.h, it_.q0[x], it_.b);
          ++qn[t];
        }
        const int n_tiles = kOne ? it_.n_kv[0] + it_.n_kv[1] : it_.n_max;
        for (int j = 0; j < n_tiles && ok; ++j, ++kc) {
          const int st = kc % kKStages;
          const uint32_t use = kc / kKStages;
          if (use > 0) {
            ok = mbar_wait(smem_u32(&bars.k_empty[st]), (use - 1) & 1, abortp);
            if (!ok) { record_timeout(p.status, 1); break; }
          }
          const uint32_t bar = smem_u32(&bars.k_full[st]);
          mbar_expect_tx(bar, kTileBytes);
          tma_load_4d(sK + st * kTileBytes, &map_k, bar, 0, it_.h / p.group, ((kMode == kSplit ? it_.j0 : 0) + j) * kTile, it_.b);
          tma_load_4d(sK + st * kTileBytes + kHalfBytes, &map_k, bar, 64, it_.h / p.group, ((kMode == kSplit ? it_.j0 : 0) + j) * kTile, it_.b);
        }
      }
      if (!ok) {
        // give copies already in flight a bounded chance to land before the CTA retires
        volatile uint32_t none = 0;
        for (uint32_t c = kc > kKStages ? kc - kKStages : 0; c < kc; ++c)
          mbar_wait(smem_u32(&bars.k_full[c % kKStages]), (c / kKStages) & 1, &none);
      }
    }
  } else if (warp == 2) {
    // ------------------------------------------------------------------ TMA producer: V
    reg_dealloc<Regs<kCap, kMode>::kUtil>();
    if (lane == 0) {
      bool ok = true;
      uint32_t vc = 0;
      for (int it = 0; it < n_waves && ok; ++it) {
        if (it == 0 && kKeepUtil ? !has_first : !get_item<kMode>(it, p, &it_)) continue;
        const int n_tiles = kOne ? it_.n_kv[0] + it_.n_kv[1] : it_.n_max;
        for (int j = 0; j < n_tiles && ok; ++j, ++vc) {
          const int st = vc % kVStages;
          const uint32_t use = vc / kVStages;
          if (use > 0) {
            ok = mbar_wait(smem_u32(&bars.v_empty[st]), (use - 1) & 1, abortp);
            if (!ok) { record_timeout(p.status, 2); break; }
          }
          const uint32_t bar = smem_u32(&bars.v_full[st]);
          mbar_expect_tx(bar, kTileBytes);
          tma_load_4d(sV + st * kTileBytes, &map_v, bar, 0, it_.h / p.group, ((kMode == kSplit ? it_.j0 : 0) + j) * kTile, it_.b);
          tma_load_4d(sV + st * kTileBytes + kHalfBytes, &map_v, bar, 64, it_.h / p.group, ((kMode == kSplit ? it_.j0 : 0) + j) * kTile, it_.b);
        }
      }
      if (!ok) {
        volatile uint32_t none = 0;
        for (uint32_t c = vc > kVStages ? vc - kVStages : 0; c < vc; ++c)
          mbar_wait(smem_u32(&bars.v_full[c % kVStages]), (c / kVStages) & 1, &none);
      }
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ QK^T issuer
    // Step j of tile 0, step j of tile 1, step j + 1 of tile 0, ...: each is issued when the softmax warps
    // have the one before it in registers.  The whole warp walks the loop (addresses and descriptors stay
    // warp-uniform, waits are converged); one elected lane issues the tcgen05.mma / commit instructions.
    // Issuing eight MMAs takes as long as they run, and a wait on a barrier that is already complete still
    // costs 130 clk beside two busy softmax warps: P.V has an issuing warp of its own so that the two
    // cover for each other (from one warp a pair of steps took 4200 clk), and the barriers of a step are
    // probed together.
    reg_dealloc<Regs<kCap, kMode>::kUtil>();
    {
      constexpr uint32_t kFmt = kBF16 ? UMMA_BF16 : UMMA_F16;
      constexpr uint32_t idesc_qk = umma_idesc_f16(kFmt, UMMA_K_MAJOR, UMMA_K_MAJOR, 128, 128);
      auto wait_all = [&](uint64_t* bar, uint32_t parity, uint32_t site) -> bool {
        const bool good = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, abortp));
        if (!good && lane == 0) record_timeout(p.status, site);
        return good;
      };
      bool ok = true;
      uint32_t kc = 0;              // K tiles consumed before this item
      uint32_t x = 0;               // uses of S so far (parity of s_free)
      uint32_t on0 = 0, on1 = 0;    // items of either tile before this one (parity of q_full)
      for (int it = 0; it < n_waves && ok; ++it) {
        if (it == 0 && kKeepUtil ? !has_first : !get_item<kMode>(it, p, &it_)) continue;
        const int n0 = it_.n_kv[0], n1 = it_.n_kv[1];
        for (int j = 0; j < it_.n_max && ok; ++j) {
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (j >= (t ? n1 : n0)) continue;
            const uint32_t kidx = kc + (kOne ? 2 * j + t : j);
            const int st = kidx % kKStages;
            const bool k_hit = mbar_try_wait(smem_u32(&bars.k_full[st]), (kidx / kKStages) & 1);
            const bool s_hit = x == 0 || mbar_try_wait(smem_u32(&bars.s_free), (x - 1) & 1);
            if (j == 0 && !kOne) ok = wait_all(&bars.q_full[t], (t ? on1 : on0) & 1, 3);
            if (j == 0 && kOne && t == 0) ok = wait_all(&bars.q_full[on0 & 1], (on0 >> 1) & 1, 3);
            if (ok && !__all_sync(0xffffffffu, k_hit)) ok = wait_all(&bars.k_full[st], (kidx / kKStages) & 1, 4);
            if (ok && !__all_sync(0xffffffffu, s_hit)) ok = wait_all(&bars.s_free, (x - 1) & 1, 13);
            if (!ok) break;
            ++x;
            tc_fence_after_sync();
            if (elect_one()) {
              const uint64_t kdesc = umma_smem_desc_sw128(sK + st * kTileBytes, 16, 1024);
              const uint64_t qdesc = umma_smem_desc_sw128(sQ + (kOne ? (on0 & 1) : t) * kTileBytes, 16, 1024);
#pragma unroll
              for (int kk = 0; kk < 8; ++kk) {
                const uint64_t off = static_cast<uint64_t>((kk & 3) * 2 + (kk >> 2) * (kHalfBytes >> 4));
                umma_ss(tbase, qdesc + off, kdesc + off, idesc_qk, kk > 0 ? 1u : 0u);
              }
              umma_commit(smem_u32(&bars.s_full[t]));
              // the K stage is free after the last QK^T that reads it; Q_t after its last QK^T
              if (kOne || t == 1 || j >= n1) umma_commit(smem_u32(&bars.k_empty[st]));
              if (kOne) {
                if (2 * j + t == n0 + n1 - 1) umma_commit(smem_u32(&bars.q_empty[on0 & 1]));
              } else if (j == (t ? n1 : n0) - 1) {
                umma_commit(smem_u32(&bars.q_empty[t]));
              }
            }
            __syncwarp();
          }
        }
        kc += kOne ? n0 + n1 : it_.n_max;
        if (n0 > 0) ++on0;
        if (n1 > 0) ++on1;
      }
    }
  } else if (warp == 3) {
    // ------------------------------------------------------------------ P.V issuer
    reg_dealloc<Regs<kCap, kMode>::kUtil>();
    {
      constexpr uint32_t kFmt = kBF16 ? UMMA_BF16 : UMMA_F16;
      constexpr uint32_t idesc_pv = umma_idesc_f16(kFmt, UMMA_K_MAJOR, UMMA_MN_MAJOR, 128, 128);
      auto wait_all = [&](uint64_t* bar, uint32_t parity, uint32_t site) -> bool {
        const bool good = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, abortp));
        if (!good && lane == 0) record_timeout(p.status, site);
        return good;
      };
      bool ok = true;
      uint32_t vc = 0;              // V tiles consumed before this item
      uint32_t sn0 = 0, sn1 = 0;    // steps of either tile before this item (parity of p_ready)
      uint32_t on0 = 0, on1 = 0;    // items of either tile before this one (parity of o_free)
      for (int it = 0; it < n_waves && ok; ++it) {
        if (it == 0 && kKeepUtil ? !has_first : !get_item<kMode>(it, p, &it_)) continue;
        const int n0 = it_.n_kv[0], n1 = it_.n_kv[1];
        for (int j = 0; j < it_.n_max && ok; ++j) {
#pragma unroll
          for (int t = 0; t < 2; ++t) {
            if (j >= (t ? n1 : n0)) continue;
            const uint32_t vidx = vc + (kOne ? 2 * j + t : j);
            const int st = vidx % kVStages;
            const uint32_t on = t ? on1 : on0, pn = (t ? sn1 : sn0) + j;
            ok = wait_all(&bars.v_full[st], (vidx / kVStages) & 1, 5);
            // the first P.V of an item overwrites O_t: the previous item's epilogue must have read it
            if (ok && j == 0 && on > 0) ok = wait_all(&bars.o_free[t], (on - 1) & 1, 12);
            if (ok) ok = wait_all(&bars.p_ready[t], pn & 1, 6);
            if (!ok) break;
            tc_fence_after_sync();
            if (elect_one()) {
              const uint64_t vdesc = umma_smem_desc_sw128(sV + st * kTileBytes, kHalfBytes, 1024);
              const uint32_t tP = tbase + 128 + t * 64, tO = tbase + 256 + t * 128;
#pragma unroll
              for (int kk = 0; kk < 8; ++kk) {
                umma_ts(tO, tP + kk * 8, vdesc + static_cast<uint64_t>(kk * (2048 >> 4)), idesc_pv,
                        (j > 0 || kk > 0) ? 1u : 0u);
              }
              umma_commit(smem_u32(&bars.pv_done[t]));
              // the V stage is free after the last P.V that reads it
              if (kOne || t == 1 || j >= n1) umma_commit(smem_u32(&bars.v_empty[st]));
            }
            __syncwarp();
          }
        }
        vc += kOne ? n0 + n1 : it_.n_max;
        sn0 += n0;
        sn1 += n1;
        if (n0 > 0) ++on0;
        if (n1 > 0) ++on1;
      }
    }
  } else {
    // ------------------------------------------------------------------ softmax + epilogue
    reg_alloc<Regs<kCap, kMode>::kSoftmax>();
    const int t = (warp - 4) >> 2;
    const int wq = warp & 3;                     // TMEM lane quarter this warp may touch
    const int r_in_tile = wq * 32 + lane;
    const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
    const uint32_t tS = tbase + lane_base;
    const uint32_t tP = tbase + lane_base + 128 + t * 64;
    const uint32_t tO = tbase + lane_base + 256 + t * 128;
    const float mul = kCap ? p.cap_out : p.scale_log2;
    bool ok = true;
    uint32_t sn = 0;  // tile steps of this tile before the current item
    for (int it = 0; it < n_waves && (ok || kOne); ++it) {
      if (it == 0 && kKeepSoftmax ? !has_first : !get_item<kMode>(it, p, &it_)) continue;
      const int n_t = it_.n_kv[t];
      if (n_t == 0 && !kOne) continue;
      const int row = it_.q0[t] + r_in_tile;
      int lim = p.Skv - 1;
      if (p.causal) lim = min(lim, row + p.diag_off);
      const int tile_min_lim = p.causal ? min(p.Skv - 1, it_.q0[t] + p.diag_off) : p.Skv - 1;

      float m_ref = -INFINITY;             // exponent reference of this row, in log2 units of the scaled logit
      float l = 0.f;                       // row sum under the current reference

      for (int j = 0; j < n_t && ok; ++j) {
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.s_full[t]), (sn + j) & 1, abortp));
        if (!ok) { if (lane == 0) record_timeout(p.status, 7); break; }
        tc_fence_after_sync();
        const int jk = (kOne ? 2 * j + t : (kMode == kSplit ? it_.j0 : 0) + j) * kTile;  // first key of this tile
        const bool masked_tile = jk + kTile - 1 > tile_min_lim;
        const int thr = lim - jk;  // columns > thr of this tile are masked for this row

        // The whole 128-wide row goes to registers at once, and S to the next QK^T.
        float e[128];
        {
          uint32_t(&u)[128] = *reinterpret_cast<uint32_t(*)[128]>(e);
          tmem_ld32(tS + 0, *reinterpret_cast<uint32_t(*)[32]>(&u[0]));
          tmem_ld32(tS + 32, *reinterpret_cast<uint32_t(*)[32]>(&u[32]));
          tmem_ld32(tS + 64, *reinterpret_cast<uint32_t(*)[32]>(&u[64]));
          tmem_ld32(tS + 96, *reinterpret_cast<uint32_t(*)[32]>(&u[96]));
          tmem_wait_ld();
        }
        tc_fence_before_sync();
        mbar_arrive(smem_u32(&bars.s_free));
        if constexpr (kCap) {
          // cap first, mask afterwards (the reference adds the mask to the capped logits)
          const float2 in2 = make_float2(2.f * p.cap_in, 2.f * p.cap_in);
          uint32_t big = 0;
#pragma unroll
          for (int i = 0; i < 64; ++i) {
            const float2 z = __fmul2_rn(make_float2(e[2 * i], e[2 * i + 1]), in2);
            e[2 * i] = z.x;
            e[2 * i + 1] = z.y;
            big |= __float_as_uint(z.x) | __float_as_uint(z.y);
          }
          if (__any_sync(0xffffffffu, (big & 0x40000000u) != 0)) {
            // (bit 30: some logit of the warp's rows is as large as the cap, infinite or NaN; the others are
            // treated as below, so that what a logit becomes depends on no other row and no masked key)
#pragma unroll
            for (int i = 0; i < 64; ++i) {
              const float2 z = make_float2(e[2 * i], e[2 * i + 1]);
              const float2 t = tanh_half2(z);
              e[2 * i] = fabsf(z.x) < 2.f ? t.x : tanh_approx(0.5f * z.x);
              e[2 * i + 1] = fabsf(z.y) < 2.f ? t.y : tanh_approx(0.5f * z.y);
            }
          } else {
#pragma unroll
            for (int i = 0; i < 64; ++i) {
              const float2 t = tanh_half2(make_float2(e[2 * i], e[2 * i + 1]));
              e[2 * i] = t.x;
              e[2 * i + 1] = t.y;
            }
          }
        }
        if (masked_tile) {
#pragma unroll
          for (int i = 0; i < 128; ++i) e[i] = (i > thr) ? -INFINITY : e[i];
        }
        // The tile's row maximum is the reference of a first tile; a later one only moves the reference up
        // (and rescales what was accumulated under the old one) when it exceeds it by too much.
        float mx4[4] = {-INFINITY, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int i = 0; i < 128; i += 8) {
          mx4[0] = max3(mx4[0], e[i], e[i + 1]);
          mx4[1] = max3(mx4[1], e[i + 2], e[i + 3]);
          mx4[2] = max3(mx4[2], e[i + 4], e[i + 5]);
          mx4[3] = max3(mx4[3], e[i + 6], e[i + 7]);
        }
        const float mx = fmaxf(fmaxf(mx4[0], mx4[1]), fmaxf(mx4[2], mx4[3])) * mul;
        if (j == 0) {
          m_ref = mx > -INFINITY ? mx : 0.f;
        } else {
          const bool need = mx > m_ref + kRescaleLimit;
          if (__any_sync(0xffffffffu, need)) {
            float alpha = 1.f;
            if (need) {
              alpha = ex2(m_ref - mx);
              m_ref = mx;
              l *= alpha;
            }
            // O_t is the sum over earlier tiles of this item, complete with their last P.V
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.pv_done[t]), (sn + j - 1) & 1, abortp));
            if (!ok) { if (lane == 0) record_timeout(p.status, 8); break; }
            tc_fence_after_sync();
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              uint32_t o[16];
              tmem_ld16(tO + c * 16, o);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 16; ++i) o[i] = __float_as_uint(__uint_as_float(o[i]) * alpha);
              tmem_st16(tO + c * 16, o);
            }
            tmem_wait_st();
          }
        }
        // two logits per FMA instruction (packed f32x2); P is packed to 16 bits right away (the compiler
        // interleaves it with the exponentials)
        const float2 mul2 = make_float2(mul, mul), neg_m2 = make_float2(-m_ref, -m_ref);
        float2 ts4[4] = {make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f), make_float2(0.f, 0.f)};
        uint32_t pk[64];
#pragma unroll
        for (int i = 0; i < 64; ++i) {
          float2 v = __ffma2_rn(make_float2(e[2 * i], e[2 * i + 1]), mul2, neg_m2);
          v.x = ex2(v.x);
          v.y = ex2(v.y);
          ts4[i & 3] = __fadd2_rn(ts4[i & 3], v);
          pk[i] = pack2<kBF16>(v.x, v.y);
        }
        const float2 ts2 = __fadd2_rn(__fadd2_rn(ts4[0], ts4[1]), __fadd2_rn(ts4[2], ts4[3]));
        l += ts2.x + ts2.y;
        if (j > 0) {  // P_t is free when the last P.V has read it (a new item: its epilogue has waited for that)
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.pv_done[t]), (sn + j - 1) & 1, abortp));
          if (!ok) { if (lane == 0) record_timeout(p.status, 8); break; }
          tc_fence_after_sync();
        }
        tmem_st32(tP, *reinterpret_cast<uint32_t(*)[32]>(&pk[0]));
        tmem_st32(tP + 32, *reinterpret_cast<uint32_t(*)[32]>(&pk[32]));
        tmem_wait_st();
        tc_fence_before_sync();
        mbar_arrive(smem_u32(&bars.p_ready[t]));
      }
      if constexpr (kOne) {
        // ---- epilogue of a one-tile item: the first slot gets the second's exponent reference and row sum
        // and hands back the factors of both accumulators; each slot writes half of the output columns
        if (n_t > 0 && ok) {
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.pv_done[t]), (sn + n_t - 1) & 1, abortp));
          if (!ok && lane == 0) record_timeout(p.status, 9);
          tc_fence_after_sync();
        }
        // (every softmax warp gets to the barriers for every item, expired waits or not)
        float f0, f1;
        if (t == 1) row_s[r_in_tile] = make_float2(l > 0.f ? m_ref : -INFINITY, l);
        tc_fence_before_sync();
        named_bar_sync(1, 256);
        if (t == 0) {
          const float2 c = row_s[r_in_tile];
          const float m0 = l > 0.f ? m_ref : -INFINITY;
          const float mm = fmaxf(m0, c.x);
          const float w0 = l > 0.f ? ex2(m0 - mm) : 0.f, w1 = c.y > 0.f ? ex2(c.x - mm) : 0.f;
          const float lsum = l * w0 + c.y * w1;
          f0 = w0 / lsum;
          f1 = w1 / lsum;
          row_s[r_in_tile] = make_float2(f0, f1);
          if (p.lse2 != nullptr && row < p.Sq)
            p.lse2[(static_cast<size_t>(it_.b) * p.H + it_.h) * p.Sq + row] = mm + log2f(lsum);
        }
        named_bar_sync(1, 256);
        tc_fence_after_sync();
        if (t == 1) {
          f0 = row_s[r_in_tile].x;
          f1 = row_s[r_in_tile].y;
        }
        const bool both = it_.n_kv[1] > 0;
        uint16_t* orow = static_cast<uint16_t*>(p.out) + static_cast<int64_t>(it_.b) * p.o_sb +
                         static_cast<int64_t>(row) * p.o_ss + static_cast<int64_t>(it_.h) * p.o_sh + t * 64;
        const uint32_t tA = tbase + lane_base + 256 + t * 64;
#pragma unroll
        for (int c4 = 0; c4 < 2; ++c4) {
          uint32_t o0[32], o1[32];
          tmem_ld32(tA + c4 * 32, o0);
          if (both) tmem_ld32(tA + 128 + c4 * 32, o1);
          tmem_wait_ld();
          if (c4 == 1) {
            // both accumulators are in registers: the next item's first P.V may overwrite them
            tc_fence_before_sync();
            mbar_arrive(smem_u32(&bars.o_free[0]));
            if (both) mbar_arrive(smem_u32(&bars.o_free[1]));
          }
          uint32_t w[16];
#pragma unroll
          for (int g = 0; g < 16; ++g) {
            float x = __uint_as_float(o0[2 * g]) * f0, y = __uint_as_float(o0[2 * g + 1]) * f0;
            if (both) {
              x = fmaf(__uint_as_float(o1[2 * g]), f1, x);
              y = fmaf(__uint_as_float(o1[2 * g + 1]), f1, y);
            }
            w[g] = pack2<kBF16>(x, y);
          }
          if (row < p.Sq) {
            if (p.out_vec32) {
              st_global_v8(orow + c4 * 32, *reinterpret_cast<const uint32_t(*)[8]>(&w[0]));
              st_global_v8(orow + c4 * 32 + 16, *reinterpret_cast<const uint32_t(*)[8]>(&w[8]));
            } else {
#pragma unroll
              for (int g = 0; g < 4; ++g)
                *reinterpret_cast<uint4*>(orow + c4 * 32 + g * 8) = make_uint4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]);
            }
          }
        }
        sn += n_t;
        continue;
      }
      if (!ok) break;

      // ---- epilogue of the item: O_t / l straight from TMEM to global memory
      ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.pv_done[t]), (sn + n_t - 1) & 1, abortp));
      if (!ok) { if (lane == 0) record_timeout(p.status, 9); break; }
      tc_fence_after_sync();
      if (kMode == kSplit && it_.nparts[t] > 1) {
        // this tile's keys are shared with other items: leave the unnormalised O, the exponent
        // reference and the row sum for the merge (a row that saw no key in this part has l = 0
        // and must not set the scale: its reference goes out as -inf)
        const size_t prow = ((static_cast<size_t>(it_.b) * p.H + it_.h) * p.Sq + row) * p.parts + it_.part;
        float* orow = p.part_o + prow * 128;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + c * 32, o);
          tmem_wait_ld();
          if (c == 3) {
            tc_fence_before_sync();
            mbar_arrive(smem_u32(&bars.o_free[t]));
          }
          if (row < p.Sq) {
#pragma unroll
            for (int g = 0; g < 4; ++g) {
              const uint32_t w[8] = {o[g * 8], o[g * 8 + 1], o[g * 8 + 2], o[g * 8 + 3],
                                     o[g * 8 + 4], o[g * 8 + 5], o[g * 8 + 6], o[g * 8 + 7]};
              st_global_v8(orow + c * 32 + g * 8, w);  // (the workspace rows are 512-byte aligned)
            }
          }
        }
        if (row < p.Sq)
          *reinterpret_cast<float2*>(p.part_ml + prow * 2) = make_float2(l > 0.f ? m_ref : -INFINITY, l);
      } else {
        const float inv_l = 1.f / l;
        uint16_t* orow = static_cast<uint16_t*>(p.out) + static_cast<int64_t>(it_.b) * p.o_sb +
                         static_cast<int64_t>(row) * p.o_ss + static_cast<int64_t>(it_.h) * p.o_sh;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          uint32_t o[32];
          tmem_ld32(tO + c * 32, o);
          tmem_wait_ld();
          if (c == 3) {
            // O_t is in registers: the next item's first P.V may overwrite it
            tc_fence_before_sync();
            mbar_arrive(smem_u32(&bars.o_free[t]));
          }
          if (row < p.Sq) {
            uint32_t w[16];
#pragma unroll
            for (int g = 0; g < 16; ++g)
              w[g] = pack2<kBF16>(__uint_as_float(o[2 * g]) * inv_l, __uint_as_float(o[2 * g + 1]) * inv_l);
            if (p.out_vec32) {
              st_global_v8(orow + c * 32, *reinterpret_cast<const uint32_t(*)[8]>(&w[0]));
              st_global_v8(orow + c * 32 + 16, *reinterpret_cast<const uint32_t(*)[8]>(&w[8]));
            } else {
#pragma unroll
              for (int g = 0; g < 4; ++g)
                *reinterpret_cast<uint4*>(orow + c * 32 + g * 8) = make_uint4(w[4 * g], w[4 * g + 1], w[4 * g + 2], w[4 * g + 3]);
            }
          }
        }
        if (p.lse2 != nullptr && row < p.Sq) {
          p.lse2[(static_cast<size_t>(it_.b) * p.H + it_.h) * p.Sq + row] = m_ref + log2f(l);
        }
      }
      sn += n_t;
    }
  }

  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tbase, 512);
  }
}

// Combines the parts of a key-range split.  A warp takes four query rows, lane = four output
// columns: every part's reference, row sum and 512-byte O row are read (they were written moments
// ago and sit in L2) with all loads of the four rows in flight at once -- the kernel is bound by
// that latency, not by the bytes -- scaled to the common reference and added in part order, so the
// result does not depend on which part finished first.
constexpr int kMaxParts = 4;
constexpr int kMergeWarps = 8;
constexpr int kMergeRowsPerWarp = 4;
constexpr int kMergeRows = kMergeWarps * kMergeRowsPerWarp;  // rows per CTA (divides the tile height)
template <bool kBF16>
__global__ void __launch_bounds__(kMergeWarps * 32) attn_merge_kernel(const FwdParams p) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int bh_count = p.B * p.H;
  const int rb = static_cast<int>(blockIdx.x) / bh_count;  // block of kMergeRows query rows
  const int bh = static_cast<int>(blockIdx.x) % bh_count;
  const int b = bh / p.H, h = bh % p.H;
  const int row0 = rb * kMergeRows + warp * kMergeRowsPerWarp;
  const int q0 = (row0 / kTile) * kTile;
  // the same arithmetic as decode_item: the parts of the 256-row block these rows' tile belongs to
  const int qa = (row0 / (2 * kTile)) * 2 * kTile;
  const int len = (max(kv_tiles_for(qa, p), kv_tiles_for(qa + kTile, p)) + p.parts - 1) / p.parts;
  const int nparts = (kv_tiles_for(q0, p) + len - 1) / len;
  griddep_wait();               // the parts are the output of the kernel ahead
  griddep_launch_dependents();
  if (nparts <= 1) return;      // (one part: the forward kernel wrote the result itself)
  float2 ml[kMergeRowsPerWarp][kMaxParts];
  float4 o[kMergeRowsPerWarp][kMaxParts];
#pragma unroll
  for (int r = 0; r < kMergeRowsPerWarp; ++r) {
    const size_t prow = (static_cast<size_t>(bh) * p.Sq + min(row0 + r, p.Sq - 1)) * p.parts;
#pragma unroll
    for (int q = 0; q < kMaxParts; ++q) {
      if (q < nparts) {
        ml[r][q] = *reinterpret_cast<const float2*>(p.part_ml + (prow + q) * 2);
        o[r][q] = *reinterpret_cast<const float4*>(p.part_o + (prow + q) * 128 + lane * 4);
      }
    }
  }
#pragma unroll
  for (int r = 0; r < kMergeRowsPerWarp; ++r) {
    const int row = row0 + r;
    if (row >= p.Sq) break;
    float m = -INFINITY;
#pragma unroll
    for (int q = 0; q < kMaxParts; ++q)
      if (q < nparts) m = fmaxf(m, ml[r][q].x);
    float l = 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int q = 0; q < kMaxParts; ++q) {
      if (q < nparts) {
        const float w = ml[r][q].x > -INFINITY ? ex2(ml[r][q].x - m) : 0.f;
        l = fmaf(w, ml[r][q].y, l);
        acc.x = fmaf(w, o[r][q].x, acc.x);
        acc.y = fmaf(w, o[r][q].y, acc.y);
        acc.z = fmaf(w, o[r][q].z, acc.z);
        acc.w = fmaf(w, o[r][q].w, acc.w);
      }
    }
    const float inv_l = 1.f / l;
    uint16_t* orow = static_cast<uint16_t*>(p.out) + static_cast<int64_t>(b) * p.o_sb +
                     static_cast<int64_t>(row) * p.o_ss + static_cast<int64_t>(h) * p.o_sh;
    uint2 v;
    v.x = pack2<kBF16>(acc.x * inv_l, acc.y * inv_l);
    v.y = pack2<kBF16>(acc.z * inv_l, acc.w * inv_l);
    *reinterpret_cast<uint2*>(orow + lane * 4) = v;
    if (p.lse2 != nullptr && lane == 0) p.lse2[static_cast<size_t>(bh) * p.Sq + row] = m + log2f(l);
  }
}

}  // namespace

// How many parts the key range of every two-tile item is cut into (kSplit).  Partial results cost about as
// much L2 traffic again as the inputs and the merge is a launch of its own, so this is only for launches
// whose query tiles would leave half of the SMs idle even at one tile per CTA, and long key ranges (S 4096,
// 2 heads: 30.9 us with one tile per CTA, 25.5 split; 100 rows over 9000 keys, 16/4 heads 58 and 30; at 1.7
// tiles per SM S 4096, 8 heads 35 and 66); it needs workspace.
int attn_fwd_parts(const AttnShape& s, int num_sms, size_t ws_bytes) {
  if (attn_decode_applies(s)) return 1;  // (attn_decode.cu splits the keys itself)
  const long long n_tiles = static_cast<long long>((s.Sq + kTile - 1) / kTile) * s.B * s.H;
  const int max_tiles = (s.Skv + kTile - 1) / kTile;
  int parts = 1;
#ifdef ASUKA_TUNE_ENV
  if (const char* e = getenv("ASUKA_FWD_PARTS")) {
    parts = atoi(e);
    while (parts > 1 && attn_fwd_split_bytes(s, parts) > ws_bytes) parts /= 2;
    return parts;
  }
#endif
  if (2 * n_tiles <= num_sms && max_tiles >= 32) parts = 4;
  while (parts > 1 && attn_fwd_split_bytes(s, parts) > ws_bytes) parts /= 2;
  return parts;
}

// One query tile per item (kSolo).  Two tiles of an item keep the tensor pipe and the MUFU busy as long as
// both have keys left, and share every K/V tile; but an item is then as long as its later tile.  One tile
// whose keys the two slots share is done in half the rounds, at twice the K/V traffic per step.  So (us, two
// tiles per item -> one):
//   - one tile per SM or fewer, three or more key tiles: always.  500 rows over 5003 keys, 32/8 heads
//     71 -> 44; S 1024, 8 heads 16.3 -> 12.6; S 512, 4 heads 11.2 -> 9.4; unmasked S 2048, 8 heads 29.7 -> 20.4
//   - with more, if the launch is a causal square, up to a number that grows with its length: the late tiles
//     are twice as long as the mean, the early ones fill in behind them, and the finer they are the better.
//     Two -> one: S 600, 32 heads (1.1 tiles per SM) 13.3 -> 12.9; S 700, 30 heads (1.2) 14.5 -> 14.2, 32 heads (1.3)
//     14.8 -> 15.0; S 1024, 25 heads (1.4) 17.4 -> 16.6, 28 heads (1.5) 17.6 -> 18.0; S 1500, 22 heads (1.8) 21.7 -> 21.5,
//     24 heads (1.9) 21.9 -> 22.2; S 2048, 20 heads (2.2) 31.5 -> 29.9, 22 heads (2.4) 31.6 -> 32.3; S 4096, 11 heads
//     (2.4) 54.3 -> 49.4; S 8000, 6 heads (2.6) 97 -> 91; beyond it S 8192, 8 heads (3.5) 112 -> 126; and not square,
//     1024 rows over 8000 keys, 32/8 heads (1.7) 108 -> 118
static bool attn_fwd_solo(const AttnShape& s, int num_sms) {
#ifdef ASUKA_TUNE_ENV
  if (const char* e = getenv("ASUKA_FWD_SOLO")) return atoi(e) != 0;
#endif
  const int nq_tiles = (s.Sq + kTile - 1) / kTile;
  const long long n_tiles = static_cast<long long>(nq_tiles) * s.B * s.H;
  if (n_tiles <= num_sms) return s.Skv > 2 * kTile;
  const int length = nq_tiles < 10 ? nq_tiles + 4 : nq_tiles < 16 ? nq_tiles + 3 : nq_tiles < 32 ? 19 : 20;
  return s.causal && 4LL * s.Skv <= 5LL * s.Sq && 8 * n_tiles <= static_cast<long long>(num_sms) * length;
}

size_t attn_fwd_split_bytes(const AttnShape& s, int parts) {
  if (parts <= 1) return 0;
  const size_t rows = static_cast<size_t>(s.B) * s.H * s.Sq;
  return rows * parts * (128 + 2) * sizeof(float);
}

cudaError_t launch_attn_fwd(const CUtensorMap& mq, const CUtensorMap& mk, const CUtensorMap& mv,
                            void* out, int64_t o_sb, int64_t o_ss, int64_t o_sh, float* lse2,
                            const AttnShape& s, int num_sms, void* split_ws, int parts, cudaStream_t stream) {
  FwdParams p;
  p.B = s.B;
  p.H = s.H;
  p.Sq = s.Sq;
  p.Skv = s.Skv;
  p.causal = s.causal;
  p.diag_off = s.Skv - s.Sq;
  p.nq_blocks = (s.Sq + 2 * kTile - 1) / (2 * kTile);
  p.parts = parts > 1 && split_ws != nullptr ? (parts < kMaxParts ? parts : kMaxParts) : 1;
  p.nq_tiles = (s.Sq + kTile - 1) / kTile;
  const bool solo = p.parts == 1 && attn_fwd_solo(s, num_sms);
  p.n_items = solo ? p.nq_tiles * s.B * s.H : p.nq_blocks * s.B * s.H * p.parts;
  {
    const double kv_bytes = 2.0 * s.B * (s.H / (s.group > 0 ? s.group : 1)) * static_cast<double>(s.Skv) * 128 * 2;
    p.unit_major = (p.parts == 1 && p.n_items > num_sms && kv_bytes > 96e6) ? 1 : 0;
  }
  const long long x_max = p.n_items;
  p.by_units = fast_div(s.B * s.H, x_max);
  p.by_heads = fast_div(s.H, s.B * s.H);
  p.by_blocks = fast_div(p.nq_blocks, x_max);
  p.by_split = fast_div(s.B * s.H * p.parts, x_max);
  p.pair_far = (p.parts == 1 && !solo && s.causal && p.n_items <= num_sms && p.nq_tiles >= 4) ? 1 : 0;
  p.group = s.group;
  p.scale_log2 = s.softmax_scale * 1.4426950408889634f;
  p.cap_in = s.softcap > 0.f ? s.softmax_scale / s.softcap : 0.f;
  p.cap_out = s.softcap * 1.4426950408889634f;
  p.lse2 = lse2;
  p.out = out;
  p.o_sb = o_sb;
  p.o_ss = o_ss;
  p.o_sh = o_sh;
  p.out_vec32 = (reinterpret_cast<uintptr_t>(out) % 32 == 0 && o_sb % 16 == 0 && o_ss % 16 == 0 && o_sh % 16 == 0) ? 1 : 0;
  p.status = device_status_words();
  p.part_o = static_cast<float*>(split_ws);
  p.part_ml = p.part_o + static_cast<size_t>(s.B) * s.H * s.Sq * p.parts * 128;
  const dim3 grid(static_cast<unsigned>(p.n_items < num_sms ? p.n_items : num_sms));
  auto pick = [&](auto mode) -> void (*)(CUtensorMap, CUtensorMap, CUtensorMap, FwdParams) {
    constexpr int kMode = decltype(mode)::value;
    if (s.softcap > 0.f) return s.bf16 ? attn_fwd_kernel<true, true, kMode> : attn_fwd_kernel<false, true, kMode>;
    return s.bf16 ? attn_fwd_kernel<true, false, kMode> : attn_fwd_kernel<false, false, kMode>;
  };
  const auto kern = p.parts > 1 ? pick(std::integral_constant<int, kSplit>())
                    : solo      ? pick(std::integral_constant<int, kSolo>())
                                : pick(std::integral_constant<int, kPair>());
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), kSmemBytes);
  if (e != cudaSuccess) return e;
  e = check_register_budget(reinterpret_cast<const void*>(kern), kThreads,
                            s.softcap > 0.f && solo ? Regs<true, kSolo>::kBlock : Regs<false, kPair>::kBlock);
  if (e != cudaSuccess) return e;
  e = launch_dependent(kern, grid, dim3(kThreads), kSmemBytes, stream, mq, mk, mv, p);
  count_launch();
  if (e != cudaSuccess || p.parts == 1) return e;
  const dim3 mgrid(static_cast<unsigned>((s.Sq + kMergeRows - 1) / kMergeRows) * s.B * s.H);
  e = launch_dependent(s.bf16 ? attn_merge_kernel<true> : attn_merge_kernel<false>, mgrid, dim3(kMergeWarps * 32), 0,
                       stream, p);
  count_launch();
  return e;
}

}  // namespace asuka
