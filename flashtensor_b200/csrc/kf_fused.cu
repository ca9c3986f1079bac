// Keyformer's score in one pass over the noise, for sm_100a:
//   kf_score = softmax((scores + g) / tau).sum(dim=2)   (cases/kernels/kf.py:36-40)
// A column's sum needs every row's denominator first, and a row's denominator all of its keys.  Taken as two
// passes (kf_rowstat_kernel, then kf_col_tma_kernel or col_scores_kernel) the noise is read, or generated, and
// its logarithms and exponentials are computed twice.  Here the exponentials of 128 query rows stay on the chip
// until their denominators are known: a cluster of CTAs shares the keys of a row, every CTA keeps its tiles
// [128 queries x 128 keys] as f32 in its tensor memory (four of them), the CTAs exchange each row's partial
// (maximum, sum) through distributed shared memory, and a second look at the tiles in tensor memory, one
// multiplication and one addition per logit, adds them up by key.
//
//   warp 0      (noise operand) TMA producer of the noise boxes [128 rows x 32 keys] f32; where TMA cannot describe the
//               operand, teller of addresses to the key warps, which copy their own shares four bytes a lane
//   warp 1      Q and K loads and the tcgen05.mma issue: S = Q K_t^T into one of four TMEM buffers
//   warps 2-3   the rows' statistics: over the four warps of a row, over the CTAs of the cluster
//   warps 4-19  four per 32 query rows, each with 32 of the 128 columns of every tile
//       pass A  S -> x = S scale - lg2(noise)/tau -> e = exp2(x - m), m the thread's running maximum; e goes back
//               to where S was, m of the tile stays in a register, the sum of the e is kept
//       then    the row's (m, sum) over the four warps, then over the CTAs of the cluster -> f = exp2(m - M) / L
//       pass B  e from TMEM in the 16x256b shape, in which a thread has 4 rows of 8 keys: sum += e * f.  The sums of
//               a CTA's keys stay in registers through all query tiles of a piece of work.
// A unit's query tiles are cut into chunks; each leaves its sums in a slab of the workspace (or directly in the score,
// with one chunk) and the kernel behind adds the slabs in order.  Chunks and cluster size follow from the sequence's
// lengths alone, how many chunks make a piece of work for a cluster from the number of units as well: a unit's scores
// are the same bits whatever other units the call has.
#include <algorithm>
#include <mutex>

#include "../../include/asuka_b200.h"
#include "kernels.h"
#include "score_math.cuh"
#include "sm100_ptx.cuh"
#include "tma_host.h"

namespace asuka {
using namespace sm100;

namespace {

constexpr int kTile = 128;
constexpr uint32_t kTileBytes = 128 * 128 * 2;
constexpr uint32_t kHalfBytes = kTileBytes / 2;
constexpr int kOwn = 4;       // tiles of a row block that a CTA holds: its 512 TMEM columns
constexpr int kKStages = 2;
constexpr int kBoxes = 7;     // noise boxes [128 rows x 32 keys]
constexpr uint32_t kBoxBytes = 128 * 32 * 4;
constexpr int kUtilWarps = 4;
constexpr int kParts = 4;              // warps to 32 query rows
constexpr int kCols = kTile / kParts;  // columns of a tile for each
constexpr int kKeyWarps = 4 * kParts;
constexpr int kThreads = (kUtilWarps + kKeyWarps) * 32;
constexpr int kMaxCluster = 8;
constexpr int kMaxChunks = 8;

enum { kNoisePlain = 0, kNoiseTma = 1, kNoiseSeeded = 2 };

struct FusedParams {
  int H, Sq, Skv;
  int causal, diag_off;
  int nq_tiles;
  float scale_log2;  // softmax_scale * log2(e) / tau
  float neg_inv_tau;
  const float* exp_rand;
  int64_t er_sb, er_sh, er_sq;
  uint64_t seed;
  uint32_t unit_off;
  uint32_t* status;
  int chained;
  int n_kt, kt_ahead;    // key tiles; of these row block i sees the first i + kt_ahead (as far as there are any)
  int chunk_tiles;       // query tiles to a chunk
  int n_pieces;          // of a unit; piece i has the chunks from first_chunk[i] to first_chunk[i + 1]
  int first_chunk[kMaxChunks + 1];
  int units, n_work;     // B * H; pieces of work in all
  float* out;            // [n_chunks][B*H][Skv]
  size_t slab;           // B * H * Skv
};

struct Tell {  // (plain noise) where a tile's noise is, and its last row and column
  const float* src;
  int last_row, last_col;
};
constexpr int kTells = 4;

struct FusedBars {
  uint64_t q_full;
  uint64_t k_full[kKStages], k_empty[kKStages];
  uint64_t s_full[kOwn], s_empty[kOwn];
  uint64_t n_full[kBoxes], n_empty[kBoxes];
  uint64_t t_full[kTells], t_empty[kTells];  // (plain noise) tell_s
  uint64_t m_full[4];     // the four warps of a row quarter have left theirs in ml_s
  uint64_t f_full[4];     // fin_s has the quarter's statistics over all keys
  uint64_t x_full[2][4];  // a row quarter's statistics of all CTAs have arrived
  uint64_t c_full, c_empty;  // the column sums of a chunk are complete; have been stored
};

__device__ __forceinline__ uint32_t mapa(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
// into another CTA's shared memory; that CTA's barrier counts the four bytes (no fence on either side)
__device__ __forceinline__ void st_async(uint32_t addr, float a, uint32_t bar) {
  asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.f32 [%0], %1, [%2];"
               ::"r"(addr), "f"(a), "r"(bar) : "memory");
}
__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory"); }

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t (&r)[8]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
      : "r"(taddr)
      : "memory");
}
// 16 lanes x 32 columns: thread t gets of every eight columns 2 (t % 4) and the next one, of lanes t / 4 and t / 4 + 8
__device__ __forceinline__ void tmem_ld_16x256b_x4(uint32_t taddr, uint32_t (&r)[16]) {
  asm volatile(
      "tcgen05.ld.sync.aligned.16x256b.x4.b32 "
      "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
      : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
        "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
      : "r"(taddr)
      : "memory");
}

// The steps of a cluster in order: its pieces of work, each a run of one unit's query tiles, latest first (with long
// and short row blocks in turn, whose tiles do not fit into tensor memory side by side, B2 H32 S1501 with seeded noise
// took 205 us instead of 189).
struct Steps {
  const FusedParams& p;
  uint32_t rank, lnc;  // (lnc: log2 of the cluster's size)
  int round, bh, chunk;
  bool more;
  int qt, qt_end, n_own;

  __device__ __forceinline__ Steps(const FusedParams& p_, uint32_t rank_, uint32_t lnc_) : p(p_), rank(rank_), lnc(lnc_) {
    round = 0;
    load_work();
  }
  __device__ __forceinline__ bool valid() const { return more; }
  __device__ __forceinline__ bool last_of_chunk() const { return qt == chunk * p.chunk_tiles; }
  // this CTA's t-th key tile: forth and back over the cluster, so that causal row blocks are shared evenly
  __device__ __forceinline__ int key_tile(int t) const {
    return (t << lnc) + static_cast<int>((t & 1) ? (1u << lnc) - 1u - rank : rank);
  }
  // Pieces are numbered latest (longest) first over all units and dealt out forth and back.
  __device__ __forceinline__ void load_work() {
    const int n = static_cast<int>(gridDim.x >> lnc), k = static_cast<int>(blockIdx.x >> lnc);
    const int w = round * n + ((round & 1) ? n - 1 - k : k);
    more = w < p.n_work;
    if (!more) return;
    const int turn = w / p.units, piece = p.n_pieces - 1 - turn;
    bh = w - turn * p.units;
    chunk = p.first_chunk[piece + 1] - 1;
    qt = min(p.nq_tiles, (chunk + 1) * p.chunk_tiles) - 1;
    qt_end = p.first_chunk[piece] * p.chunk_tiles;
    count_own();
  }
  __device__ __forceinline__ void count_own() {
    const int n_kv = min(qt + p.kt_ahead, p.n_kt);  // key tiles that the row block sees
    const int two = 2 << lnc, rem = n_kv & (two - 1);
    n_own = 2 * (n_kv >> (lnc + 1)) + (rem > static_cast<int>(rank) ? 1 : 0) + (rem > two - 1 - static_cast<int>(rank) ? 1 : 0);
  }
  __device__ __forceinline__ void next() {
    if (qt > qt_end) {
      if (last_of_chunk()) --chunk;
      --qt;
      count_own();
    } else {
      ++round;
      load_work();
    }
  }
};

template <bool kBF16, int kNoise>
__global__ void __launch_bounds__(kThreads, 1)
kf_fused_kernel(const __grid_constant__ CUtensorMap map_q, const __grid_constant__ CUtensorMap map_k,
                const __grid_constant__ CUtensorMap map_n, const FusedParams p) {
  extern __shared__ uint8_t smem_raw[];
  __shared__ __align__(8) FusedBars bars;
  __shared__ Tell tell_s[kNoise == kNoisePlain ? kTells : 1];
  __shared__ uint32_t tmem_base_s;
  __shared__ uint32_t abort_s;

  const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
  uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
  // Q tile | K tiles | noise boxes | partial statistics | column sums | statistics | exchange
  const uint32_t sQ = smem_base;
  const uint32_t sK = sQ + kTileBytes;
  constexpr uint32_t kOffNoise = kTileBytes + kKStages * kTileBytes;
  constexpr uint32_t kOffMl = kOffNoise + (kNoise == kNoiseSeeded ? 0u : kBoxes * kBoxBytes);
  constexpr uint32_t kOffRed = kOffMl + 4 * kTile * 8;
  constexpr uint32_t kOffFin = kOffRed + 4 * kOwn * kTile * 4;
  constexpr uint32_t kOffEx = kOffFin + kTile * 8;
  float2* ml_s = reinterpret_cast<float2*>(smem_gen + kOffMl);                 // [column quarter][row]
  float* red_s = reinterpret_cast<float*>(smem_gen + kOffRed);                 // column sums [row quarter][tile][key]
  float2* fin_s = reinterpret_cast<float2*>(smem_gen + kOffFin);               // [row] maximum, 1 / sum
  float* ex_s = reinterpret_cast<float*>(smem_gen + kOffEx);                   // [parity][rank][row]

  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  volatile uint32_t* abortp = &abort_s;
  const uint32_t rank = __clusterRelativeBlockRank(), nc = __clusterSizeInBlocks(), lnc = 31 - __clz(nc);

  if (!p.chained) griddep_wait();
  griddep_launch_dependents();

  if (tid == 0) {
    abort_s = 0;
    mbar_init(smem_u32(&bars.q_full), 1);
    for (int i = 0; i < kKStages; ++i) {
      mbar_init(smem_u32(&bars.k_full[i]), 1);
      mbar_init(smem_u32(&bars.k_empty[i]), 1);
    }
    for (int i = 0; i < kOwn; ++i) {
      mbar_init(smem_u32(&bars.s_full[i]), 1);
      mbar_init(smem_u32(&bars.s_empty[i]), kKeyWarps);
    }
    for (int i = 0; i < kBoxes; ++i) {
      mbar_init(smem_u32(&bars.n_full[i]), 1);
      mbar_init(smem_u32(&bars.n_empty[i]), 4);
    }
    for (int i = 0; i < kTells; ++i) {
      mbar_init(smem_u32(&bars.t_full[i]), 1);
      mbar_init(smem_u32(&bars.t_empty[i]), kKeyWarps);
    }
    for (int i = 0; i < 4; ++i) {
      mbar_init(smem_u32(&bars.m_full[i]), kParts);
      mbar_init(smem_u32(&bars.f_full[i]), 1);
    }
    mbar_init(smem_u32(&bars.c_full), kKeyWarps);
    mbar_init(smem_u32(&bars.c_empty), 2);
    for (int i = 0; i < 8; ++i) mbar_init(smem_u32(&bars.x_full[i >> 2][i & 3]), 1);
    mbar_fence_init();
    tma_prefetch_desc(&map_q);
    tma_prefetch_desc(&map_k);
    if (kNoise == kNoiseTma) tma_prefetch_desc(&map_n);
  }
  if (warp == 1) {
    __syncwarp();
    tmem_alloc(smem_u32(&tmem_base_s), 512);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  // (no CTA may signal another's barriers before they are initialised)
  cluster_arrive();
  cluster_wait();
  tc_fence_after_sync();
  const uint32_t tbase = tmem_base_s;

  Steps it(p, rank, lnc);
  auto signal = [&](uint64_t* bar) {  // this warp is done with something that no copy writes
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(bar));
  };

  if (warp == 0) {
    // ------------------------------------------------------------------ noise producer
    if (kNoise == kNoiseTma && lane == 0) {
      uint32_t n = 0;  // boxes
      bool ok = true;
      const uint64_t stream_once = l2_policy_evict_first();
      for (; it.valid() && ok; it.next()) {
        const int b = it.bh / p.H, h = it.bh % p.H;
        for (int t = 0; t < it.n_own && ok; ++t) {
          const int kv0 = it.key_tile(t) * kTile;
          for (int c4 = 0; c4 < kParts; ++c4, ++n) {
            const uint32_t slot = n % kBoxes, use = n / kBoxes;
            if (use > 0 && !mbar_wait(smem_u32(&bars.n_empty[slot]), (use - 1) & 1, abortp)) {
              record_timeout(p.status, 71);
              ok = false;
              break;
            }
            const uint32_t bar = smem_u32(&bars.n_full[slot]);
            mbar_expect_tx(bar, kBoxBytes);
            tma_load_4d_hint(smem_base + kOffNoise + slot * kBoxBytes, &map_n, bar, kv0 + c4 * 32, it.qt * kTile, h, b,
                             stream_once);
          }
        }
      }
      if (!ok) {
        // copies still in flight get a bounded chance to land before the CTA retires
        volatile uint32_t none = 0;
        for (uint32_t x = n > kBoxes ? n - kBoxes : 0; x < n; ++x)
          mbar_wait(smem_u32(&bars.n_full[x % kBoxes]), (x / kBoxes) & 1, &none);
      }
    } else if (kNoise == kNoisePlain && lane == 0) {
      // Noise that TMA cannot describe: the key warps copy their own 32 x 32 values, four bytes a lane, and learn here
      // where the next tile's are.
      uint32_t n = 0;  // tiles
      bool ok = true;
      auto tell = [&](const float* src, int last_row, int last_col) {
        const uint32_t slot = n % kTells, use = n / kTells;
        if (use > 0 && !mbar_wait(smem_u32(&bars.t_empty[slot]), (use - 1) & 1, abortp)) {
          record_timeout(p.status, 71);
          return false;
        }
        tell_s[slot].src = src;
        tell_s[slot].last_row = last_row;
        tell_s[slot].last_col = last_col;
        mbar_arrive(smem_u32(&bars.t_full[slot]));
        ++n;
        return true;
      };
      for (; it.valid() && ok; it.next()) {
        const int b = it.bh / p.H, h = it.bh % p.H, q0 = it.qt * kTile;
        const float* rows = p.exp_rand + b * p.er_sb + h * p.er_sh + q0 * p.er_sq;
        for (int t = 0; t < it.n_own && ok; ++t) {
          const int kv0 = it.key_tile(t) * kTile;
          ok = tell(rows + kv0, p.Sq - 1 - q0, p.Skv - 1 - kv0);
        }
      }
      if (ok) tell(nullptr, 0, 0);
    }
  } else if (warp == 1) {
    // ------------------------------------------------------------------ Q and K loads, MMA issue (whole warp)
    constexpr uint32_t kFmt = kBF16 ? UMMA_BF16 : UMMA_F16;
    constexpr uint32_t idesc = umma_idesc_f16(kFmt, UMMA_K_MAJOR, UMMA_K_MAJOR, 128, 128);
    auto wait_all = [&](uint64_t* bar, uint32_t parity, uint32_t site) -> bool {
      const bool good = __all_sync(0xffffffffu, mbar_wait(smem_u32(bar), parity, abortp));
      if (!good && lane == 0) record_timeout(p.status, site);
      return good;
    };
    // K tiles run ahead of the MMAs by the ring
    Steps kit = it;
    int kt = 0;             // next tile of kit to load
    uint32_t k_loaded = 0;  // tiles requested
    auto load_k = [&]() {
      while (kit.valid() && kt == kit.n_own) {
        kit.next();
        kt = 0;
      }
      if (!kit.valid()) return;
      const int st = k_loaded % kKStages;
      if (lane == 0) {
        const int b = kit.bh / p.H, h = kit.bh % p.H;
        const int kv0 = kit.key_tile(kt) * kTile;
        const uint32_t bar = smem_u32(&bars.k_full[st]);
        mbar_expect_tx(bar, kTileBytes);
        tma_load_4d(sK + st * kTileBytes, &map_k, bar, 0, h, kv0, b);
        tma_load_4d(sK + st * kTileBytes + kHalfBytes, &map_k, bar, 64, h, kv0, b);
      }
      __syncwarp();
      ++k_loaded;
      ++kt;
    };
    for (int i = 0; i < kKStages; ++i) load_k();
    bool ok = true;
    uint32_t n = 0, q_loads = 0;  // tiles issued, Q tiles
    const uint64_t qdesc = umma_smem_desc_sw128(sQ, 16, 1024);
    for (; it.valid() && ok; it.next()) {
      for (int t = 0; t < it.n_own && ok; ++t, ++n) {
        const int st = n % kKStages, buf = n % kOwn;
        if (t == 0) {
          if (lane == 0) {  // (every MMA of the query tile before is done, see below)
            const int b = it.bh / p.H, h = it.bh % p.H;
            const uint32_t bar = smem_u32(&bars.q_full);
            mbar_expect_tx(bar, kTileBytes);
            tma_load_4d(sQ, &map_q, bar, 0, h, it.qt * kTile, b);
            tma_load_4d(sQ + kHalfBytes, &map_q, bar, 64, h, it.qt * kTile, b);
          }
          __syncwarp();
          ++q_loads;
          ok = wait_all(&bars.q_full, (q_loads - 1) & 1, 73);
        }
        ok = ok && wait_all(&bars.k_full[st], (n / kKStages) & 1, 74);
        if (ok && n >= kOwn) ok = wait_all(&bars.s_empty[buf], (n / kOwn - 1) & 1, 75);
        if (!ok) break;
        tc_fence_after_sync();
        const uint64_t kdesc = umma_smem_desc_sw128(sK + st * kTileBytes, 16, 1024);
        if (elect_one()) {
#pragma unroll
          for (int kk = 0; kk < 8; ++kk) {
            const uint64_t off = static_cast<uint64_t>((kk & 3) * 2 + (kk >> 2) * (kHalfBytes >> 4));
            umma_ss(tbase + buf * 128, qdesc + off, kdesc + off, idesc, kk > 0 ? 1u : 0u);
          }
          umma_commit(smem_u32(&bars.k_empty[st]));
          umma_commit(smem_u32(&bars.s_full[buf]));
        }
        __syncwarp();
        // the stage is free when these are done, and Q when they were the last of their query tile
        ok = wait_all(&bars.k_empty[st], (n / kKStages) & 1, 72);
        if (ok) load_k();
      }
    }
    if (!ok && lane == 0) {
      volatile uint32_t none = 0;
      for (uint32_t x = k_loaded > kKStages ? k_loaded - kKStages : 0; x < k_loaded; ++x)
        mbar_wait(smem_u32(&bars.k_full[x % kKStages]), (x / kKStages) & 1, &none);
      if (q_loads > 0) mbar_wait(smem_u32(&bars.q_full), (q_loads - 1) & 1, &none);
    }
  } else if (warp < kUtilWarps) {
    // ------------------------------------------------------------------ the rows' statistics, two quarters to a warp
    const int quarter0 = (warp - 2) * 2;
    bool ok = true;
    uint32_t chunks = 0;
    for (uint32_t item = 0; it.valid() && ok; it.next(), ++item) {
      const uint32_t par = item & 1;
      for (int x = 0; x < 2 && ok; ++x) {
        const int wq = quarter0 + x, r = wq * 32 + lane;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.m_full[wq]), item & 1, abortp));
        if (!ok) { if (lane == 0) record_timeout(p.status, 80); break; }
        float2 v[kParts];
#pragma unroll
        for (int c = 0; c < kParts; ++c) v[c] = ml_s[c * kTile + r];
        float M = v[0].x;
#pragma unroll
        for (int c = 1; c < kParts; ++c) M = fmaxf(M, v[c].x);
        float L = 0.f;
#pragma unroll
        for (int c = 0; c < kParts; ++c) L += v[c].y * (v[c].x > -INFINITY ? ex2(v[c].x - M) : 0.f);
        const float lse = M + lg2(L);
        const uint32_t bar = smem_u32(&bars.x_full[par][wq]);
        if (lane == 0) mbar_expect_tx(bar, nc * 32 * 4);
        const uint32_t slot = smem_base + kOffEx + ((par * nc + rank) * kTile + r) * 4;
        for (uint32_t c = 0; c < nc; ++c) st_async(mapa(slot, c), lse, mapa(bar, c));
      }
      for (int x = 0; x < 2 && ok; ++x) {
        const int wq = quarter0 + x, r = wq * 32 + lane;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.x_full[par][wq]), (item >> 1) & 1, abortp));
        if (!ok) { if (lane == 0) record_timeout(p.status, 76); break; }
        float lse[kMaxCluster];
#pragma unroll
        for (int c = 0; c < kMaxCluster; ++c) lse[c] = c < static_cast<int>(nc) ? ex_s[(par * nc + c) * kTile + r] : -INFINITY;
        float M = lse[0];
#pragma unroll
        for (int c = 1; c < kMaxCluster; ++c) M = fmaxf(M, lse[c]);
        float L = 0.f;
#pragma unroll
        for (int c = 0; c < kMaxCluster; ++c) L += ex2(lse[c] - M);
        fin_s[r] = make_float2(M, it.qt * kTile + r < p.Sq ? __fdividef(1.f, L) : 0.f);
        signal(&bars.f_full[wq]);
      }
      if (ok && it.last_of_chunk()) {
        // ---- a chunk is done: the column sums over the row quarters, half of the tiles to a warp, go out
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.c_full), chunks & 1, abortp));
        if (!ok) { if (lane == 0) record_timeout(p.status, 79); break; }
        if (chunks == 0) griddep_wait();  // (the kernel ahead may still be reading what the slabs held)
        ++chunks;
        float* out = p.out + it.chunk * p.slab + static_cast<size_t>(it.bh) * p.Skv;
        for (int x = 0; x < kOwn / 2 * kTile; x += 32) {
          const int s = (warp - 2) * (kOwn / 2) + x / kTile, k = x % kTile + lane;
          float* r = red_s + s * kTile + k;
          const float v = (r[0] + r[kOwn * kTile]) + (r[2 * kOwn * kTile] + r[3 * kOwn * kTile]);
#pragma unroll
          for (int c = 0; c < 4; ++c) r[c * kOwn * kTile] = 0.f;
          const int key = it.key_tile(s) * kTile + k;
          if (key < p.Skv) out[key] = v;
        }
        signal(&bars.c_empty);
      }
    }
  } else {
    // ------------------------------------------------------------------ rows and columns
    const int wq = warp & 3;           // TMEM lane quarter: query rows
    const int part = (warp - kUtilWarps) >> 2;  // columns of every tile
    const int r_in_tile = wq * 32 + lane;
    const uint32_t tcol = tbase + (static_cast<uint32_t>(wq * 32) << 16) + part * kCols;
    const float scale = p.scale_log2;
    const uint32_t row_off = sw128_offset(r_in_tile, 0);  // (chunk c of the row: ^ 16 c)
    // this thread's sums: of each tile the key 8 (lane >> 3) + 2 (lane & 3) + (lane >> 2 & 1) of its warp's 32
    float* acc = red_s + wq * kOwn * kTile + part * kCols + 8 * (lane >> 3) + 2 * (lane & 3) + (lane >> 2 & 1);
#pragma unroll
    for (int s = 0; s < kOwn; ++s) acc[s * kTile] = 0.f;
    bool ok = true;
    uint32_t n = 0;     // tiles of pass A
    uint32_t item = 0;  // query tiles whose statistics were sent
    // the query tile whose pass B is still to come
    int pend_own = -1, pend_qt = 0;  // (-1: none)
    uint32_t chunks = 0;      // twice the chunks done, + 1 while the sums of the last may still be on their way out
    float mr[kOwn] = {0.f, 0.f, 0.f, 0.f};  // what the exponentials in each TMEM buffer are relative to
    // (plain noise) this warp's values of tile i start on their way
    auto fetch = [&](uint32_t i) -> bool {
      if (!__all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.t_full[i % kTells]), (i / kTells) & 1, abortp))) {
        if (lane == 0) record_timeout(p.status, 83);
        return false;
      }
      const Tell tell = tell_s[i % kTells];
      signal(&bars.t_empty[i % kTells]);
      if (tell.src == nullptr) return true;
      // (columns and rows beyond the end repeat the last one; a row's address is one multiply-add that waits for no other)
      const char* src = reinterpret_cast<const char*>(tell.src + min(part * kCols + lane, tell.last_col));
      const uint32_t row_bytes = static_cast<uint32_t>(p.er_sq) * 4u;
      const uint32_t dst = smem_base + kOffNoise + part * kBoxBytes + wq * 32 * 128;
      const uint32_t col = (lane >> 2) * 16 + (lane & 3) * 4;
      const int last = tell.last_row - wq * 32;
#pragma unroll 16
      for (int r = 0; r < 32; ++r)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;"
                     ::"r"(dst + r * 128 + (col ^ ((r & 7) * 16))),
                       "l"(src + static_cast<uint64_t>(static_cast<uint32_t>(wq * 32 + min(r, last))) * row_bytes) : "memory");
      return true;
    };
    if (kNoise == kNoisePlain) ok = fetch(0);

    while (true) {
      const bool more = it.valid();
      if (!more && pend_own < 0) break;
      const int n_own = more ? it.n_own : 0;
      const int q0 = it.qt * kTile;
      // last key that the first row of the block sees (no row beyond the end sees any)
      const int min_lim = q0 + kTile > p.Sq ? -1 : p.causal ? min(p.Skv - 1, q0 + p.diag_off) : p.Skv - 1;
      const uint32_t head_key = kNoise == kNoiseSeeded ? seeded_head_key(p.seed, static_cast<uint32_t>(it.bh) + p.unit_off) : 0u;
      float m = -INFINITY, l = 0.f;
      const int ahead = min(kOwn - pend_own, n_own);  // tiles that fit beside the ones still to be added up
      for (int t = 0; ok; ++t) {
        if (pend_own >= 0 && t == ahead) {
          // ---- pass B of the query tile before
          ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.f_full[wq]), (item - 1) & 1, abortp));
          if (!ok) { if (lane == 0) record_timeout(p.status, 81); break; }
          const float2 fin = fin_s[r_in_tile];
          if (chunks & 1) {
            ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.c_empty), ((chunks >> 1) - 1) & 1, abortp));
            if (!ok) { if (lane == 0) record_timeout(p.status, 82); break; }
            --chunks;
          }
          tmem_wait_st();
          __syncwarp();
#pragma unroll 1
          for (int s = 0; s < pend_own; ++s) {
              const uint32_t buf = (n - ahead - pend_own + s) & 3;
              const float pm = buf & 2 ? (buf & 1 ? mr[3] : mr[2]) : (buf & 1 ? mr[1] : mr[0]);
              const float fr = fin.y != 0.f ? ex2(pm - fin.x) * fin.y : 0.f;
              uint32_t g[32];
              tmem_ld_16x256b_x4(tcol + buf * 128, *reinterpret_cast<uint32_t(*)[16]>(&g[0]));
              tmem_ld_16x256b_x4(tcol + buf * 128 + (16u << 16), *reinterpret_cast<uint32_t(*)[16]>(&g[16]));
              float f[4];
#pragma unroll
              for (int k = 0; k < 4; ++k) f[k] = __shfl_sync(0xffffffffu, fr, (lane >> 2) + 8 * k);
              tmem_wait_ld();
              tc_fence_before_sync();
              signal(&bars.s_empty[buf]);
              const int kv = it.key_tile(s) * kTile + part * kCols;
              const bool has_mask = p.causal && kv + kCols - 1 > (pend_qt >> 1) * kTile + p.diag_off;
              float v[8];  // sums over this thread's rows: key 8 (i >> 1) + 2 (lane & 3) + (i & 1)
              if (has_mask) {  // keys that some row does not see: what is masked is zero whatever the row's factor is
                const int vis = (pend_qt >> 1) * kTile + wq * 32 + (lane >> 2) + p.diag_off + 1 - (kv + 2 * (lane & 3));
#pragma unroll
                for (int i = 0; i < 8; ++i) {
                  v[i] = 0.f;
#pragma unroll
                  for (int k = 0; k < 4; ++k) {  // (columns 8 x + y < vis, eight more in every further row)
                    const float e = __uint_as_float(g[(k >> 1) * 16 + 4 * (i >> 1) + 2 * (k & 1) + (i & 1)]);
                    v[i] += 8 * (i >> 1) + (i & 1) < vis + 8 * k ? e * f[k] : 0.f;
                  }
                }
              } else {
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                  float2 a = make_float2(0.f, 0.f);
#pragma unroll
                  for (int k = 0; k < 4; ++k) {
                    const int o = (k >> 1) * 16 + 4 * x + 2 * (k & 1);
                    a = __ffma2_rn(make_float2(__uint_as_float(g[o]), __uint_as_float(g[o + 1])), make_float2(f[k], f[k]), a);
                  }
                  v[2 * x] = a.x;
                  v[2 * x + 1] = a.y;
                }
              }
              // over the eight lanes with the same keys; lane 4 i + x of them keeps v[i]
#pragma unroll
              for (int w = 4; w > 0; w >>= 1) {
                const bool up = (lane & (4 * w)) != 0;
#pragma unroll
                for (int i = 0; i < w; ++i) {
                  const float keep = up ? v[i + w] : v[i], send = up ? v[i] : v[i + w];
                  v[i] = keep + __shfl_xor_sync(0xffffffffu, send, 4 * w);
                }
              }
              acc[s * kTile] += v[0];
          }
          pend_own = -1;
          if (pend_qt & 1) {  // the last query tile of its chunk
            signal(&bars.c_full);
            chunks += 3;
          }
        }
        if (t >= n_own) break;
        // ---- pass A of one tile
        const uint32_t buf = n & 3;
        const int kv0 = it.key_tile(t) * kTile + part * kCols;
        ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.s_full[buf]), (n >> 2) & 1, abortp));
        if (!ok) { if (lane == 0) record_timeout(p.status, 77); break; }
        tc_fence_after_sync();
        float x[kCols];
        uint32_t word = 0;  // (seeded) the row and the first column after the mix's first xor-shift
        if constexpr (kNoise == kNoiseSeeded) {
          word = ((static_cast<uint32_t>(q0 + r_in_tile) << 16) ^ static_cast<uint32_t>(kv0)) ^ head_key;
          word ^= word >> 16;
        }
        constexpr int kG = kNoise == kNoiseSeeded ? 8 : 16;
        // (in two halves: what is live at once has to fit beside the column sums)
#pragma unroll
        for (int hf = 0; hf < kCols / kG; ++hf) {
          uint32_t u[kG];
          if constexpr (kG == 16) tmem_ld16(tcol + buf * 128 + hf * kG, *reinterpret_cast<uint32_t(*)[16]>(u));
          else tmem_ld8(tcol + buf * 128 + hf * kG, *reinterpret_cast<uint32_t(*)[8]>(u));
          float* xh = x + hf * kG;
          if constexpr (kNoise != kNoiseSeeded) {
            const uint32_t box_i = n * kParts + part, box_slot = kNoise == kNoisePlain ? part : box_i % kBoxes;
            if (hf == 0) {
              if constexpr (kNoise == kNoisePlain) {
                asm volatile("cp.async.wait_all;" ::: "memory");
                __syncwarp();
              } else {
                ok = __all_sync(0xffffffffu, mbar_wait(smem_u32(&bars.n_full[box_slot]), (box_i / kBoxes) & 1, abortp));
                if (!ok) { if (lane == 0) record_timeout(p.status, 78); break; }
              }
            }
            const uint8_t* box = smem_gen + kOffNoise + box_slot * kBoxBytes;
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              const float4 v = *reinterpret_cast<const float4*>(box + (row_off ^ ((hf * 4 + c) * 16)));
              xh[4 * c] = v.x; xh[4 * c + 1] = v.y; xh[4 * c + 2] = v.z; xh[4 * c + 3] = v.w;
            }
            if (hf == 1) {
              if (kNoise == kNoiseTma) {
                fence_proxy_async_smem();  // (the reads above before the copy that refills the box)
                __syncwarp();
                if (lane == 0) mbar_arrive(smem_u32(&bars.n_empty[box_slot]));
              } else {
                __syncwarp();
                ok = fetch(n + 1);
                if (!ok) break;
              }
            }
          }
          tmem_wait_ld();
#pragma unroll
          for (int e = 0; e < kG; e += 2) {
            float2 l2;
            // (columns kv0 + x, x < 32: the first xor-shift of the mix leaves x where it is)
            if constexpr (kNoise == kNoiseSeeded) l2 = seeded_lg2_exp_rand2(word ^ (hf * kG + e), word ^ (hf * kG + e + 1));
            else l2 = make_float2(lg2(xh[e]), lg2(xh[e + 1]));
            const float2 v = __ffma2_rn(make_float2(__uint_as_float(u[e]), __uint_as_float(u[e + 1])), make_float2(scale, scale),
                                        __fmul2_rn(l2, make_float2(p.neg_inv_tau, p.neg_inv_tau)));
            xh[e] = v.x;
            xh[e + 1] = v.y;
          }
        }
        if (!ok) break;
        if (kv0 + kCols - 1 > min_lim) {
          const int row = q0 + r_in_tile;
          const int lim = row >= p.Sq ? -1 : p.causal ? min(p.Skv - 1, row + p.diag_off) : p.Skv - 1;
#pragma unroll
          for (int e = 0; e < kCols; ++e) x[e] = e > lim - kv0 ? -INFINITY : x[e];
        }
        float mt[4] = {m, -INFINITY, -INFINITY, -INFINITY};
#pragma unroll
        for (int e = 0; e < kCols; e += 8) {
#pragma unroll
          for (int g = 0; g < 4; ++g) mt[g] = max3(mt[g], x[e + 2 * g], x[e + 2 * g + 1]);
        }
        const float m_new = fmaxf(fmaxf(mt[0], mt[1]), fmaxf(mt[2], mt[3]));
        // (a row that has seen nothing yet: exponentials of -inf - 0)
        const float neg_m = m_new > -INFINITY ? -m_new : 0.f;
        float2 l01 = make_float2(l * (m > -INFINITY ? ex2(m + neg_m) : 0.f), 0.f), l23 = make_float2(0.f, 0.f);
        const float2 neg_m2 = make_float2(neg_m, neg_m);
#pragma unroll
        for (int e = 0; e < kCols; e += 4) {
          const float2 a = __fadd2_rn(make_float2(x[e], x[e + 1]), neg_m2), c = __fadd2_rn(make_float2(x[e + 2], x[e + 3]), neg_m2);
          x[e] = ex2(a.x); x[e + 1] = ex2(a.y); x[e + 2] = ex2(c.x); x[e + 3] = ex2(c.y);
          l01 = __fadd2_rn(l01, make_float2(x[e], x[e + 1]));
          l23 = __fadd2_rn(l23, make_float2(x[e + 2], x[e + 3]));
        }
        l = (l01.x + l01.y) + (l23.x + l23.y);
        m = m_new;
        tmem_st32(tcol + buf * 128, reinterpret_cast<uint32_t(&)[32]>(x));
#pragma unroll
        for (int s = 0; s < kOwn; ++s) mr[s] = s == static_cast<int>(buf) ? m : mr[s];
        ++n;
      }
      if (!ok || !more) break;
      ml_s[part * kTile + r_in_tile] = make_float2(m, l);
      signal(&bars.m_full[wq]);
      ++item;
      pend_own = it.n_own;
      pend_qt = 2 * it.qt + (it.last_of_chunk() ? 1 : 0);
      it.next();
    }
    if (!ok) *abortp = 1u;
  }

  if (kNoise == kNoisePlain) asm volatile("cp.async.wait_all;" ::: "memory");  // (given up: none is left under way)
  griddep_wait();  // (whatever waits for this grid waits for the one ahead as well)
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    __syncwarp();
    tmem_dealloc(tbase, 512);
  }
  // no CTA leaves while another may still signal its barriers
  __syncwarp();
  cluster_arrive();
  cluster_wait();
}

constexpr uint32_t fused_smem(int noise, int cluster) {
  return kTileBytes + kKStages * kTileBytes + (noise == kNoiseSeeded ? 0 : kBoxes * kBoxBytes) + 5 * kTile * 8 +
         4 * kOwn * kTile * 4 + 2 * cluster * kTile * 4 + 1024;
}

typedef void (*FusedKernel)(CUtensorMap, CUtensorMap, CUtensorMap, FusedParams);
FusedKernel fused_kernel(bool bf16, int noise) {
  if (noise == kNoiseSeeded) return bf16 ? kf_fused_kernel<true, kNoiseSeeded> : kf_fused_kernel<false, kNoiseSeeded>;
  if (noise == kNoisePlain) return bf16 ? kf_fused_kernel<true, kNoisePlain> : kf_fused_kernel<false, kNoisePlain>;
  return bf16 ? kf_fused_kernel<true, kNoiseTma> : kf_fused_kernel<false, kNoiseTma>;
}

// how many clusters of `cluster` CTAs the current device runs at once
int resident_clusters(FusedKernel kern, int cluster, uint32_t smem) {
  struct Entry { const void* k; int dev, cluster, n; };
  static std::mutex mu;
  static Entry seen[64];
  static int n_seen = 0;
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess) return 0;
  const void* id = reinterpret_cast<const void*>(kern);
  std::lock_guard<std::mutex> lock(mu);
  for (int i = 0; i < n_seen; ++i)
    if (seen[i].k == id && seen[i].dev == dev && seen[i].cluster == cluster) return seen[i].n;
  if (ensure_dynamic_smem(id, static_cast<int>(smem)) != cudaSuccess) return 0;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(static_cast<unsigned>(cluster));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = smem;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = static_cast<unsigned>(cluster);
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  int n = 0;
  if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
    (void)cudaGetLastError();
    return 0;
  }
  if (n_seen < 64) seen[n_seen++] = Entry{id, dev, cluster, n};
  return n;
}

int noise_kind(const ScoreArgs& a) {
  if (a.exp_rand == nullptr) return kNoiseSeeded;
  // TMA needs a 16-byte aligned base and strides that are multiples of 16 bytes
  return (reinterpret_cast<uintptr_t>(a.exp_rand) & 15u) == 0 && a.er_stride_q % 4 == 0 && a.er_stride_h % 4 == 0 &&
                 a.er_stride_b % 4 == 0 && a.er_stride_q > 0 && a.er_stride_h > 0 && a.er_stride_b > 0
             ? kNoiseTma : kNoisePlain;
}

}  // namespace

// Cluster: CTAs enough for their tensor memory to hold a row block's tiles, and more where few row blocks would leave SMs
// idle (whole case in us, two passes / 1 / 2 / 4 CTAs; noise operand: B1 H4 S512 25.5 / 22.3 / 18.8 / 15.6, B2 H40
// S512 60.2 / 48.7 / 49.9 / 57.7, B2 H40 S1000 141 / - / 104 / 113; seeded: B2 H40 S300 49.9 / 39.0 / 52.8 / 53.8, B2 H32
// S1024 114 / - / 94.6 / 108).  Clusters of other sizes than powers of two run with fewer at once than the occupancy
// query says (three CTAs, B2 H32 S1501: 293 us, four 204).  Chunks: the pieces of work can be no smaller, see cut_pieces.
// Two passes remain for
// - more than 2048 keys with a noise operand (no shared memory for the exchange of eight CTAs) or up to 3968 with
//   seeded noise, and from there more than 8 units: clusters of eight leave a fifth of the SMs idle (B1 S4096: 2 heads
//   165 / 83, 8 heads 221 / 205, 16 heads 315 / 353; S3000: B2 H40 832 / 868);
// - a workspace without room for the chunks' sums.
FusedPlan kf_fused_plan(const ScoreArgs& a, const AttnShape& s, size_t ws_bytes) {
  FusedPlan plan = {0, 0, 0};
  const int noise = noise_kind(a);
  const int n_kt = (s.Skv + kTile - 1) / kTile, nq = (s.Sq + kTile - 1) / kTile;
  const long long units = static_cast<long long>(s.B) * s.H;
  const int cluster = n_kt <= 3 ? 1 : n_kt <= 8 ? 2 : n_kt <= 16 ? 4 : 8;
  const int chunk_tiles = nq <= 4 ? 1 : std::max(2, (nq + kMaxChunks - 1) / kMaxChunks);
  const int chunks = (nq + chunk_tiles - 1) / chunk_tiles;
  if (s.group != 1 || n_kt > kOwn * cluster) return plan;
  if (noise == kNoisePlain && a.er_stride_q >= (1ll << 30)) return plan;  // (32-bit row strides in bytes)
  if (cluster == 8 && (noise != kNoiseSeeded || nq < 32 || units > 8)) return plan;
  if (chunks > 1 && static_cast<size_t>(units) * s.Skv * sizeof(float) * chunks > ws_bytes) return plan;
  // (a device or a partition of one on which such a cluster does not fit)
  if (resident_clusters(fused_kernel(s.bf16, noise), cluster, fused_smem(noise, cluster)) <= 0) return plan;
  plan.cluster = cluster;
  plan.chunks = chunks;
  plan.chunk_tiles = chunk_tiles;
  return plan;
}

// A unit's chunks to pieces of work: the more pieces, the better they fill the clusters that run at once, `resident`;
// but a cluster that goes on with the same unit saves what a change costs.  The deal is played through with a model of
// what a cluster does one after the other: 2.2 us for a query tile (exchange, second look), 1.15 us for a key tile of the
// CTA that has most (2.0 with seeded noise), 2 us for a piece of work.  Whole case in us, 1 / 2 / 4 / 8 pieces: noise
// operand B1 H4 S2048 106 / 70.8 / 54.6 / 42.8, B4 H32 S2048 482 / 482 / 481 / 482, B2 H40 S1500 221 / 199 / 199 / 225;
// seeded B2 H32 S1501 192 / 196 / 197 / 222.  Longest pieces first over all units, dealt forth and back, against unit
// by unit: B2 H16 S1000 60.9 -> 52.6, B1 H8 S2048 60 -> 51, seeded B1 H16 S600 30.1 -> 25.0 (B2 H40 S512 44.8 -> 46.7).
void cut_pieces(FusedParams& p, int chunks, int noise, int cluster, int resident, long long units) {
  const double per_tile = noise == kNoiseSeeded ? 2.0 : 1.15, per_item = 2.2, per_work = 2.0;
  double chunk[kMaxChunks] = {}, total = 0.;
  for (int i = 0; i < p.nq_tiles; ++i) {
    const double t = per_item + per_tile * ((std::min(i + p.kt_ahead, p.n_kt) + cluster - 1) / cluster);
    chunk[i / p.chunk_tiles] += t;
    total += t;
  }
  double best = 0.;
  for (int n = 1; n <= chunks; ++n) {
    // n runs of chunks, each up to its share of the total
    int first[kMaxChunks + 1] = {0};
    double run[kMaxChunks], done = 0.;
    for (int x = 0, c = 0; x < n; ++x) {
      run[x] = per_work;
      const double until = total * (x + 1) / n;
      do {
        run[x] += chunk[c];
        done += chunk[c++];
      } while (c < chunks - (n - 1 - x) && (x == n - 1 || done + 0.5 * chunk[c] <= until));
      first[x + 1] = c;
    }
    // the longest of a few of the clusters, dealt their pieces as Steps does (many rounds: all of them alike)
    double cost = 0.;
    const long long works = units * n, rounds = (works + resident - 1) / resident;
    for (int x = 0; x < 16; ++x) {
      const long long k = (resident - 1) * x / 15;
      double t = 0.;
      for (long long r = 0; r < std::min(rounds, 32ll); ++r) {
        const long long w = r * resident + ((r & 1) ? resident - 1 - k : k);
        if (w < works) t += run[n - 1 - w / units];
      }
      cost = std::max(cost, t);
    }
    if (rounds > 32) cost = (total + n * per_work) * units / resident;
    if (n == 1 || cost < best) {
      best = cost;
      p.n_pieces = n;
      std::copy(first, first + n + 1, p.first_chunk);
    }
  }
}

cudaError_t launch_kf_fused(const CUtensorMap& mq, const CUtensorMap& mk, const ScoreArgs& a, const AttnShape& s,
                            const FusedPlan& plan, void* split_ws, cudaStream_t stream, PendingChunkSum* pending) {
  const int noise = noise_kind(a);
  if (plan.chunks > 1 && split_ws == nullptr) return cudaErrorInvalidValue;
  FusedParams p;
  p.H = s.H;
  p.Sq = s.Sq;
  p.Skv = s.Skv;
  p.causal = s.causal;
  p.diag_off = s.Skv - s.Sq;
  p.nq_tiles = (s.Sq + kTile - 1) / kTile;
  p.scale_log2 = s.softmax_scale * 1.4426950408889634f / a.tau;
  p.neg_inv_tau = -1.0f / a.tau;
  p.exp_rand = a.exp_rand;
  p.er_sb = a.er_stride_b;
  p.er_sh = a.er_stride_h;
  p.er_sq = a.er_stride_q;
  p.seed = a.seed;
  p.unit_off = a.unit_offset;
  p.status = device_status_words();
  p.chained = a.chained;
  p.n_kt = (s.Skv + kTile - 1) / kTile;
  p.kt_ahead = s.causal ? (kTile - 1 + p.diag_off) / kTile + 1 : p.n_kt;
  p.chunk_tiles = plan.chunk_tiles;
  p.slab = static_cast<size_t>(s.B) * s.H * s.Skv;
  p.out = plan.chunks > 1 ? static_cast<float*>(split_ws) : a.score;
  CUtensorMap mn = mq;
  if (noise == kNoiseTma) {
    const uint64_t dims[4] = {static_cast<uint64_t>(s.Skv), static_cast<uint64_t>(s.Sq), static_cast<uint64_t>(s.H),
                              static_cast<uint64_t>(s.B)};
    const uint64_t strides[3] = {static_cast<uint64_t>(a.er_stride_q) * 4, static_cast<uint64_t>(a.er_stride_h) * 4,
                                 static_cast<uint64_t>(a.er_stride_b) * 4};
    const uint32_t box[4] = {32, 128, 1, 1};
    if (tma_host::make_f32_map_sw128(&mn, a.exp_rand, dims, strides, box) != 0) return cudaErrorInvalidValue;
  }
  const FusedKernel kern = fused_kernel(s.bf16, noise);
  const uint32_t smem = fused_smem(noise, plan.cluster);
  const int resident = resident_clusters(kern, plan.cluster, smem);
  if (resident <= 0) return cudaErrorInvalidValue;
  cudaError_t e = ensure_dynamic_smem(reinterpret_cast<const void*>(kern), static_cast<int>(smem));
  if (e != cudaSuccess) return e;
  cut_pieces(p, plan.chunks, noise, plan.cluster, resident, static_cast<long long>(s.B) * s.H);
  p.units = s.B * s.H;
  p.n_work = p.units * p.n_pieces;
  const int clusters = std::min(p.n_work, resident);
  e = launch_dependent_cluster(kern, dim3(static_cast<unsigned>(clusters * plan.cluster)), dim3(kThreads), smem,
                               static_cast<unsigned>(plan.cluster), stream, mq, mk, mn, p);
  count_launch();
  if (e != cudaSuccess) return e;
  pending->part = p.out;
  pending->part_sq = nullptr;
  pending->n_chunks = plan.chunks > 1 ? plan.chunks : 0;
  return e;
}
}  // namespace asuka
