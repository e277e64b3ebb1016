// Prefill attention forward for sm_100a: tcgen05 tensor cores, TMEM accumulators,
// TMA-staged K/V ring, online softmax in registers.
//
// Replaces the reference's partial + merge launch pair (kernels/attention.py:430-746).
//
// Persistent kernel, one CTA per SM.  A work item is two 128-row query tiles ("slots") that share a KV head.
// Warp roles (576 threads):
//   warps 0-15 : softmax; warp w serves slot w / 8, TMEM lane quadrant w % 4 and 16 of its 32 query rows.  Tensor
//                memory is read in the 16x256b layout, which puts the 128 scores of a row into the four threads of
//                a quad: row maxima and sums are two shuffles away, nothing is exchanged through shared memory
//   warp  16   : scheduler + TMA producer (draws work items, loads Q, then the K_j / V_j tiles of 128 keys in pairs
//                {V_j, K_j+1} through two stages of two buffers; paged caches are fetched one page-sized box at a
//                time from the block table)
//   warp  17   : tcgen05.mma issuer and TMEM owner; the warp stays converged, one elected lane issues
// TMEM (512 columns): S0 | S1 | O0 | O1.  Per KV tile j and slot s:
//   S_s = Q_s K_j^T   (SS MMA, 128x128xD)            -> commit s_full[s]
//   the slot's warps exponentiate S_s (exp2 domain) against each row's reference, keep the row sums, and write P_s as
//   packed 16-bit (16x128b layout) over the first 32 columns of each 64-column half of S_s -> arrive p_ready[s]
//   (a row's reference, the maximum when it was set, moves only when the sums say that it has to; O_s is then rescaled)
//   O_s += P_s V_j    (TS MMA, A from TMEM, V is the MN-major B operand) -> commit o_done[s]
// The two slots are interleaved so that one slot's softmax overlaps the other's MMAs.  At the end of an item the
// MMA warp issues the first score tile of the next item behind the last PVs, and the softmax warps read O out, normalise
// and store it while that tile is computed.  Launches of few items may cut an item's keys over the CTAs of a cluster (kParts,
// cluster_plan): each runs its part as an item of its own, and the parts meet in the tile buffers at the end.
//
// What bounds it.  Long launches run at the board's 1 000 W (1.6 GHz instead of 1.97): there the time is the energy of a
// tile, and an instruction left out per score counts in full, a shorter chain of waits half.  The softmax is therefore as
// few instructions per pair of scores as there can be: one packed FMA, two exponentials, one packed add, one conversion,
// and no row maximum.  Against a pass for the maximum before them and a quarter of the exponentials as polynomials on the
// FMA pipes: 2 x 2 048 causal tokens, 32/8 heads, D 128, 86.2 -> 81.1 us; sixteen ragged sequences of 128 to 4 096
// 1 077 -> 1 001; 8 x 2 048 without a mask 586 -> 546.
//
// Every mbarrier wait is bounded; on expiry the role records DEV_ERR_WAIT_EXPIRED
// in the workspace header and falls through to the common teardown (TMEM is freed, rows that are not known become NaN).
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "cast.cuh"
#include "cluster_residency.h"
#include "common.cuh"
#include "launch.cuh"
#include "prefill_launch.h"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace b200attn {

namespace {

using namespace ptx;

constexpr int kBM = 128;           // query rows per slot
constexpr int kBN = 128;           // keys per K/V tile
constexpr int kSlots = 2;
constexpr int kRing = 4;           // K/V tile buffers: two stages of one V buffer and one K buffer
constexpr int kStages = 2;         // a stage holds the pair {V_j, K_j+1}: one barrier to wait for, one to release
constexpr int kSoftmaxWarps = 16;  // 4 warpgroups: (slot 0 | slot 1) x (columns 0-63 | 64-127)
constexpr int kThreads = 576;
constexpr int kProducerWarp = 16;
constexpr int kMmaWarp = 17;
constexpr int kQBufs = 3;          // Q tiles: the two of the current item and the first of the next
// A tile's exponentials against the reference that stands are good as long as a thread's 32 of them, of a row, sum up to
// no more than kMaxPartialSum (P then fits 16 bits, and so does every one of them).  When that is not so the row's maximum
// lies five powers of two or more above its reference; a reference moves when the maximum is kRescaleThreshold above it.
constexpr float kMaxPartialSum = 1024.0f;
constexpr float kRescaleThreshold = 3.0f;  // log2 units
// Everything one work item needs; decoded once by the scheduler warp.  An item is two 128-row query tiles
// ("slots") that share one KV head: with an even GQA group the same 128 rows of two neighbouring q heads (equal
// causal extents, so both slots always have work), otherwise two consecutive row tiles of one q head.
struct ItemWork {
  bool valid;
  int len_q, len_k;
  long long kv_row0;   // first kv row this item reads (dense / ragged)
  int kv_tok0;         // first key of the sequence this item reads (non-zero only when the KV range is split)
  long long out_row0[kSlots];   // first output row (the partial buffer's rows when the KV range is split)
  int kv_head_coord;
  int b;
  int q_head[kSlots];
  long long q_row0[kSlots];   // first q row of the sequence on the token axis of the q tensor map
  int q_head_coord[kSlots];
  int m0[kSlots];      // first query row of each slot inside the sequence
  int nkv[kSlots];     // 128-key tiles each slot visits
  int nkv_max;
};

// shared-memory control block placed after the tiles
struct __align__(8) Control {
  uint64_t q_full[kQBufs];
  uint64_t q_empty[kQBufs];
  uint64_t kv_full[kStages];     // pair {V_j, K_j+1} (or K_0 alone / V_last alone) has landed
  uint64_t kv_empty[kStages];    // ... has been consumed by the MMAs
  uint64_t s_full[kSlots];
  uint64_t p_ready[kSlots];
  uint64_t o_done[kSlots];
  uint64_t drained;              // the MMAs of an issuer that gave up
  uint64_t sched_full[2];
  uint64_t sched_empty[2];
  int sched_item[2];
  ItemWork sched_work[2];   // decoded by the scheduler, read by every other warp
  uint32_t tmem_base;
  int abort_flag;
  bool cut;                 // parts in clusters: see finish_item
};

template <int D>
struct SmemPlan {
  static constexpr int kChunks = D / 64;                   // 128-byte column blocks per row
  static constexpr int kChunkBytes = kBN * 128;            // one column block of a 128-row tile
  static constexpr int kTileBytes = kChunks * kChunkBytes; // 128 x D 16-bit tile
  // K and V of pages lie in groups of eight rows, [group][column block][row][128 B], so that one copy brings a page's rows whole (see
  // make_kv_groups_map); all other tiles as [column block][row][128 B].
  static constexpr int kGroupBytes = kChunks * 1024;
  static constexpr int kQOff = 0;
  static constexpr int kRingOff = kQBufs * kTileBytes;
  static constexpr int kCtrlOff = kRingOff + kRing * kTileBytes;
  static constexpr int kTotal = kCtrlOff + static_cast<int>(sizeof(Control));
  static_assert(kTotal + 1024 <= 227 * 1024, "shared memory of an SM (1 KiB for the alignment of the tiles)");
};

// K and V of pages: whether a box (a page's rows, up to a tile's) comes whole, by the 5-D map of make_kv_groups_map, instead of one
// 64-column block at a time.  A box costs the producer a hundred cycles whatever it holds, and the sixteen copies of a tile of
// 16-key pages at head_dim 128, twice a step, were as long as the step: causal, 4 x 2 048 tokens, 32/8 heads 166 -> 156 us, 2 x 4 096 289
// -> 270, 4 x 252 11.8 -> 11.1; 128 queries over 2 048 keys 27.5 -> 26.4.  At head_dim 64 there is one block, and nothing to
// gain; boxes of less than a group would come in pieces (four keys 61 -> 66).
__host__ __device__ constexpr bool group_boxes(int D, int box_rows) { return D > 64 && box_rows >= 8; }

// The waits of a tile.  At head_dim 128 the first look is straight-line code (cycles per tile 1 807 -> 1 785); at 64 the softmax,
// not the chain of waits, is what a step takes, and that costs (4 x 4 096 causal 362 -> 368 us).
template <int D> __device__ __forceinline__ bool tile_wait(uint32_t bar, uint32_t parity) {
  if constexpr (D == 128) return mbar_wait_ready(bar, parity);
  else return mbar_wait(bar, parity);
}

// bounded mbarrier wait whose verdict is uniform over the (converged) warp
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
  const bool ok = mbar_wait(bar, parity);
  return __all_sync(0xffffffffu, ok);
}

__device__ __forceinline__ int blocks_of(int len_q, int rows) { return (len_q + rows - 1) / rows; }

// Ragged layout: warp-cooperative search of the (sequence, row block) that owns flat block index x.
__device__ __forceinline__ bool find_ragged_work(const PrefillParams& p, int x, int rows, int lane, int* out_b, int* out_pair) {
  int base = 0;
  for (int b0 = 0; b0 < p.batch; b0 += 32) {
    const int b = b0 + lane;
    int cnt = 0;
    if (b < p.batch) {
      const long long a = load_index(p.q_indptr, p.indptr_is_i64, b);
      const long long e = load_index(p.q_indptr, p.indptr_is_i64, b + 1);
      const long long n = e > a ? e - a : 0;
      cnt = blocks_of(static_cast<int>(n), rows);
    }
    int incl = cnt;
    for (int o = 1; o < 32; o <<= 1) {
      const int n = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += n;
    }
    const int excl = incl - cnt;
    const bool hit = (x >= base + excl) && (x < base + incl);
    const unsigned mask = __ballot_sync(0xffffffffu, hit);
    if (mask) {
      const int src = __ffs(mask) - 1;
      *out_b = b0 + src;
      *out_pair = x - (base + __shfl_sync(0xffffffffu, excl, src));
      return true;
    }
    base += __shfl_sync(0xffffffffu, incl, 31);
  }
  return false;
}

// An item is decoded in two steps.  locate_item is arithmetic on the launch's sizes and reads no memory, so that a CTA does
// it for its first item before it waits for earlier launches (a microsecond, most of it the first fetch of the code);
// finish_item reads the lengths, and for packed sequences, whose row blocks cannot be placed without them, does all of it.
__device__ __forceinline__ void place_heads(const PrefillParams& p, ItemWork& w, int wblock, int wunit) {
#pragma unroll
  for (int s = 0; s < kSlots; ++s) {
    w.q_head[s] = p.head_pair ? wunit * 2 + s : wunit;
    w.m0[s] = p.head_pair ? wblock * kBM : (wblock * kSlots + s) * kBM;
  }
}

template <bool kParts> __device__ __forceinline__ ItemWork locate_item(const PrefillParams& p, int item) {
  ItemWork w;
  w.valid = false;
  w.len_q = w.len_k = 0;
  w.kv_row0 = 0;
  w.kv_tok0 = 0;
  w.kv_head_coord = 0;
  w.b = 0;
  w.nkv_max = 0;
#pragma unroll
  for (int s = 0; s < kSlots; ++s) {
    w.q_row0[s] = w.out_row0[s] = 0;
    w.q_head[s] = w.q_head_coord[s] = w.m0[s] = w.nkv[s] = 0;
  }
  if (p.layout == B200ATTN_RAGGED) return w;
  const int heads_per_item = p.head_pair ? 2 : 1;
  const int head_units = p.q_heads / heads_per_item;
  const int rows = p.head_pair ? kBM : 2 * kBM;      // query rows an item covers
  // row blocks are the slowest-varying index and, under a causal mask, are handed out heaviest first;
  // the q heads of one KV head are neighbours and share its K/V in L2
  // with a split KV range every (sequence, KV part) pair is a sequence of its own here ("virtual" batch index)
  // (in clusters: the parts of an item are the CTAs of one)
  int part = 0;
  if constexpr (kParts) { part = item % p.cluster_parts; item /= p.cluster_parts; }
  const int per_block = head_units * p.batch * p.kv_split;
  const int nblocks = blocks_of(p.max_q, rows);
  const int blk = item / per_block, rest = item - blk * per_block;
  const int wblock = p.is_causal ? (nblocks - 1 - blk) : blk;
  const int wunit = rest % head_units;
  const int vb = rest / head_units;                    // virtual batch index: rows of the partial buffer
  w.valid = true;
  w.b = vb;
  if (p.kv_split > 1) { part = vb % p.kv_split; w.b = vb / p.kv_split; }
  w.kv_tok0 = part * p.kv_split_len;
  place_heads(p, w, wblock, wunit);
  const int kv_head = w.q_head[0] / p.group;
  w.len_q = p.max_q;
#pragma unroll
  for (int s = 0; s < kSlots; ++s) {
    w.q_row0[s] = (static_cast<long long>(w.b) * p.q_heads + w.q_head[s]) * p.max_q;
    w.out_row0[s] = (static_cast<long long>(vb) * p.q_heads + w.q_head[s]) * p.max_q;
  }
  if (p.layout == B200ATTN_DENSE) {
    w.len_k = p.max_kv;
    w.kv_row0 = (static_cast<long long>(w.b) * p.kv_heads + kv_head) * p.max_kv + w.kv_tok0;
  } else {
    w.kv_head_coord = kv_head;
  }
  return w;
}

// Whether the CTAs of a cluster share the sequence's keys; if not the first of them does the item alone.
template <bool kPaged, bool kParts> __device__ __forceinline__ bool finish_item(const PrefillParams& p, ItemWork& w, int item, int lane) {
  bool cut = kParts;
  if (p.layout == B200ATTN_RAGGED) {
    const int heads_per_item = p.head_pair ? 2 : 1;
    const int head_units = p.q_heads / heads_per_item;
    const int rows = p.head_pair ? kBM : 2 * kBM;
    int wb = -1, wblock = 0;
    const int wunit = item % head_units;
    // Under a causal mask the row blocks are handed out from the end of the packed tensor backwards: the later
    // blocks of a sequence are the heavier ones, and the blocks left for the drain of the grid are then the first,
    // light ones of the first sequences (the sizes are not known on the host, so there is no global order by weight).
    const int nflat = p.total_items / head_units;
    const int flat = item / head_units;
    w.valid = find_ragged_work(p, p.is_causal ? nflat - 1 - flat : flat, rows, lane, &wb, &wblock);
    place_heads(p, w, wblock, wunit);
    if (w.valid) {
      w.b = wb;
      const long long qa = load_index(p.q_indptr, p.indptr_is_i64, wb);
      const long long qe = load_index(p.q_indptr, p.indptr_is_i64, wb + 1);
      const long long ka = load_index(p.kv_indptr, p.indptr_is_i64, wb);
      const long long ke = load_index(p.kv_indptr, p.indptr_is_i64, wb + 1);
      w.len_q = static_cast<int>(qe > qa ? qe - qa : 0);
      w.len_k = static_cast<int>(ke > ka ? ke - ka : 0);
      w.kv_row0 = ka;
      w.kv_head_coord = w.q_head[0] / p.group;
#pragma unroll
      for (int s = 0; s < kSlots; ++s) { w.q_row0[s] = qa; w.out_row0[s] = qa; w.q_head_coord[s] = w.q_head[s]; }
    }
  } else {
    if (p.layout == B200ATTN_PAGED) {
      long long n = load_index(p.kv_indptr, p.indptr_is_i64, w.b);
      const long long cap = p.table_stride * static_cast<long long>(p.page_size);
      n = n < 0 ? 0 : (n > cap ? cap : n);
      w.len_k = static_cast<int>(n);
    }
    // Parts in clusters: what the host cut is the longest that a sequence can be.  This one may be shorter, and its items not worth
    // what the parts cost: every CTA of the cluster sees that by the same numbers, and the first takes the whole.  (64 queries over 100
    // keys in a table of 768, 8/2 heads, D 64: cut 11.1 us, not cut 7.4, a launch without clusters 7.3; over 700 in one of 1 536 13.0, 15.2
    // and, cut into parts in the workspace, 16.8.  Short items of a long sequence, under the diagonal, are cut with the others: their
    // parts are through before those are.)
    if constexpr (kParts && kPaged) {
      int tiles = (w.len_k + kBN - 1) / kBN;
      if (p.is_causal) tiles = min(tiles, (w.len_q + kBN - 1) / kBN);
      cut = tiles >= p.cut_tiles;
      if (!cut && w.kv_tok0 > 0) w.len_k = 0;
    }
    if (kParts ? cut : p.kv_split_len > 0) {
      // this item sees the keys [kv_tok0, kv_tok0 + kv_split_len) of the sequence only
      int local = w.len_k - w.kv_tok0;
      local = local < 0 ? 0 : (local > p.kv_split_len ? p.kv_split_len : local);
      w.len_k = local;
    }
  }
  w.nkv_max = 0;
#pragma unroll
  for (int s = 0; s < kSlots; ++s) {
    int n = 0;
    if (w.valid && w.m0[s] < w.len_q) {
      int kv_hi = w.len_k;
      if (p.is_causal) kv_hi = min(kv_hi, min(w.m0[s] + kBM, w.len_q) - w.kv_tok0);
      n = kv_hi > 0 ? (kv_hi + kBN - 1) / kBN : 0;
    }
    w.nkv[s] = n;
    w.nkv_max = max(w.nkv_max, n);
  }
  return cut;
}

// Parts in clusters: what a CTA sends of a strip of sixteen rows, a 16-byte piece per thread and register group: {references,
// sums} of its two rows, then its columns.
template <int D> constexpr int kStripPieces = (1 + D / 8) * 32;
template <int D> __device__ __forceinline__ uint4* peer_strip(unsigned char* smem, int n) {
  // (in clusters of eight a CTA owns two strips, of which seven others send it their parts)
  static_assert(kSoftmaxWarps / 8 * 7 * kStripPieces<D> * 16 <= kRing * SmemPlan<D>::kTileBytes, "the tile buffers hold them");
  return reinterpret_cast<uint4*>(smem + SmemPlan<D>::kRingOff) + n * kStripPieces<D>;
}
// weight of a part whose reference is m beside the largest one (a part that saw no key has -inf)
__device__ __forceinline__ float part_weight(float m, float largest) { return m == -INFINITY ? 0.f : fast_exp2(m - largest); }

// Persistent kernel: one CTA per SM; work items are drawn from a global counter (heaviest first).
// The producer warp is also the scheduler: it publishes item indices through a 2-deep ring, so it can fetch Q
// and the first K/V tiles of the next item while the other roles finish the current one.
// kPaged: the instantiation launched for paged K/V; only it carries the block-table read-ahead of the producer (in
// the dense / ragged kernel that code, though never run, cost 1 % on the dense benchmark configuration).  The other
// layout checks stay run-time checks.  kParts: the one launched in clusters that share an item (its epilogue costs the others
// registers; at the cap of 96 the forms for head_dim 128 spill, 8 bytes dense and 16 over pages.  That is not what they wait for: a
// build whose form for 64 spilled 72 took 10.48 us for 512 causal tokens, the present one, which spills none, 10.46).
template <typename T, int D, typename OutT, bool kPaged, bool kParts>
__global__ void __launch_bounds__(kThreads, 1)
prefill_kernel(const __grid_constant__ CUtensorMap tm_q, const __grid_constant__ CUtensorMap tm_k,
               const __grid_constant__ CUtensorMap tm_v, const PrefillParams p) {
  using Plan = SmemPlan<D>;
  extern __shared__ unsigned char smem_raw[];
  // 128-byte-swizzled tiles need 1024-byte alignment
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  Control* ctrl = reinterpret_cast<Control*>(smem + Plan::kCtrlOff);
  const uint32_t smem_base = smem_u32(smem);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

  // The scheduler / producer warp sets the barriers up itself and goes straight on to draw and decode its first item
  // and to issue the first copies: it only arrives at the start-up barrier, it does not wait there for the TMEM
  // allocation of the MMA warp (it never touches tensor memory).  Everybody else waits until both are done.
  if (warp == kProducerWarp) {
    if (lane == 0) {
      for (int i = 0; i < kQBufs; ++i) { mbar_init(smem_u32(&ctrl->q_full[i]), 1); mbar_init(smem_u32(&ctrl->q_empty[i]), 1); }
      for (int i = 0; i < kStages; ++i) { mbar_init(smem_u32(&ctrl->kv_full[i]), 1); mbar_init(smem_u32(&ctrl->kv_empty[i]), 1); }
      for (int s = 0; s < kSlots; ++s) {
        mbar_init(smem_u32(&ctrl->s_full[s]), 1);
        mbar_init(smem_u32(&ctrl->p_ready[s]), 8);         // one arrival per softmax warp of the slot
        mbar_init(smem_u32(&ctrl->o_done[s]), 1);
      }
      mbar_init(smem_u32(&ctrl->drained), 1);
      for (int i = 0; i < 2; ++i) {
        mbar_init(smem_u32(&ctrl->sched_full[i]), 1);
        mbar_init(smem_u32(&ctrl->sched_empty[i]), kSoftmaxWarps + 1);
      }
      ctrl->abort_flag = 0;
      ctrl->sched_item[0] = ctrl->sched_item[1] = -1;
      mbar_fence_init();
    }
    __syncwarp();
    named_bar_arrive(1, kThreads);
  } else {
    // ---------------- TMEM allocation (MMA warp owns it) ----------------
    if (warp == kMmaWarp) {
      tmem_alloc(smem_u32(&ctrl->tmem_base), 512);
      tmem_relinquish();
    }
    tc_fence_before();
    named_bar_sync(1, kThreads);
    tc_fence_after();
    // (by the MMA warp, once this CTA holds its tensor memory: a later kernel's CTA that took it first would wait for this
    // grid while this grid waits for it)
    if (warp == kMmaWarp) ptx::grid_dep_launch_dependents();
  }
  const uint32_t tmem = warp == kProducerWarp ? 0u : ctrl->tmem_base;   // (the producer never uses it)
  volatile int* abort_flag = &ctrl->abort_flag;
  // (the host knows the lengths of dense tensors: what it has cut is cut)
  constexpr bool kMayBeWhole = kParts && kPaged;
  // Parts in clusters: every warp of the cluster takes part in two barriers (at the end of this kernel) whatever happens, so that none
  // can wait for one that is not coming.  Where the item is not cut there is nothing to meet for: the warps arrive early and
  // find the barriers completed later (both at the end cost that item 1.0 us, both at its start 1.3, as placed 0.1).
  auto meet_arrive = [] { __syncwarp(); cluster_arrive_relaxed(); };
  auto meet_again = [] { __syncwarp(); cluster_wait(); cluster_arrive_relaxed(); };
  int met = 0;         // halves of the two barriers that this warp has been through

  if (warp == kProducerWarp) {
    // =========================== scheduler + TMA producer ===========================
    if (lane == 0) { prefetch_tensormap(&tm_q); prefetch_tensormap(&tm_k); prefetch_tensormap(&tm_v); }
    // the first item of a CTA is its own index (the grid never exceeds the item count); later ones are drawn
    ItemWork w = locate_item<kParts>(p, static_cast<int>(blockIdx.x));
    // The first tiles of a dense item start for L2 here, while this CTA waits for the launches in front: where they lie follows from the
    // arguments alone, and bringing lines into L2 reads nothing that a later write would not replace there.  (3 x 522 causal tokens, 32/8
    // heads, 18.5 -> 18.3 us, 16 x 600 92.8 -> 92.0.)
    if (!kPaged && p.layout == B200ATTN_DENSE && p.max_kv > 0 && lane == 0) {
      const int kv_row = static_cast<int>(w.kv_row0);
      tma_prefetch_4d(&tm_q, 0, static_cast<int>(w.q_row0[0] + w.m0[0]), 0, w.q_head_coord[0]);
      tma_prefetch_4d(&tm_k, 0, kv_row, 0, w.kv_head_coord);
      tma_prefetch_4d(&tm_q, 0, static_cast<int>(w.q_row0[1] + w.m0[1]), 0, w.q_head_coord[1]);
      tma_prefetch_4d(&tm_v, 0, kv_row, 0, w.kv_head_coord);
    }
    // everything the other warps read or write outside this CTA follows an item published or a tile loaded below
    ptx::grid_dep_wait();
    bool ok = true;
    // Paged K/V with at most 32 boxes per tile: the warp holds the raw block-table entries of 32 boxes of the item, one per
    // lane, for K and for V, and those of the next 32, read when the first became current, so that no table read stands
    // between "stage free" and "copies issued" (the ring is only two pairs deep).  Against a read per pair, one pair ahead,
    // causal with 16-key pages: 4 x 2 048 tokens, 32/8 heads, head_dim 128 187 -> 165 us, 2 x 4 096 325 -> 280, 5 x 8 181
    // at head_dim 64 600 -> 523 (dense K/V: 146, 255, 503).  (Plain registers: an array indexed by a loop counter would
    // live in local memory.)
    constexpr int kNoPage = static_cast<int>(0x80000000u);
    const int box_shift = kPaged ? 31 - __clz(p.box_rows) : 0;
    const int pf_boxes = kPaged ? kBN >> box_shift : 0;
    const bool pf = kPaged && pf_boxes <= 32;
    const bool page_pow2 = (p.page_size & (p.page_size - 1)) == 0;
    const int page_shift = 31 - __clz(p.page_size);
    int pg_k = kNoPage, pg_v = kNoPage, pg_k_next = kNoPage, pg_v_next = kNoPage;
    int pair_e = 0;       // K/V pairs issued so far, across items
    int q_uses = 0;       // Q tiles issued (or skipped) so far
    int pair_lo = 0;      // first pair of the current item
    // where row r of a tile of pages lies, and whether a box comes in one copy
    auto row_dst = [](int r) -> int { return Plan::kChunks == 1 ? r * 128 : (r >> 3) * Plan::kGroupBytes + (r & 7) * 128; };
    const bool whole_boxes = group_boxes(D, p.box_rows);
    auto first_pages = [&](const int* table, const ItemWork& it) -> int {
      const long long tg = static_cast<long long>(lane << box_shift) + it.kv_tok0;
      const long long lp = page_pow2 ? tg >> page_shift : tg / p.page_size;
      return lp < p.table_stride ? __ldcg(table + static_cast<long long>(it.b) * p.table_stride + lp) : kNoPage;
    };
    for (int k = 0; ok; ++k) {
      if (k >= 2) {
        ok = warp_wait(smem_u32(&ctrl->sched_empty[k & 1]), ((k >> 1) - 1) & 1);
        if (!ok || *abort_flag) { ok = false; break; }
      }
      int item = -1;
      bool cut = kParts;
      if (lane == 0) {
        item = k == 0 ? static_cast<int>(blockIdx.x) : static_cast<int>(gridDim.x) + atomicAdd(p.work_counter, 1);
        if (item >= p.total_items) item = -1;
      }
      item = __shfl_sync(0xffffffffu, item, 0);
      if (item >= 0) {
        if (k > 0) w = locate_item<kParts>(p, item);
        // (the entries of a table row may be read before the sequence's length is known: which of them count is decided later)
        if (pf) {
          pg_k = first_pages(p.k_table, w);
          pg_v = first_pages(p.v_table, w);
        }
        cut = finish_item<kPaged, kParts>(p, w, item, lane);
      }
      if (lane == 0) {
        if (item >= 0) ctrl->sched_work[k & 1] = w;
        if (kMayBeWhole && item >= 0) ctrl->cut = cut;
        ctrl->sched_item[k & 1] = item;
        mbar_arrive(smem_u32(&ctrl->sched_full[k & 1]));
      }
      if (item < 0) break;
      if (kMayBeWhole && !cut) { meet_arrive(); met = 1; }
      const int* vtab = kPaged ? p.v_table + static_cast<long long>(w.b) * p.table_stride : nullptr;
      const int* ktab = kPaged ? p.k_table + static_cast<long long>(w.b) * p.table_stride : nullptr;
      auto read_page = [&](const int* tab, int first_box) -> int {
        const int t = (first_box + lane) << box_shift, tg = t + w.kv_tok0;
        return t < w.len_k ? __ldcg(tab + (page_pow2 ? tg >> page_shift : tg / p.page_size)) : kNoPage;
      };
      // (a cache without a whole page: no entry can be right, and the tiles have no boxes whose entries would be checked)
      if (pf && p.num_pages <= 0 && w.nkv_max > 0 && lane == 0) p.header[0] = DEV_ERR_PAGE_RANGE;
      if (pf && w.nkv_max > 0) {
        if (w.len_k > (32 << box_shift)) {
          pg_k_next = read_page(ktab, 32);
          pg_v_next = read_page(vtab, 32);
        }
      }
      // Q tile of slot s: use 2 k + s of the three Q buffers, so the first tile of an item never waits for the item before
      // it, and the second only for that item's first slot
      auto load_q = [&](int s) -> bool {
        const int use = 2 * k + s, buf = use % kQBufs, n = use / kQBufs;
        if (n > 0 && (!warp_wait(smem_u32(&ctrl->q_empty[buf]), (n - 1) & 1) || *abort_flag)) return false;
        if (lane == 0) {
          const uint32_t bar = smem_u32(&ctrl->q_full[buf]);
          if (w.nkv[s] > 0) {
            mbar_arrive_expect_tx(bar, Plan::kTileBytes);
            tma_load_4d(smem_base + Plan::kQOff + buf * Plan::kTileBytes, &tm_q, bar, 0, static_cast<int>(w.q_row0[s] + w.m0[s]), 0,
                        w.q_head_coord[s]);
          } else {
            mbar_arrive(bar);   // keeps one q_full phase per use
          }
        }
        q_uses = use + 1;
        __syncwarp();
        return true;
      };
      if (k >= 1 && lane == 0 && w.nkv[1] > 0) {
        // pull the second slot's Q into L2 now, so the copies issued once its buffer is free only pay an L2 round trip
        tma_prefetch_4d(&tm_q, 0, static_cast<int>(w.q_row0[1] + w.m0[1]), 0, w.q_head_coord[1]);
      }
      ok = load_q(0);
      if (!ok) break;
      if (w.nkv_max == 0) {
        ok = load_q(1);
        if (!ok) break;
      }
      // K/V tiles travel in pairs that share one barrier: pair 0 of an item is K_0 alone, pair j + 1 is {V_j, K_j+1}
      // (the last one V alone).  Stage = pair % 2; its V buffer is ring buffer 2 * stage, its K buffer 2 * stage + 1.
      pair_lo = pair_e;
      const int npairs = w.nkv_max > 0 ? w.nkv_max + 1 : 0;
      for (int pi = 0; pi < npairs && ok; ++pi, ++pair_e) {
        const int stage = pair_e % kStages;
        const int use = pair_e / kStages;
        if (use > 0) {
          ok = warp_wait(smem_u32(&ctrl->kv_empty[stage]), (use - 1) & 1);
          if (!ok || *abort_flag) { ok = false; break; }
        }
        const uint32_t bar = smem_u32(&ctrl->kv_full[stage]);
        const bool has_v = pi >= 1, has_k = pi < w.nkv_max;
        const int jv = pi - 1, jk = pi;               // tile indices of the V and the K of this pair
        const uint32_t vdst = smem_base + Plan::kRingOff + (2 * stage) * Plan::kTileBytes;
        const uint32_t kdst = vdst + Plan::kTileBytes;
        if (!kPaged) {
          if (lane == 0) {
            mbar_arrive_expect_tx(bar, (has_v ? Plan::kTileBytes : 0) + (has_k ? Plan::kTileBytes : 0));
            if (has_v) tma_load_4d(vdst, &tm_v, bar, 0, static_cast<int>(w.kv_row0 + static_cast<long long>(jv) * kBN), 0, w.kv_head_coord);
            if (has_k) tma_load_4d(kdst, &tm_k, bar, 0, static_cast<int>(w.kv_row0 + static_cast<long long>(jk) * kBN), 0, w.kv_head_coord);
          }
        } else if (pf) {
          // one box per lane and operand from the entries read ahead
          if (has_k && pi > 0 && ((pi * pf_boxes) & 31) == 0) {
            pg_k = pg_k_next;
            pg_k_next = read_page(ktab, pi * pf_boxes + 32);
          }
          if (jv > 0 && ((jv * pf_boxes) & 31) == 0) {
            pg_v = pg_v_next;
            pg_v_next = read_page(vtab, jv * pf_boxes + 32);
          }
          auto boxes_of = [&](int t0) -> int { return min(pf_boxes, (w.len_k - t0 + p.box_rows - 1) >> box_shift); };
          const int nk = has_k && p.num_pages > 0 ? boxes_of(jk * kBN) : 0;
          const int nv = has_v && p.num_pages > 0 ? boxes_of(jv * kBN) : 0;
          auto row_of = [&](int page, int t) -> int {
            // an entry outside the cache is reported and replaced by page 0: never dereferenced, output stays finite
            const bool bad = page < 0 || page >= p.num_pages;
            if (bad) p.header[0] = DEV_ERR_PAGE_RANGE;
            const int tg = t + w.kv_tok0;
            return (bad ? 0 : page) * p.page_size + (page_pow2 ? tg & (p.page_size - 1) : tg % p.page_size);
          };
          const int ek = __shfl_sync(0xffffffffu, pg_k, (jk * pf_boxes + lane) & 31);
          const int ev = __shfl_sync(0xffffffffu, pg_v, (jv * pf_boxes + lane) & 31);
          const int rk = lane < nk ? row_of(ek, jk * kBN + (lane << box_shift)) : -1;
          const int rv = lane < nv ? row_of(ev, jv * kBN + (lane << box_shift)) : -1;
          if (lane == 0) mbar_arrive_expect_tx(bar, static_cast<uint32_t>(nk + nv) * p.box_rows * 128 * Plan::kChunks);
          __syncwarp();
          const int dst = row_dst(lane << box_shift);
          if (whole_boxes) {
            if (rv >= 0) tma_load_5d(vdst + dst, &tm_v, bar, 0, 0, 0, rv >> 3, w.kv_head_coord);
            if (rk >= 0) tma_load_5d(kdst + dst, &tm_k, bar, 0, 0, 0, rk >> 3, w.kv_head_coord);
          } else {
            for (int c = 0; c < Plan::kChunks; ++c) {
              if (rv >= 0) tma_load_3d(vdst + dst + c * 1024, &tm_v, bar, c * 64, w.kv_head_coord, rv);
              if (rk >= 0) tma_load_3d(kdst + dst + c * 1024, &tm_k, bar, c * 64, w.kv_head_coord, rk);
            }
          }
        } else {
          // one box of `box_rows` tokens per lane per round and operand; only pages that exist are fetched
          const int boxes = kBN / p.box_rows;
          int rows_v[4], rows_k[4];
          int nmine = 0;
          int count = 0;
          auto page_row = [&](const int* table, int t) -> int {
            if (t >= w.len_k) return -1;
            const int tg = t + w.kv_tok0;          // position in the whole sequence
            const int lp = tg / p.page_size;
            const int page = __ldcg(table + lp);
            // an entry outside the cache is reported and replaced by page 0: never dereferenced, output stays finite
            const bool bad = page < 0 || page >= p.num_pages;
            if (bad) p.header[0] = DEV_ERR_PAGE_RANGE;
            return p.num_pages > 0 ? (bad ? 0 : page) * p.page_size + (tg - lp * p.page_size) : -1;
          };
          for (int i = lane; i < boxes; i += 32) {
            const int rv = has_v ? page_row(vtab, jv * kBN + i * p.box_rows) : -1;
            const int rk = has_k ? page_row(ktab, jk * kBN + i * p.box_rows) : -1;
            rows_v[nmine] = rv;
            rows_k[nmine] = rk;
            ++nmine;
            count += (rv >= 0) + (rk >= 0);
          }
          for (int o = 16; o > 0; o >>= 1) count += __shfl_xor_sync(0xffffffffu, count, o);
          if (lane == 0) mbar_arrive_expect_tx(bar, static_cast<uint32_t>(count) * p.box_rows * 128 * Plan::kChunks);
          __syncwarp();
          int kk = 0;
          for (int i = lane; i < boxes; i += 32, ++kk) {
            const int rv = rows_v[kk], rk = rows_k[kk], dst = row_dst(i * p.box_rows);    // (fewer than four rows)
            for (int c = 0; c < Plan::kChunks; ++c) {
              if (rv >= 0) tma_load_3d(vdst + dst + c * 1024, &tm_v, bar, c * 64, w.kv_head_coord, rv);
              if (rk >= 0) tma_load_3d(kdst + dst + c * 1024, &tm_k, bar, c * 64, w.kv_head_coord, rk);
            }
          }
        }
        if (pi == 0) ok = load_q(1);
        if (kMayBeWhole && pi == 1 && met == 1) { meet_again(); met = 3; }
      }
    }
    if (!ok) {
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
      // drain: wait (bounded) for the copies still in flight before the CTA may exit
      for (int e = max(pair_lo, pair_e - kStages); e < pair_e; ++e) mbar_wait(smem_u32(&ctrl->kv_full[e % kStages]), (e / kStages) & 1);
      for (int u = max(0, q_uses - kQBufs); u < q_uses; ++u) mbar_wait(smem_u32(&ctrl->q_full[u % kQBufs]), (u / kQBufs) & 1);
    }
    if (lane == 0) {
      // This CTA draws no more items.  The last CTA to get here puts both counters back to zero for the next
      // launch on this workspace (every other CTA's draws are ordered before its own increment by the fence).
      __threadfence();
      if (atomicAdd(p.work_counter + 1, 1) == static_cast<int>(gridDim.x) - 1) {
        atomicExch(p.work_counter, 0);
        atomicExch(p.work_counter + 1, 0);
      }
    }
  } else if (warp == kMmaWarp) {
    // =========================== MMA issuer ===========================
    constexpr int kFmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    constexpr uint32_t idesc_s = make_idesc_f16(kBM, kBN, kFmt, 0);
    constexpr uint32_t idesc_o = make_idesc_f16(kBM, D, kFmt, 1);
    const uint32_t tmem_S[kSlots] = {tmem, tmem + kBN};
    const uint32_t tmem_O[kSlots] = {tmem + 2 * kBN, tmem + 2 * kBN + D};
    bool ok = true;
    // Descriptor words are prepared once: the high words never change, the low words are a base
    // (start address >> 4) plus small constants, so issuing one MMA costs the single thread a few adds.
    constexpr int kGroup = kPaged ? Plan::kGroupBytes : 1024;           // between groups of eight keys
    constexpr int kBlock = kPaged ? 1024 : Plan::kChunkBytes;           // between column blocks
    const uint64_t qdesc = make_smem_desc_sw128(smem_base, 16);                    // K-major operands (Q, K)
    const uint64_t kdesc = make_smem_desc_sw128(smem_base, 16, kGroup);
    const uint64_t vdesc = make_smem_desc_sw128(smem_base, kBlock, kGroup);        // MN-major operand (V)
    int pair_base = 0;            // pair that holds K_0 of the current item (pair j + 1 holds V_j and K_j+1)
    // per-slot state as scalars (an array indexed by the slot would live in local memory)
    int tiles_done0 = 0, tiles_done1 = 0;       // score tiles issued per slot so far (barrier phases run across items)
    bool pre_issued0 = false, pre_issued1 = false;   // first score tile of the coming item already issued
    // This warp's instructions between P and the commit of the next scores are part of every step's chain.  Inside the tile loop a
    // wait that ran out is noticed after the MMAs behind it have been issued (on whatever is there, into this CTA's own tensor
    // memory; should that be read out for an item's product, the teardown takes it back), one vote for three waits: cycles per 128 x 128 tile and SM, 8 x 2 048 without a mask 1 840 -> 1 807, 2 x 2 048 causal
    // 2 144 -> 2 103 (all-zero inputs, so at full clock); at the power limit 74.7 -> 73.9 us.  Tried beside it: the code once per stage
    // of the ring, so that descriptors are constants in uniform registers (9 cycles, but 64 / 8 heads of 22 tokens took 2 % longer
    // with it), the commit of the P V behind that of the scores (nothing).
    bool good = true;
    auto pair_full_wait = [&](int pr) -> bool {
      return warp_wait(smem_u32(&ctrl->kv_full[pr % kStages]), (pr / kStages) & 1);
    };
    // The warp stays converged while it issues: every lane runs the descriptor arithmetic, one elected lane
    // issues the tensor-core instructions and their commits.
    const uint32_t lead = elect_one();
    auto uniform = [](uint64_t x) -> uint64_t {
      const uint32_t lo = __shfl_sync(0xffffffffu, static_cast<uint32_t>(x), 0), hi = __shfl_sync(0xffffffffu, static_cast<uint32_t>(x >> 32), 0);
      return (static_cast<uint64_t>(hi) << 32) | lo;
    };
    // operand descriptors of the K and the V buffer of a pair's stage
    auto k_desc_of = [&](int pr) -> uint64_t {
      return uniform(kdesc + static_cast<uint64_t>((Plan::kRingOff + (2 * (pr % kStages) + 1) * Plan::kTileBytes) >> 4));
    };
    auto v_desc_of = [&](int pr) -> uint64_t {
      return uniform(vdesc + static_cast<uint64_t>((Plan::kRingOff + (2 * (pr % kStages)) * Plan::kTileBytes) >> 4));
    };
    auto q_desc_of = [&](int buf) -> uint64_t {
      return uniform(qdesc + static_cast<uint64_t>((Plan::kQOff + buf * Plan::kTileBytes) >> 4));
    };
    auto issue_s = [&](int s, uint64_t qa, uint64_t kb) {
      // S_s = Q_s K^T : K-major A and B, D/16 k-steps
      mma_ss_batch<D / 16, kBlock / 16>(tmem_S[s], qa, kb, idesc_s, 0u, lead);
      mma_commit_lead(smem_u32(&ctrl->s_full[s]), lead);
    };
    auto issue_pv = [&](int s, uint64_t vb, bool first) {
      // O_s (+)= P_s V : A = packed 16-bit P, 32 TMEM columns at the start of each 64-column half of the S tile;
      // B = V, MN-major
      mma_ts_batch8<2 * kGroup / 16>(tmem_O[s], tmem_S[s], vb, idesc_o, first ? 0u : 1u, lead);
      mma_commit_lead(smem_u32(&ctrl->o_done[s]), lead);
    };

    // First score tile of slot s of item kk, whose K_0 is pair `pr`: once its Q tile and K_0 have landed.  A slot without
    // tiles only takes its turn at the Q buffer.
    auto start_slot = [&](int s, int kk, int nkv_s, int pr) -> bool {
      const int use = 2 * kk + s, buf = use % kQBufs;
      if (!warp_wait(smem_u32(&ctrl->q_full[buf]), (use / kQBufs) & 1)) return false;
      if (nkv_s > 0) {
        if (!pair_full_wait(pr)) return false;
        tc_fence_after();
        issue_s(s, q_desc_of(buf), k_desc_of(pr));
        if (nkv_s == 1) mma_commit_lead(smem_u32(&ctrl->q_empty[buf]), lead);    // the slot's last use of its Q tile
      } else if (lane == 0) {
        mbar_arrive(smem_u32(&ctrl->q_empty[buf]));
      }
      __syncwarp();
      return true;
    };

    for (int k = 0; ok; ++k) {
      ok = warp_wait(smem_u32(&ctrl->sched_full[k & 1]), (k >> 1) & 1);
      if (!ok || *abort_flag) { ok = false; break; }
      const int item = ctrl->sched_item[k & 1];
      if (item < 0) break;
      const ItemWork& wr = ctrl->sched_work[k & 1];
      if (kMayBeWhole && !ctrl->cut) { meet_arrive(); met = 1; }
      const int nkv0 = wr.nkv[0], nkv1 = wr.nkv[1], nkv_max = wr.nkv_max, len_k = wr.len_k;
      const int qbuf0 = (2 * k) % kQBufs, qbuf1 = (2 * k + 1) % kQBufs;
      const uint64_t qd0 = q_desc_of(qbuf0), qd1 = q_desc_of(qbuf1);
      // (slots whose first score tile was already issued while the previous item finished are skipped)
      if (!pre_issued0) ok = start_slot(0, k, nkv0, pair_base);
      if (ok && !pre_issued1) ok = start_slot(1, k, nkv1, pair_base);
      if (!ok) break;
      if (nkv_max > 0) mma_commit_lead(smem_u32(&ctrl->kv_empty[pair_base % kStages]), lead);
      if (kMayBeWhole && met == 1) { meet_again(); met = 3; }
      pre_issued0 = pre_issued1 = false;
      for (int j = 0; j < nkv_max && ok; ++j) {
        const int pr = pair_base + 1 + j;     // the pair {V_j, K_j+1}
        const bool last_iter = j + 1 == nkv_max;
        // Everything that does not depend on the softmax warps is waited for and computed before their P is: the
        // pair {V_j, K_j+1} (one barrier; in steady state loaded long ago) and the operand descriptors.  Between a slot's
        // P and its two batches of MMAs the warp then only runs the issue.
        good = tile_wait<D>(smem_u32(&ctrl->kv_full[pr % kStages]), (pr / kStages) & 1);
        {
          const int valid = len_k - j * kBN;
          if (valid < kBN) {
            // keys past the sequence end carry P == 0 but their V rows may hold anything (stale
            // shared memory, the next sequence, poisoned page tails): zero them so 0 * x stays 0
            unsigned char* vbuf = smem + Plan::kRingOff + (2 * (pr % kStages)) * Plan::kTileBytes;
            const int first = valid > 0 ? valid : 0;
            if constexpr (kGroup == 1024) {
              const int n16 = (kBN - first) * 8;  // 16-byte pieces per column block
              for (int c = 0; c < Plan::kChunks; ++c) {
                // (written out for this case: with the indices of the other one, never run in a whole tile, 3 x 8 192 causal tokens,
                // 32/8 heads, head_dim 64, took 1 120 us instead of 1 064)
                uint4* dst = reinterpret_cast<uint4*>(vbuf + c * kBlock + first * 128);
                for (int i = lane; i < n16; i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
              }
            } else {
              // the rest of a group, then whole groups, which lie one behind the other (piece by piece, with an index for each, 7 x 20 tokens
              // took 8.8 us instead of 8.2)
              for (int c = 0; c < Plan::kChunks; ++c) {
                uint4* dst = reinterpret_cast<uint4*>(vbuf + c * kBlock + (first >> 3) * kGroup + (first & 7) * 128);
                for (int i = lane; i < (-first & 7) * 8; i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
              }
              uint4* dst = reinterpret_cast<uint4*>(vbuf + ((first + 7) >> 3) * kGroup);
              for (int i = lane; i < (kBN / 8 - ((first + 7) >> 3)) * (kGroup / 16); i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
            }
            fence_proxy_async_smem();
            __syncwarp();
          }
        }
        const uint64_t vb = v_desc_of(pr);
        const uint64_t kb = k_desc_of(pr);
        auto slot_step = [&](const int s, const int nkv_s, const int qbuf, const uint64_t qd, int& tiles_done) {
          if (j >= nkv_s) return;
          // (P of an item's first tile also says that the previous item's O has been read out: the softmax warps hand it
          // over after that)
          if (!tile_wait<D>(smem_u32(&ctrl->p_ready[s]), tiles_done & 1)) good = false;
          tc_fence_after();
          issue_pv(s, vb, j == 0);
          if (j + 1 < nkv_s) {
            issue_s(s, qd, kb);
            if (j + 2 == nkv_s) mma_commit_lead(smem_u32(&ctrl->q_empty[qbuf]), lead);   // the slot's last use of its Q tile
          }
          ++tiles_done;
        };
        if (!last_iter) {
          slot_step(0, nkv0, qbuf0, qd0, tiles_done0);
          slot_step(1, nkv1, qbuf1, qd1, tiles_done1);
          // V_j and K_j+1 have been read by everything that will read them: one commit releases the stage
          mma_commit_lead(smem_u32(&ctrl->kv_empty[pr % kStages]), lead);
          ok = __all_sync(0xffffffffu, good);
        } else {
          // The item's last tile: each slot's first score tile of the next item is issued right behind its final PV, so
          // that the tensor cores have work while the softmax warps read O out.  What is waited for here (the next item
          // published, its Q tiles and its first K tile) depends only on work this warp has already issued: the first
          // slot's Q has a buffer of its own, the second's takes the one this item's first slot gave back a tile ago.
          slot_step(0, nkv0, qbuf0, qd0, tiles_done0);
          ok = __all_sync(0xffffffffu, good) && warp_wait(smem_u32(&ctrl->sched_full[(k + 1) & 1]), ((k + 1) >> 1) & 1);
          if (!ok) break;
          const bool more = ctrl->sched_item[(k + 1) & 1] >= 0;
          const ItemWork& wn = ctrl->sched_work[(k + 1) & 1];
          if (more) {
            ok = start_slot(0, k + 1, wn.nkv[0], pair_base + nkv_max + 1);
            if (!ok) break;
          }
          slot_step(1, nkv1, qbuf1, qd1, tiles_done1);
          ok = __all_sync(0xffffffffu, good);
          if (!ok) break;
          mma_commit_lead(smem_u32(&ctrl->kv_empty[pr % kStages]), lead);
          if (more) {
            ok = start_slot(1, k + 1, wn.nkv[1], pair_base + nkv_max + 1);
            if (!ok) break;
          }
          pre_issued0 = pre_issued1 = more;
        }
      }
      if (nkv_max > 0) pair_base += nkv_max + 1;
      if (lane == 0 && ok) mbar_arrive(smem_u32(&ctrl->sched_empty[k & 1]));      // (else the teardown reads the slot)
      __syncwarp();
    }
    if (!ok) {
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
      // (what has been issued ends before tensor memory is given back)
      mma_commit_lead(smem_u32(&ctrl->drained), lead);
      warp_wait(smem_u32(&ctrl->drained), 0);
    }
  } else if (warp < kSoftmaxWarps) {
    // =========================== softmax warps ===========================
    // Warp w serves slot w / 8, the TMEM lane quadrant w % 4 (the only lanes it may touch) and, inside the quadrant,
    // the sixteen query rows 16 h .. 16 h + 15 with h = (w / 4) % 2.  Tensor memory is read in the 16x256b layout:
    // thread t holds the columns 8 i + 2 (t % 4) + {0, 1} (i = 0 .. 15) of row A = t / 4 and of row B = A + 8, so the
    // 128 scores of a row live in the four threads of a quad and row maxima and sums are two shuffles away: no
    // exchange through shared memory, no barrier inside a tile.
    const int s = warp >> 3;
    const int qd = warp & 3;
    const int h = (warp >> 2) & 1;
    const int q = lane & 3;
    const int rowA = qd * 32 + h * 16 + (lane >> 2);    // 0..127 inside the slot; row B = row A + 8
    const uint32_t lane_off = static_cast<uint32_t>(qd * 32 + h * 16) << 16;
    const uint32_t tS = tmem + s * kBN + lane_off;
    const uint32_t tO = tmem + 2 * kBN + s * D + lane_off;
    const float sl2 = p.scale_log2;
    int tile_cnt = 0;     // score tiles of this slot consumed so far (barrier phases run across items)
    bool ok = true;
    // The epilogue of an item runs while the first score tile of the slot's next item is computed.
    bool out_acc = false;     // the item has an accumulator (false: the slot had no keys, the output is zero)
    int out_phase = 0;       // o_done phase of its last PV
    int out_rows = 0;        // rows of the tile that exist in the sequence
    float out_la = 0.f, out_lb = 0.f;   // row sums of rows A and B
    float out_ma = -INFINITY, out_mb = -INFINITY;   // ... and their references (kept for a merge)
    long long out_off = 0;   // element offset of row A's first output column
    long long out_stride = 0;   // elements between consecutive rows of the output
    bool seen = false, cut = true;      // (parts in clusters; a CTA that never saw its item sends NaN)
    constexpr bool k16 = !std::is_same<OutT, float>::value;
    auto quad_max = [](float v) {
      v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 1));
      return fmaxf(v, __shfl_xor_sync(0xffffffffu, v, 2));
    };
    auto quad_sum = [](float v) {
      v += __shfl_xor_sync(0xffffffffu, v, 1);
      return v + __shfl_xor_sync(0xffffffffu, v, 2);
    };
    // 4 x 4 transpose of two-word items across the four threads of a quad (lane bits 0-1): on return item m of
    // thread q is what item q of thread m was.  x[2m], x[2m+1] are the words of item m.
    auto quad_transpose = [&](uint32_t (&x)[8]) {
      const bool b1 = (lane & 2) != 0, b0 = (lane & 1) != 0;
#pragma unroll
      for (int m = 0; m < 2; ++m) {
#pragma unroll
        for (int wd = 0; wd < 2; ++wd) {
          uint32_t& lo = x[2 * m + wd];
          uint32_t& hi = x[2 * (m + 2) + wd];
          const uint32_t recv = __shfl_xor_sync(0xffffffffu, b1 ? lo : hi, 2);
          if (b1) lo = recv; else hi = recv;
        }
      }
#pragma unroll
      for (int m = 0; m < 4; m += 2) {
#pragma unroll
        for (int wd = 0; wd < 2; ++wd) {
          uint32_t& lo = x[2 * m + wd];
          uint32_t& hi = x[2 * (m + 1) + wd];
          const uint32_t recv = __shfl_xor_sync(0xffffffffu, b0 ? lo : hi, 1);
          if (b0) lo = recv; else hi = recv;
        }
      }
    };
    // kMerge: with the parts that the other CTAs of the cluster have put into this CTA's tile buffers (see the end of the kernel)
    auto write_out = [&](auto merging) -> bool {
      constexpr bool kMerge = decltype(merging)::value;
      if (out_acc && !kMerge) {
        if (!warp_wait(smem_u32(&ctrl->o_done[s]), out_phase)) return false;
      }
      tc_fence_after();
      const int n_peers = kMerge ? p.cluster_parts - 1 : 0;
      const uint4* const strip = kMerge ? peer_strip<D>(smem, warp / p.cluster_parts * n_peers) + lane : nullptr;
      float self_a = 1.f, self_b = 1.f, ref_a = out_ma, ref_b = out_mb;     // weights of this CTA's part; largest references
      if constexpr (kMerge) {
        for (int k = 0; k < n_peers; ++k) {
          const float4 ml = *reinterpret_cast<const float4*>(strip + k * kStripPieces<D>);
          ref_a = fmaxf(ref_a, ml.x);
          ref_b = fmaxf(ref_b, ml.y);
        }
        self_a = part_weight(out_ma, ref_a);
        self_b = part_weight(out_mb, ref_b);
        out_la *= self_a;
        out_lb *= self_b;
        for (int k = 0; k < n_peers; ++k) {
          const float4 ml = *reinterpret_cast<const float4*>(strip + k * kStripPieces<D>);
          out_la += ml.z * part_weight(ml.x, ref_a);
          out_lb += ml.w * part_weight(ml.y, ref_b);
        }
      }
      // (a sum that is no number shows in its own row, also where no part has an accumulator)
      const float inv_a = out_la > 0.f ? 1.f / out_la : kMerge ? 0.f * out_la : 0.f;
      const float inv_b = out_lb > 0.f ? 1.f / out_lb : kMerge ? 0.f * out_lb : 0.f;
      // the 64 columns of block c: rows A and B as tmem_ld_16x256b_x8 gives them
      auto merge_parts = [&](uint32_t (&v)[32], int c) {
        if constexpr (kMerge) {
#pragma unroll
          for (int i = 0; i < 32; ++i) v[i] = __float_as_uint(__uint_as_float(v[i]) * (i & 2 ? self_b : self_a));
          for (int k = 0; k < n_peers; ++k) {
            const uint4* const piece = strip + k * kStripPieces<D>;
            const float4 ml = *reinterpret_cast<const float4*>(piece);
            const float wa = part_weight(ml.x, ref_a), wb = part_weight(ml.y, ref_b);
#pragma unroll
            for (int i = 0; i < 8; ++i) {
              const uint4 x = piece[(1 + c * 8 + i) * 32];
              v[4 * i] = __float_as_uint(fmaf(__uint_as_float(x.x), wa, __uint_as_float(v[4 * i])));
              v[4 * i + 1] = __float_as_uint(fmaf(__uint_as_float(x.y), wa, __uint_as_float(v[4 * i + 1])));
              v[4 * i + 2] = __float_as_uint(fmaf(__uint_as_float(x.z), wb, __uint_as_float(v[4 * i + 2])));
              v[4 * i + 3] = __float_as_uint(fmaf(__uint_as_float(x.w), wb, __uint_as_float(v[4 * i + 3])));
            }
          }
        }
      };
      constexpr int kChunksO = D / 64;
      if constexpr (k16) {
        // 16-bit output: 64 columns of a row are one 128-byte line.  A quad holds 8 consecutive columns per group;
        // transposed inside the quad, every thread owns 32 contiguous bytes and a store instruction writes 8 full
        // lines instead of one piece of 32 different lines.
        uint32_t line[kChunksO][2][8];     // [64-column chunk][row A / row B][32 bytes of the row's line]
#pragma unroll
        for (int c = 0; c < kChunksO; ++c) {
          uint32_t v[32];
          if (out_acc) {
            tmem_ld_16x256b_x8(tO + c * 64, v);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          merge_parts(v, c);
          uint32_t a[8], b[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            a[i] = ElemTraits<T>::pack2(__uint_as_float(v[4 * i]) * inv_a, __uint_as_float(v[4 * i + 1]) * inv_a);
            b[i] = ElemTraits<T>::pack2(__uint_as_float(v[4 * i + 2]) * inv_b, __uint_as_float(v[4 * i + 3]) * inv_b);
          }
          // thread q of the quad holds word q of each 16-byte block i; it ends up with blocks 2q and 2q+1 whole
          quad_transpose(a);
          quad_transpose(b);
#pragma unroll
          for (int m = 0; m < 4; ++m) {
            line[c][0][m] = a[2 * m];  line[c][0][4 + m] = a[2 * m + 1];
            line[c][1][m] = b[2 * m];  line[c][1][4 + m] = b[2 * m + 1];
          }
        }
#pragma unroll
        for (int ab = 0; ab < 2; ++ab) {
          if (rowA + 8 * ab < out_rows) {
#pragma unroll
            for (int c = 0; c < kChunksO; ++c) {
              T* out = static_cast<T*>(p.out) + out_off + ab * 8 * out_stride + c * 64 + q * 16;
              const uint32_t (&u)[8] = line[c][ab];
              if (p.out_align32) {
                st_global_v8(out, u[0], u[1], u[2], u[3], u[4], u[5], u[6], u[7]);
              } else {
                *reinterpret_cast<uint4*>(out) = make_uint4(u[0], u[1], u[2], u[3]);
                *reinterpret_cast<uint4*>(out + 8) = make_uint4(u[4], u[5], u[6], u[7]);
              }
            }
          }
        }
      } else {
        // fp32 output: a thread holds two consecutive columns per group, a quad 32 contiguous bytes of a row
#pragma unroll
        for (int c = 0; c < kChunksO; ++c) {
          uint32_t v[32];
          if (out_acc) {
            tmem_ld_16x256b_x8(tO + c * 64, v);
            tmem_wait_ld();
          } else {
#pragma unroll
            for (int i = 0; i < 32; ++i) v[i] = 0u;
          }
          merge_parts(v, c);
          float* out = static_cast<float*>(p.out) + out_off + c * 64 + q * 2;
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            if (rowA < out_rows)
              *reinterpret_cast<float2*>(out + i * 8) = make_float2(__uint_as_float(v[4 * i]) * inv_a, __uint_as_float(v[4 * i + 1]) * inv_a);
            if (rowA + 8 < out_rows)
              *reinterpret_cast<float2*>(out + 8 * out_stride + i * 8) =
                  make_float2(__uint_as_float(v[4 * i + 2]) * inv_b, __uint_as_float(v[4 * i + 3]) * inv_b);
          }
        }
      }
      return true;
    };
    for (int k = 0; ok; ++k) {
      ok = warp_wait(smem_u32(&ctrl->sched_full[k & 1]), (k >> 1) & 1);
      if (!ok || *abort_flag) { ok = false; break; }
      const int item = ctrl->sched_item[k & 1];
      if (item < 0) break;
      if (kMayBeWhole && !ctrl->cut) { meet_arrive(); meet_again(); }
      // (the few fields needed are read from shared memory where they are used, not held across the tile loop)
      const ItemWork& w = ctrl->sched_work[k & 1];
      const int n = w.nkv[s];
      const int m0s = w.m0[s];
      const int len_k = w.len_k;
      const int row0_abs = m0s + qd * 32 + h * 16 - w.kv_tok0;   // query index of the warp's first row relative to the item's first key
      float m_a = -INFINITY, m_b = -INFINITY;   // exponent references currently baked into O and l
      float l_a = 0.f, l_b = 0.f;               // partial row sums over this thread's columns
      for (int j = 0; j < n; ++j, ++tile_cnt) {
        // (whether the wait ran out is asked with the verdict on the references: a vote of its own is thirty cycles)
        const bool here = tile_wait<D>(smem_u32(&ctrl->s_full[s]), tile_cnt & 1);
        tc_fence_after();
        // Last visible column of the tile for the first and for the last of the warp's sixteen rows (the same for all rows
        // without a causal mask): hidden columns exist only on the tile that holds the sequence end or the diagonal.
        int lo = len_k - 1 - j * kBN, hi = lo;
        if (p.is_causal) { lo = min(lo, row0_abs - j * kBN); hi = min(hi, row0_abs + 15 - j * kBN); }
        uint64_t rs_a = pack_f2(0.f, 0.f), rs_b = pack_f2(0.f, 0.f);
        const uint64_t sl2_2 = pack_f2(sl2, sl2);
        uint64_t nega_2, negb_2;     // minus the exponent references of rows A and B
        auto exp_pair = [&](uint32_t x0, uint32_t x1, uint64_t neg2, uint64_t& rs) -> uint32_t {
          const uint64_t t2 = fma_f2(pack_f2(__uint_as_float(x0), __uint_as_float(x1)), sl2_2, neg2);
          float a, b;
          unpack_f2(t2, a, b);
          const float p0 = fast_exp2(a), p1 = fast_exp2(b);
          rs = add_f2(rs, pack_f2(p0, p1));
          return ElemTraits<T>::pack2(p0, p1);
        };
        // 32 columns of both rows: exponentials, row sums, P as packed 16-bit in the 16x128b layout (the pair of columns
        // 8 i + 2 q + {0, 1} is packed column 4 i + q)
        auto exp_quarter = [&](const uint32_t (&v)[16], uint32_t* pq) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            pq[2 * i] = exp_pair(v[4 * i], v[4 * i + 1], nega_2, rs_a);
            pq[2 * i + 1] = exp_pair(v[4 * i + 2], v[4 * i + 3], negb_2, rs_b);
          }
        };
        float mx_a = -INFINITY, mx_b = -INFINITY;       // maxima over this thread's columns
        auto max_quarter = [&](const uint32_t (&v)[16]) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            mx_a = max3(mx_a, __uint_as_float(v[4 * i]), __uint_as_float(v[4 * i + 1]));
            mx_b = max3(mx_b, __uint_as_float(v[4 * i + 2]), __uint_as_float(v[4 * i + 3]));
          }
        };
        float sum_a, sum_b;     // row sums over this thread's columns
        auto pair_sum = [](uint64_t v) {
          float x, y;
          unpack_f2(v, x, y);
          return x + y;
        };
        // One pass where no row's exponent reference has to move, which is nearly every tile: the
        // scores are exponentiated, as they arrive, against the reference that stands, and the sums, needed anyhow, tell
        // afterwards whether it could stand: no maximum is computed, no exponential waits for one, nothing is exchanged
        // between threads, and the tile is read from tensor memory once.  P stays in registers until the verdict: if a row
        // has to move, the scores are still there for the two passes below.
        // An item's first tile is read once more for its maximum: the largest weight is then exactly one.  (Against the maximum of
        // the first 32 columns it was rounded like all others, and outputs came out up to 1 % further from 64 bits.)
        bool done = false;
        // (columns hidden from a row are -inf)
        auto mask_quarter = [&](uint32_t (&v)[16], int c) {
          const int ta = min(len_k - 1, p.is_causal ? row0_abs + (lane >> 2) : 0x7fffffff) - j * kBN - c * 32 - 2 * q;
          const int tb = min(len_k - 1, p.is_causal ? row0_abs + (lane >> 2) + 8 : 0x7fffffff) - j * kBN - c * 32 - 2 * q;
#pragma unroll
          for (int i = 0; i < 4; ++i) {
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              v[4 * i + e] = (8 * i + e > ta) ? 0xff800000u : v[4 * i + e];           // -inf
              v[4 * i + 2 + e] = (8 * i + e > tb) ? 0xff800000u : v[4 * i + 2 + e];
            }
          }
        };
        if (lo >= kBN - 1) {
          uint32_t pk[2][16];
          uint32_t v0[16], v1[16];
          if (j == 0) {
#pragma unroll 1
            for (int c = 0; c < 4; c += 2) {
              tmem_ld_16x256b_x4(tS + c * 32, v0);
              tmem_ld_16x256b_x4(tS + c * 32 + 32, v1);
              tmem_wait_ld_regs(v0);
              tmem_wait_ld_regs(v1);
              max_quarter(v0);
              max_quarter(v1);
            }
            m_a = quad_max(mx_a) * sl2;
            m_b = quad_max(mx_b) * sl2;
          }
          tmem_ld_16x256b_x4(tS, v0);
          tmem_wait_ld_regs(v0);
          tmem_ld_16x256b_x4(tS + 32, v1);
          // (a row without a reference yet has -inf here: its sum is then no number and the verdict is no)
          nega_2 = pack_f2(-m_a, -m_a);
          negb_2 = pack_f2(-m_b, -m_b);
          exp_quarter(v0, pk[0]);
          tmem_wait_ld_regs(v1);
          tmem_ld_16x256b_x4(tS + 64, v0);
          exp_quarter(v1, pk[0] + 8);
          tmem_wait_ld_regs(v0);
          tmem_ld_16x256b_x4(tS + 96, v1);
          exp_quarter(v0, pk[1]);
          tmem_wait_ld_regs(v1);
          exp_quarter(v1, pk[1] + 8);
          sum_a = pair_sum(rs_a);
          sum_b = pair_sum(rs_b);
          done = __all_sync(0xffffffffu, here && sum_a <= kMaxPartialSum && sum_b <= kMaxPartialSum);   // (false for NaN)
          if (done) {
            tmem_st_16x128b_x8(tS, pk[0]);
            tmem_st_16x128b_x8(tS + ptx::kPHalfStride, pk[1]);
          }
        }
        if (!done) {
          ok = __all_sync(0xffffffffu, here);
          if (!ok) break;
          if (kParts && !kPaged && lo < kBN - 1) {
            // A tile with hidden columns (the diagonal, the sequence's end) in one pass too, 32 columns at a time; those hidden from all sixteen
            // rows are neither read nor exponentiated.  Only in the form for dense parts in clusters, whose calls are a few tiles long: one
            // fp32 prompt of 512 tokens 12.1 -> 11.85 us, in bf16 10.5 -> 10.2, 100 queries over 2 x 1 300 keys 15.8 -> 15.5.  In the other
            // forms the code that a whole tile does not run slows it: at full clock 8 x 2 048 without a mask 398.8 -> 402.5, head_dim 64
            // 945 -> 969, for 5 packed prompts of up to 224 tokens 10.6 -> 9.9.
            uint32_t pk[2][16];
            uint32_t v0[16];
            auto load_quarter = [&](int c) {
              tmem_ld_16x256b_x4(tS + c * 32, v0);
              tmem_wait_ld_regs(v0);
              if (lo < c * 32 + 31) mask_quarter(v0, c);
            };
            if (j == 0) {
#pragma unroll 1
              for (int c = 0; c < 4 && c * 32 <= hi; ++c) {
                load_quarter(c);
                max_quarter(v0);
              }
              m_a = quad_max(mx_a) * sl2;
              m_b = quad_max(mx_b) * sl2;
            }
            nega_2 = pack_f2(-m_a, -m_a);
            negb_2 = pack_f2(-m_b, -m_b);
#pragma unroll
            for (int c = 0; c < 4; ++c) {
              uint32_t* const pq = pk[c >> 1] + (c & 1) * 8;
              if (c * 32 <= hi) {
                load_quarter(c);
                exp_quarter(v0, pq);
              } else {
#pragma unroll
                for (int i = 0; i < 8; ++i) pq[i] = 0u;
              }
            }
            sum_a = pair_sum(rs_a);
            sum_b = pair_sum(rs_b);
            done = __all_sync(0xffffffffu, here && sum_a <= kMaxPartialSum && sum_b <= kMaxPartialSum);   // (false for NaN)
            if (done) {
              tmem_st_16x128b_x8(tS, pk[0]);
              tmem_st_16x128b_x8(tS + ptx::kPHalfStride, pk[1]);
            }
          }
        }
        if (!done) {
          // Two passes, 32 columns at a time: a row whose reference moves, or has none.
          mx_a = mx_b = -INFINITY;
          rs_a = rs_b = pack_f2(0.f, 0.f);
#pragma unroll 1
          for (int c = 0; c < 4 && c * 32 <= hi; ++c) {
            uint32_t v[16];
            tmem_ld_16x256b_x4(tS + c * 32, v);
            tmem_wait_ld_regs(v);
            if (lo < c * 32 + 31) mask_quarter(v, c);
            max_quarter(v);
          }
          mx_a = quad_max(mx_a);
          mx_b = quad_max(mx_b);
          const float mn_a = fmaxf(m_a, mx_a * sl2), mn_b = fmaxf(m_b, mx_b * sl2);
          const bool need_a = (mn_a - m_a) > kRescaleThreshold;   // false for NaN / (-inf)-(-inf)
          const bool need_b = (mn_b - m_b) > kRescaleThreshold;
          float alpha_a = 1.f, alpha_b = 1.f;
          if (need_a) { alpha_a = fast_exp2(m_a - mn_a); m_a = mn_a; l_a *= alpha_a; }
          if (need_b) { alpha_b = fast_exp2(m_b - mn_b); m_b = mn_b; l_b *= alpha_b; }
          if (j > 0 && __any_sync(0xffffffffu, need_a || need_b)) {
            // PV(j-1) has landed in O once S(j) is visible (the MMAs complete in issue order); waiting on its
            // barrier phase is then immediate, and skipping the wait on other tiles is harmless because the
            // barrier can never run two phases ahead of this warp
            ok = warp_wait(smem_u32(&ctrl->o_done[s]), (tile_cnt - 1) & 1);
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int c = 0; c < D / 16; ++c) {
              uint32_t ov[8];
              tmem_ld_16x256b_x2(tO + c * 16, ov);
              tmem_wait_ld();
#pragma unroll
              for (int i = 0; i < 2; ++i) {
                ov[4 * i] = __float_as_uint(__uint_as_float(ov[4 * i]) * alpha_a);
                ov[4 * i + 1] = __float_as_uint(__uint_as_float(ov[4 * i + 1]) * alpha_a);
                ov[4 * i + 2] = __float_as_uint(__uint_as_float(ov[4 * i + 2]) * alpha_b);
                ov[4 * i + 3] = __float_as_uint(__uint_as_float(ov[4 * i + 3]) * alpha_b);
              }
              tmem_st_16x256b_x2(tO + c * 16, ov);
            }
          }
          const float neg_a = (m_a == -INFINITY) ? 0.f : -m_a, neg_b = (m_b == -INFINITY) ? 0.f : -m_b;
          nega_2 = pack_f2(neg_a, neg_a);
          negb_2 = pack_f2(neg_b, neg_b);
          // P of a quarter goes over scores that have been read: quarters 0 and 1 over the first 32 columns, 2 and 3 over
          // the first 32 of the upper half
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t pq[8];
            if (c * 32 <= hi) {
              uint32_t v[16];
              tmem_ld_16x256b_x4(tS + c * 32, v);
              tmem_wait_ld_regs(v);
              if (lo < c * 32 + 31) mask_quarter(v, c);
              exp_quarter(v, pq);
            } else {
#pragma unroll
              for (int i = 0; i < 8; ++i) pq[i] = 0u;
            }
            tmem_st_16x128b_x4(tS + (c >> 1) * ptx::kPHalfStride + (c & 1) * 16, pq);
          }
          sum_a = pair_sum(rs_a);
          sum_b = pair_sum(rs_b);
        }
        l_a += sum_a;
        l_b += sum_b;
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->p_ready[s]));
      }
      if constexpr (kParts) { seen = true; cut = !kMayBeWhole || ctrl->cut; }
      if (!ok) break;
      // ---------------- the item's epilogue ----------------
      const int len_q = w.len_q;
      const bool slot_live = w.valid && m0s < len_q;
      const long long qrow0 = w.out_row0[s];
      const int qhead = w.q_head[s];
      out_acc = n > 0;
      out_phase = (tile_cnt - 1) & 1;
      out_rows = slot_live ? min(kBM, len_q - m0s) : 0;
      out_la = quad_sum(l_a);
      out_lb = quad_sum(l_b);
      out_ma = m_a;
      out_mb = m_b;
      if (p.lse != nullptr && q == 0) {
        // split KV range: the merge needs every row's log-sum-exp (log2 domain; -inf for a row that saw no key)
        float* lse = p.lse + qrow0 + m0s + rowA;
        if (rowA < (slot_live ? min(kBM, len_q - m0s) : 0)) lse[0] = out_la > 0.f ? m_a + log2f(out_la) : -INFINITY;
        if (rowA + 8 < (slot_live ? min(kBM, len_q - m0s) : 0)) lse[8] = out_lb > 0.f ? m_b + log2f(out_lb) : -INFINITY;
      }
      if (p.layout == B200ATTN_RAGGED) {
        out_stride = static_cast<long long>(p.q_heads) * D;
        out_off = ((qrow0 + m0s + rowA) * p.q_heads + qhead) * D;
      } else {
        out_stride = D;
        out_off = (qrow0 + m0s + rowA) * D;
      }
      __syncwarp();
      if (lane == 0) mbar_arrive(smem_u32(&ctrl->sched_empty[k & 1]));
      if constexpr (kParts) break;       // (its only item: written when the parts have met)
      else ok = write_out(std::false_type{});
    }
    if constexpr (kParts) {
      // Parts of a KV range in a cluster: every warp's sixteen rows ("strip") have an owner among the CTAs.  The others send it
      // their accumulator, row sums and references in fp32 into its tile buffers, register by register as the warp of the same
      // number there holds its own; one barrier of the cluster says that all tile buffers are done with, a second that the
      // parts have arrived.  (Every warp of the cluster meets at both; no wait before them is without a limit.)  A part that
      // gave up sends NaN, and fills the rows that are its own with it.
      const int rank = static_cast<int>(cluster_rank()), parts = p.cluster_parts;
      if (kMayBeWhole && !cut) {
        __syncwarp();
        cluster_wait();
        if (ok && rank == 0) ok = write_out(std::false_type{});
      } else {
        if (ok && out_acc) ok = warp_wait(smem_u32(&ctrl->o_done[s]), out_phase) && !__any_sync(0xffffffffu, *abort_flag);
        if (!ok) {
          out_la = out_lb = __int_as_float(0x7fc00000);
          if (seen) {
            const ItemWork& w = ctrl->sched_work[0];
            out_rows = min(kBM, w.len_q - w.m0[s]);
            out_stride = D;
            out_off = (w.out_row0[s] + w.m0[s] + rowA) * D;
          }
        }
        tc_fence_after();
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        const int owner = warp % parts;
        if (owner != rank) {
          const int from = rank < owner ? rank : rank - 1;
          const uint4* const strip = peer_strip<D>(smem, warp / parts * (parts - 1) + from) + lane;
          const uint32_t to = map_to_rank(smem_u32(strip), static_cast<uint32_t>(owner));
          st_cluster_v4(to, __float_as_uint(out_ma), __float_as_uint(out_mb), __float_as_uint(out_la), __float_as_uint(out_lb));
#pragma unroll
          for (int c = 0; c < D / 64; ++c) {
            uint32_t v[32];
            if (out_acc) {
              tmem_ld_16x256b_x8(tO + c * 64, v);
              tmem_wait_ld();
            } else {
#pragma unroll
              for (int i = 0; i < 32; ++i) v[i] = 0u;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) st_cluster_v4(to + (1 + c * 8 + i) * 512, v[4 * i], v[4 * i + 1], v[4 * i + 2], v[4 * i + 3]);
          }
        }
        __syncwarp();
        cluster_arrive();
        cluster_wait();
        if (owner == rank) write_out(std::true_type{});
      }
    }
    if (!ok && lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
  }

  // ---------------- teardown ----------------
  if (kParts && warp >= kSoftmaxWarps) {
    __syncwarp();
    if (met < 1) cluster_arrive();
    if (met < 2) cluster_wait();
    if (met < 3) cluster_arrive();
    if (met < 4) cluster_wait();
  }
  tc_fence_before();
  __syncthreads();
  if (warp == kMmaWarp) {
    tc_fence_after();
    tmem_dealloc(tmem, 512);
  }
  {
    // A wait that ran out: the rows of the items in the scheduler's two slots, those that some warp has not done with among them, are
    // unknown, and NaN says so.  (An item that its cluster shares is marked where its parts meet.  The thread and the control block
    // are read anew: kept from above they cost every tile half a percent.)
    unsigned t;
    asm volatile("mov.u32 %0, %%tid.x;" : "=r"(t));
    uintptr_t at = reinterpret_cast<uintptr_t>(smem_raw);
    asm volatile("" : "+l"(at));
    const Control* const c = reinterpret_cast<const Control*>(((at + 1023) & ~uintptr_t(1023)) + Plan::kCtrlOff);
    if (c->abort_flag && !(kParts && (!kMayBeWhole || c->cut || c->sched_work[0].kv_tok0 > 0))) {
      const OutT nan = ElemTraits<OutT>::from_float(__int_as_float(0x7fc00000));
#pragma unroll 1
      for (int k = 0; k < 2 * kSlots; ++k) {
        if (c->sched_item[k & 1] < 0) continue;
        const ItemWork& w = c->sched_work[k & 1];
        const int s = k >> 1, rows = w.valid ? min(kBM, w.len_q - w.m0[s]) : 0;
        const long long stride = p.layout == B200ATTN_RAGGED ? p.q_heads : 1;
        OutT* const out = static_cast<OutT*>(p.out) + ((w.out_row0[s] + w.m0[s]) * stride + (stride > 1 ? w.q_head[s] : 0)) * D;
#pragma unroll 1
        for (int r = t / D; r < rows; r += kThreads / D) out[r * stride * D + t % D] = nan;
      }
    }
  }
}

}  // namespace

namespace {

// Merge of the parts of a split KV range.  part[(b * parts + s)][h][r][:] holds the normalised output of part s and
// lse[...] its log-sum-exp (log2 domain): out = sum_s 2^(lse_s - max) part_s / sum_s 2^(lse_s - max)
// (the reference's merge kernel, kernels/attention.py:659-746, on normalised instead of raw accumulators).
constexpr int kMaxParts = 8;       // split_plan cuts no finer
// kParts: parts that registers are held for (two parts in the form for eight are 1 % slower: 70 registers a thread)
template <typename OutT, int D, int kParts>
__global__ void __launch_bounds__(256) prefill_merge_kernel(const OutT* part, const float* lse, OutT* out,
                                                            long long rows_per_batch, int batch, int parts) {
  ptx::grid_dep_launch_dependents();
  ptx::grid_dep_wait();
  constexpr int VEC = 16 / sizeof(OutT);          // elements per 16-byte piece
  constexpr int PIECES = D / VEC;
  const long long total = static_cast<long long>(batch) * rows_per_batch * PIECES;
  for (long long idx = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; idx < total;
       idx += static_cast<long long>(gridDim.x) * blockDim.x) {
    const int piece = static_cast<int>(idx % PIECES);
    const long long row = idx / PIECES;                    // (b, h, r) flattened
    const long long b = row / rows_per_batch, hr = row - b * rows_per_batch;
    // (all reads of a piece are on their way at once: a loop over the parts was a chain of L2 round trips.  128 queries over
    // 8 192 keys, eight parts: 23.1 -> 21.7 us)
    float l[kParts];
    uint4 u[kParts];
#pragma unroll
    for (int sp = 0; sp < kParts; ++sp) {
      if (sp < parts) {
        const long long prow = (b * parts + sp) * rows_per_batch + hr;
        l[sp] = __ldcg(lse + prow);
        u[sp] = __ldcg(reinterpret_cast<const uint4*>(part + prow * D) + piece);
      }
    }
    float mx = -INFINITY;
#pragma unroll
    for (int sp = 0; sp < kParts; ++sp)
      if (sp < parts) mx = fmaxf(mx, l[sp]);
    float acc[VEC];
#pragma unroll
    for (int i = 0; i < VEC; ++i) acc[i] = 0.f;
    float wsum = 0.f;
#pragma unroll
    for (int sp = 0; sp < kParts; ++sp) {
      if (sp < parts) {
        const float w = (l[sp] == -INFINITY) ? 0.f : fast_exp2(l[sp] - mx);
        wsum += w;
        const OutT* e = reinterpret_cast<const OutT*>(&u[sp]);
#pragma unroll
        for (int i = 0; i < VEC; ++i) acc[i] += w * ElemTraits<OutT>::to_float(e[i]);
      }
    }
    const float inv = wsum > 0.f ? 1.f / wsum : 0.f;
    uint4 o;
    OutT* oe = reinterpret_cast<OutT*>(&o);
#pragma unroll
    for (int i = 0; i < VEC; ++i) oe[i] = ElemTraits<OutT>::from_float(acc[i] * inv);
    reinterpret_cast<uint4*>(out + row * D)[piece] = o;
  }
}

// How a launch with few work items cuts every sequence's KV range, so that more SMs than there are (query tile, head
// pair, sequence) items have work: the reference splits KV when B x QH < SMs (kernels/attention.py:836-841).  Dense and
// paged layouts only: a ragged problem's lengths are not known on the host.
struct SplitPlan {
  int parts;        // 1: no split
  int part_len;     // keys per part, a multiple of 128
};
SplitPlan split_plan(const b200attn_prefill_args_t& a, int sm_count) {
  SplitPlan sp{1, 0};
  if (a.layout == B200ATTN_RAGGED || a.batch <= 0 || a.max_q <= 0 || sm_count <= 0) return sp;
  const int group = a.q_heads / a.kv_heads;
  const bool head_pair = group % 2 == 0;
  const int item_rows = head_pair ? kBM : 2 * kBM;
  const long long head_units = head_pair ? a.q_heads / 2 : a.q_heads;
  const long long nblocks = (a.max_q + item_rows - 1) / item_rows;
  const long long items = nblocks * head_units * a.batch;
  const long long kv_cap = a.layout == B200ATTN_DENSE ? a.max_kv : a.table_stride * static_cast<long long>(a.page_size);
  const long long tiles = (kv_cap + kBN - 1) / kBN;            // longest item, in 128-key steps
  if (items <= 0 || tiles < 8) return sp;
  // steps of all items: under a causal mask row block r stops at its diagonal
  long long total = 0;
  for (long long r = 0; r < nblocks; ++r) {
    const long long reach = a.is_causal ? std::min<long long>(tiles, ((r + 1) * item_rows + kBN - 1) / kBN) : tiles;
    total += reach;
  }
  total *= head_units * a.batch;
  // Estimated duration in units of one 128-key step of both slots: the longest item or the average load of an SM,
  // whichever is larger, with about two steps of fixed cost per item (pipeline fill, masked tile, epilogue) and two
  // more for the merge launch.  Measured anchors on B200: B = 16, 8/2 heads, 128 x 2 048 cross attention (64 items)
  // 45 -> 36 us in two parts; a 512-key range in two parts is slower than unsplit (hence four tiles per part at least).
  auto cost = [&](long long parts) -> double {
    const double longest = static_cast<double>((tiles + parts - 1) / parts) + 2.0;
    const double load = (static_cast<double>(total) + 2.0 * static_cast<double>(items * parts)) / sm_count;
    return std::max(longest, load) + (parts > 1 ? 2.0 : 0.0);
  };
  long long best = 1;
  double best_cost = cost(1);
  for (long long parts = 2; parts <= kMaxParts && tiles / parts >= 4; parts *= 2) {
    const double c = cost(parts);
    if (c < 0.85 * cost(1) && c < best_cost) { best = parts; best_cost = c; }
  }
  if (best < 2) return sp;
  const long long per = (tiles + best - 1) / best;
  sp.part_len = static_cast<int>(per * kBN);
  sp.parts = static_cast<int>((tiles + per - 1) / per);
  if (sp.parts < 2) sp.parts = 1;
  return sp;
}

// The same with the parts of an item in a cluster, merged through distributed shared memory: for launches whose clusters are
// all resident at once (one CTA to an SM).  There is no second launch, and items
// of four to seven tiles are worth cutting; but what a CTA sends, fp32 accumulators of 64 KB and more at head_dim 128, takes as
// long as some tiles, so the costs below, in 128-key steps of 1.6 us.  Queries of one block of rows over 4, 6 and 12 tiles, four items,
// head_dim 64 12.2 -> 11.0, 15.4 -> 12.6, 17.4 -> 13.2 us; at head_dim 128 12 tiles 18.3 -> 16.7 (in eight parts), 16 tiles 15.6 -> 16.8, so
// those keep their parts in the workspace.  (Two parts at head_dim 128 are never the cheapest: below eight tiles they do not pay, from
// there on the workspace has them.  What a launch costs, and how short a part may be, is counted otherwise in split_plan: twelve tiles
// could go in four workspace parts of three.)
struct ClusterPlan : SplitPlan { int cut_tiles; };     // (cut_tiles: see finish_item)
// `ask`: see clusters_held.
ClusterPlan cluster_plan(const b200attn_prefill_args_t& a, int sm_count, const SplitPlan& other, bool ask) {
  ClusterPlan sp{{1, 0}, 0};
  if (a.layout == B200ATTN_RAGGED || a.batch <= 0 || a.max_q <= 0 || sm_count <= 0) return sp;
  const bool head_pair = (a.q_heads / a.kv_heads) % 2 == 0;
  const int item_rows = head_pair ? kBM : 2 * kBM;
  const long long items = (a.max_q + item_rows - 1ll) / item_rows * (head_pair ? a.q_heads / 2 : a.q_heads) * a.batch;
  const long long kv_cap = a.layout == B200ATTN_DENSE ? a.max_kv : a.table_stride * static_cast<long long>(a.page_size);
  long long tiles = (kv_cap + kBN - 1) / kBN;
  if (a.is_causal) tiles = std::min<long long>(tiles, (a.max_q + kBN - 1ll) / kBN);
  // steps of the longest item, and what the parts cost beside them
  static const double cluster_cost[2][3] = {{1.7, 2.3, 2.9}, {2.6, 3.8, 4.5}};
  constexpr double kLaunchCost = 1.5, kGain = 0.4;
  const long long whole = (tiles + other.parts - 1) / other.parts;
  double best = static_cast<double>(whole) + (other.parts > 1 ? kLaunchCost : 0.0) - kGain;
  for (int i = 0; i < 3; ++i) {
    const int parts = 2 << i;
    if (tiles < parts || items > clusters_held(parts, /*per_sm=*/1, sm_count, ask)) break;
    const long long per = (tiles + parts - 1) / parts;
    const double cost = static_cast<double>(per) + cluster_cost[a.head_dim == 128][i];
    if (cost < best) {
      best = cost;
      sp.parts = parts;
      sp.part_len = static_cast<int>(per * kBN);
      // (beside one CTA alone, without a second launch, the parts at head_dim 128 cost a step less than the figures above)
      sp.cut_tiles = static_cast<int>(std::min(tiles, static_cast<long long>(cost - (a.head_dim == 128 ? 1.0 : 0.0)) + 1));
    }
  }
  return sp;
}

struct CastPlan {
  size_t q_elems, kv_elems, q_off, k_off, v_off, total;
};
CastPlan cast_plan(const b200attn_prefill_args_t& a) {
  CastPlan c{};
  auto up = [](size_t x) { return (x + 255) & ~static_cast<size_t>(255); };
  const size_t D = static_cast<size_t>(a.head_dim);
  if (a.layout == B200ATTN_RAGGED) {
    c.q_elems = static_cast<size_t>(a.total_q) * a.q_heads * D;
    c.kv_elems = static_cast<size_t>(a.total_kv) * a.kv_heads * D;
  } else {
    c.q_elems = static_cast<size_t>(a.batch) * a.q_heads * a.max_q * D;
    c.kv_elems = a.layout == B200ATTN_DENSE ? static_cast<size_t>(a.batch) * a.kv_heads * a.max_kv * D
                                            : static_cast<size_t>(a.total_kv) * a.kv_heads * D;
  }
  c.q_off = kHeaderBytes;
  c.k_off = up(c.q_off + c.q_elems * 2);
  c.v_off = up(c.k_off + c.kv_elems * 2);
  c.total = up(c.v_off + c.kv_elems * 2);
  return c;
}
}  // namespace

namespace {
// workspace: header | fp32 inputs rounded to fp16 (fp32 calls) | parts of a split KV range and their log-sum-exps
struct WsPlan {
  size_t part_off, lse_off, total;
  SplitPlan split;
};
WsPlan ws_plan(const b200attn_prefill_args_t& a, int sm_count) {
  WsPlan w{};
  auto up = [](size_t x) { return (x + 255) & ~static_cast<size_t>(255); };
  size_t off = a.dtype == B200ATTN_F32 ? cast_plan(a).total : static_cast<size_t>(kHeaderBytes);
  w.split = split_plan(a, sm_count);
  if (w.split.parts > 1) {
    const size_t rows = static_cast<size_t>(a.batch) * w.split.parts * a.q_heads * a.max_q;
    const size_t esz = a.dtype == B200ATTN_F32 ? 4 : 2;
    w.part_off = off; off = up(off + rows * a.head_dim * esz);
    w.lse_off = off;  off = up(off + rows * sizeof(float));
  }
  w.total = off;
  return w;
}
}  // namespace

size_t prefill_workspace_bytes(const b200attn_prefill_args_t& a, int sm_count) { return ws_plan(a, sm_count).total; }

int prefill_route(const b200attn_prefill_args_t& a, int sm_count) {
  const SplitPlan split = ws_plan(a, sm_count).split;
  if (const int parts = cluster_plan(a, sm_count, split, /*ask=*/false).parts; parts > 1) return parts;
  return split.parts > 1 ? B200ATTN_ROUTE_WORKSPACE + split.parts : 1;
}

int launch_prefill(const b200attn_prefill_args_t& a_in, int sm_count, cudaStream_t stream) {
  const WsPlan wsp = ws_plan(a_in, sm_count);
  const size_t need = wsp.total;
  if (a_in.workspace == nullptr || a_in.workspace_bytes < need || (reinterpret_cast<uintptr_t>(a_in.workspace) & 255)) {
    set_error("prefill: workspace needs %zu bytes, 256-byte aligned (got %zu)", need, a_in.workspace_bytes);
    return B200ATTN_E_WORKSPACE;
  }
  b200attn_prefill_args_t a = a_in;
  const bool f32 = a_in.dtype == B200ATTN_F32;
  if (f32) {
    const CastPlan c = cast_plan(a_in);
    unsigned char* ws = static_cast<unsigned char*>(a_in.workspace);
    const long long q4 = static_cast<long long>(c.q_elems / 4), kv4 = static_cast<long long>(c.kv_elems / 4);
    const CastJob job = {{static_cast<const float4*>(a_in.q), static_cast<const float4*>(a_in.k), static_cast<const float4*>(a_in.v)},
                         {reinterpret_cast<uint2*>(ws + c.q_off), reinterpret_cast<uint2*>(ws + c.k_off),
                          reinterpret_cast<uint2*>(ws + c.v_off)},
                         {q4, kv4, kv4}};
    const cudaError_t ce = launch_cast(job, sm_count, stream);
    if (ce != cudaSuccess) return cuda_fail(ce, "cast kernel launch");
    a.q = ws + c.q_off; a.k = ws + c.k_off; a.v = ws + c.v_off;
    a.dtype = B200ATTN_F16;
  }
  const int D = a.head_dim;
  PrefillParams p;
  p.out = a.out; p.q_indptr = a.q_indptr; p.kv_indptr = a.kv_indptr;
  p.k_table = a.k_table; p.v_table = a.v_table;
  p.header = static_cast<int*>(a.workspace);
  p.work_counter = p.header + 8;
  p.table_stride = a.table_stride;
  p.layout = a.layout; p.indptr_is_i64 = a.indptr_is_i64;
  p.batch = a.batch; p.q_heads = a.q_heads; p.kv_heads = a.kv_heads; p.group = a.q_heads / a.kv_heads;
  p.max_q = a.max_q; p.max_kv = a.max_kv;
  p.page_size = a.layout == B200ATTN_PAGED ? a.page_size : 1;
  p.box_rows = kBN;
  p.num_pages = 0;
  p.is_causal = a.is_causal ? 1 : 0;
  p.head_pair = (p.group % 2 == 0) ? 1 : 0;
  p.out_align32 = (reinterpret_cast<uintptr_t>(a.out) & 31) == 0 ? 1 : 0;
  const int item_rows = p.head_pair ? kBM : 2 * kBM;
  const int head_units = p.head_pair ? a.q_heads / 2 : a.q_heads;
  p.scale_log2 = a.sm_scale * 1.4426950408889634f;
  p.kv_split = wsp.split.parts;
  p.kv_split_len = wsp.split.part_len;
  p.lse = nullptr;
  p.cluster_parts = 1;
  p.cut_tiles = 0;
  if (const ClusterPlan cp = cluster_plan(a, sm_count, wsp.split, /*ask=*/true); cp.parts > 1) {
    p.cluster_parts = cp.parts;
    p.cut_tiles = cp.cut_tiles;
    p.kv_split = 1;
    p.kv_split_len = cp.part_len;
  }
  if (p.kv_split > 1) {
    // the kernel writes every part's normalised output and log-sum-exp into the workspace; a merge kernel follows
    unsigned char* ws = static_cast<unsigned char*>(a_in.workspace);
    p.out = ws + wsp.part_off;
    p.lse = reinterpret_cast<float*>(ws + wsp.lse_off);
    p.out_align32 = 1;
  }

  CUtensorMap tq, tk, tv;
  int rc;
  dim3 grid;
  const long long row_bytes = D * 2ll;
  long long total_items = 0;
  if (a.layout == B200ATTN_RAGGED) {
    if ((rc = make_kv_rows_map(&tq, a.dtype, a.q, a.total_q, a.q_heads, D, kBM, a.q_heads * row_bytes, row_bytes))) return rc;
    if ((rc = make_kv_rows_map(&tk, a.dtype, a.k, a.total_kv, a.kv_heads, D, kBN, a.kv_heads * row_bytes, row_bytes))) return rc;
    if ((rc = make_kv_rows_map(&tv, a.dtype, a.v, a.total_kv, a.kv_heads, D, kBN, a.kv_heads * row_bytes, row_bytes))) return rc;
    const long long pairs = a.total_q / item_rows + a.batch;
    total_items = pairs * head_units;
  } else {
    const long long q_rows = static_cast<long long>(a.batch) * a.q_heads * a.max_q;
    if ((rc = make_kv_rows_map(&tq, a.dtype, a.q, q_rows, 1, D, kBM, row_bytes, row_bytes))) return rc;
    if (a.layout == B200ATTN_DENSE) {
      const long long kv_rows = static_cast<long long>(a.batch) * a.kv_heads * a.max_kv;
      if ((rc = make_kv_rows_map(&tk, a.dtype, a.k, kv_rows, 1, D, kBN, row_bytes, row_bytes))) return rc;
      if ((rc = make_kv_rows_map(&tv, a.dtype, a.v, kv_rows, 1, D, kBN, row_bytes, row_bytes))) return rc;
    } else {
      // largest power of two that divides the page size, capped at the tile: every box stays inside one page
      int box = 1;
      while (box < kBN && (a.page_size % (box * 2)) == 0) box *= 2;
      p.box_rows = box;
      p.num_pages = static_cast<int>(std::min<long long>(a.total_kv / a.page_size, 0x7fffffff));
      if (group_boxes(D, box)) {
        if ((rc = make_kv_groups_map(&tk, a.dtype, a.k, a.total_kv, a.kv_heads, D, box, a.kv_heads * row_bytes, row_bytes))) return rc;
        if ((rc = make_kv_groups_map(&tv, a.dtype, a.v, a.total_kv, a.kv_heads, D, box, a.kv_heads * row_bytes, row_bytes))) return rc;
      } else {
        if ((rc = make_token_map(&tk, a.dtype, a.k, a.total_kv, a.kv_heads, D, box))) return rc;
        if ((rc = make_token_map(&tv, a.dtype, a.v, a.total_kv, a.kv_heads, D, box))) return rc;
      }
    }
    total_items = static_cast<long long>((a.max_q + item_rows - 1) / item_rows) * head_units * a.batch * p.kv_split * p.cluster_parts;
  }
  if (total_items <= 0) return B200ATTN_OK;
  if (total_items > 0x7fffffff) { set_error("prefill: too many work items"); return B200ATTN_E_UNSUPPORTED; }
  p.total_items = static_cast<int>(total_items);
  grid = dim3(static_cast<unsigned>(p.cluster_parts > 1 ? total_items : std::min<long long>(total_items, sm_count)), 1, 1);
  // The two counters in the header (next item, CTAs finished) are zero here: the workspace starts zeroed and
  // the last CTA of every launch puts them back.

  cudaError_t e;
#define B200ATTN_LAUNCH_PREFILL_AS(TYPE, DIM, OUT, PAGED, PARTS)                                         \
  do {                                                                                                   \
    const size_t smem = std::max<size_t>(SmemPlan<DIM>::kTotal + 1024, 120 * 1024);                      \
    if ((rc = ensure_dynamic_smem(reinterpret_cast<const void*>(prefill_kernel<TYPE, DIM, OUT, PAGED, PARTS>), smem))) return rc; \
    launch_dependent(prefill_kernel<TYPE, DIM, OUT, PAGED, PARTS>, grid, kThreads, smem, stream,         \
                     static_cast<unsigned>(p.cluster_parts), tq, tk, tv, p);                             \
  } while (0)
#define B200ATTN_LAUNCH_PREFILL(TYPE, DIM, OUT)                                                          \
  do {                                                                                                   \
    if (a.layout == B200ATTN_PAGED) {                                                                    \
      if (p.cluster_parts > 1) B200ATTN_LAUNCH_PREFILL_AS(TYPE, DIM, OUT, true, true);                   \
      else B200ATTN_LAUNCH_PREFILL_AS(TYPE, DIM, OUT, true, false);                                      \
    } else if (p.cluster_parts > 1) {                                                                    \
      B200ATTN_LAUNCH_PREFILL_AS(TYPE, DIM, OUT, false, true);                                           \
    } else {                                                                                             \
      B200ATTN_LAUNCH_PREFILL_AS(TYPE, DIM, OUT, false, false);                                          \
    }                                                                                                    \
  } while (0)
  if (f32) {
    if (D == 128) B200ATTN_LAUNCH_PREFILL(__half, 128, float); else B200ATTN_LAUNCH_PREFILL(__half, 64, float);
  } else if (a.dtype == B200ATTN_BF16) {
    if (D == 128) B200ATTN_LAUNCH_PREFILL(__nv_bfloat16, 128, __nv_bfloat16); else B200ATTN_LAUNCH_PREFILL(__nv_bfloat16, 64, __nv_bfloat16);
  } else {
    if (D == 128) B200ATTN_LAUNCH_PREFILL(__half, 128, __half); else B200ATTN_LAUNCH_PREFILL(__half, 64, __half);
  }
#undef B200ATTN_LAUNCH_PREFILL
#undef B200ATTN_LAUNCH_PREFILL_AS
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "prefill kernel launch");
  if (p.kv_split > 1) {
    const long long rows_per_batch = static_cast<long long>(a.q_heads) * a.max_q;
    const long long pieces = static_cast<long long>(a.batch) * rows_per_batch * (D / (f32 ? 4 : 8));
    const int blocks = static_cast<int>(std::min<long long>((pieces + 255) / 256, static_cast<long long>(sm_count) * 8));
#define B200ATTN_LAUNCH_MERGE(OUT, DIM)                                                                              \
    launch_dependent(p.kv_split <= 2 ? prefill_merge_kernel<OUT, DIM, 2> : prefill_merge_kernel<OUT, DIM, kMaxParts>, \
                     dim3(static_cast<unsigned>(blocks)), 256, 0, stream, 1,                                          \
                     static_cast<const OUT*>(p.out), static_cast<const float*>(p.lse), static_cast<OUT*>(a_in.out),   \
                     rows_per_batch, a.batch, p.kv_split)
    if (f32) { if (D == 128) B200ATTN_LAUNCH_MERGE(float, 128); else B200ATTN_LAUNCH_MERGE(float, 64); }
    else if (a.dtype == B200ATTN_BF16) { if (D == 128) B200ATTN_LAUNCH_MERGE(__nv_bfloat16, 128); else B200ATTN_LAUNCH_MERGE(__nv_bfloat16, 64); }
    else { if (D == 128) B200ATTN_LAUNCH_MERGE(__half, 128); else B200ATTN_LAUNCH_MERGE(__half, 64); }
#undef B200ATTN_LAUNCH_MERGE
    e = cudaGetLastError();
    if (e != cudaSuccess) return cuda_fail(e, "prefill merge kernel launch");
  }
  return B200ATTN_OK;
}

}  // namespace b200attn
