// Decode and speculative-decode attention for sm_100a (HBM-bound path).
//
// One launch family replaces the reference's split kernel + merge kernel pairs
// (kernels/decode.py:22-200, kernels/speculative_decode.py:22-226):
//
//   decode_plan_kernel : 1 CTA.  Reads the sequence lengths on the device (no host sync), picks the KV chunk size
//       (the smallest of 32 candidates that keeps the batch at or below `target_items` work items, a whole number of
//       waves of resident CTAs - or of a single wave, when the batch cuts into that few near-equal items and an
//       estimate of the run time favours it), splits every sequence into equal items and writes one record per item
//       in execution order, longest first.  A work item is (sequence, KV chunk); a unit is (item, kv head), heads
//       fastest.
//   decode_mma_kernel  : up to 16 q rows per KV head.  All q rows that share the KV head (group size G x draft
//       tokens M) are packed into 16-row MMA tiles, so every K/V byte is read from HBM once per KV head (the
//       reference re-reads it once per q head).  A producer warp stages K/V tiles of 64 keys by TMA (one 4-D box per
//       page and operand) through a 2- or 3-stage mbarrier ring; block-table entries outside the cache are reported
//       and never dereferenced, V rows past the sequence end are zeroed in shared memory.  QK^T and PV run on
//       bf16/fp16 mma.sync with fp32 accumulation and an online softmax in the exp2 domain.
//   decode_umma_kernel : more than 16 q rows per KV head (speculative decode).  One 128-row tcgen05 tile: Q is
//       written to tensor memory once per unit, P once per 64-key tile, so both MMAs take their A operand from TMEM
//       and shared memory is read once per K/V byte.  Persistent: one wave of CTAs walks the unit list, the producer
//       runs ahead across units.  Same planner and partial format; merges are claimed in the CTAs' teardown.
//   decode_keyrows_kernel (decode_keyrows.cuh) : 17 to 64 q rows over long sequences.  The tensor-core tiles have keys as their rows
//       and the q rows as their columns, so nothing is multiplied for rows that are not there.
//   decode_simt_kernel : the fp32-input variant, fp32 FMA arithmetic like the reference's decode kernel.
//   A unit whose sequence has a single chunk writes the output directly; otherwise it writes an (m, l, acc) partial
//       and takes a ticket.  In the one-CTA-per-unit kernels (emit_and_merge) the CTA that draws the last ticket of
//       its (sequence, kv head) performs the log-sum-exp merge; in the persistent kernel a CTA that has run out of
//       units claims complete pairs and merges them.  No CTA ever waits for another.
//   Calls that are all latency (short sequences, cluster_size) skip planner, partials and tickets: a cluster of up to eight
//       CTAs of the warp-level or the fp32 kernel shares a (sequence, kv head) pair and merges through distributed shared
//       memory; there, and only there, a CTA waits (with a limit) for the others of its cluster.
#include <algorithm>
#include <mutex>
#include <type_traits>

#include "cast.cuh"
#include "common.cuh"
#include "cluster_residency.h"
#include "decode_launch.h"
#include "launch.cuh"
#include "sm100_ptx.cuh"
#include "tensor_map.h"

namespace b200attn {

namespace {

constexpr int kTileN = 64;
constexpr int kMaxStages = 4;
constexpr int kPlanThreads = 1024;
constexpr int kPlanBuckets = 32;    // size classes of the execution order (longest items first)
constexpr int kPlanLenCache = 4096; // sequences whose lengths the planner keeps in shared memory
constexpr int kGroupedChunks = 26;  // chunks of a pair from which they are merged in two steps
constexpr int kGroupedChunksFew = 40; // ... where a thread has one element and takes eight chunks at a time
constexpr int kPlanMaxSlots = 512;  // slots of the persistent kernel that the planner deals out

struct SeqInfo {
  long long start;  // ragged: first row of the sequence
  int len;
};

__device__ __forceinline__ SeqInfo seq_info(const DecodeParams& p, int b) {
  SeqInfo s;
  s.start = 0;
  if (p.layout == B200ATTN_DENSE) {
    s.len = p.max_kv;
  } else if (p.layout == B200ATTN_RAGGED) {
    long long a = load_index(p.kv_indptr, p.indptr_is_i64, b);
    long long e = load_index(p.kv_indptr, p.indptr_is_i64, b + 1);
    a = a < 0 ? 0 : (a > p.total_kv ? p.total_kv : a);
    e = e < a ? a : (e > p.total_kv ? p.total_kv : e);
    s.start = a;
    s.len = static_cast<int>(e - a);
  } else {
    long long n = load_index(p.kv_indptr, p.indptr_is_i64, b);
    long long cap = p.table_stride * static_cast<long long>(p.page_size);
    n = n < 0 ? 0 : (n > cap ? cap : n);
    s.len = static_cast<int>(n);
  }
  return s;
}

// A CTA's work item: from the planner's records, worked out by the CTA itself, or its part of a pair in a cluster.
struct DecodeItem {
  long long start;            // ragged: first row of the sequence
  int b, c, n_chunks, item0;  // sequence, chunk, chunks of the sequence, item number of its first chunk
  int len, t_begin, t_end;    // keys of the sequence, the item's keys
};

// Fills `rows` combined rows with NaN accumulators and (m, l) = (0, 1); every thread of the CTA takes part.
__device__ __forceinline__ void poison_rows(float* comb_o, float* comb_ml, int rows, int d) {
  const float nan = __int_as_float(0x7fc00000);
  for (int i = threadIdx.x; i < rows * d; i += blockDim.x) comb_o[i] = nan;
  for (int i = threadIdx.x; i < rows; i += blockDim.x) { comb_ml[2 * i] = 0.f; comb_ml[2 * i + 1] = 1.f; }
}

// ---------------------------------------------------------------------------
// Merge of published partials of one (sequence, kv head), into its output rows or into one partial, by the `nt` threads
// t = 0 .. nt-1 of the CTA that drew the last ticket: g = max m; O = sum 2^(m-g) acc / sum 2^(m-g) l
// (kernels/decode.py:186-197).
// ---------------------------------------------------------------------------
// Where the header holds a pair's tickets in a call without a planner launch (`i`: 0, or 1 + the group of chunks).  (In the library's own
// array the planner, which runs in every call there, puts them at zero.)
struct TicketPlace { unsigned* word; int shift, bits; };
__device__ __forceinline__ TicketPlace ticket_place(const DecodeParams& p, int pair, int i) {
  unsigned* const words = reinterpret_cast<unsigned*>(p.header) + kTicketWord;
  if (p.pair_tickets) {
    const int at = pair * p.pair_tickets + i;
    return {words + (at >> 2), (at & 3) * 8, 8};
  }
  const int log_per_word = p.inline_plan == 8 ? 2 : 1;
  return {words + (pair >> log_per_word), (pair & ((1 << log_per_word) - 1)) * p.inline_plan, p.inline_plan};
}
// Draws the next merge ticket of a (sequence, kv head) pair.
__device__ __forceinline__ int draw_ticket(const DecodeParams& p, int pair, int i = 0) {
  if (!p.inline_plan && !p.pair_tickets) return atomicAdd(p.counters + pair, 1);
  const TicketPlace t = ticket_place(p, pair, i);
  return (atomicAdd(t.word, 1u << t.shift) >> t.shift) & ((1u << t.bits) - 1);
}
// Leaves the pair's ticket counter at zero for the next call; `n` tickets were drawn.
__device__ __forceinline__ void reset_ticket(const DecodeParams& p, int pair, int n, int i = 0) {
  if (!p.inline_plan && !p.pair_tickets) p.counters[pair] = 0;
  else { const TicketPlace t = ticket_place(p, pair, i); atomicSub(t.word, static_cast<unsigned>(n) << t.shift); }
}
// Chunks of a group where a pair's chunks are merged in two steps, 0 where they are not (see publish_and_merge).
__device__ __forceinline__ int merge_group(const DecodeParams& p, int n_chunks, bool few) {
  if (!p.pair_tickets || n_chunks < (few ? kGroupedChunksFew : kGroupedChunks)) return 0;
  const int groups = min(p.pair_tickets - 1, __float2int_rn(sqrtf(static_cast<float>(n_chunks))));
  return (n_chunks + groups - 1) / groups;
}

// The partials are in the slots slot0, slot0 + step, ...  `s_ml` not null: their merge goes to the first of them (shared memory for two
// floats per row; every thread of the CTA takes part then), else to `out`.
//
// One pass with a running maximum, E output elements and 8 / E chunks per step: the loads of a step do not depend on each other or on
// the running state, so they are in flight together (the merge is a chain of L2 round trips otherwise).  With eight chunks of one element
// everywhere the kernels of many rows spill (40 rows, 8 x 2 500 keys 26.8 -> 29.4 us).
// What a step reads in the place of a chunk that is not there.  (Zeros; a constant would let the compiler make branches of the loads:
// 16 x 9 943 keys of two heads, twelve rows, 42.0 -> 43.4 us, 1 x 30 000 of one head 19.4 -> 20.1.)
__device__ float4 g_no_chunk;
template <typename T, int D, int E>
__device__ __forceinline__ void merge_elements(const DecodeParams& p, long long slot0, int step, int n_chunks, T* out, int t, int nt, float* s_ml) {
  constexpr int D4 = D / 4, CH = 8 / E;
  const int R = p.rows;
  const int total = R * D4;
  for (int idx0 = t; idx0 < total; idx0 += nt * E) {
    int r[E], d4[E];
    bool live[E];
    float mg[E], l[E];
    float4 acc[E];
#pragma unroll
    for (int e = 0; e < E; ++e) {
      const int idx = idx0 + e * nt;
      live[e] = idx < total;
      const int id = live[e] ? idx : idx0;
      r[e] = id / D4;
      d4[e] = id - r[e] * D4;
      mg[e] = -INFINITY;
      l[e] = 0.f;
      acc[e] = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    for (int k0 = 0; k0 < n_chunks; k0 += CH) {
      float mk[E][CH], lk[E][CH];
      float4 o[E][CH];
#pragma unroll
      for (int e = 0; e < E; ++e) {
#pragma unroll
        for (int j = 0; j < CH; ++j) {
          const bool on = k0 + j < n_chunks;
          const long long s = slot0 + static_cast<long long>(on ? k0 + j : k0) * step;
          const float2 ml = __ldcg(reinterpret_cast<const float2*>(p.part_ml + (s * R + r[e]) * 2));
          // (zeros where there is no chunk, not another chunk with a weight of 0: that may hold infinities)
          const float4* const from = on ? reinterpret_cast<const float4*>(p.part_o + (s * R + r[e]) * D + d4[e] * 4) : &g_no_chunk;
          o[e][j] = __ldcg(from);
          mk[e][j] = on ? ml.x : -INFINITY;
          lk[e][j] = ml.y;
        }
      }
#pragma unroll
      for (int e = 0; e < E; ++e) {
        float mn = mg[e];
#pragma unroll
        for (int j = 0; j < CH; ++j) mn = fmaxf(mn, mk[e][j]);
        const float keep = (mg[e] == -INFINITY) ? 0.f : fast_exp2(mg[e] - mn);
        acc[e].x *= keep; acc[e].y *= keep; acc[e].z *= keep; acc[e].w *= keep;
        l[e] *= keep;
#pragma unroll
        for (int j = 0; j < CH; ++j) {
          const float w = (mk[e][j] == -INFINITY) ? 0.f : fast_exp2(mk[e][j] - mn);
          acc[e].x += w * o[e][j].x; acc[e].y += w * o[e][j].y; acc[e].z += w * o[e][j].z; acc[e].w += w * o[e][j].w;
          l[e] += w * lk[e][j];
        }
        mg[e] = mn;
      }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
      if (!live[e]) continue;
      if (s_ml) {
        // (this thread alone has read and writes these four elements)
        *reinterpret_cast<float4*>(p.part_o + (slot0 * R + r[e]) * D + d4[e] * 4) = acc[e];
        if (d4[e] == 0) { s_ml[2 * r[e]] = mg[e]; s_ml[2 * r[e] + 1] = l[e]; }
        continue;
      }
      const float inv = l[e] > 0.f ? 1.f / l[e] : 0.f;
      T* dst = out + static_cast<long long>(r[e]) * D + d4[e] * 4;
      if constexpr (sizeof(T) == 2) {
        uint2 u;
        u.x = ElemTraits<T>::pack2(acc[e].x * inv, acc[e].y * inv);
        u.y = ElemTraits<T>::pack2(acc[e].z * inv, acc[e].w * inv);
        *reinterpret_cast<uint2*>(dst) = u;
      } else {
        *reinterpret_cast<float4*>(dst) = make_float4(acc[e].x * inv, acc[e].y * inv, acc[e].z * inv, acc[e].w * inv);
      }
    }
  }
}
// kFew: the kernel may have so few rows that a thread has one element; it then takes eight chunks at a time (55 chunks of one sequence
// of 8 000 keys, 32/8 heads, 20.8 -> 19.7 us).
template <typename T, int D, bool kFew>
__device__ __forceinline__ void merge_chunks(const DecodeParams& p, long long slot0, int step, int n_chunks, T* out, int t, int nt, float* s_ml) {
  __threadfence();
  if (kFew && p.rows * (D / 4) <= nt) merge_elements<T, D, 1>(p, slot0, step, n_chunks, out, t, nt, s_ml);
  else merge_elements<T, D, 2>(p, slot0, step, n_chunks, out, t, nt, s_ml);
  if (s_ml) {
    __syncthreads();                 // (every thread has read the references and sums that are written over)
    for (int i = t; i < 2 * p.rows; i += nt) p.part_ml[slot0 * p.rows * 2 + i] = s_ml[i];
  }
}

// Publishes chunk c of a pair, whose partial this CTA's threads have written, by a ticket; the last arrival merges (nobody waits).
// A merge is one CTA's chain of L2 round trips, four chunks each, so that one long sequence alone was mostly that: its chunks are merged
// in groups, about as many as a group has chunks, each by the last of its CTAs to arrive, and the groups by the last of those.
// One sequence of 30 000 keys, us: 8/1 heads (235 chunks) 44.6 -> 19.9, 32/8 heads 37.1 -> 32.8; 6 of 30 271, 8/1 heads, 35.7 -> 30.9; 6 of
// 6 607 to 26 430, 40 rows of one head 59.2 -> 33.6.  With fewer chunks the second ticket costs more than the shorter chains save; in one step and
// in groups, us: 22 chunks, 20 rows, D 128 18.0, 18.7; 23 25.9, 26.7; 24, 16 rows 24.7, 25.0; 27 24.2, 23.4; 30, 32 rows 22.9, 21.1; with eight
// chunks a step, 4 rows, D 128, 27 15.5, 16.6; 30 17.0, 17.9; 36 17.9, 17.9; 55 18.0, 16.9; fp32 21 18.8, 20.5; 33 20.3, 20.9.
// `s_word`, `s_ml` (two floats per row): shared memory.
template <typename T, int D, bool kFew>
__device__ __forceinline__ void publish_and_merge(const DecodeParams& p, int b, int h, int c, int n_chunks, int item0, T* out, int* s_word,
                                                  float* s_ml) {
  const int t = static_cast<int>(threadIdx.x), nt = static_cast<int>(blockDim.x), pair = b * p.kv_heads + h;
  const long long slot0 = static_cast<long long>(item0) * p.kv_heads + h;   // chunk k lives in slot0 + k * kv_heads
  __threadfence();
  __syncthreads();
  const int group = merge_group(p, n_chunks, kFew && p.rows * (D / 4) <= nt);
  int n = n_chunks, step = p.kv_heads;
  if (group > 0) {
    const int g = c / group, size = min(group, n_chunks - g * group);
    if (t == 0) *s_word = draw_ticket(p, pair, 1 + g);
    __syncthreads();
    if (*s_word != size - 1) return;
    merge_chunks<T, D, kFew>(p, slot0 + static_cast<long long>(g * group) * step, step, size, out, t, nt, s_ml);
    if (t == 0) reset_ticket(p, pair, size, 1 + g);
    __threadfence();
    __syncthreads();
    n = (n_chunks + group - 1) / group;
    step *= group;
  }
  if (t == 0) *s_word = draw_ticket(p, pair);
  __syncthreads();
  if (*s_word != n - 1) return;
  merge_chunks<T, D, kFew>(p, slot0, step, n, out, t, nt, nullptr);
  if (t == 0) reset_ticket(p, pair, n);
}

// ---------------------------------------------------------------------------
// Emit the CTA's combined (m, l, acc) rows, then merge if this CTA is the last
// of its (sequence, kv head).  `comb_o` is smem [KS][rows_pad][D] fp32,
// `comb_ml` is smem [KS][rows_pad][2] = (m in log2 units, l).
// ---------------------------------------------------------------------------
template <typename T, int D>
__device__ __forceinline__ void emit_and_merge(const DecodeParams& p, int b, int h, int c, int n_chunks,
                                               int item0, const float* comb_o, float* comb_ml,
                                               int KS, int rows_pad, int* s_ticket) {
  constexpr int D4 = D / 4;
  const int R = p.rows;
  T* out = static_cast<T*>(p.out) +
           ((static_cast<long long>(b) * p.q_heads + static_cast<long long>(h) * p.head_stride + p.head0) * p.q_len) * D;
  const long long slot = (static_cast<long long>(item0) + c) * p.kv_heads + h;
  for (int idx = threadIdx.x; idx < R * D4; idx += blockDim.x) {
    const int r = idx / D4, d4 = idx - r * D4;
    float mg = -INFINITY;
    for (int k = 0; k < KS; ++k) mg = fmaxf(mg, comb_ml[(k * rows_pad + r) * 2]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
    for (int k = 0; k < KS; ++k) {
      const float mk = comb_ml[(k * rows_pad + r) * 2];
      const float w = (mk == -INFINITY) ? 0.f : fast_exp2(mk - mg);
      const float4 o = *reinterpret_cast<const float4*>(comb_o + (static_cast<size_t>(k) * rows_pad + r) * D + d4 * 4);
      acc.x += w * o.x; acc.y += w * o.y; acc.z += w * o.z; acc.w += w * o.w;
      l += w * comb_ml[(k * rows_pad + r) * 2 + 1];
    }
    if (n_chunks == 1) {
      const float inv = l > 0.f ? 1.f / l : 0.f;
      T* dst = out + static_cast<long long>(r) * D + d4 * 4;
      if constexpr (sizeof(T) == 2) {
        uint2 u;
        u.x = ElemTraits<T>::pack2(acc.x * inv, acc.y * inv);
        u.y = ElemTraits<T>::pack2(acc.z * inv, acc.w * inv);
        *reinterpret_cast<uint2*>(dst) = u;
      } else {
        *reinterpret_cast<float4*>(dst) = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
      }
    } else {
      *reinterpret_cast<float4*>(p.part_o + (slot * R + r) * D + d4 * 4) = acc;
      if (d4 == 0) {
        p.part_ml[(slot * R + r) * 2] = mg;
        p.part_ml[(slot * R + r) * 2 + 1] = l;
      }
    }
  }
  if (n_chunks == 1) return;

  publish_and_merge<T, D, true>(p, b, h, c, n_chunks, item0, out, s_ticket, comb_ml);
}

// ---------------------------------------------------------------------------
// Short sequences: no plan, no partials in global memory, no tickets.
//
// The CTAs of a cluster cut a (sequence, kv head) pair's keys into equal parts of whole tiles, and every output element
// has an owner among them: each CTA sends its partial of the element, and the (m, l) of its row, into the owner's shared
// memory by asynchronous stores that count on the owner's mbarrier, and the owner merges and writes.  In a planned call of
// 12 us (16 sequences of 2 048 keys, two KV heads, D 64) planning took 3.3 us, publishing a partial and drawing its ticket
// 1.5, and the merge by the CTA that drew the last one 3.3: 12.8 -> 8.0 us a call.
// ---------------------------------------------------------------------------
struct ClusterPart {
  int rank, size;        // of this CTA in its cluster, of the cluster
  int total, share;      // 16-byte pieces of the pair's output rows in fp32, pieces of a CTA's share
};

template <int D>
__device__ __forceinline__ ClusterPart cluster_part(const DecodeParams& p) {
  ClusterPart c;
  c.size = p.cluster;
  c.rank = static_cast<int>(blockIdx.x) % c.size;
  c.total = p.rows * (D / 4);
  c.share = (c.total + c.size - 1) / c.size;
  return c;
}

// Before anything else: the receiving barrier, armed with the bytes that will be sent to this CTA.  The second half of the
// cluster barrier (cluster_emit) tells that every CTA has got this far.
template <int D>
__device__ __forceinline__ void cluster_begin(const DecodeParams& p, const ClusterPart& c, uint64_t* bar) {
  if (threadIdx.x == 0) {
    const int first = c.rank * c.share, n = min(c.share, c.total - first);
    ptx::mbar_init(smem_u32(bar), 1);
    ptx::mbar_fence_init();
    if (n > 0) {
      const int rows = (first + n - 1) / (D / 4) - first / (D / 4) + 1;
      ptx::mbar_arrive_expect_tx(smem_u32(bar), static_cast<uint32_t>(c.size * (n * 16 + rows * 8)));
    }
  }
  __syncwarp();
  ptx::cluster_arrive();
}

// The keys of sequence b that are this CTA's.
__device__ __forceinline__ void cluster_item(const DecodeParams& p, const ClusterPart& c, int b, DecodeItem& it) {
  const SeqInfo si = seq_info(p, b);
  const int tiles = (si.len + kTileN - 1) / kTileN, per = ((tiles + c.size - 1) / c.size) * kTileN;
  it.start = si.start;
  it.b = b;
  it.c = c.rank;
  it.n_chunks = 1;
  it.item0 = 0;
  it.len = si.len;
  it.t_begin = min(si.len, c.rank * per);
  it.t_end = min(si.len, it.t_begin + per);
}

// `recv`: shared memory for the pieces ([CTA][share] of 16 bytes) and the rows' (m, l) ([CTA][row]) sent to this CTA.
// Every CTA of the cluster comes here, also one that gave up on a copy: it sends its rows as NaN.  `tries`: limit of a wait.
template <typename T, int D>
__device__ __forceinline__ void cluster_emit(const DecodeParams& p, const ClusterPart& cp, int b, int h, const float* comb_o,
                                             const float* comb_ml, int KS, int rows_pad, unsigned char* recv, uint64_t* bar,
                                             uint32_t tries = ptx::kWaitTries) {
  constexpr int D4 = D / 4;
  const int R = p.rows;
  const uint32_t bar_s = smem_u32(bar), recv_o = smem_u32(recv), recv_ml = recv_o + cp.size * cp.share * 16;
  ptx::cluster_wait();
  for (int idx = threadIdx.x; idx < cp.total; idx += blockDim.x) {
    const int r = idx / D4, d4 = idx - r * D4;
    float mg = -INFINITY;
    for (int k = 0; k < KS; ++k) mg = fmaxf(mg, comb_ml[(k * rows_pad + r) * 2]);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
    for (int k = 0; k < KS; ++k) {
      const float mk = comb_ml[(k * rows_pad + r) * 2];
      const float w = (mk == -INFINITY) ? 0.f : fast_exp2(mk - mg);
      const float4 o = *reinterpret_cast<const float4*>(comb_o + (static_cast<size_t>(k) * rows_pad + r) * D + d4 * 4);
      acc.x += w * o.x; acc.y += w * o.y; acc.z += w * o.z; acc.w += w * o.w;
      l += w * comb_ml[(k * rows_pad + r) * 2 + 1];
    }
    const int owner = idx / cp.share, j = idx - owner * cp.share;
    const uint32_t slot = recv_o + (cp.rank * cp.share + j) * 16;
    ptx::st_async_pair(slot, bar_s, owner, acc.x, acc.y);
    ptx::st_async_pair(slot + 8, bar_s, owner, acc.z, acc.w);
    if (d4 == 0 || j == 0) ptx::st_async_pair(recv_ml + (cp.rank * R + r) * 8, bar_s, owner, mg, l);
  }
  const int first = cp.rank * cp.share, n = min(cp.share, cp.total - first);
  if (n <= 0) return;                    // (nothing is sent to this CTA)
  const bool ok = __all_sync(0xffffffffu, ptx::mbar_wait_limit(bar_s, 0, 4 * tries));
  if (!ok) {
    // A peer is late by more than that (one that gives up on a copy first drains its others, a limit each, and limits of
    // different CTAs do not compare).  This CTA may not leave: the peer still stores into its shared memory.  Each peer either
    // comes to the cluster's barrier here, having sent everything, or has left after doing so, and every wait on its way
    // has a limit; what has been sent then only has to land.
    p.header[0] = DEV_ERR_WAIT_EXPIRED;
    ptx::cluster_arrive();
    ptx::cluster_wait();
    ptx::mbar_wait_limit(bar_s, 0, tries);
  }
  T* out = static_cast<T*>(p.out) +
           ((static_cast<long long>(b) * p.q_heads + static_cast<long long>(h) * p.head_stride + p.head0) * p.q_len) * D;
  const float4* po = reinterpret_cast<const float4*>(recv);
  const float2* pm = reinterpret_cast<const float2*>(recv + static_cast<size_t>(cp.size) * cp.share * 16);
  for (int j = threadIdx.x; j < n; j += blockDim.x) {
    const int r = (first + j) / D4, d4 = first + j - r * D4;
    float mg = -INFINITY;
    for (int c = 0; c < cp.size; ++c) mg = fmaxf(mg, pm[c * R + r].x);
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float l = 0.f;
    for (int c = 0; c < cp.size; ++c) {
      const float2 ml = pm[c * R + r];
      const float4 o = po[c * cp.share + j];
      const float w = (ml.x == -INFINITY) ? 0.f : fast_exp2(ml.x - mg);
      acc.x += w * o.x; acc.y += w * o.y; acc.z += w * o.z; acc.w += w * o.w;
      l += w * ml.y;
    }
    const float inv = !ok ? __int_as_float(0x7fc00000) : (l > 0.f ? 1.f / l : (l == l ? 0.f : l));
    T* dst = out + static_cast<long long>(r) * D + d4 * 4;
    if constexpr (sizeof(T) == 2) {
      uint2 u;
      u.x = ElemTraits<T>::pack2(acc.x * inv, acc.y * inv);
      u.y = ElemTraits<T>::pack2(acc.z * inv, acc.w * inv);
      *reinterpret_cast<uint2*>(dst) = u;
    } else {
      *reinterpret_cast<float4*>(dst) = make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
    }
  }
}

// ---------------------------------------------------------------------------
// Planner
// ---------------------------------------------------------------------------
// Keys per work item of a sequence of `len` keys that is split into `n` items: every item covers the same number of
// keys (a multiple of the 64-key tile), the last takes what is left.
__device__ __forceinline__ int seq_chunk(int len, int n) {
  const int per = (len + n - 1) / n;
  const int c = ((per + kTileN - 1) / kTileN) * kTileN;
  return c < kTileN ? kTileN : c;
}

// ceil(a / b) for a >= 0, b > 0 with `inv_b` = 1 / b in float: exact (the float quotient is at most one off for
// a < 2^22, and is corrected; larger a take the integer division).
__device__ __forceinline__ int ceil_div_fast(int a, int b, float inv_b) {
  if (a >= (1 << 22)) return static_cast<int>((static_cast<long long>(a) + b - 1) / b);
  int q = __float2int_ru(static_cast<float>(a) * inv_b);
  if (q * b < a) ++q;
  else if (q > 0 && (q - 1) * b >= a) --q;
  return q;
}

__global__ void __launch_bounds__(kPlanThreads) decode_plan_kernel(const DecodeParams p) {
  __shared__ unsigned long long s_tot[32];
  __shared__ int s_warp[32];
  __shared__ int s_carry;
  __shared__ int s_chunk;
  // per candidate, of several waves [0] and of a single one [1]: chunk, items; largest item of a single wave
  __shared__ int s_cand_chunk[2][kPlanThreads / 32], s_cand_items[2][kPlanThreads / 32], s_cand_max[kPlanThreads / 32];
  __shared__ int s_slots;                            // > 0: the batch is dealt out to that many slots
  __shared__ int s_rank[kPlanMaxSlots];              // cuts inside sequences among the slot boundaries 1 .. i
  __shared__ int s_cut[kPlanMaxSlots];               // their keys, in order
  __shared__ int s_hist[kPlanBuckets];     // items per size class, then the class's first execution slot
  __shared__ int s_cursor[kPlanBuckets];
  __shared__ int s_len[kPlanLenCache];      // sequence lengths, read from global memory once
  __shared__ int s_first[kPlanLenCache + 1]; // item prefix per sequence (a copy of item_start that needs no round trip)
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  // The attention kernel behind this one may be scheduled now: its CTAs set themselves up and wait (grid_dep_wait)
  // until this grid has completed.
  ptx::grid_dep_launch_dependents();
  ptx::grid_dep_wait();      // (the call before may still be using the records and tickets that are written below)
  if (tid < kPlanBuckets) { s_hist[tid] = 0; s_cursor[tid] = 0; }
  const bool cached = p.batch <= kPlanLenCache;
  auto len_of = [&](int b) -> int { return cached ? s_len[b] : seq_info(p, b).len; };

  // keys, and above kKeyBits the items that the smallest chunk would make (more than a wave's only matter, see try_wave)
  constexpr int kKeyBits = 44;
  const float inv_min = 1.f / static_cast<float>(p.min_chunk);
  unsigned long long tot = 0;
  SeqInfo mine;                             // of sequence tid: kept, the records need it again
  mine.start = 0;
  mine.len = 0;
  for (int b = tid; b < p.batch; b += kPlanThreads) {
    const SeqInfo si = seq_info(p, b);
    if (b == tid) mine = si;
    if (cached) s_len[b] = si.len;
    tot += static_cast<unsigned long long>(si.len) +
           (static_cast<unsigned long long>(max(1, ceil_div_fast(si.len, p.min_chunk, inv_min))) << kKeyBits);
  }
  for (int o = 16; o > 0; o >>= 1) tot += __shfl_xor_sync(0xffffffffu, tot, o);
  if (lane == 0) s_tot[warp] = tot;
  __syncthreads();
  // Chunk size: the smallest of 32 candidates between total / target_items and twice that for which the batch
  // splits into at most target_items items.  target_items is a whole number of waves of resident CTAs, so the grid
  // never spills a few CTAs into one more wave (measured: 2.9 waves run 8 % faster than 3.4).  One warp per candidate.
  // Then the same for a single wave (wave_items): when every sequence can be cut into near-equal items that are all
  // resident at once, nothing is started or merged a second or third time on an SM, which is worth more than the
  // finer grain of several waves if the lengths allow it (measured, 32 x 8 192 keys, 40 rows per KV head: 212 us
  // against 245 us; one KV head of that batch: 91 us against 159 us).  The two plans are compared by an estimate
  // of their run time in keys: the largest item plus the per-item overhead for one wave, the average load of a
  // resident CTA plus half an item for several.
  unsigned long long sum = 0;
  for (int w = 0; w < kPlanThreads / 32; ++w) sum += s_tot[w];
  const long long t = static_cast<long long>(sum & ((1ull << kKeyBits) - 1));
  const int at_most = static_cast<int>(sum >> kKeyBits);
  // (the two divisions per sequence go through a float reciprocal, corrected to the exact quotient: a pass over 256
  // lengths with integer divisions cost 2 us, and the pass runs once or twice per call)
  // Both kinds of candidate are evaluated in one pass, and what one thread used to decide in loops over shared memory
  // warp 0 decides in ballots; with that, 32-bit divisions and the lengths kept in registers a call of 16 fp32 sequences of
  // 100 to 4 096 keys, 8 heads, takes 35.1 us instead of 36.3 (in two passes, the second where it is needed, 37.1).  But 32 warps
  // that look at every length keep the SM busy: the second kind is left out where even the smallest chunk makes no more items
  // than a wave has CTAs, and of a dense batch one length is looked at.  Without that 200 fp32 sequences of 250 keys, 8/1
  // heads, D 128, took 35.1 us instead of 32.5, 64 of 20 keys with 8 drafts, 8/1 heads, D 64 in 16 bits, 12.5 instead of 11.2.
  auto candidate = [&](int target) -> int {
    long long base = t <= 0x7fffffff ? (static_cast<unsigned>(t) + target - 1) / static_cast<unsigned>(target) : (t + target - 1) / target;
    base = ((base + kTileN - 1) / kTileN) * kTileN;
    if (base < p.min_chunk) base = p.min_chunk;
    if (base > (1 << 29)) base = 1 << 29;
    const long long cand = base + (base * warp) / 32;
    return static_cast<int>(((cand + kTileN - 1) / kTileN) * kTileN);
  };
  // (a batch of more sequences than a wave has CTAs cannot fit one: every sequence is at least one item)
  const bool try_wave = p.wave_items > 0 && p.wave_items < p.target_items && p.batch <= p.wave_items &&
                        at_most > p.wave_items;
  {
    const int ck0 = candidate(p.target_items), ck1 = try_wave ? candidate(p.wave_items) : ck0;
    const float inv0 = 1.f / static_cast<float>(ck0), inv1 = 1.f / static_cast<float>(ck1);
    long long n0 = 0, n1 = 0;
    int biggest = 0;
    // (sequences of a dense batch are all alike)
    const bool dense = p.layout == B200ATTN_DENSE;
    const int looked_at = dense ? 1 : p.batch, weight = dense ? p.batch : 1;
    for (int b = lane; b < looked_at; b += 32) {
      const int len = len_of(b);
      n0 += max(1, ceil_div_fast(len, ck0, inv0)) * weight;
      if (try_wave) {
        const int v = max(1, ceil_div_fast(len, ck1, inv1));
        n1 += v * weight;
        const int per = ((ceil_div_fast(len, v, __frcp_rn(static_cast<float>(v))) + kTileN - 1) / kTileN) * kTileN;
        biggest = max(biggest, min(len, max(per, kTileN)));
      }
    }
    for (int o = 16; o > 0; o >>= 1) {
      n0 += __shfl_xor_sync(0xffffffffu, n0, o);
      if (try_wave) {
        n1 += __shfl_xor_sync(0xffffffffu, n1, o);
        biggest = max(biggest, __shfl_xor_sync(0xffffffffu, biggest, o));
      }
    }
    if (lane == 0) {
      s_cand_chunk[0][warp] = ck0;
      s_cand_chunk[1][warp] = ck1;
      s_cand_items[0][warp] = n0 > 0x7fffffff ? 0x7fffffff : static_cast<int>(n0);
      s_cand_items[1][warp] = n1 > 0x7fffffff ? 0x7fffffff : static_cast<int>(n1);
      s_cand_max[warp] = biggest;
    }
  }
  __syncthreads();
  // Dealing out: the persistent kernel's CTAs of a KV head ("slots") each take one stretch of the sequences laid end to
  // end, all of the same length with item_overhead keys added per item, cutting sequences where a stretch ends.  That is
  // about one item per sequence and one per slot instead of three per slot, and no slot ends later than another.
  const long long line = t + static_cast<long long>(p.batch + p.slots - 1) * p.item_overhead;
  if (warp == 0) {
    const unsigned fit0 = __ballot_sync(0xffffffffu, s_cand_items[0][lane] <= p.target_items);
    const unsigned fit1 = __ballot_sync(0xffffffffu, s_cand_items[1][lane] <= p.wave_items);
    if (lane == 0) {
      const int pick0 = fit0 ? __ffs(fit0) - 1 : kPlanThreads / 32 - 1, items0 = s_cand_items[0][pick0];
      int pick_chunk = s_cand_chunk[0][pick0];
      // Estimated run time of a plan in several waves, in keys: the average load of a resident CTA plus half an item.
      const float ovh = static_cast<float>(p.item_overhead), n = static_cast<float>(items0);
      float best = p.wave_items > 0 ? (static_cast<float>(t) + n * ovh) / static_cast<float>(p.wave_items) +
                                          0.5f * (static_cast<float>(t) / n + ovh)
                                    : 0.f;
      if (try_wave && items0 > p.wave_items && fit1) {
        const int pick1 = __ffs(fit1) - 1;
        const float one = static_cast<float>(s_cand_max[pick1]) + ovh;
        if (one < best) { best = one; pick_chunk = s_cand_chunk[1][pick1]; }
      }
      s_chunk = pick_chunk;
      s_carry = 0;
      // (a cut moved to the end of a sequence makes a stretch up to min_chunk longer: without that in the estimate 47
      // sequences of 350 to 5 600 keys on one KV head were dealt out and took 48 us instead of 45)
      // (One CTA to an SM: equal items end with the last round of CTAs, not half an item behind the average.  CTAs of a batch that is
      // dealt out cannot take over from one another, as those that draw units longest first do: where the estimates alone favoured it, it took
      // 0.90 to 1.17 of the time, 1.007 over 45 batches, and they did not tell which.  So it has to be ahead by about as much as they are
      // wrong, a tenth and one item's overhead, some 500 keys.  What is left are long, very uneven batches: 2 of the 45, 0.99 of the time each.)
      if (p.one_cta) {
        const float rounds = static_cast<float>((items0 + p.wave_items - 1) / p.wave_items) * (static_cast<float>(pick_chunk) + ovh);
        best = 0.89f * fminf(best, rounds) - 500.f;
      }
      const bool deal = p.slots > 1 && p.slots <= kPlanMaxSlots && cached && line < (1 << 30) && items0 > p.wave_items &&
                        static_cast<float>(line) / static_cast<float>(p.slots) + static_cast<float>(p.min_chunk) < best;
      s_slots = deal ? p.slots : 0;
    }
  }
  for (int i = tid; i < p.batch * p.kv_heads; i += kPlanThreads) p.counters[i] = 0;
  __syncthreads();
  const int chunk = s_chunk;

  // inclusive prefix sums over 0 .. n - 1, in thread order
  auto prefix = [&](int n, auto value, auto put) {
    for (int base = 0; base < n; base += kPlanThreads) {
      const int b = base + tid;
      int incl = b < n ? value(b) : 0;
      for (int o = 1; o < 32; o <<= 1) {
        const int x = __shfl_up_sync(0xffffffffu, incl, o);
        if (lane >= o) incl += x;
      }
      if (lane == 31) s_warp[warp] = incl;
      __syncthreads();
      if (warp == 0) {
        int w = s_warp[lane];
        for (int o = 1; o < 32; o <<= 1) {
          const int x = __shfl_up_sync(0xffffffffu, w, o);
          if (lane >= o) w += x;
        }
        s_warp[lane] = w;  // inclusive over warps
      }
      __syncthreads();
      const int carry = s_carry;
      const int before = warp > 0 ? s_warp[warp - 1] : 0;
      if (b < n) put(b, carry + before + incl);
      __syncthreads();
      if (tid == 0) s_carry = carry + s_warp[31];
      if (base + kPlanThreads < n) __syncthreads();      // (the last pass: the caller's next barrier)
    }
  };
  const int slots = s_slots;
  if (slots > 0) {
    // s_first[b]: where sequence b starts on the line
    prefix(p.batch, [&](int b) { return s_len[b] + p.item_overhead; }, [&](int b, int incl) { s_first[b + 1] = incl; });
    __syncthreads();
    if (tid == 0) { s_first[0] = 0; s_carry = 0; }
    __syncthreads();
    const int end = s_first[p.batch];
    int stretch = ((static_cast<int>(line) + slots - 1) / slots + kTileN - 1) / kTileN * kTileN;
    if (stretch < p.min_chunk) stretch = p.min_chunk;
    // boundary `tid` between slot tid - 1 and slot tid: key cut_t of sequence cut_b; a piece shorter than min_chunk is
    // left with the rest of its sequence
    int cut_b = p.batch, cut_t = 0;
    const long long x = static_cast<long long>(tid) * stretch;
    if (tid < slots && x < end) {
      int lo = 0, hi = p.batch;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (s_first[mid] <= x) lo = mid; else hi = mid;
      }
      cut_b = lo;
      const int off = static_cast<int>(x) - s_first[lo] - p.item_overhead;
      cut_t = off > 0 ? (off + kTileN / 2) / kTileN * kTileN : 0;
      if (cut_t < p.min_chunk) cut_t = 0;
      else if (s_len[lo] - cut_t < p.min_chunk) { cut_b = lo + 1; cut_t = 0; }
    }
    prefix(slots, [&](int) { return cut_t > 0 ? 1 : 0; }, [&](int i, int incl) {
      s_rank[i] = incl;
      if (cut_t > 0) s_cut[incl - 1] = cut_t;
    });
    __syncthreads();
    int* slot_first = reinterpret_cast<int*>(p.item_info + 2 * static_cast<long long>(p.max_items)) - (slots + 1);   // behind the records in use
    if (tid < slots) slot_first[tid] = cut_b + s_rank[tid];
    // cuts before sequence b, i.e. at boundaries that lie before its start
    auto cuts_before = [&](int b) -> int {
      const int pos = s_first[b];
      const int k = min(slots - 1, (pos + stretch - 1) / stretch - 1);
      return k > 0 ? s_rank[k] : 0;
    };
    for (int b = tid; b < p.batch; b += kPlanThreads) {
      const SeqInfo si = b == tid ? mine : seq_info(p, b);
      const int r = cuts_before(b), first = b + r, n = cuts_before(b + 1) - r + 1;
      p.item_start[b + 1] = first + n;
      for (int c = 0; c < n && first + c < p.max_items; ++c) {
        p.item_info[2 * (first + c)] = make_int4(b, c | (n << 16), first, c > 0 ? s_cut[r + c - 1] : 0);
        p.item_info[2 * (first + c) + 1] = make_int4(si.len, c + 1 < n ? s_cut[r + c] : si.len,
                                                     static_cast<int>(si.start & 0xffffffffll), static_cast<int>(si.start >> 32));
      }
    }
    if (tid == 0) {
      const int n_items = p.batch + s_rank[slots - 1];
      slot_first[slots] = n_items;
      p.item_start[0] = 0;
      p.header[1] = p.min_chunk;   // (the smallest item: a batch that is dealt out has no chunk size)
      p.header[2] = n_items;
      p.header[3] = 0;
      p.header[4] = 0;
      p.header[5] = slots;
    }
    return;
  }
  prefix(p.batch, [&](int b) { return max(1, (len_of(b) + chunk - 1) / chunk); }, [&](int b, int incl) {
    p.item_start[b + 1] = incl;
    if (cached) s_first[b + 1] = incl;
  });
  __syncthreads();
  // Per-item records, so that a CTA learns everything about its work item from one 32-byte read.  Records are laid
  // out in execution order: longest items first (by size class), so that the CTAs still running when the grid
  // drains are the short ones.  item_start keeps the per-sequence (logical) numbering, which is what the partial
  // results and the merge use.
  const float class_of_key = static_cast<float>(kPlanBuckets) / static_cast<float>(chunk + 1);
  auto size_class = [&](int item_len) -> int {
    const int q = kPlanBuckets - 1 - static_cast<int>(static_cast<float>(item_len) * class_of_key);
    return q < 0 ? 0 : (q > kPlanBuckets - 1 ? kPlanBuckets - 1 : q);
  };
  // (a sequence's first n - 1 items have the same size, its last one takes the remainder: two size classes)
  for (int b = tid; b < p.batch; b += kPlanThreads) {
    const int len = len_of(b);
    const int first = b == 0 ? 0 : (cached ? s_first[b] : p.item_start[b]);
    const int n = (cached ? s_first[b + 1] : p.item_start[b + 1]) - first;
    const int per = seq_chunk(len, n);
    const int rem = max(0, len - (n - 1) * per);
    if (n > 1) atomicAdd(&s_hist[size_class(per)], n - 1);
    atomicAdd(&s_hist[size_class(rem)], 1);
  }
  __syncthreads();
  if (warp == 0) {
    static_assert(kPlanBuckets == 32, "one class per lane");
    const int c = s_hist[lane];
    int incl = c;
    for (int o = 1; o < 32; o <<= 1) {
      const int x = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += x;
    }
    s_hist[lane] = incl - c;
  }
  __syncthreads();
  for (int b = tid; b < p.batch; b += kPlanThreads) {
    const SeqInfo si = b == tid ? mine : seq_info(p, b);
    const int first = b == 0 ? 0 : (cached ? s_first[b] : p.item_start[b]);
    const int n = (cached ? s_first[b + 1] : p.item_start[b + 1]) - first;
    const int per = seq_chunk(si.len, n);
    const int rem = max(0, si.len - (n - 1) * per);
    auto put = [&](int slot, int c) {
      const int t0 = c * per;
      p.item_info[2 * slot] = make_int4(b, c | (n << 16), first, t0);
      p.item_info[2 * slot + 1] = make_int4(si.len, min(si.len, t0 + per), static_cast<int>(si.start & 0xffffffffll),
                                            static_cast<int>(si.start >> 32));
    };
    if (n > 1) {
      const int q = size_class(per);
      const int pos = s_hist[q] + atomicAdd(&s_cursor[q], n - 1);
      for (int c = 0; c < n - 1 && pos + c < p.max_items; ++c) put(pos + c, c);
    }
    const int q = size_class(rem);
    const int pos = s_hist[q] + atomicAdd(&s_cursor[q], 1);
    if (pos < p.max_items) put(pos, n - 1);
  }
  if (tid == 0) {
    p.item_start[0] = 0;
    int n_items = s_carry;
    if (n_items > p.max_items) {
      p.header[0] = DEV_ERR_PLAN;
      n_items = 0;
    }
    p.header[1] = chunk;
    p.header[2] = n_items;
    p.header[3] = 0;          // tickets drawn and not merged yet (tcgen05 kernel)
    p.header[4] = 0;          // units drawn beyond the CTAs' first ones (tcgen05 kernel)
    p.header[5] = 0;
  } else if (p.pair_tickets && tid >= 64 && tid < 128 - kTicketWord) {
    p.header[kTicketWord + tid - 64] = 0;      // (the library's own array)
  }
}

// What the CTAs of a call without a planner launch work their items out in.
struct InlinePlan {
  long long tot[kInlineBatch / 32];
  int len[kInlineBatch], n[kInlineBatch], per[kInlineBatch];
  int items[2][32], biggest[32];
  DecodeItem mine;
  int found, over;
};

// The planner's choices (same candidates, same estimate) made by a CTA of at least kInlineBatch threads for itself.
// Items are numbered sequence by sequence, the sequences with the longest items first.  Returns false when there is no
// item of that number.
__device__ __forceinline__ bool plan_inline(const DecodeParams& p, int item, InlinePlan& s, DecodeItem& out) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  SeqInfo mine;
  mine.start = 0;
  mine.len = 0;
  if (tid < p.batch) mine = seq_info(p, tid);
  if (tid < kInlineBatch) {
    s.len[tid] = mine.len;
    long long w = mine.len;
    for (int o = 16; o > 0; o >>= 1) w += __shfl_xor_sync(0xffffffffu, w, o);
    if (lane == 0) s.tot[warp] = w;
  }
  if (tid < 32) { s.items[0][tid] = 0; s.items[1][tid] = 0; s.biggest[tid] = 0; }
  if (tid == 0) { s.found = 0; s.over = 0; }
  __syncthreads();
  long long t = 0;
#pragma unroll
  for (int w = 0; w < kInlineBatch / 32; ++w) t += s.tot[w];
  // The grid is as large as the longest sequences that there can be ask for, in pages by the table's width.  There are at most
  // t / min_chunk + batch items: a CTA that these lengths leave nothing for goes without the plan.  (12 sequences of 142 keys in tables of
  // 2 848, 64/8 heads, D 128, 5 drafts, 944 CTAs: 17.3 -> 12.1 us, behind the planner 15.0.)
  if (static_cast<long long>(item - p.batch + 1) * p.min_chunk > t) return false;
  // candidate `lane` of either target; the warps share the sequences
  auto candidate = [&](int target) -> int {
    long long base = t <= 0x7fffffff ? (static_cast<unsigned>(t) + target - 1) / static_cast<unsigned>(target) : (t + target - 1) / target;
    base = ((base + kTileN - 1) / kTileN) * kTileN;
    if (base < p.min_chunk) base = p.min_chunk;
    if (base > (1 << 29)) base = 1 << 29;
    const long long cand = base + (base * lane) / 32;
    return static_cast<int>(((cand + kTileN - 1) / kTileN) * kTileN);
  };
  const bool try_wave = p.wave_items > 0 && p.wave_items < p.target_items && p.batch <= p.wave_items;
  const int ck0 = candidate(p.target_items), ck1 = try_wave ? candidate(p.wave_items) : ck0;
  {
    const float inv0 = 1.f / static_cast<float>(ck0), inv1 = 1.f / static_cast<float>(ck1);
    int n0 = 0, n1 = 0, big = 0;
    for (int b = warp; b < p.batch; b += nwarps) {
      const int len = s.len[b];
      n0 += max(1, ceil_div_fast(len, ck0, inv0));
      const int v = max(1, ceil_div_fast(len, ck1, inv1));
      n1 += v;
      const int per = ((ceil_div_fast(len, v, __frcp_rn(static_cast<float>(v))) + kTileN - 1) / kTileN) * kTileN;
      big = max(big, min(len, max(per, kTileN)));
    }
    if (warp < p.batch) {
      atomicAdd(&s.items[0][lane], n0);
      atomicAdd(&s.items[1][lane], n1);
      atomicMax(&s.biggest[lane], big);
    }
  }
  __syncthreads();
  int chunk;
  {
    const int n0 = s.items[0][lane], n1 = s.items[1][lane];
    const unsigned fit0 = __ballot_sync(0xffffffffu, n0 <= p.target_items);
    const int pick0 = fit0 ? __ffs(fit0) - 1 : 31;
    chunk = __shfl_sync(0xffffffffu, ck0, pick0);
    const int items0 = __shfl_sync(0xffffffffu, n0, pick0);
    const unsigned fit1 = __ballot_sync(0xffffffffu, n1 <= p.wave_items);
    if (try_wave && items0 > p.wave_items && fit1) {
      const int pick1 = __ffs(fit1) - 1;
      const float ovh = static_cast<float>(p.item_overhead);
      const float n_several = static_cast<float>(items0);
      const float several = (static_cast<float>(t) + n_several * ovh) / static_cast<float>(p.wave_items) +
                            0.5f * (static_cast<float>(t) / n_several + ovh);
      const float one = static_cast<float>(s.biggest[pick1]) + ovh;
      const int ck = __shfl_sync(0xffffffffu, ck1, pick1);
      if (one < several) chunk = ck;
    }
  }
  int n = 0, per = 0;
  if (tid < p.batch) {
    n = max(1, ceil_div_fast(mine.len, chunk, 1.f / static_cast<float>(chunk)));
    per = seq_chunk(mine.len, n);
    s.n[tid] = n;
    s.per[tid] = per;
  }
  __syncthreads();
  if (tid < p.batch) {
    int first = 0, total = 0;
    for (int b = 0; b < p.batch; ++b) {
      const int pb = s.per[b], nb = s.n[b];
      total += nb;
      if (pb > per || (pb == per && b < tid)) first += nb;
    }
    if (blockIdx.x == 0 && tid == 0) { p.header[1] = chunk; p.header[2] = total; }   // (for inspection)
    if (item >= first && item < first + n) {
      s.mine = DecodeItem{mine.start, tid, item - first, n, first, mine.len, (item - first) * per,
                          min(mine.len, (item - first + 1) * per)};
      s.found = 1;
    }
    // more items than the grid was sized for (prefix sums that are not monotonic): reported, and no item is run
    if (first + n > static_cast<int>(gridDim.x) / p.kv_heads) {
      p.header[0] = DEV_ERR_PLAN;
      s.over = 1;
    }
  }
  __syncthreads();
  out = s.mine;
  return s.found != 0 && s.over == 0;
}

__device__ __forceinline__ bool decode_item(const DecodeParams& p, int item, InlinePlan& s, DecodeItem& out) {
  if (p.inline_plan) return plan_inline(p, item, s, out);
  if (item >= p.header[2]) return false;
  const int4 rec0 = p.item_info[2 * item];
  const int4 rec1 = p.item_info[2 * item + 1];
  out.b = rec0.x; out.c = rec0.y & 0xffff; out.n_chunks = static_cast<unsigned>(rec0.y) >> 16; out.item0 = rec0.z;
  out.len = rec1.x; out.t_begin = rec0.w; out.t_end = rec1.y;
  out.start = (static_cast<long long>(rec1.w) << 32) | static_cast<unsigned int>(rec1.z);
  return true;
}

// ---------------------------------------------------------------------------
// bf16 / fp16 tensor-core kernel.
// Warps 0 .. n_mtiles*key_slices-1 consume; the last warp is the TMA producer.
// A stage holds 64 keys: K as D/64 column blocks of [64 rows][128 B] (128-byte swizzle, as
// written by the TMA), then V in the same form.
// ---------------------------------------------------------------------------
struct __align__(8) DecodeCtrl {
  uint64_t full[kMaxStages];
  uint64_t empty[kMaxStages];
  int ticket;
  int abort_flag;
};

// Byte offset of the 128-byte row (key t of the tile, column block cb) inside a K or V tile.  A tile is a
// sequence of TMA boxes of `1 << box_shift` keys, each stored as [column block][key][128 B].
template <int CHUNKS>
__device__ __forceinline__ uint32_t tile_row_offset(int t, int cb, int box_shift) {
  const int box = t >> box_shift, r = t & ((1 << box_shift) - 1);
  return static_cast<uint32_t>((((box * CHUNKS + cb) << box_shift) + r) << 7);
}
// address of 16-byte piece `pc` (0..7) of that row under the 128-byte swizzle (tile base 1024-byte aligned)
__device__ __forceinline__ uint32_t swz_piece(uint32_t row_off, int pc) {
  return row_off + (((pc ^ (row_off >> 7)) & 7) << 4);
}

__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity) {
  const bool ok = ptx::mbar_wait(bar, parity);
  return __all_sync(0xffffffffu, ok);
}

// Block-table read-ahead of a producer warp for paged caches (`on`: a 64-key tile has at most 32 boxes).  The warp holds
// the raw entries of 32 boxes of its item, one per lane, for K and for V, and those of the next 32, read when the first
// became current: a table read is waited for once in 32 boxes, long after it was issued, instead of a tile after it
// (32 x 16 384 keys in 16-key pages, head_dim 128: 388 -> 365 us with 40 rows per KV head, 483 -> 417 with
// 128; dense K/V of that size 341 and 380).
// Entries are checked when they are used, so that nothing waits for the read before.  Registers are plain scalars: an
// array indexed by a loop counter would live in local memory.
constexpr int kNoPage = static_cast<int>(0x80000000u);
struct PageAhead {
  const int* ktab;
  const int* vtab;
  int lane, boxes, box_shift, page_shift, page_size;
  bool on;
  int t_begin, t_end;          // the item's keys
  int kp, vp, kp_next, vp_next;
  __device__ __forceinline__ PageAhead(const DecodeParams& p, int lane_) : lane(lane_) {
    box_shift = p.box_shift;
    boxes = kTileN >> box_shift;
    on = p.layout == B200ATTN_PAGED && boxes <= 32;
    page_shift = p.page_shift;
    page_size = p.page_size;
    ktab = vtab = nullptr;
    t_begin = t_end = 0;
    kp = vp = kp_next = vp_next = kNoPage;
  }
  __device__ __forceinline__ void read(int first_box, int& k, int& v) const {
    const int t = t_begin + ((first_box + lane) << box_shift);
    k = v = kNoPage;
    if (t < t_end) {
      // (page size known only at run time; a shift when it is a power of two)
      const int lp = page_shift >= 0 ? (t >> page_shift) : t / page_size;
      k = __ldcg(ktab + lp);
      v = __ldcg(vtab + lp);
    }
  }
  __device__ __forceinline__ void start(const DecodeParams& p, int b, int begin, int end) {
    if (!on) return;
    ktab = p.k_table + static_cast<long long>(b) * p.table_stride;
    vtab = p.v_table + static_cast<long long>(b) * p.table_stride;
    t_begin = begin;
    t_end = end;
    // (a cache without a whole page: no entry can be right, and the tiles have no boxes whose entries would be checked)
    if (p.num_pages <= 0 && begin < end && lane == 0) p.header[0] = DEV_ERR_PAGE_RANGE;
    read(0, kp, vp);
    read(32, kp_next, vp_next);
  }
  // cache row of an entry's box at key t, -1 when there is none
  __device__ __forceinline__ int row(const DecodeParams& p, int page, int t) const {
    const int off = page_shift >= 0 ? (t & (page_size - 1)) : t % page_size;
    // an entry outside the cache is reported and replaced by page 0: never dereferenced, output stays finite
    const bool bad = page < 0 || page >= p.num_pages;
    if (bad) p.header[0] = DEV_ERR_PAGE_RANGE;
    return (bad ? 0 : page) * p.page_size + off;
  }
  // entries for tile number `tile` of the item become current (called for every tile, in order); returns the boxes that
  // the tile has
  __device__ __forceinline__ int advance(const DecodeParams& p, int tile) {
    if (((tile * boxes) & 31) == 0 && tile > 0) {
      kp = kp_next;
      vp = vp_next;
      read(tile * boxes + 32, kp_next, vp_next);
    }
    const int t0 = t_begin + tile * kTileN;
    return p.num_pages > 0 ? min(boxes, (t_end - t0 + (1 << box_shift) - 1) >> box_shift) : 0;
  }
  // rows of the lane's box of that tile, for K and for V
  __device__ __forceinline__ int tile_rows(const DecodeParams& p, int tile, int& kr, int& vr) {
    const int n = advance(p, tile), at = (tile * boxes) & 31;
    const int k = __shfl_sync(0xffffffffu, kp, (at + lane) & 31), v = __shfl_sync(0xffffffffu, vp, (at + lane) & 31);
    const int t0 = t_begin + tile * kTileN;
    kr = vr = -1;
    if (lane < n) {
      kr = row(p, k, t0 + (lane << box_shift));
      vr = row(p, v, t0 + (lane << box_shift));
    }
    return n;
  }
  // row of any box of that tile (of the first `n`), of K (op 0) or of V; -1 beyond
  __device__ __forceinline__ int box_row(const DecodeParams& p, int tile, int n, int box, int op) const {
    const int at = (tile * boxes) & 31;
    const int k = __shfl_sync(0xffffffffu, kp, (at + box) & 31), v = __shfl_sync(0xffffffffu, vp, (at + box) & 31);
    return box < n && op < 2 ? row(p, op ? v : k, t_begin + tile * kTileN + (box << box_shift)) : -1;
  }
};

// The Q fragments are re-read from shared memory at every k-step instead of living in 4*D/16 registers per thread:
// that keeps the kernel at 128 registers, so two or three CTAs share an SM.
// NB: 16-key blocks a consumer warp handles per step (2 when a warp owns 32 or more keys of a stage).
// T: element type of q, k, v as the kernel reads them; OutT: element type of the output rows (T, or float when the
// inputs are fp16 copies of fp32 tensors).
// kCluster: a cluster of CTAs per (sequence, kv head) pair, nothing planned (see ClusterPart).
template <typename T, int D, int kStages, int NB, int kMaxThreads, int kMinBlocks, typename OutT, bool kCluster>
__global__ void __launch_bounds__(kMaxThreads, kMinBlocks) decode_mma_kernel(const __grid_constant__ CUtensorMap tm_k,
                                                         const __grid_constant__ CUtensorMap tm_v,
                                                         const DecodeParams p) {
  extern __shared__ unsigned char smem_raw[];
  constexpr int CPR = D * 2 / 16;            // 16-byte pieces per row
  constexpr int ROW_BYTES = D * 2;
  constexpr int CHUNKS = D / 64;             // 128-byte column blocks
  constexpr int CHUNK_BYTES = kTileN * 128;  // one column block of a 64-key tile
  constexpr int TILE_BYTES = CHUNKS * CHUNK_BYTES;
  constexpr int STAGE_BYTES = 2 * TILE_BYTES;
  constexpr int KSTEPS = D / 16;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int NMT = p.n_mtiles;
  const int n_cwarps = (blockDim.x >> 5) - 1;   // consumer warps
  const int KS = n_cwarps / NMT;
  const int mt = warp % NMT, ks = warp / NMT;   // meaningful for consumer warps only
  const int rows_pad = NMT * 16;
  const bool is_producer = warp == n_cwarps;
  // (a part of a few tiles: the ring is as long as they are, or as shared memory allows)
  const int n_stages = kCluster ? p.stages : kStages;

  // smem: [stages (1024-byte aligned)] [Q rows] [control]
  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  unsigned char* stage_base = smem;
  unsigned char* q_smem = smem + n_stages * STAGE_BYTES;
  DecodeCtrl* ctrl = reinterpret_cast<DecodeCtrl*>(q_smem + rows_pad * ROW_BYTES);
  const uint32_t stage_s = smem_u32(stage_base);
  const uint32_t q_s = smem_u32(q_smem);

  // Everything that needs nothing from earlier launches comes before the wait for them.
  if (tid == 0) {
    for (int i = 0; i < n_stages; ++i) {
      ptx::mbar_init(smem_u32(&ctrl->full[i]), 1);
      ptx::mbar_init(smem_u32(&ctrl->empty[i]), n_cwarps);
    }
    ctrl->abort_flag = 0;
    ptx::mbar_fence_init();
  }
  if (is_producer && lane == 0) { ptx::prefetch_tensormap(&tm_k); ptx::prefetch_tensormap(&tm_v); }
  ClusterPart part = {};
  __shared__ uint64_t recv_bar;
  if constexpr (kCluster) {
    part = cluster_part<D>(p);
    if (part.size > 1) cluster_begin<D>(p, part, &recv_bar);
  }
  __syncthreads();
  ptx::grid_dep_launch_dependents();
  ptx::grid_dep_wait();      // what earlier launches wrote (the planner's records among it) is visible from here on
  // heads vary fastest across CTAs: the CTAs that run side by side walk the same pages and read
  // neighbouring head slices of each token row, which keeps DRAM rows open
  DecodeItem it;
  int h;
  if constexpr (kCluster) {
    const int pair = blockIdx.x / part.size;
    h = pair % p.kv_heads;
    cluster_item(p, part, pair / p.kv_heads, it);
  } else {
    __shared__ InlinePlan s_plan;
    const int item = blockIdx.x / p.kv_heads;
    if (!decode_item(p, item, s_plan, it)) return;
    h = blockIdx.x - item * p.kv_heads;
  }
  const int b = it.b, c = it.c, n_chunks = it.n_chunks, item0 = it.item0;
  const int len = it.len;
  const int t_begin = it.t_begin, t_end = it.t_end;
  const int ntiles = t_end > t_begin ? (t_end - t_begin + kTileN - 1) / kTileN : 0;

  float m_used[2] = {-INFINITY, -INFINITY};  // exponent reference baked into o[] and l_run[]
  float l_run[2] = {0.f, 0.f};
  float o[D / 8][4];
#pragma unroll
  for (int i = 0; i < D / 8; ++i) { o[i][0] = 0.f; o[i][1] = 0.f; o[i][2] = 0.f; o[i][3] = 0.f; }
  const int r0 = mt * 16 + (lane >> 2);
  const int r1 = r0 + 8;

  if (is_producer) {
    // =========================== TMA producer ===========================
    int h_coord = h;
    long long row0 = it.start;               // ragged
    if (p.layout == B200ATTN_DENSE) { h_coord = 0; row0 = (static_cast<long long>(b) * p.kv_heads + h) * p.max_kv; }
    bool ok = true;
    int issued = 0;
    PageAhead ahead(p, lane);
    ahead.start(p, b, t_begin, t_end);
    int stage = 0, use = 0;
    for (int tile = 0; tile < ntiles; ++tile, stage = stage + 1 < n_stages ? stage + 1 : 0, use += stage == 0) {
      if (use > 0) {
        ok = warp_wait(smem_u32(&ctrl->empty[stage]), (use - 1) & 1);
        if (!ok) break;
      }
      const int t0 = t_begin + tile * kTileN;
      const uint32_t kdst = stage_s + stage * STAGE_BYTES;
      const uint32_t vdst = kdst + TILE_BYTES;
      const uint32_t bar = smem_u32(&ctrl->full[stage]);
      if (p.layout != B200ATTN_PAGED) {
        if (lane == 0) {
          ptx::mbar_arrive_expect_tx(bar, STAGE_BYTES);
          const int row = static_cast<int>(row0 + t0);
          ptx::tma_load_4d(kdst, &tm_k, bar, 0, row, 0, h_coord);
          ptx::tma_load_4d(vdst, &tm_v, bar, 0, row, 0, h_coord);
        }
      } else if (ahead.on) {
        int kr, vr;
        const int count = ahead.tile_rows(p, tile, kr, vr);
        const uint32_t box_bytes = 128u * CHUNKS << ahead.box_shift;
        if (lane == 0) ptx::mbar_arrive_expect_tx(bar, static_cast<uint32_t>(2 * count) * box_bytes);
        __syncwarp();
        const uint32_t boff = static_cast<uint32_t>(lane) * box_bytes;
        if (kr >= 0) ptx::tma_load_4d(kdst + boff, &tm_k, bar, 0, kr, 0, h_coord);
        if (vr >= 0) ptx::tma_load_4d(vdst + boff, &tm_v, bar, 0, vr, 0, h_coord);
      } else {
        // one box of box_rows keys per (lane, round); only pages that hold keys of this chunk are fetched
        const int boxes = kTileN >> p.box_shift;
        const int box_rows = 1 << p.box_shift;
        const int* ktab = p.k_table + static_cast<long long>(b) * p.table_stride;
        const int* vtab = p.v_table + static_cast<long long>(b) * p.table_stride;
        int krow[2], vrow[2];
        int count = 0, n = 0;
        for (int i = lane; i < boxes; i += 32, ++n) {
          const int t = t0 + i * box_rows;
          int kr = -1, vr = -1;
          if (t < t_end) {
            int lp, off;
            if (p.page_shift >= 0) { lp = t >> p.page_shift; off = t & (p.page_size - 1); }
            else { lp = t / p.page_size; off = t - lp * p.page_size; }
            const int kp = __ldcg(ktab + lp), vp = __ldcg(vtab + lp);
            // an entry outside the cache is reported and replaced by page 0: never dereferenced, output stays finite
            const bool kbad = kp < 0 || kp >= p.num_pages, vbad = vp < 0 || vp >= p.num_pages;
            if (kbad || vbad) p.header[0] = DEV_ERR_PAGE_RANGE;
            if (p.num_pages > 0) {
              kr = (kbad ? 0 : kp) * p.page_size + off;
              vr = (vbad ? 0 : vp) * p.page_size + off;
            }
          }
          krow[n] = kr; vrow[n] = vr;
          count += (kr >= 0) + (vr >= 0);
        }
        for (int off = 16; off > 0; off >>= 1) count += __shfl_xor_sync(0xffffffffu, count, off);
        if (lane == 0) ptx::mbar_arrive_expect_tx(bar, static_cast<uint32_t>(count) * box_rows * 128 * CHUNKS);
        __syncwarp();
        n = 0;
        for (int i = lane; i < boxes; i += 32, ++n) {
          const uint32_t boff = static_cast<uint32_t>(i) * box_rows * 128 * CHUNKS;
          if (krow[n] >= 0) ptx::tma_load_4d(kdst + boff, &tm_k, bar, 0, krow[n], 0, h_coord);
          if (vrow[n] >= 0) ptx::tma_load_4d(vdst + boff, &tm_v, bar, 0, vrow[n], 0, h_coord);
        }
      }
      issued = tile + 1;
    }
    if (!ok) {
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; ctrl->abort_flag = 1; }
      // bounded drain of the copies still in flight before the CTA may exit
      for (int t = max(0, issued - n_stages); t < issued; ++t)
        ptx::mbar_wait(smem_u32(&ctrl->full[t % n_stages]), (t / n_stages) & 1);
    }
  } else {
    // =========================== consumers ===========================
    // Q rows (group x drafts, contiguous in memory) -> smem, zero padded to 16-row tiles (the producer does not wait for them)
    {
      const T* qg = static_cast<const T*>(p.q) +
                    ((static_cast<long long>(b) * p.q_heads + static_cast<long long>(h) * p.head_stride + p.head0) * p.q_len) * D;
      for (int idx = tid; idx < rows_pad * CPR; idx += n_cwarps * 32) {
        const int row = idx / CPR, ch = idx % CPR;
        uint4 val = make_uint4(0u, 0u, 0u, 0u);
        if (row < p.rows) val = *reinterpret_cast<const uint4*>(qg + static_cast<long long>(row) * D + ch * 8);
        *reinterpret_cast<uint4*>(q_smem + row * ROW_BYTES + ((ch ^ (row & 7)) << 4)) = val;
      }
      ptx::named_bar_sync(1, n_cwarps * 32);
    }
    uint32_t qf[4];
    const int q_row = mt * 16 + ((lane >> 3) & 1) * 8 + (lane & 7);
    const uint32_t q_rbase = q_s + q_row * ROW_BYTES;
    int lim0 = len - 1, lim1 = len - 1;  // last visible key index for each of this lane's two rows
    if (p.causal) {
      lim0 = len - p.q_len + (r0 % p.q_len);
      lim1 = len - p.q_len + (r1 % p.q_len);
    }
    const int lim_min = min(lim0, lim1);
    const float sl2 = p.scale_log2;
    bool ok = true;

    int stage = 0, use = 0;
    for (int tile = 0; tile < ntiles; ++tile, stage = stage + 1 < n_stages ? stage + 1 : 0, use += stage == 0) {
      ok = warp_wait(smem_u32(&ctrl->full[stage]), use & 1);
      if (!ok) break;
      const uint32_t ks_base = stage_s + stage * STAGE_BYTES;
      const uint32_t vs_base = ks_base + TILE_BYTES;
      const int tile_t0 = t_begin + tile * kTileN;
      const int valid = len - tile_t0;  // keys of this tile that belong to the sequence

      // one step = NB consecutive 16-key blocks: the softmax bookkeeping (max, shuffles, rescale test) and the
      // Q fragment reads are shared by the NB blocks
      for (int sb = ks * NB; sb < kTileN / 16; sb += KS * NB) {
        const int tok0 = sb * 16;             // within tile
        const int abs0 = tile_t0 + tok0;      // within sequence
        if (abs0 >= t_end) break;
        if (valid < tok0 + 16 * NB) {
          // keys past the sequence end get P == 0, but their V rows may hold anything (page tails,
          // the next sequence, stale shared memory): zero them so that 0 * x stays 0
          unsigned char* vtile = stage_base + stage * STAGE_BYTES + TILE_BYTES;
          const int first = max(valid, tok0);
          const int npieces = (tok0 + 16 * NB - first) * CHUNKS * 8;
          for (int i = lane; i < npieces; i += 32) {
            const int t = first + i / (CHUNKS * 8), cb = (i >> 3) % CHUNKS;
            *reinterpret_cast<uint4*>(vtile + tile_row_offset<CHUNKS>(t, cb, p.box_shift) + ((i & 7) << 4)) = make_uint4(0u, 0u, 0u, 0u);
          }
          __syncwarp();
        }
        float s[2 * NB][4];
#pragma unroll
        for (int i = 0; i < 2 * NB; ++i) { s[i][0] = 0.f; s[i][1] = 0.f; s[i][2] = 0.f; s[i][3] = 0.f; }
        {
          const int mat = lane >> 3;
          uint32_t roff[NB][CHUNKS];
#pragma unroll
          for (int nb = 0; nb < NB; ++nb) {
            const int trow = tok0 + nb * 16 + (mat >> 1) * 8 + (lane & 7);
#pragma unroll
            for (int cb = 0; cb < CHUNKS; ++cb) roff[nb][cb] = tile_row_offset<CHUNKS>(trow, cb, p.box_shift);
          }
#pragma unroll
          for (int kk = 0; kk < KSTEPS; ++kk) {
            const int ch = kk * 2 + (mat & 1);   // 16-byte piece index along D
            const int qch = kk * 2 + (lane >> 4);
            ldmatrix_x4(qf, q_rbase + ((qch ^ (q_row & 7)) << 4));
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
              uint32_t kb[4];
              ldmatrix_x4(kb, ks_base + swz_piece(roff[nb][ch >> 3], ch & 7));
              mma_m16n8k16<T>(s[2 * nb], qf, kb[0], kb[1]);
              mma_m16n8k16<T>(s[2 * nb + 1], qf, kb[2], kb[3]);
            }
          }
        }
        // scale, mask (only where the step reaches a row's last visible key), online softmax in the exp2 domain
        float mx0 = -INFINITY, mx1 = -INFINITY;
        const bool all_visible = __all_sync(0xffffffffu, abs0 + 16 * NB - 1 <= lim_min);
        if (all_visible) {
#pragma unroll
          for (int nt = 0; nt < 2 * NB; ++nt) {
            s[nt][0] *= sl2; s[nt][1] *= sl2; s[nt][2] *= sl2; s[nt][3] *= sl2;
            mx0 = fmaxf(mx0, fmaxf(s[nt][0], s[nt][1]));
            mx1 = fmaxf(mx1, fmaxf(s[nt][2], s[nt][3]));
          }
        } else {
#pragma unroll
          for (int nt = 0; nt < 2 * NB; ++nt) {
            const int col = abs0 + nt * 8 + 2 * (lane & 3);
            s[nt][0] = (col <= lim0) ? s[nt][0] * sl2 : -INFINITY;
            s[nt][1] = (col + 1 <= lim0) ? s[nt][1] * sl2 : -INFINITY;
            s[nt][2] = (col <= lim1) ? s[nt][2] * sl2 : -INFINITY;
            s[nt][3] = (col + 1 <= lim1) ? s[nt][3] * sl2 : -INFINITY;
            mx0 = fmaxf(mx0, fmaxf(s[nt][0], s[nt][1]));
            mx1 = fmaxf(mx1, fmaxf(s[nt][2], s[nt][3]));
          }
        }
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 1));
        mx0 = fmaxf(mx0, __shfl_xor_sync(0xffffffffu, mx0, 2));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 1));
        mx1 = fmaxf(mx1, __shfl_xor_sync(0xffffffffu, mx1, 2));
        // the accumulators are rescaled only when a row's max grew by more than 2^8; until then the
        // older reference keeps being used (exact: the same reference normalises the row at the end).  In a cluster a row has
        // fewer warps than a plan's shortest items give it, with more keys each, and fewer weights that are exactly one: there a
        // warp follows its maximum more closely.  Error against 64 bits of one user of 1 500 keys, over that of its planned call:
        // 1.03 at eight powers of two, 1.02 at three, 0.96 at one, 0.93 at none; the last costs up to a tenth of a short call.
        constexpr float kMove = kCluster ? 1.f : 8.f;
        const bool need0 = (mx0 - m_used[0]) > kMove, need1 = (mx1 - m_used[1]) > kMove;
        if (__any_sync(0xffffffffu, need0 || need1)) {
          float a0 = 1.f, a1 = 1.f;
          if (need0) { a0 = fast_exp2(m_used[0] - mx0); m_used[0] = mx0; }
          if (need1) { a1 = fast_exp2(m_used[1] - mx1); m_used[1] = mx1; }
          l_run[0] *= a0; l_run[1] *= a1;
#pragma unroll
          for (int i = 0; i < D / 8; ++i) { o[i][0] *= a0; o[i][1] *= a0; o[i][2] *= a1; o[i][3] *= a1; }
        }
        const float ms0 = (m_used[0] == -INFINITY) ? 0.f : m_used[0];
        const float ms1 = (m_used[1] == -INFINITY) ? 0.f : m_used[1];
        uint32_t pa[NB][4];
#pragma unroll
        for (int nt = 0; nt < 2 * NB; ++nt) {
          const float p0 = fast_exp2(s[nt][0] - ms0), p1 = fast_exp2(s[nt][1] - ms0);
          const float p2 = fast_exp2(s[nt][2] - ms1), p3 = fast_exp2(s[nt][3] - ms1);
          l_run[0] += p0 + p1;   // per-lane partial row sums; reduced over the quad at the end
          l_run[1] += p2 + p3;
          pa[nt >> 1][(nt & 1) * 2 + 0] = ElemTraits<T>::pack2(p0, p1);
          pa[nt >> 1][(nt & 1) * 2 + 1] = ElemTraits<T>::pack2(p2, p3);
        }
        {
          const int mat = lane >> 3;
          uint32_t roff[NB][CHUNKS];
#pragma unroll
          for (int nb = 0; nb < NB; ++nb) {
            const int trow = tok0 + nb * 16 + (mat & 1) * 8 + (lane & 7);
#pragma unroll
            for (int cb = 0; cb < CHUNKS; ++cb) roff[nb][cb] = tile_row_offset<CHUNKS>(trow, cb, p.box_shift);
          }
#pragma unroll
          for (int n0 = 0; n0 < D / 16; ++n0) {
            const int ch = n0 * 2 + (mat >> 1);
#pragma unroll
            for (int nb = 0; nb < NB; ++nb) {
              uint32_t vb[4];
              ldmatrix_x4_trans(vb, vs_base + swz_piece(roff[nb][ch >> 3], ch & 7));
              mma_m16n8k16<T>(o[2 * n0], pa[nb], vb[0], vb[1]);
              mma_m16n8k16<T>(o[2 * n0 + 1], pa[nb], vb[2], vb[3]);
            }
          }
        }
      }
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(smem_u32(&ctrl->empty[stage]));
    }
    if (!ok && lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; ctrl->abort_flag = 1; }
  }
  __syncthreads();  // every tile consumed (or the CTA gave up): the stage ring is free for the cross-warp combine

  float* comb_o = reinterpret_cast<float*>(stage_base);
  float* comb_ml = comb_o + static_cast<size_t>(KS) * rows_pad * D;
  if (!is_producer) {
    l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], 1);
    l_run[0] += __shfl_xor_sync(0xffffffffu, l_run[0], 2);
    l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], 1);
    l_run[1] += __shfl_xor_sync(0xffffffffu, l_run[1], 2);
    float* o0 = comb_o + (static_cast<size_t>(ks) * rows_pad + r0) * D;
    float* o1 = comb_o + (static_cast<size_t>(ks) * rows_pad + r1) * D;
#pragma unroll
    for (int i = 0; i < D / 8; ++i) {
      const int col = i * 8 + 2 * (lane & 3);
      *reinterpret_cast<float2*>(o0 + col) = make_float2(o[i][0], o[i][1]);
      *reinterpret_cast<float2*>(o1 + col) = make_float2(o[i][2], o[i][3]);
    }
    if ((lane & 3) == 0) {
      comb_ml[(ks * rows_pad + r0) * 2] = m_used[0];
      comb_ml[(ks * rows_pad + r0) * 2 + 1] = l_run[0];
      comb_ml[(ks * rows_pad + r1) * 2] = m_used[1];
      comb_ml[(ks * rows_pad + r1) * 2 + 1] = l_run[1];
    }
  }
  __syncthreads();
  if (ctrl->abort_flag) {
    // A bounded wait ran out: the CTA's rows are unknown.  It still emits and draws its ticket, so that the
    // (sequence, kv head) is merged and its counter returns to zero, but with NaN rows: the failure shows in the
    // output as well as in the error word.
    poison_rows(comb_o, comb_ml, KS * rows_pad, D);
    __syncthreads();
  }
  if constexpr (kCluster) {
    // (behind the control block, rounded up to 16 bytes)
    unsigned char* recv = reinterpret_cast<unsigned char*>(ctrl) + ((sizeof(DecodeCtrl) + 15) & ~size_t(15));
    if (part.size > 1) {
      cluster_emit<OutT, D>(p, part, b, h, comb_o, comb_ml, KS, rows_pad, recv, &recv_bar);
      return;
    }
  }
  emit_and_merge<OutT, D>(p, b, h, c, n_chunks, item0, comb_o, comb_ml, KS, rows_pad, &ctrl->ticket);
}

// ---------------------------------------------------------------------------
// tcgen05 kernel for many q rows per KV head (speculative decode: group x drafts > 16 rows).
//
// With 17..128 rows the warp-level MMA kernel above is bound by shared-memory bandwidth: every K/V fragment is
// re-read by ldmatrix once per 16-row tile.  Here the rows are padded to one 128-row tcgen05 tile whose A operands
// live in tensor memory (Q is written there once per work unit, P once per key tile), so shared memory is read
// exactly once per K/V byte, by the tensor core.  Per 64-key tile: S = Q K^T (TS MMA, 128 x 64 x D) -> the softmax
// warps (thread = q row, only the warps that hold real rows work) exponentiate S against the row's standing reference,
// keep the row sums, write P as packed 16-bit over S -> O += P V (TS MMA, V is the MN-major B operand).  Two CTAs share
// an SM (256 TMEM columns, 3 stages of 64 keys each), which overlaps one CTA's softmax with the other's MMAs.
//
// What bounds it.  A tile is a chain: scores seen 270 cycles after the issue, 830 of softmax, 550 of MMAs; and a stage is
// away for 360 (freed and noticed) + 600 to 1 200 (its copies issued by three warps) + 2 200 (under load).  Long batches run
// at the board's power limit on top of that (32 sequences of 1 000 to 33 000 keys: 1.37 GHz).  Against one issuing warp, a
// pass for the maximum, and stages given back only when the next had arrived: 8 x 8 192 keys of one head, D 64, 28.5 -> 25.1
// us; 4 x 8 192, D 128, 50.6 -> 48.2; 16 x 16 384 and 128 rows 75 -> 68; one sequence of 8 192 in pages 43.5 -> 40.2.
//
// The kernel is persistent: the grid is one wave (two CTAs per SM); a CTA starts with unit (item, kv head) number
// blockIdx.x of the planner's longest-first list and its producer warp draws further units from a counter in the
// workspace header, publishing them to the MMA and softmax warps through a four-deep ring in shared memory.  The
// producer runs ahead into the next unit while the last tiles of the current one are still being consumed: the stage
// ring - the bytes the SM keeps in flight, which is what bounds this kernel - never drains between units, and tensor
// memory, barriers and tensor maps are set up once per CTA.  For that the epilogue leaves shared memory alone: each
// softmax thread writes its O row from registers to the output (single-chunk sequences) or to the partials; merges
// are claimed by CTAs in their teardown.  Planner and partial / ticket formats are shared with the kernels above.
// ---------------------------------------------------------------------------
constexpr int kUmmaStages = 3;
constexpr int kUmmaTmemCols = 256;
// A tile's 64 exponentials of a row against the reference that stands are good as long as their sum is at most this (P then
// fits 16 bits); when it is not, the row's maximum lies four powers of two or more above its reference, and a reference
// moves when the maximum is kMoveThreshold above it.
constexpr float kMaxRowSum = 1024.0f;
constexpr float kMoveThreshold = 3.0f;   // log2 units
constexpr int kUmmaThreads = 256;     // four softmax warps, three that issue copies, the MMA warp
constexpr int kUmmaIssuers = 3;       // warps that share the copies of a stage of pages
constexpr int kUmmaUnitRing = 4;      // units the producer may be ahead of the slowest consumer
constexpr int kUmmaMaxClaims = 1;     // merges a CTA takes per sweep of the ticket counters in its teardown
constexpr int kMergeClaimed = 1 << 30; // added to a pair's ticket counter by the CTA that merges it

struct __align__(8) UmmaCtrl {
  uint64_t full[kUmmaStages];
  uint64_t empty[kUmmaStages];
  uint64_t q_ready;   // softmax warps -> MMA warp: the unit's Q rows are in tensor memory
  uint64_t s_full;    // MMA warp -> softmax warps (commit): S of a tile
  uint64_t p_ready;   // softmax warps -> MMA warp: P of a tile
  uint64_t o_done;    // MMA warp -> softmax warps (commit): PV of a tile
  uint64_t o_free;    // softmax warps -> MMA warp: the finished unit's O has been read out of tensor memory
  uint64_t drained;   // the MMAs of an issuer that gave up
  uint64_t rows_out;  // softmax threads: my partial rows of the unit are written and fenced
  uint64_t unit_full[kUmmaUnitRing];    // producer -> MMA and softmax warps: slot r % ring holds the CTA's r-th unit
  uint64_t unit_empty[kUmmaUnitRing];   // MMA warp + softmax warps -> producer: done with that slot
  int unit_ring[kUmmaUnitRing];         // unit indices (n_units or more: the CTA has no r-th unit)
  int published;                        // units published so far, the end mark included
  uint32_t tmem_base;
  int abort_flag;
  int abort_round;    // first round (unit of this CTA) whose output may be incomplete after a wait ran out
  int ready;          // teardown: (sequence, kv head) pairs whose chunks are all published and that nobody merges yet
  int n_reserved;     // teardown: claim attempts of this sweep
  int n_claimed;      // teardown: pairs this CTA claimed in this sweep
  int claimed[kUmmaMaxClaims];
};

// One (work item, kv head) unit as every role of the CTA reads it from the planner's records.
struct UmmaUnit {
  long long seq_start;
  int b, h, c, n_chunks, item0, len, t_begin, t_end, ntiles;
};

__device__ __forceinline__ UmmaUnit umma_unit(const DecodeParams& p, int u) {
  UmmaUnit w;
  const int item = u / p.kv_heads;
  w.h = u - item * p.kv_heads;
  const int4 rec0 = p.item_info[2 * item];
  const int4 rec1 = p.item_info[2 * item + 1];
  w.b = rec0.x; w.c = rec0.y & 0xffff; w.n_chunks = static_cast<unsigned>(rec0.y) >> 16; w.item0 = rec0.z;
  w.len = rec1.x;
  w.seq_start = (static_cast<long long>(rec1.w) << 32) | static_cast<unsigned int>(rec1.z);
  w.t_begin = rec0.w;
  w.t_end = rec1.y;
  w.ntiles = w.t_end > w.t_begin ? (w.t_end - w.t_begin + kTileN - 1) / kTileN : 0;
  return w;
}

// Merges.  A (sequence, kv head) pair whose chunks have all drawn their tickets is merged by whichever CTA claims
// it while sweeping the ticket counters in its teardown, with all of its threads: CTAs that finish early take the pairs that
// are complete, the CTA that draws a pair's last ticket sweeps after it did, so every pair is merged by the time
// the last CTA leaves, and no CTA waits for another.  A CTA takes one pair per sweep and sweeps again as long as it
// saw a complete pair; header[3] (tickets drawn and not merged) lets a CTA skip the sweep when there is nothing.
template <typename OutT, int D, typename Ctrl>
__device__ __forceinline__ void claim_merges(const DecodeParams& p, Ctrl* ctrl, int me) {
  if (ctrl->abort_flag) return;
  const int tid = threadIdx.x;
  const int n_pairs = p.batch * p.kv_heads;
  for (int sweep = 0; sweep < n_pairs + 64; ++sweep) {
    if (tid == 0) {
      ctrl->ready = *reinterpret_cast<volatile int*>(p.header + 3);
      ctrl->n_reserved = 0;
      ctrl->n_claimed = 0;
    }
    __syncthreads();
    if (ctrl->ready <= 0) break;
    for (int e = tid; e < n_pairs; e += static_cast<int>(blockDim.x)) {
      const int pair = (e + me * 61) % n_pairs;            // CTAs start their sweeps at different pairs
      const int b = pair / p.kv_heads;
      const int n = p.item_start[b + 1] - p.item_start[b];
      if (n > 1 && *reinterpret_cast<volatile int*>(p.counters + pair) == n &&
          atomicAdd(&ctrl->n_reserved, 1) < kUmmaMaxClaims &&
          atomicCAS(p.counters + pair, n, n + kMergeClaimed) == n) {
        atomicSub(p.header + 3, n);
        ctrl->claimed[atomicAdd(&ctrl->n_claimed, 1)] = pair;
      }
    }
    __syncthreads();
    if (ctrl->n_reserved == 0) break;                      // no complete pair in sight: whoever completes one sweeps
    const int n_claimed = ctrl->n_claimed;
    for (int i = 0; i < n_claimed; ++i) {
      const int pair = ctrl->claimed[i];
      const int b = pair / p.kv_heads, h = pair - b * p.kv_heads;
      const int item0 = p.item_start[b];
      OutT* out = static_cast<OutT*>(p.out) +
                  ((static_cast<long long>(b) * p.q_heads + static_cast<long long>(h) * p.head_stride + p.head0) * p.q_len) * D;
      const int n = p.item_start[b + 1] - item0;
      merge_chunks<OutT, D, false>(p, static_cast<long long>(item0) * p.kv_heads + h, p.kv_heads, n, out, tid, static_cast<int>(blockDim.x), nullptr);
      if (tid == 0) reset_ticket(p, pair, n);
    }
    __syncthreads();
  }
}

// A bounded wait ran out: the rows of the unit whose rows were being written, and of the units this CTA had not
// reached, are unknown.  They are filled with NaN (and their tickets are not drawn, so nobody merges over them):
// the failure shows in the output as well as in the error word.  `unit_of(r)`: the CTA's r-th unit.
template <typename OutT, int D, typename Ctrl, typename UnitOf>
__device__ __forceinline__ void poison_units(const DecodeParams& p, Ctrl* ctrl, int n_units, UnitOf unit_of) {
  const OutT nan_t = ElemTraits<OutT>::from_float(__int_as_float(0x7fc00000));
  // The slots of units that are not finished cannot have been reused, so those units are among the ring's: from its oldest on, where
  // abort_round lies further back (0: nobody knows), and in their order, in which the end mark is the last.
  for (int r = max(ctrl->abort_round, ctrl->published - kUmmaUnitRing); r < ctrl->published; ++r) {
    if (ctrl->unit_ring[r % kUmmaUnitRing] >= n_units) break;
    const UmmaUnit w = unit_of(r);
    OutT* out = static_cast<OutT*>(p.out) +
                ((static_cast<long long>(w.b) * p.q_heads + static_cast<long long>(w.h) * p.head_stride + p.head0) * p.q_len) * D;
    for (int i = threadIdx.x; i < p.rows * D; i += static_cast<int>(blockDim.x)) out[i] = nan_t;
  }
}

// T: element type of q, k, v as the kernel reads them; OutT: element type of the output rows (T, or float when the
// inputs are fp16 copies of fp32 tensors).  kOwnPlan: no planner has run, and every CTA works out the one unit that is its own.
template <typename T, int D, typename OutT, bool kOwnPlan>
__global__ void __launch_bounds__(kUmmaThreads, 2) decode_umma_kernel(const __grid_constant__ CUtensorMap tm_k,
                                                             const __grid_constant__ CUtensorMap tm_v,
                                                             const DecodeParams p) {
  using namespace ptx;
  extern __shared__ unsigned char smem_raw[];
  __shared__ InlinePlan s_plan;
  __shared__ UmmaUnit s_unit;
  constexpr int CHUNKS = D / 64;
  constexpr int CHUNK_BYTES = kTileN * 128;
  constexpr int TILE_BYTES = CHUNKS * CHUNK_BYTES;
  constexpr int STAGE_BYTES = 2 * TILE_BYTES;
  constexpr int kQCols = D / 2;               // TMEM columns of the packed 16-bit Q tile
  constexpr int kSCol = kQCols;               // S (64 fp32 columns); P overwrites its first 32
  constexpr int kOCol = kQCols + kTileN;      // O (D fp32 columns)
  static_assert(kOCol + D <= kUmmaTmemCols, "TMEM budget");
  // (with up to 64 rows only the first two softmax warps work: the producer and the MMA warp are not among their neighbours
  // in the SM's four partitions)
  constexpr int kHelper = 4, kProducer = 6, kMma = 7;

  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int R = p.rows;
  const int active_warps = (R + 31) >> 5;      // softmax warps that own real rows
  const int n_softmax = active_warps * 32;
  // A warp issues a box every 95 to 130 cycles, whatever the box's size, and different warps do not hold one another up: the
  // sixteen boxes of a stage of 16-key pages took one warp 1 580 of the 2 540 cycles that a CTA had for a tile.  (Pages that
  // are cut into more boxes than a warp has lanes are left to the producer.)  The two or four boxes of a dense or packed tile
  // are the producer's alone: what a further warp saves there is less than its way to the unit's record and the arrivals cost
  // (64 sequences of 20 keys, 64/8 heads, D 128, 16.0 -> 15.4 us, of 600 41.5 -> 41.2; 16 of 20 to 60 13.1 -> 12.6).
  const int boxes_log2 = p.layout == B200ATTN_PAGED ? 6 - p.box_shift : 0;
  const bool shared_issue = boxes_log2 <= 5;
  const int issuers = p.layout == B200ATTN_PAGED && shared_issue ? kUmmaIssuers : 1;

  unsigned char* smem = reinterpret_cast<unsigned char*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  UmmaCtrl* ctrl = reinterpret_cast<UmmaCtrl*>(smem + kUmmaStages * STAGE_BYTES);
  const uint32_t smem_base = smem_u32(smem);

  if (tid == 0) {
    for (int i = 0; i < kUmmaStages; ++i) {
      mbar_init(smem_u32(&ctrl->full[i]), issuers);
      mbar_init(smem_u32(&ctrl->empty[i]), 1);
    }
    mbar_init(smem_u32(&ctrl->q_ready), n_softmax);
    mbar_init(smem_u32(&ctrl->s_full), 1);
    mbar_init(smem_u32(&ctrl->p_ready), active_warps);
    mbar_init(smem_u32(&ctrl->o_done), 1);
    mbar_init(smem_u32(&ctrl->o_free), n_softmax);
    mbar_init(smem_u32(&ctrl->rows_out), n_softmax);
    mbar_init(smem_u32(&ctrl->drained), 1);
    for (int i = 0; i < kUmmaUnitRing; ++i) {
      mbar_init(smem_u32(&ctrl->unit_full[i]), 1);
      mbar_init(smem_u32(&ctrl->unit_empty[i]), active_warps + issuers);
    }
    ctrl->published = 0;
    ctrl->abort_flag = 0;
    ctrl->abort_round = 0x7fffffff;
    mbar_fence_init();
  }
  if (warp == kMma) {
    tmem_alloc(smem_u32(&ctrl->tmem_base), kUmmaTmemCols);
    tmem_relinquish();
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = ctrl->tmem_base;
  volatile int* abort_flag = &ctrl->abort_flag;

  // (no launch_dependents here: with the next call's planner waiting beside it this kernel ran 3 % slower, 363 us
  // instead of 352 on 32 sequences of 1 to 33 thousand keys)
  // (Nor without a planner: the next call's CTAs take the SMs that this one leaves empty, and then share some while others
  // stay empty: one sequence of 8 000 keys, 64/8 heads, 8 drafts 36.0 us instead of 28.4, of 2 000 with 5 drafts 20.8 and 17.6.)
  ptx::grid_dep_wait();      // the planner's records are complete and visible from here on
  const int G = static_cast<int>(gridDim.x), me = static_cast<int>(blockIdx.x);
  int n_units;
  if constexpr (kOwnPlan) {
    // a CTA per unit, which it works out itself: unit `me` is its only one
    DecodeItem mine;
    const bool have = plan_inline(p, me / p.kv_heads, s_plan, mine);
    if (tid == 0 && have) {
      UmmaUnit w;
      w.seq_start = mine.start;
      w.b = mine.b; w.h = me % p.kv_heads; w.c = mine.c; w.n_chunks = mine.n_chunks; w.item0 = mine.item0; w.len = mine.len;
      w.t_begin = mine.t_begin; w.t_end = mine.t_end;
      w.ntiles = w.t_end > w.t_begin ? (w.t_end - w.t_begin + kTileN - 1) / kTileN : 0;
      s_unit = w;
    }
    __syncthreads();
    n_units = have ? me + 1 : 0;
  } else {
    n_units = p.header[2] * p.kv_heads;
  }
  auto unit_of = [&](int u) -> UmmaUnit {
    if constexpr (kOwnPlan) return s_unit;
    else return umma_unit(p, u);
  };
  // Units are handed out dynamically, longest first: a CTA's first unit is its own index, later ones are drawn from a
  // counter in the workspace header by the producer warp, which publishes them to the other warps through a small
  // ring in shared memory (a static deal cannot follow a batch of a few long and many short sequences: the CTAs that
  // were dealt one more long unit finish last).  unit_at(r): the CTA's r-th unit, n_units or more when there is
  // none, -1 when the (bounded) wait for the producer ran out.
  auto unit_at = [&](int r) -> int {
    if (!warp_wait(smem_u32(&ctrl->unit_full[r % kUmmaUnitRing]), (r / kUmmaUnitRing) & 1)) return -1;
    return *reinterpret_cast<volatile int*>(&ctrl->unit_ring[r % kUmmaUnitRing]);
  };
  auto unit_done = [&](int r) {   // this warp will not read slot r again
    __syncwarp();
    if (lane == 0) mbar_arrive(smem_u32(&ctrl->unit_empty[r % kUmmaUnitRing]));
  };

  // Issuing warp `part`'s share of a stage: of the tile's (box, operand, column block) every `issuers`-th.
  auto issue_share = [&](const UmmaUnit& w, PageAhead& ahead, int tile, int stage, int part) {
    const bool paged = p.layout == B200ATTN_PAGED;
    const int t0 = w.t_begin + tile * kTileN;
    const int boxes = 1 << boxes_log2, total = 2 * CHUNKS << boxes_log2;
    const uint32_t box_bytes = static_cast<uint32_t>(kTileN >> boxes_log2) * 128;
    const uint32_t bar = smem_u32(&ctrl->full[stage]);
    const int n = paged ? ahead.advance(p, tile) : 1;
    int h_coord = w.h;
    long long row0 = w.seq_start;
    if (p.layout == B200ATTN_DENSE) { h_coord = 0; row0 = (static_cast<long long>(w.b) * p.kv_heads + w.h) * p.max_kv; }
    // boxes of the share in this tile: the indices part, part + issuers, ... whose box is one of the first n
    int count = 0;
    for (int base = 0; base < total; base += 32 * issuers) {
      const int idx = base + lane * issuers + part;
      count += __popc(__ballot_sync(0xffffffffu, idx < total && (idx & (boxes - 1)) < n));
    }
    if (lane == 0) {
      if (count > 0) mbar_arrive_expect_tx(bar, static_cast<uint32_t>(count) * box_bytes);
      else mbar_arrive(bar);
    }
    __syncwarp();
    for (int base = 0; base < total; base += 32 * issuers) {
      const int idx = base + lane * issuers + part;
      const int box = idx & (boxes - 1), rest = idx >> boxes_log2, op = rest & 1, cc = rest >> 1;
      const int row = paged ? ahead.box_row(p, tile, n, box, idx < total ? op : 2) : (idx < total ? static_cast<int>(row0 + t0) : -1);
      const uint32_t dst = smem_base + stage * STAGE_BYTES + op * TILE_BYTES + cc * CHUNK_BYTES + box * box_bytes;
      if (row >= 0) tma_load_3d(dst, op ? &tm_v : &tm_k, bar, cc * 64, h_coord, row);
    }
  };

  if (warp == kProducer) {
    // =========================== TMA producer ===========================
    if (lane == 0) { prefetch_tensormap(&tm_k); prefetch_tensormap(&tm_v); }
    bool ok = true;
    int g = 0;                                   // tiles issued so far, over all units
    PageAhead ahead(p, lane);                    // (a unit's first entries are read when it is drawn)
    auto publish = [&](int r, int u) {            // lane 0
      ctrl->unit_ring[r % kUmmaUnitRing] = u;
      ctrl->published = r + 1;
      mbar_arrive(smem_u32(&ctrl->unit_full[r % kUmmaUnitRing]));
    };
    // Dealt out (slots > 0): the CTA's units are the items of its slot, in order.  Else its first unit is its own index.
    const int slots = kOwnPlan ? 0 : p.header[5];
    int u = me, u_end = n_units;
    if (slots > 0) {
      const int slot = me / p.kv_heads;
      const int* slot_first = reinterpret_cast<const int*>(p.item_info + 2 * static_cast<long long>(p.max_items)) - (slots + 1);
      u = n_units;
      if (slot < slots) {
        u = __ldcg(slot_first + slot) * p.kv_heads + me % p.kv_heads;
        u_end = __ldcg(slot_first + slot + 1) * p.kv_heads;
      }
    }
    if (u >= u_end) u = n_units;
    if (lane == 0) publish(0, u);
    for (int r = 0; ok && u < n_units; ++r) {
      const UmmaUnit w = unit_of(u);
      if (r == 0) ahead.start(p, w.b, w.t_begin, w.t_end);
      for (int tile = 0; tile < w.ntiles; ++tile) {
        const int stage = g % kUmmaStages, use = g / kUmmaStages;
        if (use > 0) {
          ok = warp_wait(smem_u32(&ctrl->empty[stage]), (use - 1) & 1);
          if (!ok || *abort_flag) { ok = false; break; }
        }
        if (shared_issue) {
          issue_share(w, ahead, tile, stage, 0);
        } else {
          const int t0 = w.t_begin + tile * kTileN;
          const uint32_t kdst = smem_base + stage * STAGE_BYTES;
          const uint32_t vdst = kdst + TILE_BYTES;
          const uint32_t bar = smem_u32(&ctrl->full[stage]);
          const int box_rows = 1 << p.box_shift;
          const int h_coord = w.h;
          const int boxes = kTileN >> p.box_shift;
          const int* ktab = p.k_table + static_cast<long long>(w.b) * p.table_stride;
          const int* vtab = p.v_table + static_cast<long long>(w.b) * p.table_stride;
          int krow[2], vrow[2];
          int count = 0, n = 0;
          for (int i = lane; i < boxes; i += 32, ++n) {
            const int t = t0 + i * box_rows;
            int kr = -1, vr = -1;
            if (t < w.t_end) {
              int lp, off;
              if (p.page_shift >= 0) { lp = t >> p.page_shift; off = t & (p.page_size - 1); }
              else { lp = t / p.page_size; off = t - lp * p.page_size; }
              const int kp = __ldcg(ktab + lp), vp = __ldcg(vtab + lp);
              // an entry outside the cache is reported and replaced by page 0: never dereferenced, output stays finite
              const bool kbad = kp < 0 || kp >= p.num_pages, vbad = vp < 0 || vp >= p.num_pages;
              if (kbad || vbad) p.header[0] = DEV_ERR_PAGE_RANGE;
              if (p.num_pages > 0) {
                kr = (kbad ? 0 : kp) * p.page_size + off;
                vr = (vbad ? 0 : vp) * p.page_size + off;
              }
            }
            krow[n] = kr; vrow[n] = vr;
            count += (kr >= 0) + (vr >= 0);
          }
          for (int off = 16; off > 0; off >>= 1) count += __shfl_xor_sync(0xffffffffu, count, off);
          if (lane == 0) mbar_arrive_expect_tx(bar, static_cast<uint32_t>(count) * box_rows * 128 * CHUNKS);
          __syncwarp();
          n = 0;
          for (int i = lane; i < boxes; i += 32, ++n) {
            const uint32_t roff = static_cast<uint32_t>(i) * box_rows * 128;
#pragma unroll
            for (int cc = 0; cc < CHUNKS; ++cc) {
              if (krow[n] >= 0) tma_load_3d(kdst + cc * CHUNK_BYTES + roff, &tm_k, bar, cc * 64, h_coord, krow[n]);
              if (vrow[n] >= 0) tma_load_3d(vdst + cc * CHUNK_BYTES + roff, &tm_v, bar, cc * 64, h_coord, vrow[n]);
            }
          }
        }
        ++g;
      }
      if (!ok) break;
      // The unit's last copy is on its way: only now draw the next unit (as late as the ring allows, so that the
      // longest-first list is dealt to whoever runs dry first), publish it, and pull what its first steps need -
      // the block-table entries of its first tile, its Q rows (into L2) - ahead of the warps that will ask for them.
      int u_next = n_units;
      if (r + 1 >= kUmmaUnitRing) {
        ok = warp_wait(smem_u32(&ctrl->unit_empty[(r + 1) % kUmmaUnitRing]), ((r + 1) / kUmmaUnitRing - 1) & 1);
        if (!ok || *abort_flag) { ok = false; break; }
      }
      if (lane == 0) {
        u_next = kOwnPlan ? n_units : slots > 0 ? u + p.kv_heads : min(G + atomicAdd(p.header + 4, 1), n_units);
        if (u_next >= u_end) u_next = n_units;
        publish(r + 1, u_next);
      }
      u_next = __shfl_sync(0xffffffffu, u_next, 0);
      if (u_next < n_units) {
        const UmmaUnit w2 = unit_of(u_next);
        ahead.start(p, w2.b, w2.t_begin, w2.t_end);
        const T* q2 = static_cast<const T*>(p.q) +
                      ((static_cast<long long>(w2.b) * p.q_heads + static_cast<long long>(w2.h) * p.head_stride + p.head0) * p.q_len) * D;
        for (int i = lane; i < (R * D * static_cast<int>(sizeof(T))) / 128; i += 32) prefetch_l2(reinterpret_cast<const char*>(q2) + i * 128);
      }
      u = u_next;
    }
    if (!ok) {
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
      // bounded drain of the copies still in flight before the CTA may exit
      for (int t = max(0, g - kUmmaStages); t < g; ++t)
        mbar_wait(smem_u32(&ctrl->full[t % kUmmaStages]), (t / kUmmaStages) & 1);
    }
  } else if (warp >= kHelper && warp < kHelper + kUmmaIssuers - 1) {
    // =========================== further issuing warps ===========================
    if (issuers > 1) {
      bool ok = true;
      int g = 0;
      PageAhead ahead(p, lane);
      for (int r = 0; ok; ++r) {
        const int u = unit_at(r);
        if (u < 0) { ok = false; break; }
        unit_done(r);
        if (u >= n_units) break;
        const UmmaUnit w = unit_of(u);
        ahead.start(p, w.b, w.t_begin, w.t_end);
        for (int tile = 0; tile < w.ntiles; ++tile, ++g) {
          const int stage = g % kUmmaStages, use = g / kUmmaStages;
          if (use > 0) {
            ok = warp_wait(smem_u32(&ctrl->empty[stage]), (use - 1) & 1);
            if (!ok || *abort_flag) { ok = false; break; }
          }
          issue_share(w, ahead, tile, stage, 1 + warp - kHelper);
        }
      }
      if (!ok) {
        if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
        for (int t = max(0, g - kUmmaStages); t < g; ++t)
          mbar_wait(smem_u32(&ctrl->full[t % kUmmaStages]), (t / kUmmaStages) & 1);
      }
    }
  } else if (warp == kMma) {
    // =========================== MMA issuer ===========================
    constexpr int kFmt = std::is_same<T, __nv_bfloat16>::value ? 1 : 0;
    constexpr uint32_t idesc_s = make_idesc_f16(128, kTileN, kFmt, 0);
    constexpr uint32_t idesc_o = make_idesc_f16(128, D, kFmt, 1);
    const uint64_t kdesc = make_smem_desc_sw128(smem_base, 16);
    const uint64_t vdesc = make_smem_desc_sw128(smem_base, CHUNK_BYTES);
    // The warp stays converged while it issues (every lane runs the descriptor arithmetic, one elected lane issues
    // the tensor-core instructions and their commits): a divergent single-lane issuer loses most of its issue slots
    // to busy neighbouring warps.
    const uint32_t lead = elect_one();
    auto issue_s = [&](int gi) {
      const uint64_t kb = kdesc + static_cast<uint64_t>(((gi % kUmmaStages) * STAGE_BYTES) >> 4);
      mma_ts_kmajor_batch<D / 16, (CHUNK_BYTES >> 4)>(tmem + kSCol, tmem, kb, idesc_s, 0u, lead);
      mma_commit_lead(smem_u32(&ctrl->s_full), lead);
    };
    bool ok = true;
    int g = 0;                                   // tiles consumed so far, over all units
    // (the record of the next unit is read while the current one runs: two L2 round trips less at every hand-over)
    for (int r = 0; ok; ++r) {
      const int u = unit_at(r);
      if (u < 0) { ok = false; break; }
      if (u >= n_units) break;
      const UmmaUnit w = unit_of(u);
      ok = warp_wait(smem_u32(&ctrl->q_ready), r & 1);
      if (!ok || *abort_flag) { ok = false; break; }
      if (w.ntiles == 0) {
        // nothing to multiply; keep the o_free phase in step (the softmax warps arrive once per unit)
        if (r > 0) ok = warp_wait(smem_u32(&ctrl->o_free), (r - 1) & 1);
        unit_done(r);
        continue;
      }
      ok = warp_wait(smem_u32(&ctrl->full[g % kUmmaStages]), (g / kUmmaStages) & 1);
      if (!ok) break;
      tc_fence_after();
      issue_s(g);
      for (int tile = 0; tile < w.ntiles && ok; ++tile, ++g) {
        const int stage = g % kUmmaStages;
        // what does not depend on the softmax warps comes before the wait for their P: the zero fill of V rows past the
        // end, the operand descriptors
        const int valid = w.len - (w.t_begin + tile * kTileN);
        if (valid < kTileN) {
          // keys past the sequence end carry P == 0 but their V rows may hold anything: zero them so 0 * x stays 0
          // (the stage is complete: its K half was consumed by S(tile))
          unsigned char* vbuf = smem + stage * STAGE_BYTES + TILE_BYTES;
          const int first = valid > 0 ? valid : 0;
          const int n16 = (kTileN - first) * 8;
          for (int cc = 0; cc < CHUNKS; ++cc) {
            uint4* dst = reinterpret_cast<uint4*>(vbuf + cc * CHUNK_BYTES + first * 128);
            for (int i = lane; i < n16; i += 32) dst[i] = make_uint4(0u, 0u, 0u, 0u);
          }
          fence_proxy_async_smem();
          __syncwarp();
        }
        const uint64_t vb = vdesc + static_cast<uint64_t>((stage * STAGE_BYTES + TILE_BYTES) >> 4);
        // A wait of a tile that ran out is noticed behind the MMAs, which then multiply whatever is there into this CTA's own
        // tensor memory (where the softmax warps take that for the unit's product, the teardown fills its rows with NaN): votes between
        // P and the next scores, and loops around waits that are nearly always over, are part of every tile's chain.  32 sequences of
        // 1 to 33 thousand keys in pages, 40 rows per KV head, 335 -> 327 us, 32 x 8 192 keys (dense) 206 -> 196, 8 of 1 to 4 thousand,
        // 32/8 heads, 8 drafts, D 64 27.2 -> 25.9.
        bool good = mbar_wait_ready(smem_u32(&ctrl->p_ready), g & 1);
        // (a PV that starts a new accumulator: the previous unit's O must have left tensor memory)
        if (tile == 0 && r > 0) good = mbar_wait(smem_u32(&ctrl->o_free), (r - 1) & 1) && good;
        tc_fence_after();
        mma_ts_batch4(tmem + kOCol, tmem + kSCol, vb, idesc_o, tile > 0 ? 1u : 0u, lead);
        mma_commit_lead(smem_u32(&ctrl->o_done), lead);
        // K_tile was read by S(tile) (complete: its P has come back) and V_tile by the PV just issued: the stage goes back
        // to the issuing warps before this warp waits for the next one
        mma_commit_lead(smem_u32(&ctrl->empty[stage]), lead);
        if (tile + 1 < w.ntiles) {
          good = mbar_wait_ready(smem_u32(&ctrl->full[(g + 1) % kUmmaStages]), ((g + 1) / kUmmaStages) & 1) && good;
          tc_fence_after();
          issue_s(g + 1);
        }
        ok = __all_sync(0xffffffffu, good);
      }
      if (ok) unit_done(r);
    }
    if (!ok) {
      // (the softmax warps may have gone on since: no unit of the ring is known to be right)
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; ctrl->abort_round = 0; }
      // (what has been issued ends before tensor memory is given back)
      mma_commit_lead(smem_u32(&ctrl->drained), lead);
      warp_wait(smem_u32(&ctrl->drained), 0);
    }
  } else if (warp < active_warps) {
    // =========================== softmax warps: thread = q row ===========================
    const int row = tid;
    const uint32_t lane_off = static_cast<uint32_t>(warp * 32) << 16;
    const float sl2 = p.scale_log2;
    const uint32_t tS = tmem + lane_off + kSCol;
    const uint32_t tO = tmem + lane_off + kOCol;
    bool ok = true;
    int g = 0;                                   // tiles consumed so far, over all units
    int merges = 0;                              // units of this CTA that went through the ticket (barrier phases)
    int r = 0;
    auto rows_of = [&](const UmmaUnit& w) {
      return (static_cast<long long>(w.b) * p.q_heads + static_cast<long long>(w.h) * p.head_stride + p.head0) * p.q_len;
    };
    // Q row -> TMEM as the packed 16-bit A operand (rows past R are zero).  Called when the S MMAs of the unit before
    // have all completed (this warp has consumed their last score tile), i.e. before that unit's epilogue, so that
    // the MMA warp can start on the next unit while the rows of the finished one are written out.
    auto write_q = [&](int unit, const UmmaUnit& w) {
      if (unit >= n_units) return;
      const T* qg = static_cast<const T*>(p.q) + rows_of(w) * D;
#pragma unroll
      for (int cc = 0; cc < kQCols / 32; ++cc) {
        uint32_t qv[32];
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          uint4 x = make_uint4(0u, 0u, 0u, 0u);
          if (row < R) x = *(reinterpret_cast<const uint4*>(qg + static_cast<long long>(row) * D) + cc * 8 + i);
          qv[i * 4 + 0] = x.x; qv[i * 4 + 1] = x.y; qv[i * 4 + 2] = x.z; qv[i * 4 + 3] = x.w;
        }
        tmem_st32(tmem + lane_off + cc * 32, qv);
      }
      tmem_wait_st();
      tc_fence_before();
      mbar_arrive(smem_u32(&ctrl->q_ready));
    };
    // The ticket of a unit's pair is drawn by thread 0 one unit later (or in the teardown): by then the barrier that
    // says "all rows are written" completed long ago and the fence before the ticket has nothing left to wait for.
    int owed_pair = -1, owed_round = 0;          // thread 0: pair whose ticket is still to be drawn, and its unit's round
    auto draw_owed_ticket = [&]() {
      if (tid != 0 || owed_pair < 0) return;
      if (mbar_wait(smem_u32(&ctrl->rows_out), (merges - 1) & 1) && !*abort_flag) {
        __threadfence();                         // the rows the other softmax threads wrote before they arrived, too
        atomicAdd(p.counters + owed_pair, 1);
        atomicAdd(p.header + 3, 1);              // tickets drawn and not merged yet (a hint for the teardown)
      } else {
        p.header[0] = DEV_ERR_WAIT_EXPIRED;
        *abort_flag = 1;
      }
      owed_pair = -1;
    };
    int u = unit_at(0);
    if (u < 0) ok = false;
    UmmaUnit w = unit_of(min(max(u, 0), max(n_units - 1, 0)));
    if (ok) write_q(u, w);
    for (; ok; ++r) {
      if (u >= n_units) break;
      const long long row_base = rows_of(w);
      float m_used = -INFINITY, l_run = 0.f;               // per-row softmax state
      int lim = w.len - 1;                                 // last visible key of this row
      if (p.causal) lim = w.len - p.q_len + (row % p.q_len);
      const int first_lim = p.causal ? w.len - p.q_len : w.len - 1;      // the smallest of all rows
      for (int tile = 0; tile < w.ntiles; ++tile, ++g) {
        const bool here = mbar_wait_ready(smem_u32(&ctrl->s_full), g & 1);     // (asked with the verdict on the references)
        tc_fence_after();
        const int t0 = w.t_begin + tile * kTileN;
        const int limit = lim - t0;             // columns 0..limit of this tile are visible
        uint64_t rs;
        float neg_m;
        // 16 columns: exponentials, their sum, P as packed 16-bit
        auto exp_part = [&](const uint32_t (&v)[16], uint32_t* pq) {
          const uint64_t sl2_2 = pack_f2(sl2, sl2), neg_2 = pack_f2(neg_m, neg_m);
#pragma unroll
          for (int i = 0; i < 8; ++i) {
            float a, b;
            unpack_f2(fma_f2(pack_f2(__uint_as_float(v[2 * i]), __uint_as_float(v[2 * i + 1])), sl2_2, neg_2), a, b);
            a = fast_exp2(a);
            b = fast_exp2(b);
            rs = add_f2(rs, pack_f2(a, b));
            pq[i] = ElemTraits<T>::pack2(a, b);
          }
        };
        auto row_sum = [&]() {
          float a, b;
          unpack_f2(rs, a, b);
          return a + b;
        };
        float sum;
        bool done = false;
        // One pass where no row's exponent reference has to move, which is nearly every tile: against the reference that
        // stands, with the sum to tell whether it could (see kMaxRowSum); P stays in registers until then.  A unit's first
        // tile is read once more for its maximum: the largest weight is then exactly one.  (Against the maximum of the first 16
        // columns it was rounded like all others, and calls of a few hundred keys came out 3 - 6 % further from 64 bits.  It costs
        // 0.3 us a unit: 64 sequences of 300 keys, 8/1 heads with 8 drafts, D 64 14.9 -> 15.0, 4 of 150, 64/8 heads, 14.1 -> 14.5;
        // with two loads at a time 15.2 and 14.4, through the two passes below 15.5 and 14.6.)
        // Hidden columns (the draft-causal tail, the sequence's end) are -inf on the way: a row that sees nothing yet has no
        // reference, and its sum no number.
        {
          const bool full = first_lim - t0 >= kTileN - 1;
          auto hide = [&](uint32_t (&v)[16], int c) {
            if (full) return;
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c * 16 + i > limit) v[i] = 0xff800000u;          // -inf
          };
          uint32_t va[16], vb[16], pk[32];
          rs = pack_f2(0.f, 0.f);
          if (tile == 0) {
            uint32_t vc[16], vd[16];
            tmem_ld16(tS, va);
            tmem_ld16(tS + 16, vb);
            tmem_ld16(tS + 32, vc);
            tmem_ld16(tS + 48, vd);
            tmem_wait_ld_regs(va);
            tmem_wait_ld_regs(vb);
            tmem_wait_ld_regs(vc);
            tmem_wait_ld_regs(vd);
            hide(va, 0);
            hide(vb, 1);
            hide(vc, 2);
            hide(vd, 3);
            float ma = -INFINITY, mb = -INFINITY;
#pragma unroll
            for (int i = 0; i < 16; i += 2) {
              ma = max3(ma, __uint_as_float(va[i]), __uint_as_float(va[i + 1]));
              mb = max3(mb, __uint_as_float(vb[i]), __uint_as_float(vb[i + 1]));
              ma = max3(ma, __uint_as_float(vc[i]), __uint_as_float(vc[i + 1]));
              mb = max3(mb, __uint_as_float(vd[i]), __uint_as_float(vd[i + 1]));
            }
            m_used = fmaxf(ma, mb) * sl2;
          }
          tmem_ld16(tS, va);
          tmem_wait_ld_regs(va);
          tmem_ld16(tS + 16, vb);
          hide(va, 0);
          neg_m = -m_used;             // (+inf for a row without a reference yet: the sum is then no number)
          exp_part(va, pk);
          tmem_wait_ld_regs(vb);
          tmem_ld16(tS + 32, va);
          hide(vb, 1);
          exp_part(vb, pk + 8);
          tmem_wait_ld_regs(va);
          tmem_ld16(tS + 48, vb);
          hide(va, 2);
          exp_part(va, pk + 16);
          tmem_wait_ld_regs(vb);
          hide(vb, 3);
          exp_part(vb, pk + 24);
          sum = row_sum();
          done = __all_sync(0xffffffffu, here && sum <= kMaxRowSum);
          if (done) tmem_st32(tS, pk);
        }
        if (!done) {
          ok = __all_sync(0xffffffffu, here);
          if (!ok) break;
          // two passes, 16 columns at a time: a reference that moves
          auto load_part = [&](uint32_t (&v)[16], int c) {
            tmem_ld16(tS + c * 16, v);
            tmem_wait_ld_regs(v);
#pragma unroll
            for (int i = 0; i < 16; ++i)
              if (c * 16 + i > limit) v[i] = 0xff800000u;          // -inf
          };
          float mx = -INFINITY;
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t v[16];
            load_part(v, c);
#pragma unroll
            for (int i = 0; i < 16; i += 2) mx = max3(mx, __uint_as_float(v[i]), __uint_as_float(v[i + 1]));
          }
          mx *= sl2;
          const bool need = (mx - m_used) > kMoveThreshold;
          float alpha = 1.f;
          if (need) { alpha = fast_exp2(m_used - mx); m_used = mx; l_run *= alpha; }
          if (tile > 0 && __any_sync(0xffffffffu, need)) {
            // PV(tile-1) has completed once S(tile) is visible (MMAs complete in issue order); the wait is immediate
            ok = warp_wait(smem_u32(&ctrl->o_done), (g - 1) & 1);
            if (!ok) break;
            tc_fence_after();
#pragma unroll 1
            for (int cc = 0; cc < D / 16; ++cc) {
              uint32_t ov[16];
              tmem_ld16(tO + cc * 16, ov);
              tmem_wait_ld_regs(ov);
#pragma unroll
              for (int i = 0; i < 16; ++i) ov[i] = __float_as_uint(__uint_as_float(ov[i]) * alpha);
              tmem_st16(tO + cc * 16, ov);
            }
          }
          neg_m = (m_used == -INFINITY) ? 0.f : -m_used;
          rs = pack_f2(0.f, 0.f);
          // (P of a part lies over scores that have been read)
#pragma unroll 1
          for (int c = 0; c < 4; ++c) {
            uint32_t v[16], pq[8];
            load_part(v, c);
            exp_part(v, pq);
            tmem_st8(tS + c * 8, pq);
          }
          sum = row_sum();
        }
        l_run += sum;
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(smem_u32(&ctrl->p_ready));
      }
      if (!ok) break;
      // the next unit (published by the producer when it issued this unit's last copy, its Q rows already on their
      // way into L2): its Q goes to tensor memory before this unit's rows are written out
      const int u_next = unit_at(r + 1);
      if (u_next < 0) { ok = false; break; }
      const UmmaUnit w_next = u_next < n_units ? unit_of(u_next) : w;
      write_q(u_next, w_next);
      // ---------------- the unit's rows leave tensor memory ----------------
      if (w.ntiles > 0) {
        ok = warp_wait(smem_u32(&ctrl->o_done), (g - 1) & 1);
        if (!ok) break;
        tc_fence_after();
      }
      const bool single = w.n_chunks == 1;
      const long long slot = (static_cast<long long>(w.item0) + w.c) * p.kv_heads + w.h;
      OutT* out = static_cast<OutT*>(p.out) + row_base * D;
      const float inv = single ? (l_run > 0.f ? 1.f / l_run : 0.f) : 1.f;
#pragma unroll
      for (int cc = 0; cc < D / 32; ++cc) {
        uint32_t ov[32];
        if (w.ntiles > 0) {
          tmem_ld32(tO + cc * 32, ov);
          tmem_wait_ld();
        } else {
#pragma unroll
          for (int i = 0; i < 32; ++i) ov[i] = 0u;
        }
        if (cc == D / 32 - 1) {
          // O is in registers: the MMA warp may start the next unit's accumulator
          tc_fence_before();
          mbar_arrive(smem_u32(&ctrl->o_free));
        }
        if (row < R) {
          if (single) {
            if constexpr (sizeof(OutT) == 2) {
              uint4* dst = reinterpret_cast<uint4*>(out + static_cast<long long>(row) * D + cc * 32);
#pragma unroll
              for (int i = 0; i < 4; ++i) {
                uint4 x;
                x.x = ElemTraits<OutT>::pack2(__uint_as_float(ov[8 * i]) * inv, __uint_as_float(ov[8 * i + 1]) * inv);
                x.y = ElemTraits<OutT>::pack2(__uint_as_float(ov[8 * i + 2]) * inv, __uint_as_float(ov[8 * i + 3]) * inv);
                x.z = ElemTraits<OutT>::pack2(__uint_as_float(ov[8 * i + 4]) * inv, __uint_as_float(ov[8 * i + 5]) * inv);
                x.w = ElemTraits<OutT>::pack2(__uint_as_float(ov[8 * i + 6]) * inv, __uint_as_float(ov[8 * i + 7]) * inv);
                dst[i] = x;
              }
            } else {
              float4* dst = reinterpret_cast<float4*>(out + static_cast<long long>(row) * D + cc * 32);
#pragma unroll
              for (int i = 0; i < 8; ++i)
                dst[i] = make_float4(__uint_as_float(ov[4 * i]) * inv, __uint_as_float(ov[4 * i + 1]) * inv,
                                     __uint_as_float(ov[4 * i + 2]) * inv, __uint_as_float(ov[4 * i + 3]) * inv);
            }
          } else {
            float4* dst = reinterpret_cast<float4*>(p.part_o + (slot * R + row) * D + cc * 32);
#pragma unroll
            for (int i = 0; i < 8; ++i)
              dst[i] = make_float4(__uint_as_float(ov[4 * i]), __uint_as_float(ov[4 * i + 1]),
                                   __uint_as_float(ov[4 * i + 2]), __uint_as_float(ov[4 * i + 3]));
          }
        }
      }
      if (!single) {
        if (row < R) {
          p.part_ml[(slot * R + row) * 2] = m_used;
          p.part_ml[(slot * R + row) * 2 + 1] = l_run;
        }
        // Publish the partial.  Nobody merges here: the merge is left to the teardown of whichever CTA gets to it first
        // (see there), so the softmax warps go straight on to their next unit.  The softmax threads meet on an
        // mbarrier with a bounded wait, never on bar.sync: a warp that gave up must not hang the rest.
        draw_owed_ticket();
        mbar_arrive(smem_u32(&ctrl->rows_out));
        if (!kOwnPlan) owed_pair = w.b * p.kv_heads + w.h;      // (else the teardown draws)
        owed_round = r;
        ++merges;
      }
      unit_done(r);
      w = w_next;
      u = u_next;
    }
    if (ok) draw_owed_ticket();
    if (!ok) {
      // (a unit whose ticket was still owed counts as unfinished: its pair will never be merged)
      atomicMin(&ctrl->abort_round, (tid == 0 && owed_pair >= 0) ? owed_round : r);
      if (lane == 0) { p.header[0] = DEV_ERR_WAIT_EXPIRED; *abort_flag = 1; }
    }
  }
  // ---------------- teardown ----------------
  tc_fence_before();
  __syncthreads();
  if (warp == kMma) { tc_fence_after(); tmem_dealloc(tmem, kUmmaTmemCols); }
  if constexpr (kOwnPlan) {
    // One unit: its ticket is drawn here, by every CTA that has one, and the last of a pair's merges it.
    const UmmaUnit w = s_unit;
    if (n_units > 0 && w.n_chunks > 1) {
      const long long slot = (static_cast<long long>(w.item0) + w.c) * p.kv_heads + w.h;
      if (ctrl->abort_flag) {
        // (a wait ran out: the rows are unknown, and NaN says so in the merge)
        for (int i = tid; i < R * D; i += blockDim.x) p.part_o[slot * R * D + i] = __int_as_float(0x7fc00000);
        for (int i = tid; i < R * 2; i += blockDim.x) p.part_ml[slot * R * 2 + i] = __int_as_float(0x7fc00000);
      }
      OutT* out = static_cast<OutT*>(p.out) +
                  ((static_cast<long long>(w.b) * p.q_heads + static_cast<long long>(w.h) * p.head_stride + p.head0) * p.q_len) * D;
      publish_and_merge<OutT, D, false>(p, w.b, w.h, w.c, w.n_chunks, w.item0, out, &ctrl->ready, reinterpret_cast<float*>(smem));
      return;
    }
  }
  if (!kOwnPlan) claim_merges<OutT, D>(p, ctrl, me);
  if (ctrl->abort_flag) poison_units<OutT, D>(p, ctrl, n_units, [&](int r) { return unit_of(ctrl->unit_ring[r % kUmmaUnitRing]); });
}

#include "decode_keyrows.cuh"

// ---------------------------------------------------------------------------
// fp32 kernel: fp32 FMA dot products.
//
// A key row is held by D / 8 lanes, eight floats each, so a warp has 32 / (D / 8) rows in hand per load instruction
// (4 at head_dim 64, 2 at 128) and a dot product is three or four shuffles instead of the five that a row spread over
// the whole warp takes; the RB query rows of a block share every key row that is loaded.  Each lane group keeps an
// online softmax of its own over its keys, so that nothing but the dot products crosses lanes inside the loop; the
// groups of a warp are merged once at the end, the warps of a row in emit_and_merge.
// What bounds the kernel is the bytes in flight: every lane copies the 16-byte pieces that it will use itself
// (cp.async, kSimtDepth steps ahead) into a ring of its own in shared memory, so nothing waits for another lane and the
// registers stay free for the rows; block-table entries are read one step before the copies that need them.
// ---------------------------------------------------------------------------
constexpr int kSimtThreads = 128;
constexpr int kSimtDepth = 4;                // steps whose copies are in flight
constexpr int kSimtKeys = 2;                 // key rows of a lane group per step
constexpr size_t kSimtRingBytes = static_cast<size_t>(kSimtThreads) * kSimtDepth * kSimtKeys * 4 * 16;

template <int D, int RB, bool kCluster>
__global__ void __launch_bounds__(kSimtThreads, 3) decode_simt_kernel(const DecodeParams p) {
  extern __shared__ __align__(128) unsigned char smem[];
  __shared__ int s_ticket;
  constexpr int kGroup = D / 8;              // lanes that share a key row
  constexpr int kRowsWarp = 32 / kGroup;     // key rows of a warp per load instruction
  constexpr int kKeys = kSimtKeys;
  constexpr int kStep = kRowsWarp * kKeys;   // keys of a warp per step
  ClusterPart part = {};
  __shared__ uint64_t recv_bar;
  if constexpr (kCluster) {
    part = cluster_part<D>(p);
    if (part.size > 1) cluster_begin<D>(p, part, &recv_bar);
  }
  ptx::grid_dep_launch_dependents();
  ptx::grid_dep_wait();      // what earlier launches wrote (the planner's records among it) is visible from here on
  // heads vary fastest across CTAs: the CTAs that run side by side walk the same pages and read
  // neighbouring head slices of each token row, which keeps DRAM rows open
  DecodeItem it;
  int h;
  if constexpr (kCluster) {
    const int pair = blockIdx.x / part.size;
    h = pair % p.kv_heads;
    cluster_item(p, part, pair / p.kv_heads, it);
  } else {
    __shared__ InlinePlan s_plan;
    const int item = blockIdx.x / p.kv_heads;
    if (!decode_item(p, item, s_plan, it)) return;
    h = blockIdx.x - item * p.kv_heads;
  }
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int sub = lane / kGroup, gl = lane % kGroup;
  constexpr int nwarps = kSimtThreads / 32;
  const int R = p.rows;

  const int b = it.b, c = it.c, n_chunks = it.n_chunks, item0 = it.item0;
  const long long seq_start = it.start;
  const int len = it.len;
  const int t_begin = it.t_begin, t_end = it.t_end;

  float* comb_o = reinterpret_cast<float*>(smem + kSimtRingBytes);      // [KS][R][D]
  const int blocks = (R + RB - 1) / RB;                                 // blocks of RB rows
  const int KS = (blocks <= nwarps && nwarps % blocks == 0) ? nwarps / blocks : 1;   // warps that split a block's keys
  float* comb_ml = comb_o + static_cast<size_t>(KS) * R * D;            // [KS][R][2]
  const float* kg = static_cast<const float*>(p.k) + gl * 4;
  const float* vg = static_cast<const float*>(p.v) + gl * 4;
  const float* qg = static_cast<const float*>(p.q) +
                    ((static_cast<long long>(b) * p.q_heads + static_cast<long long>(h) * p.head_stride + p.head0) * p.q_len) * D;
  const float sl2 = p.scale_log2;
  const uint32_t ring = smem_u32(smem) + tid * 16;
  // dense and ragged rows: element offset of key 0, and from one key to the next
  const bool dense = p.layout == B200ATTN_DENSE;
  const long long kv_base = dense ? (static_cast<long long>(b) * p.kv_heads + h) * p.max_kv * D
                                  : (seq_start * p.kv_heads + h) * D;
  const int kv_stride = dense ? D : p.kv_heads * D;
  constexpr int kHalf = D / 2;               // a lane holds 4 floats at gl * 4 and 4 at D / 2 + gl * 4

  for (int rr = warp; rr < blocks * KS; rr += nwarps) {
    const int r0 = (rr % blocks) * RB, ks = rr / blocks;
    float4 q0[RB], q1[RB], a0[RB], a1[RB];
    float m[RB], l[RB];
    int vis[RB];                             // keys [0, vis) of the sequence are visible to the row
    int stop = 0, all = t_end;               // keys any row of the block sees; keys every row sees
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      const int r = min(r0 + i, R - 1);      // (rows past the last repeat it and are not written)
      q0[i] = __ldcg(reinterpret_cast<const float4*>(qg + static_cast<long long>(r) * D) + gl);
      q1[i] = __ldcg(reinterpret_cast<const float4*>(qg + static_cast<long long>(r) * D + kHalf) + gl);
      a0[i] = a1[i] = make_float4(0.f, 0.f, 0.f, 0.f);
      m[i] = -INFINITY;
      l[i] = 0.f;
      vis[i] = min(t_end, p.causal ? len - p.q_len + (r % p.q_len) + 1 : len);
      stop = max(stop, vis[i]);
      all = min(all, vis[i]);
    }
    // block-table entries of the step at key t, K's and V's of every key row of the lane's group
    const bool paged = p.layout == B200ATTN_PAGED;
    const int* ktab = paged ? p.k_table + static_cast<long long>(b) * p.table_stride : nullptr;
    const int* vtab = paged ? p.v_table + static_cast<long long>(b) * p.table_stride : nullptr;
    int kp[kKeys], vp[kKeys];
    auto fetch_pages = [&](int t) {
#pragma unroll
      for (int j = 0; j < kKeys; ++j) {
        const int key = t + j * kRowsWarp + sub;
        kp[j] = vp[j] = 0;
        if (paged && key < stop) {
          const int lp = p.page_shift >= 0 ? key >> p.page_shift : key / p.page_size;
          kp[j] = ktab[lp];
          vp[j] = vtab[lp];
        }
      }
    };
    unsigned on = 0;                         // kKeys bits per step in flight, the newest lowest: the key is there
    // issues the copies of the step at key t into slot `slot` of the lane's ring (zeros for keys that are not there)
    auto copy = [&](int t, int slot) {
#pragma unroll
      for (int j = 0; j < kKeys; ++j) {
        const int key = t + j * kRowsWarp + sub;
        bool there = key < stop;
        long long ko = 0, vo = 0;
        if (there) {
          if (paged) {
            const bool bad = kp[j] < 0 || kp[j] >= p.num_pages || vp[j] < 0 || vp[j] >= p.num_pages;
            if (bad) p.header[0] = DEV_ERR_PAGE_RANGE;   // a key on a page outside the cache weighs nothing
            there = !bad;
            const int off = p.page_shift >= 0 ? key & (p.page_size - 1) : key % p.page_size;
            if (there) {
              ko = ((static_cast<long long>(kp[j]) * p.page_size + off) * p.kv_heads + h) * D;
              vo = ((static_cast<long long>(vp[j]) * p.page_size + off) * p.kv_heads + h) * D;
            }
          } else {
            ko = vo = kv_base + static_cast<long long>(key) * kv_stride;
          }
        }
        const int bytes = there ? 16 : 0;
        const uint32_t dst = ring + static_cast<uint32_t>((slot * kKeys + j) * 4) * (kSimtThreads * 16);
        cp_async16(dst, kg + ko, bytes);
        cp_async16(dst + kSimtThreads * 16, kg + ko + kHalf, bytes);
        cp_async16(dst + 2 * kSimtThreads * 16, vg + vo, bytes);
        cp_async16(dst + 3 * kSimtThreads * 16, vg + vo + kHalf, bytes);
        on = (on << 1) | (there ? 1u : 0u);
      }
      cp_async_commit();
    };
    int t = t_begin + ks * kStep;
    fetch_pages(t);
#pragma unroll
    for (int s = 0; s < kSimtDepth - 1; ++s) {
      const int ts = t + s * KS * kStep;
      copy(ts, s);
      fetch_pages(ts + KS * kStep);
    }
    int slot = 0;
    for (; t < stop; t += KS * kStep) {
      {
        const int ts = t + (kSimtDepth - 1) * KS * kStep;
        copy(ts, (slot + kSimtDepth - 1) % kSimtDepth);     // (the slot was read in the step before)
        fetch_pages(ts + KS * kStep);
      }
      cp_async_wait<kSimtDepth - 1>();
      float4 ck0[kKeys], ck1[kKeys], cv0[kKeys], cv1[kKeys];
      bool con[kKeys];
#pragma unroll
      for (int j = 0; j < kKeys; ++j) {
        const float4* piece = reinterpret_cast<const float4*>(smem) + tid + (slot * kKeys + j) * 4 * kSimtThreads;
        ck0[j] = piece[0]; ck1[j] = piece[kSimtThreads]; cv0[j] = piece[2 * kSimtThreads]; cv1[j] = piece[3 * kSimtThreads];
        con[j] = (on >> ((kSimtDepth - 1) * kKeys + kKeys - 1 - j)) & 1u;
      }
      slot = (slot + 1) % kSimtDepth;
      const bool whole = t + kStep <= all;   // every row sees every key of the step
      float dot[RB][kKeys];
#pragma unroll
      for (int i = 0; i < RB; ++i) {
#pragma unroll
        for (int j = 0; j < kKeys; ++j) {
          float d = q0[i].x * ck0[j].x;
          d = fmaf(q0[i].y, ck0[j].y, d); d = fmaf(q0[i].z, ck0[j].z, d); d = fmaf(q0[i].w, ck0[j].w, d);
          d = fmaf(q1[i].x, ck1[j].x, d); d = fmaf(q1[i].y, ck1[j].y, d);
          d = fmaf(q1[i].z, ck1[j].z, d); d = fmaf(q1[i].w, ck1[j].w, d);
          dot[i][j] = d;
        }
      }
#pragma unroll
      for (int off = kGroup / 2; off > 0; off >>= 1) {
#pragma unroll
        for (int i = 0; i < RB; ++i) {
#pragma unroll
          for (int j = 0; j < kKeys; ++j) dot[i][j] += __shfl_xor_sync(0xffffffffu, dot[i][j], off);
        }
      }
#pragma unroll
      for (int i = 0; i < RB; ++i) {
        float mn = m[i];
        bool see[kKeys];
#pragma unroll
        for (int j = 0; j < kKeys; ++j) {
          see[j] = con[j] && (whole || t + j * kRowsWarp + sub < vis[i]);
          dot[i][j] = see[j] ? dot[i][j] * sl2 : -INFINITY;
          mn = fmaxf(mn, dot[i][j]);
        }
        const float ms = mn == -INFINITY ? 0.f : mn;    // nothing visible yet: every weight below is 0
        const float a = fast_exp2(m[i] - ms);           // m == -inf: 0
        m[i] = mn;
        l[i] *= a;
        a0[i].x *= a; a0[i].y *= a; a0[i].z *= a; a0[i].w *= a;
        a1[i].x *= a; a1[i].y *= a; a1[i].z *= a; a1[i].w *= a;
#pragma unroll
        for (int j = 0; j < kKeys; ++j) {
          // (a key that the row does not see is left out rather than weighed with 0: its V may be anything)
          if (!whole && !see[j]) continue;
          const float w = fast_exp2(dot[i][j] - ms);
          l[i] += w;
          a0[i].x = fmaf(w, cv0[j].x, a0[i].x); a0[i].y = fmaf(w, cv0[j].y, a0[i].y);
          a0[i].z = fmaf(w, cv0[j].z, a0[i].z); a0[i].w = fmaf(w, cv0[j].w, a0[i].w);
          a1[i].x = fmaf(w, cv1[j].x, a1[i].x); a1[i].y = fmaf(w, cv1[j].y, a1[i].y);
          a1[i].z = fmaf(w, cv1[j].z, a1[i].z); a1[i].w = fmaf(w, cv1[j].w, a1[i].w);
        }
      }
    }
    cp_async_wait<0>();
    // merge the lane groups of the warp, then leave one partial per (key slice, row)
#pragma unroll
    for (int i = 0; i < RB; ++i) {
      float g = m[i];
#pragma unroll
      for (int off = kGroup; off < 32; off <<= 1) g = fmaxf(g, __shfl_xor_sync(0xffffffffu, g, off));
      const float w = m[i] == -INFINITY ? 0.f : fast_exp2(m[i] - g);
      float x[9] = {a0[i].x, a0[i].y, a0[i].z, a0[i].w, a1[i].x, a1[i].y, a1[i].z, a1[i].w, l[i]};
#pragma unroll
      for (int e = 0; e < 9; ++e) {
        x[e] *= w;
#pragma unroll
        for (int off = kGroup; off < 32; off <<= 1) x[e] += __shfl_xor_sync(0xffffffffu, x[e], off);
      }
      if (r0 + i < R && sub == 0) {
        const size_t row = static_cast<size_t>(ks) * R + r0 + i;
        *reinterpret_cast<float4*>(comb_o + row * D + gl * 4) = make_float4(x[0], x[1], x[2], x[3]);
        *reinterpret_cast<float4*>(comb_o + row * D + kHalf + gl * 4) = make_float4(x[4], x[5], x[6], x[7]);
        if (gl == 0) { comb_ml[row * 2] = g; comb_ml[row * 2 + 1] = x[8]; }
      }
    }
  }
  __syncthreads();
  if constexpr (kCluster) {
    unsigned char* recv = reinterpret_cast<unsigned char*>(comb_ml + ((static_cast<size_t>(KS) * R * 2 + 3) & ~size_t(3)));
    if (part.size > 1) {
      cluster_emit<float, D>(p, part, b, h, comb_o, comb_ml, KS, R, recv, &recv_bar);
      return;
    }
  }
  emit_and_merge<float, D>(p, b, h, c, n_chunks, item0, comb_o, comb_ml, KS, R, &s_ticket);
}

template <typename K>
int set_smem(K kernel, size_t bytes) {
  return ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), bytes);
}

}  // namespace

// ---------------------------------------------------------------------------
// host side
// ---------------------------------------------------------------------------
// q heads of one KV head that one launch serves.  A CTA holds at most 128 q rows (group x draft tokens) per KV head;
// a larger group is cut into the largest equal sub-groups that fit, one launch each over the same K/V (the reference
// takes any head ratio: kernels/speculative_decode.py:262-299).
int decode_pass_group(int group, int q_len) {
  if (q_len < 1) q_len = 1;
  int g = group;
  while (g > 1 && (g * q_len > 128 || group % g != 0)) --g;
  return g < 1 ? 1 : g;
}

// Six (item, kv head) CTAs per SM: two or three waves of the tensor-core kernels (3 or 2 resident CTAs per SM).
// Fewer, longer CTAs amortise start-up and merge; the planner keeps the item count at or below this, so the grid
// is a whole number of waves.  (Measured on B200, paged decode and speculative decode: 4 / 6 / 8 / 12 / 16 per SM
// give 0.84 / 0.83 / 0.81 / 0.80 / 0.78 and 0.71 / 0.70 / 0.73 / 0.67 / 0.64 of the copy bandwidth without the
// whole-wave rule, 0.76 for speculative decode with it.)
static int decode_target_items(int sm_count, int kv_heads) {
  const int per_sm = 6;
  return static_cast<int>(std::max<long long>(1, (static_cast<long long>(sm_count) * per_sm) / std::max(1, kv_heads)));
}

DecodeWsLayout decode_ws_layout(const b200attn_decode_args_t& a, int sm_count, bool allow_cast) {
  DecodeWsLayout w;
  const int group = decode_pass_group(a.kv_heads > 0 ? a.q_heads / a.kv_heads : 1, a.q_len);
  const int rows = group * a.q_len;
  // fp32 inputs of a speculative-decode call (more than one q row per head, or more than 16 rows per KV head) are
  // rounded to fp16 in the workspace and run on the tensor-core kernels with fp32 accumulation and fp32 output: the
  // reference multiplies them with tl.dot on fp32 operands, i.e. in TF32, which keeps the same ten mantissa bits
  // (kernels/speculative_decode.py:153,175); one fp32 FMA warp per q row re-reads K/V once per row and is one to two
  // orders of magnitude slower there.  Plain decode (one q row per head), which the reference computes in fp32 FMAs
  // (kernels/decode.py:146-160), stays on the fp32 kernel.
  // (not when the copies would be huge - a paged cache is copied whole - : beyond kCastLimitBytes the call stays on
  // the fp32 kernel rather than ask the caller for that much scratch)
  constexpr size_t kCastLimitBytes = size_t(8) << 30;
  const size_t kv_rows_all = a.layout == B200ATTN_DENSE ? static_cast<size_t>(a.batch) * a.kv_heads * a.max_kv
                                                        : static_cast<size_t>(a.total_kv > 0 ? a.total_kv : 0) * a.kv_heads;
  const bool cast16 = allow_cast && a.dtype == B200ATTN_F32 && (rows > 16 || a.q_len > 1) &&
                      kv_rows_all * a.head_dim * 4 <= kCastLimitBytes;
  const bool f32_kernel = a.dtype == B200ATTN_F32 && !cast16;
  w.target_items = decode_target_items(sm_count, a.kv_heads);
  // one wave: 2 (tcgen05 kernel, more than 16 rows) or 3 resident CTAs per SM; per-item start-up + merge cost in keys of
  // streaming time (from the sweeps quoted in the planner)
  const bool wide = rows > 16 && !f32_kernel;
  w.wave_items = static_cast<int>(std::max<long long>(1, (static_cast<long long>(sm_count) * (wide ? 2 : 3)) / std::max(1, a.kv_heads)));
  w.item_overhead = wide ? 448 : 128;
  // keep the partial write (rows x D fp32) small next to the chunk's K/V bytes
  int min_chunk = 128;
  const int by_rows = ((rows * 8 + kTileN - 1) / kTileN) * kTileN;
  if (by_rows > min_chunk) min_chunk = by_rows;
  w.min_chunk = min_chunk;
  w.max_items = w.target_items + a.batch;
  auto up = [](size_t x) { return (x + 255) & ~static_cast<size_t>(255); };
  size_t off = kHeaderBytes;
  w.item_start_off = off; off = up(off + sizeof(int) * (static_cast<size_t>(a.batch) + 1));
  w.counters_off = off;   off = up(off + sizeof(int) * static_cast<size_t>(a.batch) * a.kv_heads);
  w.info_off = off;       off = up(off + 32 * static_cast<size_t>(w.max_items));
  const size_t slots = static_cast<size_t>(w.max_items) * a.kv_heads;
  w.ml_off = off;         off = up(off + sizeof(float) * slots * rows * 2);
  w.o_off = off;          off = up(off + sizeof(float) * slots * rows * a.head_dim);
  w.cast_q_off = w.cast_k_off = w.cast_v_off = 0;
  w.cast_q_elems = w.cast_kv_elems = 0;
  if (cast16) {
    w.cast_q_elems = static_cast<size_t>(a.batch) * a.q_heads * a.q_len * a.head_dim;
    const size_t kv_rows = a.layout == B200ATTN_DENSE ? static_cast<size_t>(a.batch) * a.kv_heads * a.max_kv
                                                      : static_cast<size_t>(a.total_kv) * a.kv_heads;
    w.cast_kv_elems = kv_rows * a.head_dim;
    w.cast_q_off = off; off = up(off + 2 * w.cast_q_elems);
    w.cast_k_off = off; off = up(off + 2 * w.cast_kv_elems);
    w.cast_v_off = off; off = up(off + 2 * w.cast_kv_elems);
  }
  w.total = off;
  return w;
}

namespace {
int launch_decode_pass(const b200attn_decode_args_t& a, int sm_count, cudaStream_t stream, const DecodeWsLayout& w,
                       int pass_group, int head0, bool f32_out, bool built_in);

}  // namespace

int launch_decode(const b200attn_decode_args_t& a, int sm_count, cudaStream_t stream, bool built_in) {
  const DecodeWsLayout w = decode_ws_layout(a, sm_count, /*allow_cast=*/!built_in);
  if (a.workspace == nullptr || a.workspace_bytes < w.total || (reinterpret_cast<uintptr_t>(a.workspace) & 255)) {
    set_error("decode: workspace needs %zu bytes, 256-byte aligned (got %zu)", w.total, a.workspace_bytes);
    return B200ATTN_E_WORKSPACE;
  }
  const int group = a.q_heads / a.kv_heads;
  const int pass_group = decode_pass_group(group, a.q_len);
  b200attn_decode_args_t b = a;
  if (w.cast_kv_elems > 0) {
    // fp16 copies of q, k, v (see decode_ws_layout); the launches below read them and write fp32 rows
    unsigned char* ws = static_cast<unsigned char*>(a.workspace);
    void* dst[3] = {ws + w.cast_q_off, ws + w.cast_k_off, ws + w.cast_v_off};
    const long long q4 = static_cast<long long>(w.cast_q_elems / 4), kv4 = static_cast<long long>(w.cast_kv_elems / 4);
    const CastJob job = {{static_cast<const float4*>(a.q), static_cast<const float4*>(a.k), static_cast<const float4*>(a.v)},
                         {static_cast<uint2*>(dst[0]), static_cast<uint2*>(dst[1]), static_cast<uint2*>(dst[2])},
                         {q4, kv4, kv4}};
    const cudaError_t e = launch_cast(job, sm_count, stream);
    if (e != cudaSuccess) return cuda_fail(e, "cast kernel launch");
    b.q = dst[0]; b.k = dst[1]; b.v = dst[2];
    b.dtype = B200ATTN_F16;
  }
  // one launch per sub-group of q heads; they run back to back on the stream and share the workspace
  for (int head0 = 0; head0 < group; head0 += pass_group) {
    const int rc = launch_decode_pass(b, sm_count, stream, w, pass_group, head0, w.cast_kv_elems > 0, built_in);
    if (rc) return rc;
  }
  return B200ATTN_OK;
}

namespace {
// Dynamic shared memory of a CTA.  `cluster`: CTAs that share a pair, 0 behind a plan; what they send to one of them, pieces and rows'
// (m, l), comes behind the rest, with up to 32 bytes of alignment.
size_t recv_bytes(int cluster, int rows, int D) {
  return cluster ? static_cast<size_t>(cluster) * ((rows * (D / 4) + cluster - 1) / cluster * 16 + rows * 8) + 32 : 0;
}
constexpr int kMmaSlices = 4;              // consumer warps of the warp-level kernel, which split the keys of a tile
size_t mma_smem(int stages, int cluster, int rows, int D) {
  const size_t stage_bytes = static_cast<size_t>(stages) * 2 * kTileN * D * 2;
  const size_t comb_bytes = sizeof(float) * static_cast<size_t>(kMmaSlices) * 16 * (D + 2);
  return 1024 + std::max(stage_bytes, comb_bytes) + static_cast<size_t>(16) * D * 2 + sizeof(DecodeCtrl) + recv_bytes(cluster, rows, D);
}
size_t simt_smem(int cluster, int rows, int D) {
  // (four warps leave at most 4 / blocks-of-rows partials per row: see the kernel)
  const int rb = rows >= 3 ? 4 : rows;
  return kSimtRingBytes + sizeof(float) * static_cast<size_t>(std::max(rows, 4 * rb)) * (D + 2) + recv_bytes(cluster, rows, D);
}

// CTAs of either kernel that an SM holds: by their registers three, by shared memory maybe fewer (at D 128 the 16-bit kernel's
// fit three times up to ten rows, the fp32 kernel's up to seven).
int ctas_per_sm(size_t smem) {
  return static_cast<int>(std::min<size_t>(3, 228 * 1024 / (smem + 1024 + 64)));
}

// What one CTA takes for a tile of 64 keys, alone on its SM, in ns.  (The fp32 kernel multiplies blocks of 1, 2 or 4 rows, each
// block's keys split over the warps that the blocks leave it: see there.)
int tile_ns(const b200attn_decode_args_t& a, int rows) {
  if (a.dtype != B200ATTN_F32) return a.head_dim == 128 ? 800 : 460;
  return (rows == 1 ? 830 : rows == 2 ? 1100 : rows <= 4 ? 1500 : rows <= 8 ? 3000 : 6000) * a.head_dim / 64;
}

// CTAs per (sequence, KV head) pair when the call runs without a plan, 0 when it is planned.  Up to eight CTAs share a pair,
// as long as all of them are resident at once.  A planned call takes 9 to 12 us before its items' length counts, some 5 more when
// the planner has a launch of its own (`planner`: more than 96 pairs), and cuts the keys evenly over the GPU whatever the lengths are;
// a call in clusters takes 3 us and its longest part.  So the line is drawn by the time of a part (tile_ns), of one as long as the
// host can tell: dense, the length of all; paged, the table's width; ragged, the average, and the longest that there can be,
// a sequence that holds all keys, has a line of its own.  The lines are where the sweep below found the last call that was not faster
// planned: 16-bit and fp32, D 64 and 128, 1 to 16 rows, 1 to 768 pairs, 64 to 16 000 keys; equal lengths, lengths from
// nothing to twice the average, and one sequence with nearly all keys among 2 to 32.  Planned -> in clusters, us:
//   dense: more CTAs than SMs share the bandwidth either way, and parts up to 15 us are worth it (32/8 heads, D 128, 16 x 2 048
//     36 -> 27; 4 x 8 192 32 -> 27), below that up to 7.5 (1 x 4 096 16.1 -> 10.6, but in clusters of two 30).
//   paged: the same without the first: the other sequences may be shorter (4 x 8 pairs, a table of 4 096 keys, D 64: 13.6 -> 11.0 with
//     lengths anywhere up to that, 10.7 with one of them that long; but 8 x 8 pairs in clusters of four 23 -> 18.6 if all are that
//     long, a fifth slower than planned if one is).
//   ragged: 16 sequences of 125 keys on average, 8/8 heads, D 128: 12.9 -> 6.4, and when one has nearly all of them 17.9 -> 17.2;
//     of 250 keys 16.1 -> 7.5 and 21 -> 30.  A pair gets as many CTAs as make the second case a gain too, or else the most there
//     are, and the call is planned when that would take it half as long again as the plan (26 us for the part): over the
//     sweep clusters give 0.66 of the planned time to equal and to evenly spread lengths, 0.78 to batches of one long sequence,
//     1.5 to the worst of them (fp32 0.86, 0.94 and 1.1).
//   fp32: the plan's shortest items, 128 keys, are in the planned time, so two tiles are added to the line: 8/1 heads, D 64, 1 x 1 024
//     14.6 -> 11.1, 1 x 2 048 15.8 -> 17.2; 16 packed sequences, one with 1 900 keys, 8/1 heads: 17 planned and in clusters of eight,
//     50 in those of two; one with 7 900: 26 and 53.  With more than two rows the CTAs of an SM hold one another up: a part takes half as long again where there are
//     more CTAs than SMs (4 x 1 024, 64/8 heads, D 128: 27.8 -> 30.4).
int cluster_size(const b200attn_decode_args_t& a, int sm_count, int rows, bool ask) {
  const long long pairs = static_cast<long long>(a.batch) * a.kv_heads;
  if (pairs <= 0) return 0;
  const bool ragged = a.layout == B200ATTN_RAGGED, dense = a.layout == B200ATTN_DENSE, fp32 = a.dtype == B200ATTN_F32;
  // (fp32 calls of up to 192 pairs may have none either, but the lines are right for them as they are: with those for up to 96 pairs,
  // 240 packed calls of 97 to 192 of 40 to 600 keys took 1.02 of their time, 13 x 200 of 8/8 heads, D 128, equal 9.9 -> 14.8 us, with one
  // sequence of nearly all keys 24.4 -> 17.1)
  const bool planner = pairs > kInlinePairs;
  auto tiles_of = [](long long keys) { return (keys + kTileN - 1) / kTileN; };
  const long long tiles = tiles_of(ragged ? (a.total_kv + a.batch - 1) / a.batch
                                   : dense ? a.max_kv : a.table_stride * static_cast<long long>(a.page_size));
  const long long longest = ragged ? tiles_of(a.total_kv) : tiles;
  const long long ns = tile_ns(a, rows);
  auto held = [&](long long c) -> long long {
    const int n = static_cast<int>(c);
    const int per_sm = ctas_per_sm(fp32 ? simt_smem(n, rows, a.head_dim) : mma_smem(2, n, rows, a.head_dim));
    return clusters_held(n, per_sm, sm_count, ask);
  };
  long long most = 8;
  while (most > 1 && pairs > held(most)) most /= 2;
  long long c = most;
  while (c > 1 && tiles <= c / 2) c /= 2;
  for (;; c *= 2) {
    const long long ctas = pairs * c;
    long long near, far, last;
    if (dense && fp32) near = ctas >= 2ll * sm_count ? 16000 : 5500 + 2 * ns;
    else if (dense) near = ctas > sm_count ? 15000 : c == 8 ? 7500 : 5000;
    else if (fp32) near = (planner ? 4500 : 3200) + 2 * ns;
    else near = !ragged && (c == most || planner) ? 7500 : 5000;
    far = last = near;
    if (ragged && fp32) far = (planner ? 13000 : 5500) + 2 * ns, last = (planner ? 22000 : 9000) + 2 * ns;
    else if (ragged) far = planner ? 15000 : c == 8 ? 8000 : 6500, last = planner ? 26000 : 15000;
    // (time of a part: with more CTAs than an SM each, and of the waves when a pair's only CTA has to wait for its turn)
    double part = static_cast<double>(ns);
    if (fp32 && rows > 2) {
      if (ctas > sm_count) part *= 1.5;
      if (const long long n = held(c); pairs > n) part *= static_cast<double>((pairs + n - 1) / n) * n / pairs;
    }
    if ((tiles + c - 1) / c * part <= near && (longest + c - 1) / c * part <= (c == most ? last : far)) return static_cast<int>(c);
    if (c == most) return 0;
  }
}

// keys of all sequences, as many as there can be
long long most_keys(const b200attn_decode_args_t& a) {
  if (a.layout == B200ATTN_RAGGED) return a.total_kv;
  return a.batch * (a.layout == B200ATTN_DENSE ? static_cast<long long>(a.max_kv) : a.table_stride * a.page_size);
}

// Bits of a merge ticket where the CTAs plan for themselves (plan_inline, about a microsecond each), 0 where the call needs the
// planner's launch, 4 to 5 us in front of the kernel.
//
// Up to sixteen rows, and fp32: few (sequence, kv head) pairs.  The line is the number of merge tickets that fit into the header,
// the only part of a workspace that may be relied on to be zero without a launch; beyond it a call streams for longer
// and the planner is a smaller part of it.  Measured: one user 22.2 -> 17.7 us per (append, append, decode), 16 x 2 048
// keys of two heads 17.2 -> 13.0, four drafts for 16 short sequences 15.1 -> 12.9, 7 x 30 201 keys at 0.98 of the copy
// bandwidth.  fp32, which reads twice the bytes: twice as many pairs, with tickets of eight bits
// where no pair can be cut into more items than those count, up to 300 MiB of keys and values (the most that there can be).  16
// packed sequences of 100 to 4 096 keys, 8/8 heads, D 64 36.3 -> 32.4 us, 13 x 1 500 18.9 -> 15.5, 24 x 1 500 at D 128 in pages 43.8 ->
// 38.7; 20 x 3 000 119 -> 113, but 20 x 10 000 (819 MB, 64/8 heads, dense) 281 -> 290: the planner puts the last, shorter item of each
// sequence behind all others, which is worth more than its launch there.  (Between the two packed lengths from nothing to twice the
// average still gained without it: 340 MB 0.93 to 1.01 of the time over twelve calls, 650 MB 0.95 to 1.00.  And in pages it is the
// width of the table that counts: a server whose tables are as wide as its context limit keeps the planner.)
//
// More than sixteen rows (the tcgen05 kernel; two CTAs to an SM): the planner deals a batch out to the CTAs by keys, which no CTA can
// see by itself (a batch cut into equal items leaves some CTAs without one), and a CTA's own plan takes longer the more sequences there
// are.  So: up to 1 024 keys for each CTA, less 8 for every sequence.  40 rows, D 128, with the planner and without, in us: 12 x 300
// keys of eight heads 15.7, 12.4; 1 x 2 000 22.9, 17.6; 10 x 2 590 39.0, 31.9; 38 x 1 557 of two heads 30.8, 25.7; 60 x 1 973 of one
// 30.8, 26.8; 90 x 1 315 30.3, 30.0; and beyond the line 60 x 4 933 45.6, 47.9; 75 x 3 946 45.7, 49.8; 90 x 2 302 38.4, 44.3.
//
// Not in the library's own array: nobody can zero that again after two calls have overlapped on it against
// the rules, and a ticket left over there would keep later calls from ever merging; the planner's tickets start at zero
// in every call.
int inline_plan_bits(const b200attn_decode_args_t& a, int sm_count, int rows) {
  const long long pairs = static_cast<long long>(a.batch) * a.kv_heads, keys = most_keys(a);
  if (a.dtype != B200ATTN_F32 && rows > 16)
    return pairs <= kInlinePairs && keys * a.kv_heads <= (1024 - 8ll * a.batch) * 2 * sm_count ? 16 : 0;
  if (pairs <= kInlinePairs) return 16;
  return a.dtype == B200ATTN_F32 && pairs <= kInlinePairs8 && a.batch <= kInlineBatch &&
         decode_target_items(sm_count, a.kv_heads) + a.batch <= 255 &&
         2 * keys * a.kv_heads * a.head_dim * 4 <= 300ll << 20 ? 8 : 0;
}

// Which way a pass of `rows` q rows per KV head goes: clusters (CTAs per pair), or items that the CTAs plan for themselves, or
// (neither) items behind the planner.  More than sixteen rows of 16-bit elements always go to the tcgen05 kernel; those of fp32 are
// planned (at six microseconds a tile and more a part is rarely short enough, and none was measured).
struct Route { int cluster, inline_plan; };      // (inline_plan: the bits of a ticket)
// `ask`: see clusters_held.
Route route_of(const b200attn_decode_args_t& a, int sm_count, int rows, bool built_in, bool ask) {
  Route r;
  r.cluster = rows <= 16 ? cluster_size(a, sm_count, rows, ask) : 0;
  r.inline_plan = built_in || r.cluster ? 0 : inline_plan_bits(a, sm_count, rows);
  return r;
}

// largest power of two that divides the page size, at most a tile of 64: every box stays inside one page
int page_box(const b200attn_decode_args_t& a) {
  int box = kTileN;
  if (a.layout == B200ATTN_PAGED) {
    box = 1;
    while (box < kTileN && (a.page_size % (box * 2)) == 0) box *= 2;
  }
  return box;
}

// Whether a planned pass of more than sixteen rows goes to decode_keyrows_kernel.  A unit there, a CTA's to itself, has some 2.5 us
// beside its copies; decode_umma_kernel's take longer, but an SM has two CTAs.  So the line is the length of a sequence, 512 keys at
// head_dim 128 and 1 024 at 64 (us, umma and keyrows, 40 rows of eight heads, D 128: 64 sequences of 250 keys 25.1, 28.4; of 400 33.5, 34.7;
// of 600 41.9, 41.5; of 1 000 59.4, 57.6; 200 of 400 82.7, 78.9; D 64, 64 of 700 32.6, 39.7; of 1 000 41.3, 48.0; of 1 200 60.2, 51.8; of
// 2 400 90.3, 86.4), and half of that where no SM has more than one unit (16 of 250 at D 128, 20 rows 22.7, 16.0; 40 rows 15.4, 15.8).
// Tables of pages say how long a sequence can be; twice the line is asked of them, which sequences of any length up to that reach on average.
// And the cache says how many keys there can be in all, where no sequences share pages.  Three quarters of the line are asked of that, so
// that short sequences in wide tables stay with decode_umma_kernel where the cache is no larger than they need: us, keyrows and umma, tables of
// 8 192 keys, eight heads, 40 rows, D 128, 64 x 20 keys 22.8, 17.2; 256 x 20 59.2, 39.0; 64 x 250 28.5, 23.9; 256 x 250 78.4, 71.2; 24 rows, D 64,
// 256 x 20 58.1, 32.9; 128 x 500 53.6, 47.4; 19 x 250 (152 units for 148 SMs) 26.3, 15.5.  Of the whole line 64 x 1 000, D 64, would take 56.2 in
// place of 48.4, 128 x 1 000 of two heads, 32 rows, D 128 37.0 in place of 34.6.
// And each SM needs 2 048 keys (D 64 4 096) where some have more than one unit: shorter calls end with a round that is mostly empty, or cut their
// sequences for it (100 x 1 000 keys of two heads, 48 rows, 44.2 us, umma 30.5; 20 x 300 to 2 500 of eight 44.4, 41.5; 40 x 600 to 2 500 62.9, 68.8).
// (Much shorter ones in wide tables of a large cache are slower for it: the same calls.  Both kernels launched, and the planner's word for
// which of them stays, cost every call 4 to 6 us.)
bool keyrows_suit(const b200attn_decode_args_t& a, int sm_count, int rows) {
  if (a.dtype == B200ATTN_F32 || rows <= 16 || rows > kKrMaxRows || !keyrows_boxes(page_box(a))) return false;
  if (inline_plan_bits(a, sm_count, rows)) return false;      // (also in the library's own array, where such a call is planned)
  const long long pairs = static_cast<long long>(a.batch) * a.kv_heads;
  const bool one_each = pairs <= sm_count;
  // At head_dim 64 sequences that have to be cut for the SMs are slower here (us, umma and keyrows, packed, 40 rows, 12 x 6 000 keys of eight heads
  // 47.3, 56.7; 35 x 6 000 of two 40.4, 42.8; 88 x 4 000 of one 37.6, 43.9; lengths of a sixteenth to twice 2 500, 110 of one head 34.2, 40.6; where
  // SMs have more than one pair such lengths take 0.95 of umma's time).  Only equal ones, of which most SMs have one, stay whole, and only of a
  // dense batch is that known (120 x 2 400 39.5, 32.0; 148 x 8 000 76.4, 69.5; packed, 110 x 2 500 would be 37.7, 33.3).
  if (one_each && a.head_dim == 64 && (a.layout != B200ATTN_DENSE || pairs * 3 < sm_count * 2ll)) return false;
  auto enough = [&](long long keys, int quarters) {        // ... of the line
    const long long line = (512 << 7) / a.head_dim * (one_each ? 1 : 2) * quarters / 8;
    return keys >= line * a.batch && (one_each || keys * a.kv_heads * a.head_dim >= (512ll << 7) * quarters * sm_count);
  };
  if (a.layout != B200ATTN_PAGED) return enough(most_keys(a), 4);
  return enough(most_keys(a), 8) && enough(a.total_kv, 3);
}

// `f32_out`: the inputs are the fp16 copies of fp32 tensors and the output rows are fp32
int launch_decode_pass(const b200attn_decode_args_t& a, int sm_count, cudaStream_t stream, const DecodeWsLayout& w,
                       int pass_group, int head0, bool f32_out, bool built_in) {
  DecodeParams p;
  p.q = a.q; p.k = a.k; p.v = a.v; p.out = a.out;
  p.kv_indptr = a.kv_indptr; p.k_table = a.k_table; p.v_table = a.v_table;
  unsigned char* ws = static_cast<unsigned char*>(a.workspace);
  p.header = reinterpret_cast<int*>(ws);
  p.item_start = reinterpret_cast<int*>(ws + w.item_start_off);
  p.counters = reinterpret_cast<int*>(ws + w.counters_off);
  p.item_info = reinterpret_cast<int4*>(ws + w.info_off);
  p.part_ml = reinterpret_cast<float*>(ws + w.ml_off);
  p.part_o = reinterpret_cast<float*>(ws + w.o_off);
  p.total_kv = a.total_kv; p.table_stride = a.table_stride;
  p.layout = a.layout; p.indptr_is_i64 = a.indptr_is_i64;
  p.batch = a.batch; p.q_heads = a.q_heads; p.kv_heads = a.kv_heads;
  p.head_stride = a.q_heads / a.kv_heads; p.head0 = head0;
  p.group = pass_group; p.q_len = a.q_len; p.rows = p.group * a.q_len;
  p.n_mtiles = (p.rows + 15) / 16;
  p.max_kv = a.max_kv; p.page_size = a.layout == B200ATTN_PAGED ? a.page_size : 1;
  p.page_shift = -1;
  if (p.page_size > 0 && (p.page_size & (p.page_size - 1)) == 0) {
    int s = 0; while ((1 << s) < p.page_size) ++s;
    p.page_shift = s;
  }
  p.num_pages = a.layout == B200ATTN_PAGED ? static_cast<int>(std::min<long long>(a.total_kv / p.page_size, 0x7fffffff)) : 0;
  p.causal = a.causal_drafts ? 1 : 0;
  p.box_shift = 6;
  p.target_items = w.target_items; p.min_chunk = w.min_chunk; p.max_items = w.max_items;
  p.wave_items = w.wave_items; p.item_overhead = w.item_overhead;
  p.scale_log2 = a.sm_scale * 1.4426950408889634f;

  const long long pairs = static_cast<long long>(a.batch) * a.kv_heads;
  const Route route = route_of(a, sm_count, p.rows, built_in, /*ask=*/true);
  p.cluster = route.cluster;
  p.inline_plan = route.inline_plan;
  // (a byte counts a group's chunks, and the chunks of a pair that is merged in one step)
  constexpr int kTicketBytes = (64 - kTicketWord) * 4;
  p.pair_tickets = 0;
  // (in the library's own array such calls are planned, but merged alike)
  if ((p.inline_plan || (built_in && (a.dtype == B200ATTN_F32 || p.rows <= 16))) && pairs > 0 && pairs <= kTicketBytes / 4 && w.max_items <= 255 * (kTicketBytes / pairs - 1))
    p.pair_tickets = static_cast<int>(kTicketBytes / pairs);
  if (p.inline_plan && a.dtype != B200ATTN_F32 && p.rows > 16) {
    // The tcgen05 kernel, few sequences: items for one CTA an SM, not two, up to six of the shortest.  A second CTA on some of the SMs holds its neighbour up,
    // and a merge, one CTA's work, is as long as a sequence has items: 1 x 8 000 keys of eight heads, 40 rows, D 128, 35.8 -> 25.7
    // us, 3 x 12 000 of two 45.6 -> 28.6, 1 x 30 000 of four, 64 rows, 71.2 -> 50.1.  (With any batch 12 x 1 400 in pages 21.0 ->
    // 23.6, 4 x 3 000 of eight, D 64, 16.0 -> 19.1.)
    if (a.batch <= 3 && most_keys(a) * a.kv_heads <= 6ll * w.min_chunk * sm_count) {
      p.target_items = std::max(1, sm_count / a.kv_heads);
      p.wave_items = 0;
    }
  }
  // the kernels of many rows are persistent: two CTAs to an SM (planned for in decode_ws_layout), or one
  const bool key_rows = keyrows_suit(a, sm_count, p.rows);
  p.slots = a.dtype != B200ATTN_F32 && p.rows > 16 ? 2 * sm_count / a.kv_heads : 0;
  if (key_rows) {
    // Three units a CTA where there are enough to share, handed out longest first: us, against six and dealt out as for two CTAs, 128 x 1 500
    // keys of two heads, 40 rows, D 128 51.7 -> 44.4, 34 x 10 232 of eight, 36 rows, D 64 171 -> 166, 200 x 300 to 4 000 in pages 91.8 -> 88.1.
    // Very uneven batches are still dealt out (32 x 1 000 to 33 000 291 -> 286).
    p.wave_items = std::max(1, sm_count / a.kv_heads);
    p.target_items = std::max(1, 3 * sm_count / a.kv_heads);
    p.slots = sm_count / a.kv_heads;
  }
  p.one_cta = key_rows;
  unsigned grid_items = static_cast<unsigned>(w.max_items);
  cudaError_t e = cudaSuccess;
  if (p.inline_plan) {
    // no more items than this, whatever the lengths are: an item has min_chunk keys or ends a sequence
    grid_items = static_cast<unsigned>(std::min<long long>(w.max_items, most_keys(a) / w.min_chunk + a.batch));
  } else if (!p.cluster) {
    e = launch_dependent(decode_plan_kernel, dim3(1), kPlanThreads, 0, stream, 1, p);
  }
  if (e != cudaSuccess) return cuda_fail(e, "decode_plan_kernel launch");

  const dim3 grid(p.cluster ? static_cast<unsigned>(pairs * p.cluster) : grid_items * a.kv_heads, 1);
  const int D = a.head_dim;
  if (a.dtype == B200ATTN_F32) {
    const int rb = p.rows >= 3 ? 4 : p.rows;
    const size_t smem = simt_smem(p.cluster, p.rows, D);
    int rc = 0;
#define B200ATTN_LAUNCH_SIMT(DIM, RB)                                                                 \
    do {                                                                                              \
      if (p.cluster) {                                                                                \
        if ((rc = set_smem(decode_simt_kernel<DIM, RB, true>, smem))) return rc;                      \
        launch_dependent(decode_simt_kernel<DIM, RB, true>, grid, kSimtThreads, smem, stream, p.cluster, p); \
      } else {                                                                                        \
        if ((rc = set_smem(decode_simt_kernel<DIM, RB, false>, smem))) return rc;                     \
        launch_dependent(decode_simt_kernel<DIM, RB, false>, grid, kSimtThreads, smem, stream, 1, p); \
      }                                                                                               \
    } while (0)
    if (D == 128) { if (rb == 1) B200ATTN_LAUNCH_SIMT(128, 1); else if (rb == 2) B200ATTN_LAUNCH_SIMT(128, 2); else B200ATTN_LAUNCH_SIMT(128, 4); }
    else          { if (rb == 1) B200ATTN_LAUNCH_SIMT(64, 1);  else if (rb == 2) B200ATTN_LAUNCH_SIMT(64, 2);  else B200ATTN_LAUNCH_SIMT(64, 4); }
#undef B200ATTN_LAUNCH_SIMT
  } else if (p.rows > 16) {
    // many q rows per KV head: one 128-row tcgen05 tile with Q and P in tensor memory
    CUtensorMap tk, tv;
    int rc = 0;
    const int box = page_box(a);
    p.box_shift = 0;
    while ((1 << p.box_shift) < box) ++p.box_shift;
    long long tokens;
    int heads;
    if (a.layout == B200ATTN_DENSE) { tokens = static_cast<long long>(a.batch) * a.kv_heads * a.max_kv; heads = 1; }
    else { tokens = a.total_kv; heads = a.kv_heads; }
    if ((rc = make_token_map(&tk, a.dtype, a.k, tokens, heads, D, box))) return rc;
    if ((rc = make_token_map(&tv, a.dtype, a.v, tokens, heads, D, box))) return rc;
    const size_t stage_bytes = static_cast<size_t>(kUmmaStages) * 2 * kTileN * D * 2;
    const size_t smem = 1024 + stage_bytes + sizeof(UmmaCtrl);
    // persistent: one wave walks the unit list (fewer CTAs when the list cannot be longer)
    auto wave_of = [&](int ctas) { return dim3(std::min(static_cast<unsigned>(w.max_items) * a.kv_heads, static_cast<unsigned>(ctas))); };
    const dim3 grid = p.inline_plan ? dim3(grid_items * a.kv_heads) : wave_of(2 * sm_count);
    CUtensorMap tq, gk = tk, gv = tv;
    if (key_rows) {
      const long long q_rows = static_cast<long long>(a.batch) * a.q_heads * a.q_len;
      if ((rc = make_token_map(&tq, a.dtype, a.q, q_rows, 1, D, (p.rows + 15) & ~15))) return rc;
      if (D == 128 && a.layout == B200ATTN_PAGED) {
        if ((rc = make_kv_groups_map(&gk, a.dtype, a.k, tokens, heads, D, box, heads * D * 2ll, D * 2ll))) return rc;
        if ((rc = make_kv_groups_map(&gv, a.dtype, a.v, tokens, heads, D, box, heads * D * 2ll, D * 2ll))) return rc;
      }
    }
#define B200ATTN_LAUNCH_UMMA(TYPE, DIM, OUT)                                  \
    do {                                                                      \
      if (key_rows) {                                                         \
        constexpr size_t bytes = KrPlan<DIM>::kTotal;                         \
        if ((rc = set_smem(decode_keyrows_kernel<TYPE, DIM, OUT>, bytes))) return rc; \
        launch_dependent(decode_keyrows_kernel<TYPE, DIM, OUT>, wave_of(sm_count), kKrThreads, bytes, stream, 1, tq, gk, gv, p); \
        break;                                                                \
      }                                                                       \
      auto* kernel = p.inline_plan ? decode_umma_kernel<TYPE, DIM, OUT, true> \
                                   : decode_umma_kernel<TYPE, DIM, OUT, false>; \
      if ((rc = set_smem(kernel, smem))) return rc;                           \
      launch_dependent(kernel, grid, kUmmaThreads, smem, stream, 1, tk, tv, p); \
    } while (0)
    if (f32_out) {
      if (D == 128) B200ATTN_LAUNCH_UMMA(__half, 128, float); else B200ATTN_LAUNCH_UMMA(__half, 64, float);
    } else if (a.dtype == B200ATTN_BF16) {
      if (D == 128) B200ATTN_LAUNCH_UMMA(__nv_bfloat16, 128, __nv_bfloat16); else B200ATTN_LAUNCH_UMMA(__nv_bfloat16, 64, __nv_bfloat16);
    } else {
      if (D == 128) B200ATTN_LAUNCH_UMMA(__half, 128, __half); else B200ATTN_LAUNCH_UMMA(__half, 64, __half);
    }
#undef B200ATTN_LAUNCH_UMMA
  } else {
    // at most 16 q rows per KV head reach this kernel (more go to the tcgen05 kernel above): one 16-row tile, four
    // consumer warps that split every K/V tile by key slice, and the producer warp
    const int nmt = p.n_mtiles;
    if (nmt != 1) { set_error("decode: %d row tiles per KV head in the warp-level kernel", nmt); return B200ATTN_E_UNSUPPORTED; }
    const int threads = 32 * (kMmaSlices + 1);
    // measured on B200 (paged decode, 32/8 heads): 2 stages with Q re-read from shared memory lets three CTAs share an
    // SM and hides each CTA's start-up and merge behind its neighbours
    int stages = 2;
    if (p.cluster) {
      // The parts are a few tiles long: as many stages as fit, so that a part's copies are under way at once (two stages made every
      // second tile wait for its copy; with that, and a producer that does not wait for the Q rows, 16 x 2 048 keys of two heads,
      // D 64, take 7.5 us instead of 8.0, one sequence of 1 500 in pages, D 128, 7.5 instead of 8.8).  Stages that cost an SM
      // a CTA are taken only where the clusters then leave a sixteenth of the GPU free: the next call's set up
      // beside them (4 x 300 keys, 32/8 heads, D 128, 32 clusters of 33: 8.2 us with three stages, 7.2 with two, 2 048 keys in
      // pages 12.6 and 11.5; 8 x 300, 64 of 71: 7.2 and 8.2).
      const int most = ctas_per_sm(mma_smem(2, p.cluster, p.rows, D));
      auto fits = [&](int n) {
        const int per_sm = ctas_per_sm(mma_smem(n, p.cluster, p.rows, D));
        if (per_sm == most) return true;
        const int held = per_sm > 0 ? clusters_held(p.cluster, per_sm, sm_count, /*ask=*/true) : 0;
        return pairs <= held - held / 16;
      };
      while (stages < kMaxStages && fits(stages + 1)) ++stages;
    }
    p.stages = stages;
    const size_t smem = mma_smem(stages, p.cluster, p.rows, D);
    // tensor maps over K and V: (D, heads, tokens), one box = 64 elements x 1 head x box_rows keys
    CUtensorMap tk, tv;
    int rc = 0;
    const int box = page_box(a);
    p.box_shift = 0;
    while ((1 << p.box_shift) < box) ++p.box_shift;
    if (a.layout == B200ATTN_DENSE) {
      const long long rows = static_cast<long long>(a.batch) * a.kv_heads * a.max_kv;
      if ((rc = make_kv_rows_map(&tk, a.dtype, a.k, rows, 1, D, box, D * 2ll, D * 2ll))) return rc;
      if ((rc = make_kv_rows_map(&tv, a.dtype, a.v, rows, 1, D, box, D * 2ll, D * 2ll))) return rc;
    } else {
      const long long rstride = static_cast<long long>(a.kv_heads) * D * 2;
      if ((rc = make_kv_rows_map(&tk, a.dtype, a.k, a.total_kv, a.kv_heads, D, box, rstride, D * 2ll))) return rc;
      if ((rc = make_kv_rows_map(&tv, a.dtype, a.v, a.total_kv, a.kv_heads, D, box, rstride, D * 2ll))) return rc;
    }
#define B200ATTN_LAUNCH_DECODE_V(TYPE, DIM, STAGES, NBLK, MAXT, MINB, OUT)                               \
    do {                                                                                                  \
      if (p.cluster) {                                                                                    \
        if ((rc = set_smem(decode_mma_kernel<TYPE, DIM, STAGES, NBLK, MAXT, MINB, OUT, true>, smem))) return rc; \
        launch_dependent(decode_mma_kernel<TYPE, DIM, STAGES, NBLK, MAXT, MINB, OUT, true>, grid, threads, smem, stream, p.cluster, tk, tv, p); \
      } else {                                                                                            \
        if ((rc = set_smem(decode_mma_kernel<TYPE, DIM, STAGES, NBLK, MAXT, MINB, OUT, false>, smem))) return rc; \
        launch_dependent(decode_mma_kernel<TYPE, DIM, STAGES, NBLK, MAXT, MINB, OUT, false>, grid, threads, smem, stream, 1, tk, tv, p); \
      }                                                                                                   \
    } while (0)
#define B200ATTN_LAUNCH_DECODE(TYPE, DIM, OUT) B200ATTN_LAUNCH_DECODE_V(TYPE, DIM, 2, 1, 160, 3, OUT)
    if (f32_out) {
      if (D == 128) B200ATTN_LAUNCH_DECODE(__half, 128, float); else B200ATTN_LAUNCH_DECODE(__half, 64, float);
    } else if (a.dtype == B200ATTN_BF16) {
      if (D == 128) B200ATTN_LAUNCH_DECODE(__nv_bfloat16, 128, __nv_bfloat16); else B200ATTN_LAUNCH_DECODE(__nv_bfloat16, 64, __nv_bfloat16);
    } else {
      if (D == 128) B200ATTN_LAUNCH_DECODE(__half, 128, __half); else B200ATTN_LAUNCH_DECODE(__half, 64, __half);
    }
#undef B200ATTN_LAUNCH_DECODE_V
#undef B200ATTN_LAUNCH_DECODE
  }
  e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "decode kernel launch");
  return B200ATTN_OK;
}
}  // namespace

// the call as its passes see it: fp32 inputs that are copied are fp16
static b200attn_decode_args_t as_launched(const b200attn_decode_args_t& a, int sm_count, bool built_in) {
  b200attn_decode_args_t b = a;
  if (decode_ws_layout(a, sm_count, /*allow_cast=*/!built_in).cast_kv_elems > 0) b.dtype = B200ATTN_F16;
  return b;
}

int decode_route(const b200attn_decode_args_t& a, int sm_count, bool built_in) {
  const Route r = route_of(as_launched(a, sm_count, built_in), sm_count, decode_pass_group(a.q_heads / a.kv_heads, a.q_len) * a.q_len, built_in,
                           /*ask=*/false);
  return r.cluster ? r.cluster : r.inline_plan ? B200ATTN_ROUTE_INLINE : B200ATTN_ROUTE_PLANNER;
}

bool decode_keys_as_rows(const b200attn_decode_args_t& a, int sm_count, bool built_in) {
  return keyrows_suit(as_launched(a, sm_count, built_in), sm_count, decode_pass_group(a.q_heads / a.kv_heads, a.q_len) * a.q_len);
}

// ---------------------------------------------------------------------------
// Decode without any caller-provided or allocated scratch memory.
//
// Some hosts of this library are not allowed to allocate device memory at the moment they need
// attention: an inference server that hands its whole HBM budget to the KV cache at start-up and
// forbids allocations afterwards, a plug-in running inside another framework's memory pool, or
// code running while that framework is recording its work and must not disturb its allocator.
// For them the planner tables, merge tickets and split-KV partials live in this fixed array,
// which is part of the loaded module: every GPU that loads the library holds kStaticScratchBytes
// of it until the process exits.
// ---------------------------------------------------------------------------
constexpr size_t kStaticScratchBytes = size_t(8) << 20;  // 8 MiB
static __device__ __align__(256) unsigned char g_decode_scratch[kStaticScratchBytes];

namespace {
constexpr int kScratchMaxDevices = 64;
std::mutex g_scratch_mutex;
void* g_scratch_ptr[kScratchMaxDevices] = {};
}  // namespace

// `a.device` must be the current device.  The first call on a device resolves the device address of
// the array (in host code `g_decode_scratch` itself is only a handle, not something a kernel may be
// given); later calls reuse the cached address.
int launch_decode_static(const b200attn_decode_args_t& a, int sm_count, cudaStream_t stream) {
  if (a.device < 0 || a.device >= kScratchMaxDevices) {
    set_error("decode_static: device ordinal %d out of range", a.device);
    return B200ATTN_E_INVALID;
  }
  const DecodeWsLayout w = decode_ws_layout(a, sm_count, /*allow_cast=*/false);
  if (w.total > kStaticScratchBytes) {
    set_error("decode_static: this problem needs %zu bytes of scratch but the built-in array holds %zu; "
              "use b200attn_decode with a caller-provided workspace", w.total, kStaticScratchBytes);
    return B200ATTN_E_WORKSPACE;
  }
  void* ptr = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_scratch_ptr[a.device] == nullptr) {
      void* resolved = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&resolved, g_decode_scratch);
      if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(decode scratch)");
      g_scratch_ptr[a.device] = resolved;
    }
    ptr = g_scratch_ptr[a.device];
  }
  b200attn_decode_args_t b = a;
  b.workspace = ptr;
  b.workspace_bytes = kStaticScratchBytes;
  // The planner kernel rewrites the item prefix and zeroes the merge tickets at the start of every
  // call, and partial slots are always written before they are read, so stale contents are harmless.
  return launch_decode(b, sm_count, stream, /*built_in=*/true);
}


// Reads and clears the device error word of the built-in array (word 0, where the kernels of
// launch_decode_static report an expired wait, an out-of-range block-table entry or a planner overflow).
// One small copy on `stream`, which it synchronises; allocates nothing.  `device` must be current.
int check_decode_static(int device, cudaStream_t stream, int32_t* code) {
  if (device < 0 || device >= kScratchMaxDevices) {
    set_error("decode_static_check: device ordinal %d out of range", device);
    return B200ATTN_E_INVALID;
  }
  void* ptr = nullptr;
  {
    std::lock_guard<std::mutex> lock(g_scratch_mutex);
    if (g_scratch_ptr[device] == nullptr) {
      void* resolved = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&resolved, g_decode_scratch);
      if (e != cudaSuccess) return cuda_fail(e, "cudaGetSymbolAddress(decode scratch)");
      g_scratch_ptr[device] = resolved;
    }
    ptr = g_scratch_ptr[device];
  }
  int32_t word = 0;
  cudaError_t e = cudaMemcpyAsync(&word, ptr, sizeof(word), cudaMemcpyDeviceToHost, stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(e, "reading the built-in array's error word");
  if (code) *code = word;
  if (word == 0) return B200ATTN_OK;
  e = cudaMemsetAsync(ptr, 0, sizeof(word), stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(stream);
  if (e != cudaSuccess) return cuda_fail(e, "clearing the built-in array's error word");
  set_error("a decode_static kernel reported device error code %d (1 = bounded wait expired, 2 = block-table entry "
            "out of range, 3 = planner overflow)", word);
  return B200ATTN_E_DEVICE;
}

// ---------------------------------------------------------------------------
// Self-test of a cluster in which one CTA is late: of two CTAs that share a row the second sends its part only after the
// first has run out of patience (a bounded wait on a barrier that nothing completes, much longer than the first's).
// out[0 .. 63]: the row, out[64]: 1 when everything sent to the first CTA had landed by the time it left cluster_emit.
// ---------------------------------------------------------------------------
namespace {
__global__ void __launch_bounds__(64) cluster_expiry_selftest_kernel(const DecodeParams p, uint32_t tries, int late) {
  constexpr int D = 64;
  __shared__ __align__(16) float comb_o[D];
  __shared__ float comb_ml[2];
  __shared__ __align__(16) unsigned char recv[2 * (D / 8) * 16 + 2 * 8];
  __shared__ uint64_t recv_bar, dead_bar;
  const ClusterPart part = cluster_part<D>(p);
  cluster_begin<D>(p, part, &recv_bar);
  ptx::grid_dep_wait();      // (the caller's zero fill of the header)
  comb_o[threadIdx.x] = static_cast<float>(part.rank + 1);
  if (threadIdx.x == 0) {
    comb_ml[0] = 0.f;
    comb_ml[1] = 1.f;
    ptx::mbar_init(smem_u32(&dead_bar), 1);
    ptx::mbar_fence_init();
  }
  __syncthreads();
  if (late && part.rank == 1) ptx::mbar_wait_limit(smem_u32(&dead_bar), 0, 64 * tries);
  __syncthreads();
  cluster_emit<float, D>(p, part, 0, 0, comb_o, comb_ml, 1, 1, recv, &recv_bar, tries);
  if (part.rank == 0 && threadIdx.x == 0) static_cast<float*>(p.out)[D] = ptx::mbar_try_wait(smem_u32(&recv_bar), 0) ? 1.f : 0.f;
}
}  // namespace

// Self-test of what a CTA of the persistent kernels does when it gives up: `published` entries, the last of them the end mark if `ended`,
// unit r being sequence r with one row of 64; the rows that its poison_units fills become NaN.
namespace {
__global__ void __launch_bounds__(64) abandoned_units_selftest_kernel(const DecodeParams p, int published, int ended, int abort_round) {
  __shared__ UmmaCtrl ctrl;
  const int n_units = published - (ended ? 1 : 0);
  if (threadIdx.x == 0) {
    for (int r = max(0, published - kUmmaUnitRing); r < published; ++r) ctrl.unit_ring[r % kUmmaUnitRing] = r;
    ctrl.published = published;
    ctrl.abort_round = abort_round;
  }
  __syncthreads();
  poison_units<float, 64>(p, &ctrl, n_units, [&](int r) { UmmaUnit w = {}; w.b = ctrl.unit_ring[r % kUmmaUnitRing]; return w; });
}
}  // namespace

int launch_abandoned_units_selftest(float* out, int published, int ended, int abort_round, cudaStream_t stream) {
  DecodeParams p = {};
  p.out = out;
  p.q_heads = p.kv_heads = p.head_stride = p.q_len = p.rows = 1;
  abandoned_units_selftest_kernel<<<1, 64, 0, stream>>>(p, published, ended, abort_round);
  const cudaError_t e = cudaGetLastError();
  return e == cudaSuccess ? B200ATTN_OK : cuda_fail(e, "abandoned-units selftest kernel launch");
}

int launch_cluster_selftest(int* header, float* out, uint32_t tries, int late, cudaStream_t stream) {
  DecodeParams p = {};
  p.header = header;
  p.out = out;
  p.cluster = 2;
  p.batch = p.q_heads = p.kv_heads = p.group = p.head_stride = p.q_len = p.rows = 1;
  const cudaError_t e = launch_dependent(cluster_expiry_selftest_kernel, dim3(2), 64, 0, stream, 2, p, tries, late);
  return e == cudaSuccess ? B200ATTN_OK : cuda_fail(e, "cluster selftest kernel launch");
}

}  // namespace b200attn
