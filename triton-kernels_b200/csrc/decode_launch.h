// Host/device shared declarations for the decode path.
#pragma once

#include <cuda_runtime.h>
#include <stddef.h>

#include "../../include/b200attn.h"

namespace b200attn {

// Merge tickets of calls without a planner launch: 16 bits per (sequence, KV head) pair in the workspace header, the
// only part of a workspace that keeps its contents between calls (every call leaves them at zero); 8 bits where a pair cannot be
// cut into more than 255 items.
constexpr int kTicketWord = 16;                     // first header word that holds tickets
constexpr int kInlinePairs = 2 * (64 - kTicketWord);
constexpr int kInlinePairs8 = 4 * (64 - kTicketWord);
constexpr int kInlineBatch = kInlinePairs;          // sequences that a CTA plans

// Kernel parameter block (passed by value).
struct DecodeParams {
  const void* q;
  const void* k;
  const void* v;
  void* out;
  const void* kv_indptr;
  const int* k_table;
  const int* v_table;
  int* header;       // [0] error code, [1] chunk tokens, [2] number of work items, [5] slots dealt out, [kTicketWord ...] inline-plan tickets
  int* item_start;   // [batch + 1] prefix of per-sequence chunk counts
  int* counters;     // [batch * kv_heads] merge tickets
  int4* item_info;   // [max_items][2]: {sequence, chunk + (chunks << 16), first item of the sequence, first key}, {len, end key, start lo, start hi}
  float* part_ml;    // [slot][rows][2]  (running max in log2 units, running sum)
  float* part_o;     // [slot][rows][D]  un-normalised accumulators
  long long total_kv;
  long long table_stride;
  int layout;
  int indptr_is_i64;
  int batch;
  int q_heads;
  int kv_heads;
  int group;         // q heads per kv head served by this launch
  int head_stride;   // q heads per kv head in the tensors
  int head0;         // first q head (inside each kv head's group) this launch serves
  int q_len;         // M
  int rows;          // group * M: q rows that share one kv head
  int n_mtiles;      // ceil(rows / 16)
  int max_kv;
  int page_size;
  int page_shift;    // log2(page_size) or -1
  int num_pages;
  int box_shift;     // log2 of the keys per TMA box (paged: the largest power of two that divides the page size, <= 64)
  int causal;
  int target_items;
  int wave_items;    // items of one KV head that are resident at once (one wave of CTAs); 0: never plan a single wave
  int item_overhead; // start-up and merge of a work item, in keys of streaming time (planner's cost estimate)
  int min_chunk;
  int max_items;
  int one_cta;       // the persistent kernel has one CTA to an SM: see the planner's estimates
  int slots;         // persistent kernel: CTAs per KV head that the planner may deal the batch out to; 0: none
  int inline_plan;   // not 0: no planner launch, every CTA works out its own item (few (sequence, KV head) pairs); the bits of a merge ticket
  int pair_tickets;  // such calls of few pairs, and those in the own array: header bytes of a pair, the first its merge ticket, the others those of groups of its chunks; else 0
  int cluster;       // CTAs that share a (sequence, KV head) pair in the kernels without a plan; 0: items are planned
  int stages;        // K/V stages of a CTA of the warp-level kernel in a cluster
  float scale_log2;  // sm_scale * log2(e)
};

struct DecodeWsLayout {
  size_t item_start_off;
  size_t counters_off;
  size_t info_off;
  size_t ml_off;
  size_t o_off;
  size_t total;
  int target_items;
  int wave_items;    // items of one KV head that are resident at once (one wave of CTAs); 0: never plan a single wave
  int item_overhead; // start-up and merge of a work item, in keys of streaming time (planner's cost estimate)
  int min_chunk;
  int max_items;
  // fp32 inputs of a speculative-decode call: fp16 copies of q, k, v that the tensor-core kernels read
  // (0 elements: no copies, the launch reads the caller's tensors)
  size_t cast_q_off, cast_k_off, cast_v_off;
  size_t cast_q_elems, cast_kv_elems;
};

int decode_pass_group(int group, int q_len);
// `allow_cast` false: plan fp32 inputs for the fp32 FMA kernel whatever the row count (no room for copies)
DecodeWsLayout decode_ws_layout(const b200attn_decode_args_t& a, int sm_count, bool allow_cast = true);
// `built_in`: the workspace is the library's own array (launch_decode_static): no casts, and always a planner launch
int launch_decode(const b200attn_decode_args_t& a, int sm_count, cudaStream_t stream, bool built_in = false);
// which way a call goes: see b200attn_decode_route
int decode_route(const b200attn_decode_args_t& a, int sm_count, bool built_in);
// whether its passes behind the planner are decode_keyrows_kernel's: see b200attn_decode_keys_as_rows
bool decode_keys_as_rows(const b200attn_decode_args_t& a, int sm_count, bool built_in);
int launch_decode_static(const b200attn_decode_args_t& a, int sm_count, cudaStream_t stream);
int check_decode_static(int device, cudaStream_t stream, int32_t* code);
int launch_cluster_selftest(int* header, float* out, uint32_t tries, int late, cudaStream_t stream);
int launch_abandoned_units_selftest(float* out, int published, int ended, int abort_round, cudaStream_t stream);

}  // namespace b200attn
