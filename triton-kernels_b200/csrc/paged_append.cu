// Paged KV-cache write side: scatters new K or V rows of every sequence into the pages its block table names.
// It is the inverse of the gather the attention kernels perform and replaces the Python double loop of the
// reference's fixtures (tests/test_attention.py:101-134, benchmarks/attention.py:351-431).  Pure byte movement:
// one warp per token row, 16-byte pieces, every source and destination byte touched once.
#include "common.cuh"
#include "launch.cuh"
#include "paged_append_launch.h"
#include "sm100_ptx.cuh"

namespace b200attn {

namespace {

// What bounds it at the sizes it runs at (a token, a chunk) is its chain of dependent reads, each an L2 round trip: the owner
// of a row is looked for by the whole warp, 32 prefix sums per step, together with the sequence's position and while the row
// itself is on its way, which leaves two round trips, those and the table's, where a binary search by every lane made seven
// of them at sixteen sequences: one user (two appends of a token and a decode call) 13.5 -> 12.3 us.
__global__ void __launch_bounds__(256) paged_append_kernel(const PagedAppendParams p) {
  const int lane = threadIdx.x & 31;
  const long long warp = (static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x) >> 5;
  const long long nwarps = (static_cast<long long>(gridDim.x) * blockDim.x) >> 5;
  const int pieces = p.row_bytes >> 4;
  constexpr int kHeld = 4;                  // 16-byte pieces of the row that a lane holds before it knows where they go
  ptx::grid_dep_launch_dependents();
  ptx::grid_dep_wait();
  for (long long row = warp; row < p.total_rows; row += nwarps) {
    const uint4* src = reinterpret_cast<const uint4*>(static_cast<const unsigned char*>(p.src) + row * p.row_bytes);
    uint4 held[kHeld];
#pragma unroll
    for (int i = 0; i < kHeld; ++i)
      if (lane + 32 * i < pieces) held[i] = __ldcg(src + lane + 32 * i);
    // sequence that owns this source row: the last b with indptr[b] <= row, among [lo, lo + n)
    int lo = 0, n = p.batch;
    while (n > 32) {
      const int step = (n + 31) >> 5, at = lane * step;
      const unsigned below = __ballot_sync(0xffffffffu, at < n && load_index(p.src_indptr, p.indptr_is_i64, lo + at) <= row);
      const int k = below ? 31 - __clz(below) : 0;
      lo += k * step;
      n = min(step, n - k * step);
    }
    long long first = 0, end = 0, pos0 = 0;
    if (lane < n) {
      first = load_index(p.src_indptr, p.indptr_is_i64, lo + lane);
      end = load_index(p.src_indptr, p.indptr_is_i64, lo + lane + 1);
      if (p.dst_pos) pos0 = load_index(p.dst_pos, p.indptr_is_i64, lo + lane);
    }
    const unsigned owner = __ballot_sync(0xffffffffu, first <= row && row < end);
    if (owner == 0) continue;                 // malformed prefix sums: nothing is written
    const int o = 31 - __clz(owner), b = lo + o;
    const long long pos = row - __shfl_sync(0xffffffffu, first, o) + __shfl_sync(0xffffffffu, pos0, o);
    const long long lp = (static_cast<unsigned long long>(pos) >> 31) == 0
                             ? static_cast<long long>(static_cast<unsigned>(pos) / static_cast<unsigned>(p.page_size)) : pos / p.page_size;
    if (pos < 0 || lp >= p.table_stride) {
      if (lane == 0) p.header[0] = DEV_ERR_PAGE_RANGE;
      continue;
    }
    const int page = __ldcg(p.table + static_cast<long long>(b) * p.table_stride + lp);
    if (page < 0 || page >= p.num_pages) {
      if (lane == 0) p.header[0] = DEV_ERR_PAGE_RANGE;   // reported, never dereferenced
      continue;
    }
    const long long dst_row = static_cast<long long>(page) * p.page_size + (pos - lp * p.page_size);
    uint4* dst = reinterpret_cast<uint4*>(static_cast<unsigned char*>(p.cache) + dst_row * p.row_bytes);
#pragma unroll
    for (int i = 0; i < kHeld; ++i)
      if (lane + 32 * i < pieces) dst[lane + 32 * i] = held[i];
    for (int i = lane + 32 * kHeld; i < pieces; i += 32) dst[i] = __ldcg(src + i);
  }
}

}  // namespace

int launch_paged_append(const b200attn_paged_append_args_t& a, int sm_count, cudaStream_t stream) {
  PagedAppendParams p;
  p.src = a.src; p.cache = a.cache; p.src_indptr = a.src_indptr; p.dst_pos = a.dst_pos; p.table = a.table;
  p.header = static_cast<int*>(a.workspace);
  p.total_rows = a.total_rows; p.table_stride = a.table_stride;
  p.row_bytes = a.row_bytes; p.indptr_is_i64 = a.indptr_is_i64; p.batch = a.batch; p.page_size = a.page_size;
  const long long pages = a.cache_rows / a.page_size;
  p.num_pages = static_cast<int>(pages > 0x7fffffff ? 0x7fffffff : pages);
  if (a.total_rows == 0) return B200ATTN_OK;
  const long long warps_needed = a.total_rows;
  long long blocks = (warps_needed + 7) / 8;              // 8 warps per block
  const long long cap = static_cast<long long>(sm_count) * 16;
  if (blocks > cap) blocks = cap;
  const cudaError_t e = launch_dependent(paged_append_kernel, dim3(static_cast<unsigned>(blocks)), 256, 0, stream, 1, p);
  if (e != cudaSuccess) return cuda_fail(e, "paged_append_kernel launch");
  return B200ATTN_OK;
}

}  // namespace b200attn
