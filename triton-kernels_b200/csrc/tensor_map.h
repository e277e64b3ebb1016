// Host helper: TMA tensor maps over token-major 16-bit tensors.
#pragma once

#include <cuda.h>

namespace b200attn {

// 3-D map over a [tokens][heads][D] 16-bit tensor (heads == 1 for tensors whose rows of one head are
// contiguous): box = 64 elements x 1 head x box_rows tokens, 128-byte swizzle, zero fill out of bounds.
// `dtype` is B200ATTN_F16 or B200ATTN_BF16.  Returns 0 or a B200ATTN_E_* code.
int make_token_map(CUtensorMap* m, int dtype, const void* base, long long tokens, int heads, int D, int box_rows);

// 4-D map used by the decode kernels: dims (64 elements, token rows, D/64 column blocks, heads) with strides
// (row_stride_bytes, 128, head_stride_bytes); box = 64 x box_rows x D/64 x 1, 128-byte swizzle.  One copy
// brings box_rows keys of one head as [column block][row][128 B] into shared memory.
int make_kv_rows_map(CUtensorMap* m, int dtype, const void* base, long long rows, int heads, int D, int box_rows,
                     long long row_stride_bytes, long long head_stride_bytes);

// 5-D map over the same rows in groups of eight: dims (64 elements, 8 rows, D/64 column blocks, groups, heads); box = 64 x 8 x D/64 x
// box_rows / 8 x 1, 128-byte swizzle, box_rows a multiple of eight.  One copy brings box_rows keys of one head as
// [group][column block][row of the group][128 B], which, unlike the 4-D map's order, a tcgen05 descriptor can address across boxes of any
// size: the groups of a column block lie at one distance in the whole tile.
int make_kv_groups_map(CUtensorMap* m, int dtype, const void* base, long long rows, int heads, int D, int box_rows,
                       long long row_stride_bytes, long long head_stride_bytes);

}  // namespace b200attn
