// Row softmax / log-softmax over the last dimension for sm_100a (HBM-bound: one read, one write).
//
// Replaces the reference's small / medium / partial + merge + finalize kernels (kernels/softmax.py:18-150 and
// :239-375): there a row longer than one block is read twice (three launches when it is split over programs).
// Here a row is read once, kept on the SM and normalised from there:
//   softmax_warp_kernel    up to 4 KiB (fp32 3 KiB): a warp per row, the row in its registers
//   softmax_reg_kernel     up to 64 KiB: one CTA per row, the row in registers
//   softmax_pipe_kernel    up to 108 KiB, most rows of whole pieces: one CTA per row, two or three rows in shared memory
//   softmax_ring_kernel    the others up to 1.75 MiB: a CTA, or a cluster of 2, 4 or 8 CTAs, per row; the row passes through
//                          a ring of shared-memory chunks filled by bulk copies, the next row loads while this one is
//                          reduced and written
// These move 16-byte pieces; the few elements of a row before its first and behind its last 16-byte boundary travel
// singly, so the row length may be anything.  Rows that are longer, or lie differently in x and out:
//   softmax_row_kernel     up to 200 KiB: one CTA per row, the row in shared memory
//   softmax_cluster_kernel up to 1.6 MB: 200 KiB per CTA in shared memory, cluster of eight
//   softmax_stream_kernel  beyond: one CTA per row, online (max, sum) pass, then a second read
// Clusters exchange their (max, sum) pairs through distributed shared memory; the ring kernel does it with
// asynchronous remote stores that count on the receiver's mbarrier, because a cluster-wide barrier also waits
// for the previous row's global stores.
// All arithmetic is fp32, like the reference's `.to(tl.float32)`.  fp32 results are expf of x - max (softmax) or x - max
// minus the logarithm of the sum, whose terms are within 2^-22 (piece_exp_sum, which says what the ring does instead);
// 16-bit rows take ex2.approx of (x - max) * log2(e), as tl.exp compiles to.  `out` may alias `x`: a row is written only after all of it has been staged
// (the streaming kernel reads element i right before it writes element i), and rows staged ahead of time are other rows.
#include <cooperative_groups.h>

#include <algorithm>
#include <atomic>
#include <type_traits>

#include "common.cuh"
#include "launch.cuh"
#include "sm100_ptx.cuh"
#include "softmax_launch.h"

namespace cg = cooperative_groups;

namespace b200attn {

namespace {

constexpr int kRowSmemBytes = 200 * 1024;   // row bytes one CTA stages
constexpr int kMaxCluster = 8;              // portable cluster size

__device__ __forceinline__ float warp_max(float v) {
  for (int o = 16; o > 0; o >>= 1) v = fmaxf(v, __shfl_xor_sync(0xffffffffu, v, o));
  return v;
}
__device__ __forceinline__ float warp_sum(float v) {
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// block-wide reductions through a 32-float scratch array; every thread gets the result
__device__ __forceinline__ float block_max(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  __syncthreads();                 // scratch may still be read from a previous reduction
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float r = lane < nw ? scratch[lane] : -INFINITY;
  return warp_max(r);
}
__device__ __forceinline__ float block_sum(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  __syncthreads();
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  float r = lane < nw ? scratch[lane] : 0.f;
  return warp_sum(r);
}

// the same without the leading barrier: the caller guarantees a barrier between the last read of `scratch` and this call
__device__ __forceinline__ float block_max_nolead(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_max(v);
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  return warp_max(lane < nw ? scratch[lane] : -INFINITY);
}
__device__ __forceinline__ float block_sum_nolead(float v, float* scratch) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nw = (blockDim.x + 31) >> 5;
  v = warp_sum(v);
  if (lane == 0) scratch[warp] = v;
  __syncthreads();
  return warp_sum(lane < nw ? scratch[lane] : 0.f);
}

template <typename T> struct Vec16 { static constexpr int kElems = 16 / sizeof(T); };

// a 32-bit word of -inf
template <typename T>
constexpr uint32_t kNegInfWord = sizeof(T) == 4 ? 0xff800000u : (std::is_same<T, __half>::value ? 0xfc00fc00u : 0xff80ff80u);

template <typename T> __device__ __forceinline__ float fast_or_exact_exp(float x) {
  // 16-bit outputs round away far more than the approximate exponential loses; fp32 outputs need expf
  if constexpr (sizeof(T) == 2) return __expf(x);
  else return expf(x);
}


// A maximum drops NaN, so a part of a row whose maximum is -inf may still hold one.  Its terms are taken against 0 then:
// exp(-inf) = 0 adds nothing and exp(NaN) reaches the sum, where a part that is skipped would lose it (a masked row with a
// NaN would come out as a distribution).  A part's sum moves to another reference the same way: 0 * 0 or NaN * 0.
__device__ __forceinline__ float exp_ref(float m) { return m == -INFINITY ? 0.f : m; }

// (max, sum of exp(x - max)) of two parts
__device__ __forceinline__ void merge_ml(float& m, float& l, float m2, float l2) {
  const float g = fmaxf(m, m2), ref = exp_ref(g);
  l = l * expf(m - ref) + l2 * expf(m2 - ref);
  m = g;
}

// Stage `n` elements of a row in shared memory and return this thread's running max.
template <typename T>
__device__ __forceinline__ float stage_row(const T* src, T* row, long long n) {
  float mx = -INFINITY;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) {
    const T v = src[i];            // (plain load: `out` may alias `x`)
    row[i] = v;
    mx = fmaxf(mx, ElemTraits<T>::to_float(v));
  }
  return mx;
}

template <typename T>
__device__ __forceinline__ float row_exp_sum(const T* row, long long n, float m) {
  const float ref = exp_ref(m);
  float s = 0.f;
  for (long long i = threadIdx.x; i < n; i += blockDim.x) s += fast_or_exact_exp<T>(ElemTraits<T>::to_float(row[i]) - ref);
  return s;
}

// softmax: exp(x - m) / l;  log-softmax: (x - m) - log l  (in this order: m + log l would lose log l next to a
// large m)
template <typename T, bool LOG>
__device__ __forceinline__ T finish(float x, float m, float k) {
  if constexpr (LOG) return ElemTraits<T>::from_float((x - m) - k);
  else return ElemTraits<T>::from_float(fast_or_exact_exp<T>(x - m) * k);
}

template <typename T, bool LOG>
__device__ __forceinline__ void write_row(const T* row, T* dst, long long n, float m, float k) {
  for (long long i = threadIdx.x; i < n; i += blockDim.x) dst[i] = finish<T, LOG>(ElemTraits<T>::to_float(row[i]), m, k);
}

// the constant the write pass needs: 1 / l for softmax, log l for log-softmax
template <bool LOG>
__device__ __forceinline__ float final_constant(float m, float l) {
  (void)m;
  if constexpr (LOG) return logf(l);
  else return 1.f / l;
}

// ---------------------------------------------------------------------------
// one CTA per row, the row in registers: thread t holds the 16-byte pieces t, t + blockDim, ... (VPT of them)
// ---------------------------------------------------------------------------

// the elements of one 32-bit word of a 16-byte piece (two 16-bit values, or one float) <-> fp32
template <typename T> __device__ __forceinline__ void word_to_floats(uint32_t w, float* f) {
  if constexpr (std::is_same<T, __nv_bfloat16>::value) {
    f[0] = __uint_as_float(w << 16);                 // a bf16 is the upper half of the fp32 with the same value
    f[1] = __uint_as_float(w & 0xffff0000u);
  } else if constexpr (std::is_same<T, __half>::value) {
    const float2 t = __half22float2(*reinterpret_cast<const __half2*>(&w));
    f[0] = t.x;
    f[1] = t.y;
  } else {
    f[0] = __uint_as_float(w);
  }
}
template <typename T> __device__ __forceinline__ uint32_t floats_to_word(const float* f) {
  if constexpr (sizeof(T) == 2) return ElemTraits<T>::pack2(f[0], f[1]);
  else return __float_as_uint(f[0]);
}

// Where a row lies relative to the 16-byte grid of memory: `head` elements before the first 16-byte boundary, `nv` whole
// 16-byte pieces, and the rest behind them.  x and out are misaligned by the same amount (the launcher checks), so the
// pieces of a row are aligned in both; the fewer than 2 E elements around them, the edges, are single loads and stores.
struct RowSplit { int head, nv, edges; };
template <typename T> __device__ __forceinline__ RowSplit split_row(const T* row, long long cols) {
  constexpr int E = Vec16<T>::kElems;
  RowSplit s;
  const int off = static_cast<int>(reinterpret_cast<uintptr_t>(row) & 15) / static_cast<int>(sizeof(T));
  s.head = static_cast<int>(min(static_cast<long long>(off ? E - off : 0), cols));
  s.nv = static_cast<int>((cols - s.head) / E);
  s.edges = static_cast<int>(cols - static_cast<long long>(s.nv) * E);
  return s;
}
// column of edge element i (0 <= i < edges)
template <typename T> __device__ __forceinline__ long long edge_col(const RowSplit& s, int i) {
  return i < s.head ? i : static_cast<long long>(s.nv) * Vec16<T>::kElems + i;
}

// exp(x) for the sums and results of rows of type T: 16-bit outputs round away far more than the approximate
// exponential loses (the difference to the maximum is taken first, so it is exact near the maximum whatever the
// magnitude); fp32 outputs need expf
template <typename T> __device__ __forceinline__ float row_exp(float d) {
  if constexpr (sizeof(T) == 2) return fast_exp2(d * 1.4426950408889634f);
  else return expf(d);
}

// maximum of a 16-byte piece (16-bit values: exact in 16 bits, one packed instruction per two elements)
template <typename T> __device__ __forceinline__ float piece_max(const uint4& u) {
  if constexpr (sizeof(T) == 2) {
    using T2 = typename std::conditional<std::is_same<T, __half>::value, __half2, __nv_bfloat162>::type;
    const T2 a = __hmax2(*reinterpret_cast<const T2*>(&u.x), *reinterpret_cast<const T2*>(&u.y));
    const T2 b = __hmax2(*reinterpret_cast<const T2*>(&u.z), *reinterpret_cast<const T2*>(&u.w));
    const T2 c = __hmax2(a, b);
    float f[2];
    word_to_floats<T>(*reinterpret_cast<const uint32_t*>(&c), f);
    return fmaxf(f[0], f[1]);
  } else {
    return fmaxf(fmaxf(__uint_as_float(u.x), __uint_as_float(u.y)), fmaxf(__uint_as_float(u.z), __uint_as_float(u.w)));
  }
}

// Sum of exp(x - m) over a piece; the difference d = x - m first (exact near the maximum whatever the magnitude), two
// elements per instruction where the hardware packs them.
//   16-bit types: ex2.approx(d log2e).  The product's rounding puts |d| 2^-24 on a term beside the 2^-22 of ex2.approx:
//     nothing next to the 2^-12 and 2^-9 to which the results are rounded.
//   RESIDUAL (fp32): that |d| 2^-24 would show in a row whose elements lie at one distance from its maximum.  With t = d log2e as it
//     was rounded, exp(d) = 2^t e^c for c = d - t ln2.  Two FMAs give c (the residual of a rounded product, Dekker 1971), and
//     e^c = 1 + c to 2^-39 while a term is above 2^-24 of the largest (|c| < 2^-19): every term that counts is within
//     ex2.approx's 2^-22.  d is held at -200 (the term is 0 from -104 on), so that -inf leaves no NaN in c; a NaN stays
//     one.  Log-sum of rows of 512, 4 096 and 16 384 elements at one distance of 5.6 to 8.5, rms against 64 bits: 1.2, 1.2
//     and 1.0e-7; with the bare ex2.approx 2.2e-7 each, with expf 1.0e-7.  expf took 262 us where this takes 252 on 16 276
//     rows of 12 288.
//   The ring takes the bare ex2.approx for fp32 too: d is the distance to the thread's own maximum there, so that equal
//     elements add 1 each and distant ones little, and the rounding of the sums is what is left.  Rows of 16 384 to 131 072
//     elements, a 32nd of them 0, the others at one distance of 5.7 to 8.5: log-sum 1.5e-7 to 2.9e-7 rms with and without
//     the residual (3e-7 to 6e-7 in the element-wise kernels that summed expf); 2 000 x 50 001 softmax 143 us with, 137 without.
// KEEP (fp32 softmax): the terms are the results, they come from expf and replace the elements.
template <typename T, bool KEEP, bool RESIDUAL = sizeof(T) == 4>
__device__ __forceinline__ float piece_exp_sum(uint4& u, float m) {
  uint32_t w[4] = {u.x, u.y, u.z, u.w};
  if constexpr (KEEP) {
    float s[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      s[q] = expf(__uint_as_float(w[q]) - m);
      w[q] = __float_as_uint(s[q]);
    }
    u = make_uint4(w[0], w[1], w[2], w[3]);
    return (s[0] + s[1]) + (s[2] + s[3]);
  } else if constexpr (RESIDUAL) {
    const uint64_t nm = ptx::pack_f2(-m, -m), log2e = ptx::pack_f2(1.4426950408889634f, 1.4426950408889634f);
    constexpr float kLn2 = 0.6931471805599453f, kLn2Rest = static_cast<float>(0.6931471805599453 - static_cast<double>(kLn2));
    const uint64_t ln2 = ptx::pack_f2(-kLn2, -kLn2), ln2_rest = ptx::pack_f2(-kLn2Rest, -kLn2Rest);
    uint64_t sum = ptx::pack_f2(0.f, 0.f);
#pragma unroll
    for (int q = 0; q < 4; q += 2) {
      float a, b;
      ptx::unpack_f2(ptx::add_f2(ptx::pack_f2(__uint_as_float(w[q]), __uint_as_float(w[q + 1])), nm), a, b);
      const uint64_t d = ptx::pack_f2(ptx::max_nan(a, -200.f), ptx::max_nan(b, -200.f));
      const uint64_t t = ptx::mul_f2(d, log2e);
      const uint64_t c = ptx::fma_f2(t, ln2_rest, ptx::fma_f2(t, ln2, d));
      ptx::unpack_f2(t, a, b);
      const uint64_t y = ptx::pack_f2(fast_exp2(a), fast_exp2(b));
      sum = ptx::fma_f2(y, c, ptx::add_f2(sum, y));
    }
    float s0, s1;
    ptx::unpack_f2(sum, s0, s1);
    return s0 + s1;
  } else {
    const uint64_t nm = ptx::pack_f2(-m, -m);
    constexpr float kLog2e = 1.4426950408889634f;
    float s0 = 0.f, s1 = 0.f;
#pragma unroll
    for (int q = 0; q < 4; q += sizeof(T) / 2) {
      float f[2] = {__uint_as_float(w[q]), __uint_as_float(w[q | 1])};
      if constexpr (sizeof(T) == 2) word_to_floats<T>(w[q], f);
      float a, b;
      ptx::unpack_f2(ptx::add_f2(ptx::pack_f2(f[0], f[1]), nm), a, b);
      s0 += fast_exp2(a * kLog2e);
      s1 += fast_exp2(b * kLog2e);
    }
    return s0 + s1;
  }
}

// What the store pass needs of a row: its maximum and log(sum) (log-softmax), 1 / sum (fp32 softmax) or -log2(sum)
// (16-bit softmax: exp(x - m) / l = exp2((x - m) log2e - log2 l), the division folded into the exponent).  A row of
// -inf only has m = -inf, and -inf - -inf makes every output NaN, like the sum over no terms it stands for.
template <typename T, bool LOG> __device__ __forceinline__ float row_constant(float l) {
  if constexpr (LOG) return logf(l);
  else if constexpr (sizeof(T) == 2) return -__log2f(l);
  else return 1.f / l;
}
// KEPT: x is exp(x - m) already (fp32 softmax of rows in registers)
template <typename T, bool LOG, bool KEPT> __device__ __forceinline__ float row_value(float x, float m, float k) {
  if constexpr (KEPT) return x * k;
  else if constexpr (LOG) return (x - m) - k;
  else if constexpr (sizeof(T) == 2) return fast_exp2(fmaf(x - m, 1.4426950408889634f, k));
  else return expf(x - m) * k;
}
template <typename T, bool LOG, bool KEPT> __device__ __forceinline__ uint4 piece_values(const uint4& u, float m, float k) {
  constexpr int W = Vec16<T>::kElems / 4;
  uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    float f[W];
    word_to_floats<T>(w[q], f);
#pragma unroll
    for (int e = 0; e < W; ++e) f[e] = row_value<T, LOG, KEPT>(f[e], m, k);
    w[q] = floats_to_word<T>(f);
  }
  return make_uint4(w[0], w[1], w[2], w[3]);
}

// ---------------------------------------------------------------------------
// short rows: a warp per row, the row's 16-byte pieces in the warp's registers (VPT per lane), no barrier of any kind.
// Bound by HBM, below it by the launch.  A CTA per row spent most of a short row in its two block reductions, and a row
// whose length is not a multiple of 16 bytes went through single-element copies: 65 536 x 128 bf16 25.0 -> 14.9 us (no
// two rows' loads overlapped before), 30 001 x 2 047 bf16 139 -> 38 us (0.98 of the copy bandwidth), 64 x 2 048 (a
// launch) 4.2 -> 2.5 us.
// ---------------------------------------------------------------------------
// Longest row: eight pieces per lane (16-bit), six (fp32, where one warp is long about a row: 195 312 x 1 024
// 263 us, with two warps per row 237); beyond, a CTA's registers were faster.
template <typename T> constexpr int kWarpPieces = 32 * (sizeof(T) == 4 ? 6 : 8);
constexpr int kWarpRows = 4;   // warps per CTA
template <typename T, bool LOG, int VPT>
__global__ void __launch_bounds__(kWarpRows * 32) softmax_warp_kernel(const T* x, T* out, long long rows, long long cols) {
  constexpr bool KEEP = sizeof(T) == 4 && !LOG;
  const int lane = threadIdx.x & 31;
  ptx::grid_dep_wait();
  ptx::grid_dep_launch_dependents();
  for (long long r = static_cast<long long>(blockIdx.x) * kWarpRows + (threadIdx.x >> 5); r < rows;
       r += static_cast<long long>(gridDim.x) * kWarpRows) {
    const T* src = x + r * cols;
    T* dst = out + r * cols;
    const RowSplit sp = split_row(src, cols);
    const uint4* s4 = reinterpret_cast<const uint4*>(src + sp.head);
    uint4* d4 = reinterpret_cast<uint4*>(dst + sp.head);
    uint4 u[VPT];
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (lane + 32 * k < sp.nv) u[k] = s4[lane + 32 * k];
    float edge = -INFINITY;
    if (lane < sp.edges) edge = ElemTraits<T>::to_float(src[edge_col<T>(sp, lane)]);
    float m = edge;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (lane + 32 * k < sp.nv) m = fmaxf(m, piece_max<T>(u[k]));
    m = warp_max(m);
    float s = lane < sp.edges ? row_exp<T>(edge - m) : 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (lane + 32 * k < sp.nv) s += piece_exp_sum<T, KEEP>(u[k], m);
    const float c = row_constant<T, LOG>(warp_sum(s));
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (lane + 32 * k < sp.nv) d4[lane + 32 * k] = piece_values<T, LOG, KEEP>(u[k], m, c);
    if (lane < sp.edges) dst[edge_col<T>(sp, lane)] = ElemTraits<T>::from_float(row_value<T, LOG, false>(edge, m, c));
  }
}

// ---------------------------------------------------------------------------
// medium rows: a CTA per row, thread t holds the four 16-byte pieces t, t + blockDim, ...: as many threads as the row
// needs, and 32 registers, so that 2 048 threads share an SM and up to 128 KiB of rows are in flight on it.  Bound by
// HBM.  With power-of-two CTAs a quarter of the threads idled on average: 20 000 x 3 001 bf16 161.7 -> 41.3 us, 5 000 x
// 8 200 fp32 80.7 -> 57.9 us, 16 384 x 16 384 bf16 200 -> 170 us (0.96 of the copy bandwidth).
// fp32: places behind the row hold -inf and every thread sums its four pieces without asking, so that their exponentials
// overlap; 16-bit rows have no registers left for that and ask (with spills: +6 %).  WHOLE: rows that are whole pieces have
// no edges.  Both together, log-softmax: 12 207 x 16 384 fp32 262 -> 244 us, 24 414 x 16 384 bf16 264 -> 241 (softmax).
// ---------------------------------------------------------------------------
template <typename T, bool LOG, bool WHOLE>
__global__ void __launch_bounds__(1024, 2) softmax_reg_kernel(const T* x, T* out, long long rows, long long cols) {
  constexpr bool KEEP = sizeof(T) == 4 && !LOG;
  constexpr bool PAD = sizeof(T) == 4;
  constexpr int VPT = 4;
  __shared__ float scratch[2][32];
  ptx::grid_dep_wait();
  ptx::grid_dep_launch_dependents();
  const int t = threadIdx.x;
  for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
    const T* src = x + r * cols;
    T* dst = out + r * cols;
    const RowSplit sp = WHOLE ? RowSplit{0, static_cast<int>(cols / Vec16<T>::kElems), 0} : split_row(src, cols);
    const uint4* s4 = reinterpret_cast<const uint4*>(src + sp.head);
    uint4* d4 = reinterpret_cast<uint4*>(dst + sp.head);
    uint4 u[VPT];
#pragma unroll
    for (int k = 0; k < VPT; ++k) {
      if (t + k * static_cast<int>(blockDim.x) < sp.nv) u[k] = s4[t + k * static_cast<int>(blockDim.x)];
      else if (PAD) u[k] = make_uint4(kNegInfWord<T>, kNegInfWord<T>, kNegInfWord<T>, kNegInfWord<T>);
    }
    float edge = -INFINITY;
    if (!WHOLE && t < sp.edges) edge = ElemTraits<T>::to_float(src[edge_col<T>(sp, t)]);
    float m = edge;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (PAD || t + k * static_cast<int>(blockDim.x) < sp.nv) m = fmaxf(m, piece_max<T>(u[k]));
    m = block_max_nolead(m, scratch[0]);   // (each scratch is rewritten only after the other's barrier)
    float s = !WHOLE && t < sp.edges ? row_exp<T>(edge - m) : 0.f;
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (PAD || t + k * static_cast<int>(blockDim.x) < sp.nv) s += piece_exp_sum<T, KEEP>(u[k], m);
    const float c = row_constant<T, LOG>(block_sum_nolead(s, scratch[1]));
#pragma unroll
    for (int k = 0; k < VPT; ++k)
      if (t + k * static_cast<int>(blockDim.x) < sp.nv) d4[t + k * static_cast<int>(blockDim.x)] = piece_values<T, LOG, KEEP>(u[k], m, c);
    if (!WHOLE && t < sp.edges) dst[edge_col<T>(sp, t)] = ElemTraits<T>::from_float(row_value<T, LOG, false>(edge, m, c));
  }
}

// ---------------------------------------------------------------------------
// one CTA per row, the row in shared memory
// ---------------------------------------------------------------------------
template <typename T, bool LOG>
__global__ void softmax_row_kernel(const T* x, T* out, long long rows, long long cols) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float scratch[32];
  T* row = reinterpret_cast<T*>(smem_raw);
  for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
    const T* src = x + r * cols;
    __syncthreads();               // the previous row has been written out of `row`
    float m = stage_row<T>(src, row, cols);
    m = block_max(m, scratch);     // (its barriers also publish the staged row)
    const float l = block_sum(row_exp_sum<T>(row, cols, m), scratch);
    write_row<T, LOG>(row, out + r * cols, cols, m, final_constant<LOG>(m, l));
  }
}

// ---------------------------------------------------------------------------
// one cluster per row: every CTA stages a slice, (max, sum) pairs meet in distributed shared memory
// ---------------------------------------------------------------------------
template <typename T, bool LOG>
__global__ void softmax_cluster_kernel(const T* x, T* out, long long rows, long long cols,
                                       long long slice) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float scratch[32];
  __shared__ float ml[2];          // this CTA's (max, sum), read by its peers
  cg::cluster_group cluster = cg::this_cluster();
  const unsigned rank = cluster.block_rank(), csize = cluster.num_blocks();
  T* row = reinterpret_cast<T*>(smem_raw);
  const long long c0 = std::min<long long>(cols, slice * rank);
  const long long n = std::min<long long>(cols - c0, slice);
  const long long nclusters = gridDim.x / csize;
  for (long long r = blockIdx.x / csize; r < rows; r += nclusters) {
    const T* src = x + r * cols + c0;
    float m = stage_row<T>(src, row, n);
    m = block_max(m, scratch);
    const float l = block_sum(row_exp_sum<T>(row, n, m), scratch);
    if (threadIdx.x == 0) { ml[0] = m; ml[1] = l; }
    cluster.sync();                // every CTA's pair is in place
    float gm = -INFINITY, gl = 0.f;
    for (unsigned p = 0; p < csize; ++p) {
      const float* peer = cluster.map_shared_rank(ml, p);
      merge_ml(gm, gl, peer[0], peer[1]);
    }
    cluster.sync();                // all pairs have been read: they may be overwritten for the next row
    write_row<T, LOG>(row, out + r * cols + c0, n, gm, final_constant<LOG>(gm, gl));
    __syncthreads();               // `row` is free again
  }
}

// ---------------------------------------------------------------------------
// Rows of which two fit an SM: the CTA keeps as many rows as fit in shared memory; the bulk copies of the next rows run
// while one is reduced and written, all 1 024 threads on the same row.  Bound by HBM.  Against the ring below it has no
// slots, so that nothing is lost to a last chunk that is not full, and more threads for two passes of exponentials;
// takes_pipe says where it is the faster one.  8 000 x 50 000 bf16 314 -> 287 us, 9 765 x 40 960 302 -> 272 (log-softmax),
// 10 526 x 19 000 fp32 287 -> 252.
// ---------------------------------------------------------------------------
constexpr int kPipeThreads = 1024;
constexpr int kPipeBytes = 108 * 1024;      // longest row (two are staged)
constexpr int kPipeStages = 3;              // shorter ones, from 64 KiB on

template <typename T, bool LOG>
__global__ void __launch_bounds__(kPipeThreads, 1)
softmax_pipe_kernel(const T* x, T* out, long long rows, long long cols, int stages /* rows staged, 2..kPipeStages */) {
  constexpr bool KEEP = sizeof(T) == 4 && !LOG;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float scratch[2][32];
  __shared__ __align__(8) uint64_t full[kPipeStages];
  uint4* const base = reinterpret_cast<uint4*>(smem_raw);
  const int tid = threadIdx.x;
  const int n = static_cast<int>(cols / Vec16<T>::kElems);
  if (tid == 0) {
    for (int i = 0; i < kPipeStages; ++i) ptx::mbar_init(smem_u32(&full[i]), 1);
    ptx::mbar_fence_init();
    // The first row starts for L2 before the wait for the launches in front: where it lies is an argument, and bringing lines into L2 reads
    // nothing that a later write would not replace there.  (Here and in the ring: 148 x 27 648 bf16 6.5 -> 4.5 us, 809 x 22 336 fp16 16.9
    // -> 16.4, 8 000 x 20 000 fp32 227 -> 223, 2 450 x 81 603 285 -> 278.  In the kernels with a row in registers, whose later CTAs would do
    // it too, 4 to 8 % slower.)
    ptx::bulk_prefetch_l2(x + blockIdx.x * cols, static_cast<uint32_t>(n) * 16u);
  }
  __syncthreads();
  ptx::grid_dep_wait();
  ptx::grid_dep_launch_dependents();
  const long long step = gridDim.x;
  auto load = [&](long long r, int stage) {
    ptx::mbar_arrive_expect_tx(smem_u32(&full[stage]), static_cast<uint32_t>(n) * 16u);
    ptx::bulk_load(smem_u32(base + static_cast<size_t>(stage) * n), x + r * cols, static_cast<uint32_t>(n) * 16u,
                   smem_u32(&full[stage]));
  };
  if (tid == 0)
    for (int s = 0; s < stages - 1 && blockIdx.x + s * step < rows; ++s) load(blockIdx.x + s * step, s);
  int stage = 0;
  unsigned phase = 0;
  bool ok = true;                                          // false: a bounded wait ran out, the rows come out as NaN
  for (long long r = blockIdx.x; r < rows; r += step) {
    // refill the stage of the row before: it was read for the last time before the barrier that ended that row
    const long long ahead = r + (stages - 1) * step;
    if (tid == 0 && ahead < rows) {
      ptx::fence_proxy_async_smem();
      load(ahead, stage == 0 ? stages - 1 : stage - 1);
    }
    ok = ptx::mbar_wait(smem_u32(&full[stage]), phase) && ok;
    uint4* const row = base + static_cast<size_t>(stage) * n;
    float m = -INFINITY;
#pragma unroll 2
    for (int i = tid; i < n; i += kPipeThreads) m = fmaxf(m, piece_max<T>(row[i]));
    m = block_max_nolead(m, scratch[0]);                   // (each scratch is rewritten only after the other's barrier)
    float s = 0.f;
#pragma unroll 2
    for (int i = tid; i < n; i += kPipeThreads) {
      uint4 u = row[i];
      s += piece_exp_sum<T, KEEP>(u, m);
      if (KEEP) row[i] = u;
    }
    if (!ok) s = __int_as_float(0x7fc00000);
    const float l = block_sum_nolead(s, scratch[1]);
    const float c = row_constant<T, LOG>(l);
    uint4* const d4 = reinterpret_cast<uint4*>(out + r * cols);
#pragma unroll 2
    for (int i = tid; i < n; i += kPipeThreads) d4[i] = piece_values<T, LOG, KEEP>(row[i], m, c);
    __syncthreads();                                       // the stage may be refilled
    if (++stage == stages) { stage = 0; phase ^= 1u; }
  }
  // (thread 0 gave up: wait, bounded, for the copies in flight before the CTA's memory goes away)
  if (tid == 0 && !ok)
    for (int i = 0; i < stages; ++i)
      for (unsigned parity = 0; parity < 2; ++parity) ptx::mbar_wait(smem_u32(&full[i]), parity);
}

// ---------------------------------------------------------------------------
// long rows: a ring of 32 KiB chunks (24 KiB, see Ring) in shared memory.  A producer warp fills it by bulk copies; the other warps take a
// chunk as soon as it has landed and keep a running (max, sum) per thread (first pass), combine them once per row, and
// go over the chunks again to write the row (second pass), handing each back to the producer, which fills it with the
// next row.  So a row is read once, loads run under both passes, and there is one barrier per row.  A row that is
// longer than the ring, or of which there are too few to keep every SM busy, is shared by a cluster of 2, 4 or 8 CTAs.
// Bound by HBM with a fixed microsecond per row (the reduction, during which nothing is stored).  The chunk is what the
// waits and the loop overhead are spread over: 4 pieces per thread against 2 and 1 gave 135, 150 and 160 us on 2 000 x
// 50 000 fp32; 512 threads against 256 and 384 gave 135, 159 and 140.  Larger clusters than a row needs only cost
// (cluster 2 / 4: 155 / 220 us).  Before (three barriers per row, a slice of the row as one copy, single-element loads
// for odd lengths) and now: 2 000 x 50 001 fp32 282 -> 138 us (0.89 of the copy bandwidth), 1 024 x 131 072 fp32
// 309 -> 198, bf16 151 -> 103, 8 192 x 24 576 fp32 268 -> 249.
// ---------------------------------------------------------------------------
constexpr int kRingThreads = 512;                   // threads that compute (the producer warp comes on top)
constexpr int kRingWarps = kRingThreads / 32;
// PER 16-byte pieces per thread and chunk.  Four; three where that lets the ring hold more rows, because a row's last
// chunk would be nearly empty and still take a slot (12 135 x 32 960 bf16 361 -> 319 us).
template <int PER> struct Ring {
  static constexpr int kChunk = kRingThreads * PER;
  static constexpr int kSlots = PER == 4 ? 7 : 9;          // 224 and 216 KiB
  static int chunks(long long slice) { return static_cast<int>((slice + kChunk - 1) / kChunk); }
};
constexpr int kRingPieces = Ring<4>::kChunk * Ring<4>::kSlots;

// (m, s) <- (m, s) + the elements of a thread's pieces of a chunk; m is the reference of s
template <typename T, int PER> __device__ __forceinline__ void online_add(float& m, float& s, uint4 (&u)[PER]) {
  float mx = piece_max<T>(u[0]);
#pragma unroll
  for (int k = 1; k < PER; ++k) mx = fmaxf(mx, piece_max<T>(u[k]));
  if (mx > m) {
    s = (sizeof(T) == 4 && m == -INFINITY) ? s : s * row_exp<T>(m - mx);   // (m == -inf: s is 0 or NaN and stays that)
    m = mx;
  }
  if (sizeof(T) == 2 || m != -INFINITY) {
    const float ref = sizeof(T) == 2 ? exp_ref(m) : m;
    float t = piece_exp_sum<T, false, false>(u[0], ref);
#pragma unroll
    for (int k = 1; k < PER; ++k) t += piece_exp_sum<T, false, false>(u[k], ref);
    s += t;
  } else {
    // fp32 rows branch where 16-bit ones select the reference (which made those 3 % faster): 6 666 x 30 000 log-softmax took
    // 272 us with the selection, 258 so; 2 000 x 50 001 137 and 135
#pragma unroll
    for (int k = 0; k < PER; ++k) s += piece_exp_sum<T, false, false>(u[k], 0.f);
  }
}

template <typename T, bool LOG, int PER>
__global__ void __launch_bounds__(kRingThreads + 32, 1)
softmax_ring_kernel(const T* x, T* out, long long rows, long long cols, int slice /* pieces of a row per CTA */, int csize) {
  constexpr int kRingPer = PER, kRingChunk = Ring<PER>::kChunk, kRingSlots = Ring<PER>::kSlots;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  __shared__ float2 scratch[2][kRingWarps];
  __shared__ __align__(8) float2 pairs[2][kMaxCluster];    // every CTA's (max, sum) of the even / odd row in work
  __shared__ __align__(8) uint64_t pair_bar[2];            // completes when all pairs of that row have landed
  __shared__ __align__(8) uint64_t full[kRingSlots], empty[kRingSlots];
  uint4* const ring = reinterpret_cast<uint4*>(smem_raw);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int rank = csize > 1 ? static_cast<int>(cg::this_cluster().block_rank()) : 0;
  if (tid == 0) {
    for (int i = 0; i < 2; ++i) ptx::mbar_init(smem_u32(&pair_bar[i]), 1);
    for (int i = 0; i < kRingSlots; ++i) {
      ptx::mbar_init(smem_u32(&full[i]), 1);
      ptx::mbar_init(smem_u32(&empty[i]), kRingWarps);
    }
    ptx::mbar_fence_init();
  }
  const long long row_step = gridDim.x / csize, r0 = blockIdx.x / csize;
  const int first = slice * rank;                          // this CTA's pieces of every row: first .. first + slice - 1
  auto my_pieces = [&](const RowSplit& sp) { return max(0, min(slice, sp.nv - first)); };
  if (tid == 0) {
    const RowSplit sp = split_row(x + r0 * cols, cols);
    const int n = min(my_pieces(sp), kRingSlots * kRingChunk);
    if (n > 0) ptx::bulk_prefetch_l2(reinterpret_cast<const uint4*>(x + r0 * cols + sp.head) + first, static_cast<uint32_t>(n) * 16u);
  }
  if (csize > 1) cg::this_cluster().sync(); else __syncthreads();
  ptx::grid_dep_wait();
  ptx::grid_dep_launch_dependents();

  if (warp == kRingWarps) {
    // ------------------------------ producer ------------------------------
    if (lane == 0) {
      int slot = 0;
      unsigned phase = 1;                                  // parity of the wait for a free slot (the first round is free)
      long long issued = 0;
      bool ok = true;
      for (long long r = r0; ok && r < rows; r += row_step) {
        const T* src = x + r * cols;
        const RowSplit sp = split_row(src, cols);
        const uint4* s4 = reinterpret_cast<const uint4*>(src + sp.head) + first;
        const int n = my_pieces(sp);
        for (int p = 0; p < n; p += kRingChunk) {
          if (issued >= kRingSlots) ok = ptx::mbar_wait(smem_u32(&empty[slot]), phase);
          if (!ok) break;
          const uint32_t bytes = static_cast<uint32_t>(min(kRingChunk, n - p)) * 16u;
          ptx::mbar_arrive_expect_tx(smem_u32(&full[slot]), bytes);
          ptx::bulk_load(smem_u32(ring + slot * kRingChunk), s4 + p, bytes, smem_u32(&full[slot]));
          ++issued;
          if (++slot == kRingSlots) { slot = 0; phase ^= 1u; }
        }
      }
      // (a consumer gave up: wait, bounded, for the copies in flight before the CTA's memory goes away)
      if (!ok)
        for (int i = 0; i < kRingSlots; ++i) {
          const unsigned done = static_cast<unsigned>((issued - 1 - i) / kRingSlots);
          if (issued - 1 - i >= 0) ptx::mbar_wait(smem_u32(&full[(issued - 1 - i) % kRingSlots]), done & 1u);
        }
    }
    return;
  }
  // ------------------------------ consumers ------------------------------
  int slot = 0;
  unsigned phase = 0, iter = 0;
  bool ok = true;                                          // false: a bounded wait ran out, the rows come out as NaN
  for (long long r = r0; r < rows; r += row_step, ++iter) {
    const T* src = x + r * cols;
    T* dst = out + r * cols;
    const RowSplit sp = split_row(src, cols);
    const int n = my_pieces(sp);
    const int edges = rank == 0 ? sp.edges : 0;
    float edge = -INFINITY;
    if (tid < edges) edge = ElemTraits<T>::to_float(src[edge_col<T>(sp, tid)]);
    const int slot0 = slot;
    float m = -INFINITY, s = 0.f;
    for (int p = 0; p < n; p += kRingChunk) {
      if (ok) ok = ptx::mbar_wait(smem_u32(&full[slot]), phase);
      const uint4* c4 = ring + slot * kRingChunk + tid;
      const int left = n - p - tid;
      uint4 u[kRingPer];
      if (n - p >= kRingChunk) {
#pragma unroll
        for (int k = 0; k < kRingPer; ++k) u[k] = c4[k * kRingThreads];
      } else {
        constexpr uint32_t w = kNegInfWord<T>;
#pragma unroll
        for (int k = 0; k < kRingPer; ++k) u[k] = k * kRingThreads < left ? c4[k * kRingThreads] : make_uint4(w, w, w, w);
      }
      online_add<T, PER>(m, s, u);
      if (++slot == kRingSlots) { slot = 0; phase ^= 1u; }
    }
    if (tid < edges) {
      const float mx = fmaxf(m, edge), ref = exp_ref(mx);
      s = s * row_exp<T>(m - ref) + row_exp<T>(edge - ref);
      m = mx;
    }
    if (!ok) { m = 0.f; s = __int_as_float(0x7fc00000); }
    // the CTA's (max, sum): warps through shuffles, warps of the CTA through shared memory
    float mw = warp_max(m);
    float sw = warp_sum(s * row_exp<T>(m - exp_ref(mw)));
    float2* sc = scratch[iter & 1u];
    if (lane == 0) sc[warp] = make_float2(mw, sw);
    ptx::named_bar_sync(1, kRingThreads);
    const float2 pw = lane < kRingWarps ? sc[lane] : make_float2(-INFINITY, 0.f);
    float gm = warp_max(pw.x);
    float gl = warp_sum(pw.y * row_exp<T>(pw.x - exp_ref(gm)));
    if (csize > 1) {
      // Thread 0 posts the CTA's pair into every CTA's `pairs` (its own included) with asynchronous remote stores that
      // count bytes on the receiver's barrier: no cluster-wide barrier, no fence that would wait for the previous
      // row's global stores.  Slot reuse is safe: a peer can send row r + 2 only after it has seen this CTA's pair
      // of row r + 1, which thread 0 sends after all threads here have read the pairs of row r (the barrier above).
      // A CTA whose own wait for a chunk ran out still waits for its peers' pairs: it would be done with its rows first
      // and leave while they post into its memory.  Such a wait happens once per CTA (the chunks after it are not waited
      // for), so that a peer is late by one limit at most, and four are allowed here.
      const unsigned parity = iter & 1u;
      const uint32_t bar = smem_u32(&pair_bar[parity]);
      if (tid == 0) {
        ptx::mbar_arrive_expect_tx(bar, static_cast<uint32_t>(csize) * 8u);
        const uint32_t to = smem_u32(&pairs[parity][rank]);
        for (int p = 0; p < csize; ++p) ptx::st_async_pair(to, bar, p, gm, gl);
      }
      ok = ptx::mbar_wait_limit(bar, (iter >> 1) & 1u, 4 * ptx::kWaitTries) && ok;
      gm = -INFINITY;
      for (int p = 0; p < csize; ++p) gm = fmaxf(gm, pairs[parity][p].x);
      gl = 0.f;
      for (int p = 0; p < csize; ++p) {
        const float2 q = pairs[parity][p];
        gl += q.y * row_exp<T>(q.x - exp_ref(gm));
      }
      if (!ok) gl = __int_as_float(0x7fc00000);
    }
    const float c = row_constant<T, LOG>(gl);
    uint4* d4 = reinterpret_cast<uint4*>(dst + sp.head) + first;
    int back = slot0;
    for (int p = 0; p < n; p += kRingChunk) {
      const uint4* c4 = ring + back * kRingChunk + tid;
      uint4* o4 = d4 + p + tid;
      const int left = n - p - tid;
      uint4 u[kRingPer];
#pragma unroll
      for (int k = 0; k < kRingPer; ++k)
        if (k * kRingThreads < left) u[k] = c4[k * kRingThreads];
      __syncwarp();
      if (lane == 0) ptx::mbar_arrive(smem_u32(&empty[back]));
#pragma unroll
      for (int k = 0; k < kRingPer; ++k)
        if (k * kRingThreads < left) o4[k * kRingThreads] = piece_values<T, LOG, false>(u[k], gm, c);
      if (++back == kRingSlots) back = 0;
    }
    if (tid < edges) dst[edge_col<T>(sp, tid)] = ElemTraits<T>::from_float(row_value<T, LOG, false>(edge, gm, c));
  }
}

// ---------------------------------------------------------------------------
// rows that do not fit a cluster: online (max, sum), then a second read
// ---------------------------------------------------------------------------
template <typename T, bool LOG>
__global__ void softmax_stream_kernel(const T* x, T* out, long long rows, long long cols) {
  __shared__ float scratch[32];
  for (long long r = blockIdx.x; r < rows; r += gridDim.x) {
    const T* src = x + r * cols;
    T* dst = out + r * cols;
    float m = -INFINITY, l = 0.f;
    for (long long i = threadIdx.x; i < cols; i += blockDim.x) {
      const float v = ElemTraits<T>::to_float(src[i]);
      if (v > m) { l *= expf(m - v); m = v; }
      l += expf(v - exp_ref(m));
    }
    const float gm = block_max(m, scratch);
    const float gl = block_sum(l * expf(m - exp_ref(gm)), scratch);
    const float k = final_constant<LOG>(gm, gl);
    for (long long i = threadIdx.x; i < cols; i += blockDim.x)
      dst[i] = finish<T, LOG>(ElemTraits<T>::to_float(src[i]), gm, k);
  }
}

template <typename K>
int set_smem_limit(K kernel, size_t bytes) {
  return ensure_dynamic_smem(reinterpret_cast<const void*>(kernel), bytes);
}

// CTAs that share a row of `nv` pieces in the ring kernel: as few as hold it, more when there are so few rows that SMs
// would stay idle (as long as a CTA still has two chunks of the row).
inline int ring_cluster(long long rows, long long nv, int sm_count) {
  int csize = 1;
  while ((nv + csize - 1) / csize > kRingPieces) csize *= 2;
  while (csize < kMaxCluster && rows * csize * 2 <= sm_count && nv > 4LL * csize * Ring<4>::kChunk) csize *= 2;
  return csize;
}

// Three pieces per thread and chunk instead of four (see Ring).
inline bool ring_of_three(long long slice) {
  const int c4 = Ring<4>::chunks(static_cast<int>(slice)), c3 = Ring<3>::chunks(static_cast<int>(slice));
  return c3 <= Ring<3>::kSlots && Ring<3>::kSlots * c4 * 5 >= Ring<4>::kSlots * c3 * 6;
}

// Rows of `nv` whole pieces, beyond what registers hold, that softmax_pipe_kernel takes: those of which two fit, but for the
// 16-bit ones of which two fit the ring as well and fill most of its slots; there the ring's second pass over one row runs
// beside the first pass over the next.  The line, measured with bf16, ring / here (us): softmax 34 000 columns (0.92 full)
// 302 / 306, 42 000 (0.85) 295 / 305, 40 960 (0.83) 298 / 283; log-softmax 36 000 (0.98) 293 / 297, 44 000 (0.90) 287 / 278;
// one and a bit rows in the ring, 50 000 and 55 296: 314 / 287 and 286 / 279.  fp32 at 18 000 (0.98): 276 / 258; but one or
// two rows per SM of fp32 softmax, where the ring's first pass need not wait for the whole row (148 x 27 648: 7.0 / 7.2).
template <typename T, bool LOG> bool takes_pipe(long long rows, long long nv, int sm_count) {
  if (nv * 16 > kPipeBytes) return false;
  if (sizeof(T) == 4) return LOG || rows > 2LL * sm_count;
  const bool three = ring_of_three(nv);
  const int chunk = three ? Ring<3>::kChunk : Ring<4>::kChunk, slots = three ? Ring<3>::kSlots : Ring<4>::kSlots;
  const int chunks = static_cast<int>((nv + chunk - 1) / chunk);
  return 2 * chunks > slots || 100 * nv < (LOG ? 92LL : 85LL) * chunks * chunk;
}

// Rows whose 16-byte pieces can be copied as they are (x and out misaligned by the same amount).
template <typename T, bool LOG>
int launch_pieces(const b200attn_softmax_args_t& a, int sm_count, cudaStream_t stream) {
  const T* x = static_cast<const T*>(a.x);
  T* out = static_cast<T*>(a.out);
  const long long rows = a.rows, cols = a.cols;
  constexpr int E = Vec16<T>::kElems;
  const long long nv = cols / E;
  const bool whole = cols % E == 0 && (reinterpret_cast<uintptr_t>(x) & 15) == 0;   // every row is whole pieces
  cudaError_t e = cudaSuccess;
  if (nv <= kWarpPieces<T>) {
    int vpt = 1;
    while (32 * vpt < nv) vpt *= 2;
    const long long max_grid = static_cast<long long>(sm_count) * (2048 / (kWarpRows * 32)) * 4;
    const dim3 grid(static_cast<unsigned>(std::min<long long>((rows + kWarpRows - 1) / kWarpRows, max_grid)));
    switch (vpt) {
      case 1: e = launch_dependent(softmax_warp_kernel<T, LOG, 1>, grid, kWarpRows * 32, 0, stream, 1, x, out, rows, cols); break;
      case 2: e = launch_dependent(softmax_warp_kernel<T, LOG, 2>, grid, kWarpRows * 32, 0, stream, 1, x, out, rows, cols); break;
      case 4: e = launch_dependent(softmax_warp_kernel<T, LOG, 4>, grid, kWarpRows * 32, 0, stream, 1, x, out, rows, cols); break;
      default: e = launch_dependent(softmax_warp_kernel<T, LOG, 8>, grid, kWarpRows * 32, 0, stream, 1, x, out, rows, cols); break;
    }
  } else if (nv <= 4 * 1024) {
    // four pieces per thread whatever the length; rows are dealt in small portions (16 resident grids' worth of CTAs),
    // which measured 2 - 7 % above 4 and keeps CTAs from running in step
    const int threads = static_cast<int>(((nv + 3) / 4 + 31) / 32 * 32);
    const long long max_grid = static_cast<long long>(sm_count) * (2048 / threads) * 16;
    const dim3 grid(static_cast<unsigned>(std::min<long long>(rows, max_grid)));
    e = launch_dependent(whole ? softmax_reg_kernel<T, LOG, true> : softmax_reg_kernel<T, LOG, false>, grid, threads, 0, stream,
                         1, x, out, rows, cols);
  } else if (whole && takes_pipe<T, LOG>(rows, nv, sm_count)) {
    const int stages = std::max(2, std::min(kPipeStages, 2 * kPipeBytes / static_cast<int>(nv * 16)));
    const size_t smem = static_cast<size_t>(nv) * 16 * stages;
    const int rc = set_smem_limit(softmax_pipe_kernel<T, LOG>, 2 * kPipeBytes);
    if (rc) return rc;
    e = launch_dependent(softmax_pipe_kernel<T, LOG>, dim3(static_cast<unsigned>(std::min<long long>(rows, sm_count))), kPipeThreads,
                         smem, stream, 1, x, out, rows, cols, stages);
  } else {
    const int csize = ring_cluster(rows, nv, sm_count);
    const int slice = static_cast<int>((nv + csize - 1) / csize);
    const size_t smem = static_cast<size_t>(kRingPieces) * 16;
    auto kernel = ring_of_three(slice) ? softmax_ring_kernel<T, LOG, 3> : softmax_ring_kernel<T, LOG, 4>;
    int rc = set_smem_limit(kernel, smem);
    if (rc) return rc;
    // one CTA per SM; how many clusters of a size the GPU holds at once is asked of the driver once (the answer depends
    // on the device model only, and only B200 is accepted)
    static std::atomic<int> resident[4];
    const int log_c = csize == 1 ? 0 : (csize == 2 ? 1 : (csize == 4 ? 2 : 3));
    int n = resident[log_c].load(std::memory_order_relaxed);
    if (n == 0) {
      n = sm_count;
      if (csize > 1) {
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(sm_count / csize * csize), 1, 1);
        cfg.blockDim = dim3(kRingThreads + 32, 1, 1);
        cfg.dynamicSmemBytes = smem;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = csize;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        cfg.attrs = attr;
        cfg.numAttrs = 1;
        e = cudaOccupancyMaxActiveClusters(&n, kernel, &cfg);
        if (e != cudaSuccess) return cuda_fail(e, "cudaOccupancyMaxActiveClusters(softmax)");
        n = std::max(1, n);
      }
      resident[log_c].store(n, std::memory_order_relaxed);
    }
    const long long clusters = std::min<long long>(rows, n);
    e = launch_dependent(kernel, dim3(static_cast<unsigned>(clusters * csize)), kRingThreads + 32, smem, stream,
                         static_cast<unsigned>(csize), x, out, rows, cols, slice, csize);
  }
  if (e != cudaSuccess) return cuda_fail(e, "softmax kernel launch");
  return B200ATTN_OK;
}

// Everything else: rows that x and out place differently on the 16-byte grid, and rows beyond what a cluster's ring holds.
template <typename T, bool LOG>
int launch_elements(const b200attn_softmax_args_t& a, int sm_count, cudaStream_t stream) {
  const T* x = static_cast<const T*>(a.x);
  T* out = static_cast<T*>(a.out);
  const long long rows = a.rows, cols = a.cols;
  const size_t row_bytes = static_cast<size_t>(cols) * sizeof(T);
  if (row_bytes <= static_cast<size_t>(kRowSmemBytes)) {
    int threads = 64;
    while (threads < 1024 && static_cast<long long>(threads) * 8 < cols) threads *= 2;
    int rc = set_smem_limit(softmax_row_kernel<T, LOG>, row_bytes);
    if (rc) return rc;
    const long long max_grid = static_cast<long long>(sm_count) * 32;
    const unsigned grid = static_cast<unsigned>(std::min<long long>(rows, max_grid));
    softmax_row_kernel<T, LOG><<<grid, threads, row_bytes, stream>>>(x, out, rows, cols);
  } else if (row_bytes <= static_cast<size_t>(kRowSmemBytes) * kMaxCluster) {
    // more CTAs per row while a slice stays above 64 KiB (fp32) / 128 KiB (16-bit), measured: smaller CTAs share an SM
    // and one's loads overlap another's stores
    int csize = 2;
    while (csize < kMaxCluster && (static_cast<size_t>(kRowSmemBytes) * csize < row_bytes || row_bytes / csize > (sizeof(T) == 4 ? 64 : 128) * 1024)) csize *= 2;
    const long long slice = (cols + csize - 1) / csize;
    const size_t smem = static_cast<size_t>(slice) * sizeof(T);
    int rc = set_smem_limit(softmax_cluster_kernel<T, LOG>, smem);
    if (rc) return rc;
    const int per_sm = std::max<int>(1, std::min<int>(2, static_cast<int>((220 * 1024) / (smem + 1024))));
    const long long clusters = std::min<long long>(rows, std::max(1, sm_count * per_sm / csize));
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(clusters * csize), 1, 1);
    cfg.blockDim = dim3(1024, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = csize;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    cudaError_t e = cudaLaunchKernelEx(&cfg, softmax_cluster_kernel<T, LOG>, x, out, rows, cols, slice);
    if (e != cudaSuccess) return cuda_fail(e, "softmax cluster kernel launch");
  } else {
    const unsigned grid = static_cast<unsigned>(std::min<long long>(rows, static_cast<long long>(sm_count) * 2));
    softmax_stream_kernel<T, LOG><<<grid, 1024, 0, stream>>>(x, out, rows, cols);
  }
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) return cuda_fail(e, "softmax kernel launch");
  return B200ATTN_OK;
}

template <typename T>
int launch_dtype(const b200attn_softmax_args_t& a, int sm_count, cudaStream_t stream) {
  const uintptr_t xa = reinterpret_cast<uintptr_t>(a.x), oa = reinterpret_cast<uintptr_t>(a.out);
  const bool pieces = (xa & 15) == (oa & 15) && xa % sizeof(T) == 0 &&
                      a.cols / Vec16<T>::kElems <= static_cast<long long>(kRingPieces) * kMaxCluster;
  if (a.log_softmax) return pieces ? launch_pieces<T, true>(a, sm_count, stream) : launch_elements<T, true>(a, sm_count, stream);
  return pieces ? launch_pieces<T, false>(a, sm_count, stream) : launch_elements<T, false>(a, sm_count, stream);
}

}  // namespace

int launch_softmax(const b200attn_softmax_args_t& a, int sm_count, cudaStream_t stream) {
  switch (a.dtype) {
    case B200ATTN_F16: return launch_dtype<__half>(a, sm_count, stream);
    case B200ATTN_BF16: return launch_dtype<__nv_bfloat16>(a, sm_count, stream);
    case B200ATTN_F32: return launch_dtype<float>(a, sm_count, stream);
    default: set_error("softmax: unknown dtype %d", a.dtype); return B200ATTN_E_UNSUPPORTED;
  }
}

}  // namespace b200attn
