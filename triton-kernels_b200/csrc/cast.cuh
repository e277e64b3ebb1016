// fp32 q, k and v rounded to fp16 copies in the workspace, for the calls that multiply fp32 inputs in 16 bits (the
// reference does the same cast in registers, kernels/attention.py:547,572,594,614).
#pragma once

#include <algorithm>

#include "common.cuh"
#include "launch.cuh"
#include "sm100_ptx.cuh"

namespace b200attn {

struct CastJob {
  const float4* src[3];
  uint2* dst[3];
  long long n4[3];     // float4 pieces (every tensor here is a whole number of head_dim rows)
};

// One launch for the three tensors, blockIdx.y names the tensor: HBM-bound when they are large, and three launches of
// their own were most of the time of a short call.
constexpr int kCastLoads = 4;      // pieces that a thread has on the way
static __global__ void __launch_bounds__(256) cast_f32_to_f16_kernel(const CastJob job) {
  ptx::grid_dep_launch_dependents();
  ptx::grid_dep_wait();
  const int t = blockIdx.y;
  const float4* src = t == 0 ? job.src[0] : (t == 1 ? job.src[1] : job.src[2]);
  uint2* dst = t == 0 ? job.dst[0] : (t == 1 ? job.dst[1] : job.dst[2]);
  const long long n4 = t == 0 ? job.n4[0] : (t == 1 ? job.n4[1] : job.n4[2]);
  // (four loads in flight per thread: one left an SM with 32 KB on the way; 4 x 4 096 tokens, 8 heads, D 64: 125.7 -> 122.4 us
  // a call)
  const long long step = static_cast<long long>(gridDim.x) * blockDim.x;
  for (long long i = blockIdx.x * static_cast<long long>(blockDim.x) + threadIdx.x; i < n4; i += kCastLoads * step) {
    float4 x[kCastLoads];
#pragma unroll
    for (int j = 0; j < kCastLoads; ++j)
      if (i + j * step < n4) x[j] = __ldcg(src + i + j * step);
#pragma unroll
    for (int j = 0; j < kCastLoads; ++j)
      if (i + j * step < n4) dst[i + j * step] = make_uint2(ElemTraits<__half>::pack2(x[j].x, x[j].y), ElemTraits<__half>::pack2(x[j].z, x[j].w));
  }
}

inline cudaError_t launch_cast(const CastJob& job, int sm_count, cudaStream_t stream) {
  const long long most = std::max(job.n4[0], std::max(job.n4[1], job.n4[2]));
  if (most == 0) return cudaSuccess;
  // (a thread's pieces are counted in: blocks for one piece per thread were four times as many to start, and were most of the
  // launch.  4 x 128 tokens, 32/8 heads, D 128: 17.6 -> 12.8 us a call, 2 x 256 19.5 -> 14.7, 100 11.4 -> 10.5)
  constexpr int kPieces = 256 * kCastLoads;
  const unsigned blocks = static_cast<unsigned>(std::min<long long>((most + kPieces - 1) / kPieces, static_cast<long long>(sm_count) * 16));
  return launch_dependent(cast_f32_to_f16_kernel, dim3(blocks, 3, 1), 256, 0, stream, 1, job);
}

}  // namespace b200attn
