// Helpers shared by the normalisation kernels: block-wide sum, 8-wide bf16 pack / unpack.
#pragma once
#include "../common/ptx.cuh"

namespace zb {

constexpr int NORM_THREADS = 256;
constexpr int NORM_MAXV = 4;  // 16-byte chunks per thread kept in registers -> H <= 8192

__device__ __forceinline__ float block_sum(float v, float* red) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
  __syncthreads();
  if (l == 0) red[w] = v;
  __syncthreads();
  float t = (threadIdx.x < (blockDim.x >> 5)) ? red[threadIdx.x] : 0.f;
  if (w == 0) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (l == 0) red[32] = t;
  }
  __syncthreads();
  return red[32];
}

// Rows a CTA works on at a time: as many teams of threads as leave each thread at most NORM_MAXV 16-byte chunks.
inline int norm_rows_per_cta(int H) { return H <= 1024 ? 8 : H <= 2048 ? 4 : H <= 4096 ? 2 : 1; }

// Barrier among the NORM_THREADS / RW threads of one team (a team of one warp needs none).
template <int RW>
__device__ __forceinline__ void team_barrier(int team) {
  if constexpr (RW == 1) __syncthreads();
  else if constexpr (RW < 8) asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(NORM_THREADS / RW) : "memory");
}

// Sum over the threads of a team; `red` holds one value per warp of the CTA and is not reused between two calls without
// a barrier in between.
template <int RW>
__device__ __forceinline__ float team_sum(float v, float* red, int team) {
  constexpr int WARPS = NORM_THREADS / RW / 32;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  if constexpr (WARPS > 1) {
    if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = v;
    team_barrier<RW>(team);
    v = 0.f;
#pragma unroll
    for (int k = 0; k < WARPS; ++k) v += red[team * WARPS + k];
  }
  return v;
}

__device__ __forceinline__ void unpack8(const uint4& u, float* f) {
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8(const float* f) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]); u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]); u.w = pack_bf16x2(f[6], f[7]);
  return u;
}

}  // namespace zb
