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

__device__ __forceinline__ float lane_add(float v, int o) { return v + __shfl_xor_sync(0xffffffffu, v, o); }
__device__ __forceinline__ float2 lane_add(float2 v, int o) {
  return make_float2(v.x + __shfl_xor_sync(0xffffffffu, v.x, o), v.y + __shfl_xor_sync(0xffffffffu, v.y, o));
}

// Barrier among the NORM_THREADS / RW threads of one team (a team of one warp needs none).
template <int RW>
__device__ __forceinline__ void team_barrier(int team) {
  if constexpr (RW == 1) __syncthreads();
  else if constexpr (RW < 8) asm volatile("bar.sync %0, %1;" ::"r"(team + 1), "n"(NORM_THREADS / RW) : "memory");
}

// Row sums keep one order whatever the split into teams, so that a result does not depend on it: 32 consecutive 16-byte
// chunks of a row (and those 256, 512, ... chunks further on) form a group, added lane by lane and then over the lanes;
// there are eight groups.  A thread holds the chunks of NORM_GROUPS<RW> groups, chunk i in v[i % NORM_GROUPS<RW>].
template <int RW>
constexpr int NORM_GROUPS = RW < NORM_MAXV ? RW : NORM_MAXV;

// Sums of the eight groups, one per call and entry of g, on every thread of the team.  `red` holds 8 values per team and is
// not reused between two calls without a barrier in between.
template <int RW, typename T>
__device__ __forceinline__ void team_group_sums(T (&v)[NORM_GROUPS<RW>], T* red, int team, T (&g)[8]) {
  constexpr int WARPS = NORM_THREADS / RW / 32, A = NORM_GROUPS<RW>;
#pragma unroll
  for (int a = 0; a < A; ++a) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v[a] = lane_add(v[a], o);
  }
  if constexpr (WARPS > 1) {
    if ((threadIdx.x & 31) == 0) {
#pragma unroll
      for (int a = 0; a < A; ++a) red[team * 8 + (threadIdx.x >> 5) % WARPS + a * WARPS] = v[a];
    }
    team_barrier<RW>(team);
#pragma unroll
    for (int k = 0; k < 8; ++k) g[k] = red[team * 8 + k];
  } else {
#pragma unroll
    for (int k = 0; k < 8; ++k) g[k] = k < A ? v[k] : T{};
  }
}
template <int RW>
__device__ __forceinline__ float team_sum(float (&v)[NORM_GROUPS<RW>], float* red, int team) {
  float g[8];
  team_group_sums<RW>(v, red, team, g);
  return ((g[0] + g[4]) + (g[2] + g[6])) + ((g[1] + g[5]) + (g[3] + g[7]));
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
