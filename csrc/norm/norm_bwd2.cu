// RMSNorm / LayerNorm backward, second version (same interface and scratch as zb_norm_bwd).
// Differences from the first version (norm.cu):
//   * a CTA works on RW rows at a time, a team of 256 / RW threads each with up to four 16-byte chunks per thread, so that
//     narrow rows keep every thread busy;
//   * x, dy and the residual gradient of the next one to three groups of rows are on their way into shared memory
//     (cp.async) while a group is reduced.  A thread reads only the chunks it has requested itself, so the ring needs no
//     barrier;
//   * one barrier per row (none where a team is one warp): the (sum g*xhat, sum g) pair is reduced in one pass;
//   * the column reduction of the per-CTA partial sums runs on H/32 CTAs of 32 x 32 threads (32
//     rows in flight per column) instead of H/256 CTAs walking all partial rows one after another.
// Bound by memory latency: with one row per CTA and the next row requested into registers 4616 x 768 took 42 us, now 24;
// 4096 x 4096 46 -> 38 us, 2048 x 5120 50 -> 34 us (operands not in L2; reduction of the partial sums included).
// Sums are formed in a fixed order, so results are deterministic; dx does not depend on the split into teams.
#include "../common/host.h"
#include "../common/ptx.cuh"
#include "norm_common.cuh"

extern "C" int zb_norm_partial_rows(int T);

namespace zb {

__device__ __forceinline__ void cp_async16(uint32_t dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() {   // all but the newest N groups of this thread have landed
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

template <int NV>   // 16-byte chunks per thread
struct NormBwdCfg {
  static constexpr int STAGES = NV == 4 ? 2 : NV == 3 ? 3 : 4;            // about 100 KB: two CTAs per SM
  static constexpr int STAGE_BYTES = 3 * NV * NORM_THREADS * 16;          // x, dy, residual gradient
  static constexpr int SMEM_BYTES = STAGES * STAGE_BYTES;
};

template <bool LN, int RW, int NV>
__global__ void __launch_bounds__(NORM_THREADS, 2)
norm_bwd2_kernel(const __nv_bfloat16* dy, const __nv_bfloat16* x,
                 const __nv_bfloat16* w, const float* stats,
                 const __nv_bfloat16* dres, __nv_bfloat16* dx,
                 float* part_dw, float* part_db, int T, int H) {
  chain_trigger();
  chain_wait();
  using Cfg = NormBwdCfg<NV>;
  constexpr int TEAM = NORM_THREADS / RW, NS = Cfg::STAGES, A = NORM_GROUPS<RW>;
  extern __shared__ __align__(128) uint8_t ring[];
  __shared__ float2 red[2][RW * 8];
  const int team = threadIdx.x / TEAM, tt = threadIdx.x % TEAM;
  const int nchunk = H >> 3;
  const uint32_t slot0 = smem_u32(ring) + threadIdx.x * 16;
  auto slot = [&](int stage, int tensor, int i) {
    return slot0 + uint32_t(stage * Cfg::STAGE_BYTES + (tensor * NV + i) * (NORM_THREADS * 16));
  };
  float aw[NV][8], ab[LN ? NV : 1][8];
  uint4 wraw[NV];
#pragma unroll
  for (int i = 0; i < NV; ++i) {
    const int c = tt + i * TEAM;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      aw[i][j] = 0.f;
      if (LN) ab[i][j] = 0.f;
    }
    wraw[i] = c < nchunk ? reinterpret_cast<const uint4*>(w)[c] : make_uint4(0u, 0u, 0u, 0u);
  }
  const int groups = (T + RW - 1) / RW;
  auto request = [&](int g, int stage) {   // this thread's chunks of its team's row of group g
    const int row = g * RW + team;
    if (g < groups && row < T) {
      const size_t base = size_t(row) * H;
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = tt + i * TEAM;
        if (c < nchunk) {
          cp_async16(slot(stage, 0, i), x + base + c * 8);
          cp_async16(slot(stage, 1, i), dy + base + c * 8);
          if (dres != nullptr) cp_async16(slot(stage, 2, i), dres + base + c * 8);
        }
      }
    }
    cp_async_commit();
  };
#pragma unroll
  for (int s = 0; s < NS; ++s) request(blockIdx.x + s * gridDim.x, s);
  float2 st = make_float2(0.f, 0.f);
  {
    const int row = blockIdx.x * RW + team;
    if (row < T) st = *reinterpret_cast<const float2*>(stats + 2 * size_t(row));
  }
  int stage = 0, buf = 0;
  for (int g = blockIdx.x; g < groups; g += gridDim.x, buf ^= 1) {
    const int row = g * RW + team;
    const float mean = st.x, rstd = st.y;
    const long nrow = long(g + gridDim.x) * RW + team;
    if (nrow < T) st = *reinterpret_cast<const float2*>(stats + 2 * nrow);
    cp_async_wait<NS - 1>();
    if (row < T) {   // the whole team
      float2 s[A] = {};
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        if (tt + i * TEAM < nchunk) {
          float xf[8], df[8], wf[8];
          unpack8(ld_shared_v4(slot(stage, 0, i)), xf);
          unpack8(ld_shared_v4(slot(stage, 1, i)), df);
          unpack8(wraw[i], wf);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xh = (xf[j] - mean) * rstd, gg = __fmul_rn(df[j], wf[j]);
            s[i % A].x += gg * xh;
            aw[i][j] += df[j] * xh;
            if (LN) {
              s[i % A].y += gg;
              ab[i][j] += df[j];
            }
          }
        }
      }
      float2 sums[8];
      team_group_sums<RW>(s, red[buf], team, sums);
      float s1 = 0.f, s2 = 0.f;
#pragma unroll
      for (int k = 0; k < 8; ++k) {
        s1 += sums[k].x;
        s2 += sums[k].y;
      }
      const float m1 = s1 / H, m2 = LN ? s2 / H : 0.f;
      uint4* dxr = reinterpret_cast<uint4*>(dx + size_t(row) * H);
#pragma unroll
      for (int i = 0; i < NV; ++i) {
        const int c = tt + i * TEAM;
        if (c < nchunk) {
          float xf[8], df[8], wf[8], rf[8], o[8];
          unpack8(ld_shared_v4(slot(stage, 0, i)), xf);
          unpack8(ld_shared_v4(slot(stage, 1, i)), df);
          unpack8(wraw[i], wf);
          if (dres != nullptr) unpack8(ld_shared_v4(slot(stage, 2, i)), rf);
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            const float xh = (xf[j] - mean) * rstd;
            o[j] = rstd * (__fmul_rn(df[j], wf[j]) - xh * m1 - m2);
            if (dres != nullptr) o[j] += rf[j];
          }
          dxr[c] = pack8(o);
        }
      }
    }
    request(g + NS * gridDim.x, stage);   // behind the stores that used the last value read from this stage
    stage = stage + 1 == NS ? 0 : stage + 1;
  }
  // column sums of this CTA: teams in order, through shared memory (the ring: every copy into it has landed)
  cp_async_wait<0>();
  auto finish = [&](auto& acc, float* part) {
    float* sm = reinterpret_cast<float*>(ring);
    float* out = part + size_t(blockIdx.x) * H;
    if (RW > 1) __syncthreads();
#pragma unroll
    for (int i = 0; i < NV; ++i) {
      const int c = tt + i * TEAM;
      if (c < nchunk) {
        float4* d = reinterpret_cast<float4*>((RW > 1 ? sm + team * H : out) + c * 8);
        d[0] = make_float4(acc[i][0], acc[i][1], acc[i][2], acc[i][3]);
        d[1] = make_float4(acc[i][4], acc[i][5], acc[i][6], acc[i][7]);
      }
    }
    if (RW > 1) {
      __syncthreads();
      for (int c = threadIdx.x; c < H / 4; c += NORM_THREADS) {
        float4 t = reinterpret_cast<const float4*>(sm)[c];
#pragma unroll
        for (int k = 1; k < RW; ++k) {
          const float4 v = reinterpret_cast<const float4*>(sm + k * H)[c];
          t.x += v.x; t.y += v.y; t.z += v.z; t.w += v.w;
        }
        reinterpret_cast<float4*>(out)[c] = t;
      }
    }
  };
  finish(aw, part_dw);
  if constexpr (LN) {
    if (part_db != nullptr) finish(ab, part_db);
  }
}

template <bool LN, int RW, int NV>
static int launch_norm_bwd2(const __nv_bfloat16* dy, const __nv_bfloat16* x, const __nv_bfloat16* w, const float* stats,
                            const __nv_bfloat16* dres, __nv_bfloat16* dx, float* part_dw, float* part_db, int T, int H,
                            int blocks, cudaStream_t stream) {
  auto kern = norm_bwd2_kernel<LN, RW, NV>;
  static bool attr_set = false;
  if (!attr_set) {
    ZB_CUDA_OK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, NormBwdCfg<NV>::SMEM_BYTES));
    attr_set = true;
  }
  ZB_CUDA_OK(launch_pass(kern, blocks, NORM_THREADS, NormBwdCfg<NV>::SMEM_BYTES, stream, dy, x, w, stats, dres, dx, part_dw,
                         part_db, T, H));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}

// out[h] (+)= sum_p part[p, h] with a 32 x 32 thread block per 32 columns: thread (tx, ty) adds rows
// ty, ty + 32, ...; the partial sums of a column are then added by a warp, lane by lane.
// blockIdx.y selects one of two such sums (weight and bias gradient in one launch).
template <typename OutT>
__global__ void __launch_bounds__(1024)
colsum_accumulate2_kernel(const float* part0, const float* part1, int P, int H,
                          OutT* out0, OutT* out1, int accumulate) {
  chain_trigger();
  chain_wait();
  __shared__ float sm[32][33];
  const float* part = blockIdx.y ? part1 : part0;
  OutT* out = blockIdx.y ? out1 : out0;
  const int tx = threadIdx.x & 31, ty = threadIdx.x >> 5;
  const int h = blockIdx.x * 32 + tx;
  float s = 0.f;
  if (h < H) {
#pragma unroll 4
    for (int p = ty; p < P; p += 32) s += part[size_t(p) * H + h];
  }
  sm[ty][tx] = s;
  __syncthreads();
  float t = sm[tx][ty];   // column ty, rows tx, tx + 32, ...
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
  const int c = blockIdx.x * 32 + ty;
  if (tx == 0 && c < H) {
    if (accumulate) t += float(out[c]);
    out[c] = OutT(t);
  }
}

// Finishes one or two column sums (out1 / part1 null: one).
int colsum_finish(const float* part0, int P, int H, void* out0, const float* part1, void* out1, int grad_f32,
                  int accumulate, cudaStream_t stream) {
  const dim3 grid((H + 31) / 32, out1 != nullptr ? 2 : 1);
  if (grad_f32)
    ZB_CUDA_OK(launch_pass(colsum_accumulate2_kernel<float>, grid, 1024, 0, stream, part0, part1, P, H,
                           static_cast<float*>(out0), static_cast<float*>(out1), accumulate));
  else
    ZB_CUDA_OK(launch_pass(colsum_accumulate2_kernel<__nv_bfloat16>, grid, 1024, 0, stream, part0, part1, P, H,
                           static_cast<__nv_bfloat16*>(out0), static_cast<__nv_bfloat16*>(out1), accumulate));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}

}  // namespace zb

// Rows of partial sums that zb_norm_bwd2 writes (of the zb_norm_partial_rows(T) it has room for).
extern "C" int zb_norm_bwd2_rows(int T, int H) {
  const int rw = zb::norm_rows_per_cta(H), groups = (T + rw - 1) / rw, cap = zb_norm_partial_rows(T);
  return groups < cap ? groups : cap;
}

extern "C" int zb_norm_bwd2(const void* dy, const void* x, const void* w, const float* stats, const void* dres,
                            void* dx, float* part_dw, float* part_db, void* dw, void* db, int T, int H, int ln,
                            int grad_f32, int accumulate, cudaStream_t stream) {
  using namespace zb;
  if (H % 8 != 0 || H > NORM_THREADS * NORM_MAXV * 8) ZB_FAIL(-1, "norm: H=%d unsupported", H);
  if (T <= 0) return 0;
  auto DY = static_cast<const __nv_bfloat16*>(dy);
  auto X = static_cast<const __nv_bfloat16*>(x);
  auto W = static_cast<const __nv_bfloat16*>(w);
  auto DR = static_cast<const __nv_bfloat16*>(dres);
  auto DX = static_cast<__nv_bfloat16*>(dx);
  const int rw = norm_rows_per_cta(H), nv = (H / 8 + NORM_THREADS / rw - 1) / (NORM_THREADS / rw);
  const int P = zb_norm_bwd2_rows(T, H);   // two CTAs per SM, a row of partial sums each
  int rc = 0;
#define ZB_NORM_BWD(RW_, NV_)                                                                                        \
  rc = ln ? launch_norm_bwd2<true, RW_, NV_>(DY, X, W, stats, DR, DX, part_dw, part_db, T, H, P, stream)              \
          : launch_norm_bwd2<false, RW_, NV_>(DY, X, W, stats, DR, DX, part_dw, nullptr, T, H, P, stream)
  if (rw == 8) {
    if (nv == 1) ZB_NORM_BWD(8, 1);
    else if (nv == 2) ZB_NORM_BWD(8, 2);
    else if (nv == 3) ZB_NORM_BWD(8, 3);
    else ZB_NORM_BWD(8, 4);
  } else if (rw == 4) {
    if (nv == 3) ZB_NORM_BWD(4, 3);
    else ZB_NORM_BWD(4, 4);
  } else if (rw == 2) {
    if (nv == 3) ZB_NORM_BWD(2, 3);
    else ZB_NORM_BWD(2, 4);
  } else {
    if (nv == 3) ZB_NORM_BWD(1, 3);
    else ZB_NORM_BWD(1, 4);
  }
#undef ZB_NORM_BWD
  if (rc) return rc;
  const bool bias = ln && db != nullptr;
  if (dw != nullptr) return colsum_finish(part_dw, P, H, dw, bias ? part_db : nullptr, bias ? db : nullptr, grad_f32, accumulate, stream);
  if (bias) return colsum_finish(part_db, P, H, db, nullptr, nullptr, grad_f32, accumulate, stream);
  return 0;
}
