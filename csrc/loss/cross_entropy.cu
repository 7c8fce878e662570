// Fused cross-entropy forward + backward over bf16 logits [T, V]:
//   loss[t]    = logsumexp(logits[t, :]) - logits[t, target[t]]
//   dlogits    = (softmax(logits[t, :]) - onehot(target[t])) * grad_scale      (bf16)
// One CTA per row; the row is read twice (the second read hits L2) and the gradient is
// written once, in place if dlogits == logits.
//
// Two exponentials per logit: the exponential unit takes 117 us of the 160 that memory takes for 2048 x 128256, so what else is
// done per logit has to stay small (packed differences and maxima) and several loads in flight.  With scalars and one load
// at a time, and now: 2048 x 128256 265 -> 209 us, 4096 x 32000 111 -> 94, 3072 x 30528 86 -> 71, 1018 x 49152 46 -> 39, 256 x
// 32000 13.7 -> 9.4.  Against 64 bits a loss is off by up to 1.4e-7 of itself (rows of 32000 to 128256 normal
// logits of size 1 and 8).
#include "../common/host.h"
#include "../common/ptx.cuh"

namespace zb {

constexpr int CE_THREADS = 512, CE_UNROLL = 4;   // 16-byte pieces of a thread in flight

// e^(x - m) = 2^((x - m) log2 e) of two values.  The difference is taken first: x log2 e - m log2 e, one operation less, would
// carry the rounding of m log2 e, which grows with m (2.6e-6 of every term at m = 80), where this one's follows x - m.
__device__ __forceinline__ float2 ce_exp2(float2 x, float m) {
  float a, b;
  ffma2(a, b, x.x, x.y, 1.f, 1.f, -m, -m);
  fmul2(a, b, a, b, 1.4426950408889634f, 1.4426950408889634f);
  return make_float2(exp2f(a), exp2f(b));
}
__device__ __forceinline__ uint32_t ce_max2(uint32_t a, uint32_t b) {
  asm("max.bf16x2 %0, %0, %1;" : "+r"(a) : "r"(b));
  return a;
}
// The gradient of a row.
__device__ __forceinline__ void ce_gradient(const uint4* xv, uint4* dv, int n, int hit, int target, float m, float inv, float gs) {
  for (int c0 = threadIdx.x; c0 < n; c0 += CE_UNROLL * CE_THREADS) {
    uint4 u[CE_UNROLL];
#pragma unroll
    for (int i = 0; i < CE_UNROLL; ++i)
      if (c0 + i * CE_THREADS < n) u[i] = xv[c0 + i * CE_THREADS];
#pragma unroll
    for (int i = 0; i < CE_UNROLL; ++i) {
      const int c = c0 + i * CE_THREADS;
      if (c >= n) break;
      const uint32_t w[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
      float2 g[4];
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        g[j] = ce_exp2(unpack_bf16x2(w[j]), m);
        fmul2(g[j].x, g[j].y, g[j].x, g[j].y, inv, inv);
      }
      if (c == hit) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (2 * j == target) g[j].x -= gs;
          if (2 * j + 1 == target) g[j].y -= gs;
        }
      }
      dv[c] = make_uint4(pack_bf16x2(g[0].x, g[0].y), pack_bf16x2(g[1].x, g[1].y), pack_bf16x2(g[2].x, g[2].y),
                         pack_bf16x2(g[3].x, g[3].y));
    }
  }
}

template <int CTAS>   // per SM
__global__ void __launch_bounds__(CE_THREADS, CTAS)
ce_fwd_bwd_kernel(const __nv_bfloat16* logits, const long* targets,
                  __nv_bfloat16* dlogits, float* loss_rows, int T, int V,
                  long ld, float grad_scale, long ignore_index) {
  chain_trigger();
  chain_wait();
  __shared__ float red_m[CE_THREADS / 32], red_s[CE_THREADS / 32];
  __shared__ float bc[3];
  const int row = blockIdx.x;
  const __nv_bfloat16* x = logits + row * ld;
  const bool vec = (V % 8 == 0) && (ld % 8 == 0);
  const int n = V / 8;
  const long tgt = targets[row];
  const bool ignored = (tgt == ignore_index) || tgt < 0 || tgt >= V;
  // The target's logit is read ahead of the last barrier: behind it other threads may have written the gradient over it.
  if (threadIdx.x == 0) bc[2] = ignored ? 0.f : __bfloat162float(x[tgt]);
  float m = -INFINITY, s = 0.f;
  if (vec) {
    const uint4* xv = reinterpret_cast<const uint4*>(x);
    for (int c0 = threadIdx.x; c0 < n; c0 += CE_UNROLL * CE_THREADS) {
      uint4 u[CE_UNROLL];
#pragma unroll
      for (int i = 0; i < CE_UNROLL; ++i) {
        u[i] = make_uint4(0xff80ff80u, 0xff80ff80u, 0xff80ff80u, 0xff80ff80u);   // minus infinities add nothing
        if (c0 + i * CE_THREADS < n) u[i] = xv[c0 + i * CE_THREADS];
      }
#pragma unroll
      for (int i = 0; i < CE_UNROLL; ++i) {
        const uint32_t w[4] = {u[i].x, u[i].y, u[i].z, u[i].w};
        const float2 t = unpack_bf16x2(ce_max2(ce_max2(w[0], w[1]), ce_max2(w[2], w[3])));
        const float cm = fmaxf(t.x, t.y);
        if (cm > m) { s *= __expf(m - cm); m = cm; }
        const float at = m == -INFINITY ? 0.f : m;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const float2 e = ce_exp2(unpack_bf16x2(w[j]), at);
          s += e.x;
          s += e.y;
        }
      }
    }
  } else {
    for (int c = threadIdx.x; c < V; c += CE_THREADS) {
      float f = __bfloat162float(x[c]);
      if (f > m) { s *= __expf(m - f); m = f; }
      s += __expf(f - m);
    }
  }
  // combine (m, s) across the CTA
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, s, o);
    float nm = fmaxf(m, om);
    s = (m == -INFINITY ? 0.f : s * __expf(m - nm)) + (om == -INFINITY ? 0.f : os * __expf(om - nm));
    m = nm;
  }
  if ((threadIdx.x & 31) == 0) { red_m[threadIdx.x >> 5] = m; red_s[threadIdx.x >> 5] = s; }
  __syncthreads();
  if (threadIdx.x < 32) {
    m = threadIdx.x < CE_THREADS / 32 ? red_m[threadIdx.x] : -INFINITY;
    s = threadIdx.x < CE_THREADS / 32 ? red_s[threadIdx.x] : 0.f;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      float om = __shfl_xor_sync(0xffffffffu, m, o), os = __shfl_xor_sync(0xffffffffu, s, o);
      float nm = fmaxf(m, om);
      s = (m == -INFINITY ? 0.f : s * __expf(m - nm)) + (om == -INFINITY ? 0.f : os * __expf(om - nm));
      m = nm;
    }
    if (threadIdx.x == 0) { bc[0] = m; bc[1] = s; }
  }
  __syncthreads();
  m = bc[0];
  s = bc[1];
  if (threadIdx.x == 0) loss_rows[row] = ignored ? 0.f : (m + __logf(s)) - bc[2];
  if (dlogits == nullptr) return;
  const float inv = ignored ? 0.f : grad_scale / s;
  const float gs = ignored ? 0.f : grad_scale;
  __nv_bfloat16* dx = dlogits + row * ld;
  if (vec) {
    const uint4* xv = reinterpret_cast<const uint4*>(x);
    uint4* dv = reinterpret_cast<uint4*>(dx);
    const int hit = ignored ? -1 : int(tgt / 8), target = int(tgt % 8);   // the piece the target lies in, and where
    ce_gradient(xv, dv, n, hit, target, m, inv, gs);
  } else {
    for (int c = threadIdx.x; c < V; c += CE_THREADS) {
      float f = __expf(__bfloat162float(x[c]) - m) * inv;
      if (c == tgt) f -= gs;
      dx[c] = __float2bfloat16(f);
    }
  }
}

}  // namespace zb

extern "C" int zb_cross_entropy(const void* logits, const long* targets, void* dlogits, float* loss_rows,
                                int T, int V, long ld, float grad_scale, long ignore_index,
                                cudaStream_t stream) {
  using namespace zb;
  if (T <= 0) return 0;
  // Two CTAs per SM, with more registers for loads, where more rows than that are not there (256 x 32000: 9.9 us, with three 12.6)
  // or would not stay in L2 until their second reading (2048 x 128256: 211 and 231 us; 2048 x 50272, 45 MB: 89 and 80).
  const bool two = T <= 2 * num_sms() || 3L * num_sms() * V * 2 > 100'000'000L;
  auto kern = ce_fwd_bwd_kernel<3>;
  if (two) kern = ce_fwd_bwd_kernel<2>;
  ZB_CUDA_OK(launch_pass(kern, T, CE_THREADS, 0, stream, static_cast<const __nv_bfloat16*>(logits), targets,
                         static_cast<__nv_bfloat16*>(dlogits), loss_rows, T, V, ld, grad_scale, ignore_index));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}
