// Memory-bound elementwise kernels (bf16 I/O, fp32 math, 16-byte accesses):
//   RoPE (rotate-half, in place on the packed QKV buffer), SwiGLU fwd/bwd,
//   GELU(tanh)/ReLU fwd/bwd, embedding gather / scatter-add (+ learned positions).
// They stand in for the ATen elementwise kernels the reference reaches through
// apply_rotary_pos_emb (models/llama_simple.py:34-58), HF LlamaMLP, gelu_new
// (models/gpt_simple.py:119-134) and nn.Embedding (models/llama_simple.py:550-552).
#include "../common/host.h"
#include "../common/ptx.cuh"
#include "act_math.cuh"
#include <type_traits>

namespace zb {

__device__ __forceinline__ void unpack8e(const uint4& u, float* f) {
  float2 a = unpack_bf16x2(u.x), b = unpack_bf16x2(u.y), c = unpack_bf16x2(u.z), d = unpack_bf16x2(u.w);
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y; f[4] = c.x; f[5] = c.y; f[6] = d.x; f[7] = d.y;
}
__device__ __forceinline__ uint4 pack8e(const float* f) {
  uint4 u;
  u.x = pack_bf16x2(f[0], f[1]); u.y = pack_bf16x2(f[2], f[3]);
  u.z = pack_bf16x2(f[4], f[5]); u.w = pack_bf16x2(f[6], f[7]);
  return u;
}

// ------------------------------- RoPE -------------------------------
// buf: [T, row_stride] bf16; heads 0..nheads-1 of width d start at column 0 (q heads then
// k heads in the packed QKV layout). cs: [S, d] fp32 = cos(d/2) | sin(d/2) per position.
// position of token t = (t % S). sign = +1 forward, -1 backward (transpose rotation).
__global__ void rope_kernel(__nv_bfloat16* buf, const float* cs, int T,
                            int S, int nheads, int d, int row_stride, float sign) {
  chain_trigger();
  chain_wait();
  const int half = d >> 1;
  const int cpr = half >> 3;  // 16-byte chunks per half head
  const long total = long(T) * nheads * cpr;
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < total; i += long(gridDim.x) * blockDim.x) {
    const int c = int(i % cpr);
    const int h = int((i / cpr) % nheads);
    const int t = int(i / (long(cpr) * nheads));
    const int pos = t % S;
    __nv_bfloat16* base = buf + size_t(t) * row_stride + h * d + c * 8;
    uint4 lo = *reinterpret_cast<uint4*>(base);
    uint4 hi = *reinterpret_cast<uint4*>(base + half);
    float a[8], b[8], oa[8], ob[8];
    unpack8e(lo, a);
    unpack8e(hi, b);
    const float4* cp = reinterpret_cast<const float4*>(cs + size_t(pos) * d + c * 8);
    const float4* sp = reinterpret_cast<const float4*>(cs + size_t(pos) * d + half + c * 8);
    float co[8], si[8];
    *reinterpret_cast<float4*>(co) = cp[0]; *reinterpret_cast<float4*>(co + 4) = cp[1];
    *reinterpret_cast<float4*>(si) = sp[0]; *reinterpret_cast<float4*>(si + 4) = sp[1];
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      float s = si[j] * sign;
      oa[j] = a[j] * co[j] - b[j] * s;
      ob[j] = b[j] * co[j] + a[j] * s;
    }
    *reinterpret_cast<uint4*>(base) = pack8e(oa);
    *reinterpret_cast<uint4*>(base + half) = pack8e(ob);
  }
}

// ------------------------------- SwiGLU -------------------------------
// gu: [T, 2F] (gate | up), out: [T, F] = silu(gate) * up
__global__ void swiglu_fwd_kernel(const __nv_bfloat16* gu, __nv_bfloat16* out,
                                  long T, int F) {
  chain_trigger();
  chain_wait();
  const int cpr = F >> 3;
  const long total = T * cpr;
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < total; i += long(gridDim.x) * blockDim.x) {
    const long t = i / cpr;
    const int c = int(i % cpr);
    const __nv_bfloat16* g = gu + t * 2 * F + c * 8;
    float a[8], b[8], o[8];
    unpack8e(ld_v4(g), a);
    unpack8e(ld_v4(g + F), b);
#pragma unroll
    for (int j = 0; j < 8; ++j) o[j] = swiglu_fwd(a[j], b[j]);
    *reinterpret_cast<uint4*>(out + t * F + c * 8) = pack8e(o);
  }
}
// dgu: [T, 2F]: dgate = dout * up * silu'(gate), dup = dout * silu(gate)
__global__ void swiglu_bwd_kernel(const __nv_bfloat16* gu, const __nv_bfloat16* dout,
                                  __nv_bfloat16* dgu, long T, int F) {
  chain_trigger();
  chain_wait();
  const int cpr = F >> 3;
  const long total = T * cpr;
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < total; i += long(gridDim.x) * blockDim.x) {
    const long t = i / cpr;
    const int c = int(i % cpr);
    const __nv_bfloat16* g = gu + t * 2 * F + c * 8;
    float a[8], b[8], d[8], da[8], db[8];
    unpack8e(ld_v4(g), a);
    unpack8e(ld_v4(g + F), b);
    unpack8e(ld_v4(dout + t * F + c * 8), d);
#pragma unroll
    for (int j = 0; j < 8; ++j) swiglu_bwd(a[j], b[j], d[j], da[j], db[j]);
    *reinterpret_cast<uint4*>(dgu + t * 2 * F + c * 8) = pack8e(da);
    *reinterpret_cast<uint4*>(dgu + t * 2 * F + F + c * 8) = pack8e(db);
  }
}

// ------------------------------- GELU / ReLU -------------------------------
__global__ void act_fwd_kernel(const __nv_bfloat16* x, __nv_bfloat16* y, long n8, int kind) {
  chain_trigger();
  chain_wait();
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < n8; i += long(gridDim.x) * blockDim.x) {
    float a[8], o[8];
    unpack8e(ld_v4(x + i * 8), a);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const float2 v = act_fwd2(make_float2(a[j], a[j + 1]), kind);
      o[j] = v.x;
      o[j + 1] = v.y;
    }
    *reinterpret_cast<uint4*>(y + i * 8) = pack8e(o);
  }
}
__global__ void act_bwd_kernel(const __nv_bfloat16* x, const __nv_bfloat16* dy,
                               __nv_bfloat16* dx, long n8, int kind) {
  chain_trigger();
  chain_wait();
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < n8; i += long(gridDim.x) * blockDim.x) {
    float a[8], d[8], o[8];
    unpack8e(ld_v4(x + i * 8), a);
    unpack8e(ld_v4(dy + i * 8), d);
#pragma unroll
    for (int j = 0; j < 8; j += 2) {
      const float2 v = act_bwd2(make_float2(a[j], a[j + 1]), kind);
      o[j] = d[j] * v.x;
      o[j + 1] = d[j + 1] * v.y;
    }
    *reinterpret_cast<uint4*>(dx + i * 8) = pack8e(o);
  }
}

// ------------------------------- embedding -------------------------------
// out[t, :] = table[ids[t], :] (+ pos_table[(t % S) + pos_offset, :])
__global__ void embedding_fwd_kernel(const long* ids, const __nv_bfloat16* table,
                                     const __nv_bfloat16* pos_table, __nv_bfloat16* out,
                                     int T, int H, int V, int S, int pos_offset) {
  chain_trigger();
  chain_wait();
  const int cpr = H >> 3;
  const long total = long(T) * cpr;
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < total; i += long(gridDim.x) * blockDim.x) {
    const int t = int(i / cpr), c = int(i % cpr);
    long id = ids[t];
    id = id < 0 ? 0 : (id >= V ? V - 1 : id);
    uint4 v = *reinterpret_cast<const uint4*>(table + id * H + c * 8);
    if (pos_table != nullptr) {
      float a[8], b[8];
      unpack8e(v, a);
      unpack8e(*reinterpret_cast<const uint4*>(pos_table + size_t((t % S) + pos_offset) * H + c * 8), b);
#pragma unroll
      for (int j = 0; j < 8; ++j) a[j] += b[j];
      v = pack8e(a);
    }
    *reinterpret_cast<uint4*>(out + size_t(t) * H + c * 8) = v;
  }
}
// dtable[ids[t], :] += dout[t, :] (atomic), dpos[(t % S) + off, :] += dout[t, :]
template <typename GT>
__device__ __forceinline__ void atomic_add2(GT* p, float a, float b);
template <>
__device__ __forceinline__ void atomic_add2<float>(float* p, float a, float b) {
  atomicAdd(p, a);
  atomicAdd(p + 1, b);
}
template <>
__device__ __forceinline__ void atomic_add2<__nv_bfloat16>(__nv_bfloat16* p, float a, float b) {
  atomicAdd(reinterpret_cast<__nv_bfloat162*>(p), __floats2bfloat162_rn(a, b));
}
// Adds of 16 bytes each (p 16-byte aligned): one request to the L2 atomic units where two- and four-byte adds made eight
// and four. 4096 x 4096 into fp32
// 98 -> 40 us, into bf16 43 -> 23.
__device__ __forceinline__ void red_add8(float* p, const uint4& u) {
  float f[8];
  unpack8e(u, f);
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p), "f"(f[0]), "f"(f[1]), "f"(f[2]), "f"(f[3]) : "memory");
  asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(p + 4), "f"(f[4]), "f"(f[5]), "f"(f[6]), "f"(f[7]) : "memory");
}
__device__ __forceinline__ void red_add8(__nv_bfloat16* p, const uint4& u) {
  asm volatile("red.global.add.noftz.v4.bf16x2 [%0], {%1, %2, %3, %4};" ::"l"(p), "r"(u.x), "r"(u.y), "r"(u.z), "r"(u.w)
               : "memory");
}
// VEC: both tables 16-byte aligned
template <typename GT, bool VEC>
__global__ void embedding_bwd_kernel(const long* ids, const __nv_bfloat16* dout,
                                     GT* dtable, GT* dpos, int T, int H, int V,
                                     int S, int pos_offset) {
  chain_trigger();
  chain_wait();
  const int cpr = H >> 3;
  const long total = long(T) * cpr;
  for (long i = blockIdx.x * long(blockDim.x) + threadIdx.x; i < total; i += long(gridDim.x) * blockDim.x) {
    const int t = int(i / cpr), c = int(i % cpr);
    long id = ids[t];
    id = id < 0 ? 0 : (id >= V ? V - 1 : id);
    const uint4 u = ld_v4(dout + size_t(t) * H + c * 8);
    GT* dst = dtable + id * H + c * 8;
    if constexpr (VEC) {
      red_add8(dst, u);
      if (dpos != nullptr) red_add8(dpos + size_t((t % S) + pos_offset) * H + c * 8, u);
      continue;
    }
    float a[8];
    unpack8e(u, a);
#pragma unroll
    for (int j = 0; j < 8; j += 2) atomic_add2<GT>(dst + j, a[j], a[j + 1]);
    if (dpos != nullptr) {
      GT* dp = dpos + size_t((t % S) + pos_offset) * H + c * 8;
#pragma unroll
      for (int j = 0; j < 8; j += 2) atomic_add2<GT>(dp + j, a[j], a[j + 1]);
    }
  }
}

// ------------------------------- image patches -------------------------------
// out[(b, py, px), (c, i, j)] = img[b, c, py p + i, px p + j] as bf16, columns from C p^2 up to kdim zero (ViT patch embedding
// as a GEMM operand).  One thread writes 16 bytes; with p a multiple of 8 its eight values are one row segment.  A pure
// copy: reads of the image and writes of the operand, both in order within a patch row.  8 images of 3 x 384 x 384, p = 16:
// 712 us with torch unfold, transpose and conversion, 19 us so.
__global__ void patches_kernel(const float* img, __nv_bfloat16* out, int C, int Hi, int Wi, int p,
                               int kdim, long total) {
  chain_trigger();
  chain_wait();
  const int cpr = kdim >> 3, nx = Wi / p, ny = Hi / p, pp = p * p;
  for (long w = blockIdx.x * long(blockDim.x) + threadIdx.x; w < total; w += long(gridDim.x) * blockDim.x) {
    const int k0 = int(w % cpr) * 8;
    const long tok = w / cpr;
    const int px = int(tok % nx), py = int((tok / nx) % ny);
    const long b = tok / (long(nx) * ny);
    float f[8];
#pragma unroll
    for (int u = 0; u < 8; ++u) {
      const int k = k0 + u;
      const int c = k / pp, r = k - c * pp, i = r / p, j = r - i * p;
      f[u] = c < C ? img[((b * C + c) * Hi + py * p + i) * long(Wi) + px * p + j] : 0.f;
    }
    *reinterpret_cast<uint4*>(out + w * 8) = pack8e(f);
  }
}
// p a multiple of 8, Wi of 4, no padding: two 16-byte loads per thread
__global__ void patches8_kernel(const float* img, __nv_bfloat16* out, int C, int Hi, int Wi, int p,
                                long total) {
  chain_trigger();
  chain_wait();
  const int pp = p * p, cpr = C * pp >> 3, nx = Wi / p, ny = Hi / p;
  for (long w = blockIdx.x * long(blockDim.x) + threadIdx.x; w < total; w += long(gridDim.x) * blockDim.x) {
    const int k = int(w % cpr) * 8;
    const long tok = w / cpr;
    const int px = int(tok % nx), py = int((tok / nx) % ny);
    const long b = tok / (long(nx) * ny);
    const int c = k / pp, r = k - c * pp, i = r / p, j = r - i * p;
    const float4* src = reinterpret_cast<const float4*>(img + ((b * C + c) * Hi + py * p + i) * long(Wi) + px * p + j);
    const float4 a = src[0], d = src[1];
    const float f[8] = {a.x, a.y, a.z, a.w, d.x, d.y, d.z, d.w};
    *reinterpret_cast<uint4*>(out + w * 8) = pack8e(f);
  }
}

static inline int grid_for(long work_items, int threads) {
  long b = (work_items + threads - 1) / threads;
  long cap = long(num_sms()) * 16;
  return int(b < 1 ? 1 : (b > cap ? cap : b));
}

static bool aligned16(const void* a, const void* b = nullptr, const void* c = nullptr) {
  return ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(b) | reinterpret_cast<uintptr_t>(c)) & 15) == 0;
}

}  // namespace zb

extern "C" {

int zb_rope(void* buf, const float* cs, int T, int S, int nheads, int d, int row_stride, int backward,
            cudaStream_t stream) {
  using namespace zb;
  if (d % 16 != 0 || row_stride % 8 != 0) ZB_FAIL(-1, "rope: head dim %d / stride %d unsupported", d, row_stride);
  if (T <= 0 || nheads <= 0) return 0;
  if (!aligned16(buf, cs)) ZB_FAIL(-4, "rope: an operand is not 16-byte aligned");
  long total = long(T) * nheads * (d / 16);
  ZB_CUDA_OK(launch_pass(rope_kernel, grid_for(total, 256), 256, 0, stream, static_cast<__nv_bfloat16*>(buf), cs, T, S,
                         nheads, d, row_stride, backward ? -1.f : 1.f));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}

int zb_swiglu_fwd(const void* gu, void* out, long T, int F, cudaStream_t stream) {
  using namespace zb;
  if (F % 8 != 0) ZB_FAIL(-1, "swiglu: F=%d not a multiple of 8", F);
  if (T <= 0) return 0;
  if (!aligned16(gu, out)) ZB_FAIL(-4, "swiglu: an operand is not 16-byte aligned");
  ZB_CUDA_OK(launch_pass(swiglu_fwd_kernel, grid_for(T * (F / 8), 256), 256, 0, stream,
                         static_cast<const __nv_bfloat16*>(gu), static_cast<__nv_bfloat16*>(out), T, F));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}
int zb_swiglu_bwd(const void* gu, const void* dout, void* dgu, long T, int F, cudaStream_t stream) {
  using namespace zb;
  if (F % 8 != 0) ZB_FAIL(-1, "swiglu: F=%d not a multiple of 8", F);
  if (T <= 0) return 0;
  if (!aligned16(gu, dout, dgu)) ZB_FAIL(-4, "swiglu: an operand is not 16-byte aligned");
  ZB_CUDA_OK(launch_pass(swiglu_bwd_kernel, grid_for(T * (F / 8), 256), 256, 0, stream,
                         static_cast<const __nv_bfloat16*>(gu), static_cast<const __nv_bfloat16*>(dout),
                         static_cast<__nv_bfloat16*>(dgu), T, F));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}
int zb_act_fwd(const void* x, void* y, long n, int kind, cudaStream_t stream) {
  using namespace zb;
  if (n % 8 != 0) ZB_FAIL(-1, "act: n=%ld not a multiple of 8", n);
  if (n <= 0) return 0;
  if (!aligned16(x, y)) ZB_FAIL(-4, "act: an operand is not 16-byte aligned");
  ZB_CUDA_OK(launch_pass(act_fwd_kernel, grid_for(n / 8, 256), 256, 0, stream, static_cast<const __nv_bfloat16*>(x),
                         static_cast<__nv_bfloat16*>(y), n / 8, kind));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}
int zb_act_bwd(const void* x, const void* dy, void* dx, long n, int kind, cudaStream_t stream) {
  using namespace zb;
  if (n % 8 != 0) ZB_FAIL(-1, "act: n=%ld not a multiple of 8", n);
  if (n <= 0) return 0;
  if (!aligned16(x, dy, dx)) ZB_FAIL(-4, "act: an operand is not 16-byte aligned");
  ZB_CUDA_OK(launch_pass(act_bwd_kernel, grid_for(n / 8, 256), 256, 0, stream, static_cast<const __nv_bfloat16*>(x),
                         static_cast<const __nv_bfloat16*>(dy), static_cast<__nv_bfloat16*>(dx), n / 8, kind));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}
// img fp32 [B, C, Hi, Wi] contiguous -> out bf16 [B (Hi / p) (Wi / p), kdim], kdim >= C p^2 a multiple of 8
int zb_patches(const float* img, void* out, int B, int C, int Hi, int Wi, int p, int kdim, cudaStream_t stream) {
  using namespace zb;
  if (p <= 0 || kdim % 8 != 0 || long(kdim) < long(C) * p * p) ZB_FAIL(-1, "patches: patch %d / row of %d unsupported", p, kdim);
  const long total = long(B) * (Hi / p) * (Wi / p) * (kdim / 8);
  if (total <= 0) return 0;
  auto O = static_cast<__nv_bfloat16*>(out);
  if (p % 8 == 0 && Wi % 4 == 0 && kdim == C * p * p && (reinterpret_cast<uintptr_t>(img) & 15) == 0)
    ZB_CUDA_OK(launch_pass(patches8_kernel, grid_for(total, 256), 256, 0, stream, img, O, C, Hi, Wi, p, total));
  else
    ZB_CUDA_OK(launch_pass(patches_kernel, grid_for(total, 256), 256, 0, stream, img, O, C, Hi, Wi, p, kdim, total));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}
int zb_embedding_fwd(const long* ids, const void* table, const void* pos_table, void* out, int T, int H, int V,
                     int S, int pos_offset, cudaStream_t stream) {
  using namespace zb;
  if (H % 8 != 0) ZB_FAIL(-1, "embedding: H=%d not a multiple of 8", H);
  if (T <= 0) return 0;
  ZB_CUDA_OK(launch_pass(embedding_fwd_kernel, grid_for(long(T) * (H / 8), 256), 256, 0, stream, ids,
                         static_cast<const __nv_bfloat16*>(table), static_cast<const __nv_bfloat16*>(pos_table),
                         static_cast<__nv_bfloat16*>(out), T, H, V, S, pos_offset));
  ZB_CUDA_OK(cudaGetLastError());
  return 0;
}
int zb_embedding_bwd(const long* ids, const void* dout, void* dtable, void* dpos, int T, int H, int V, int S,
                     int pos_offset, int grad_f32, cudaStream_t stream) {
  using namespace zb;
  if (H % 8 != 0) ZB_FAIL(-1, "embedding: H=%d not a multiple of 8", H);
  if (T <= 0) return 0;
  const int g = grid_for(long(T) * (H / 8), 256);
  const bool vec = ((reinterpret_cast<uintptr_t>(dtable) | reinterpret_cast<uintptr_t>(dpos)) & 15) == 0;
  auto D = static_cast<const __nv_bfloat16*>(dout);
  auto launch = [&](auto* table, auto* pos) -> int {
    using GT = std::remove_pointer_t<decltype(table)>;
    if (vec) ZB_CUDA_OK(launch_pass(embedding_bwd_kernel<GT, true>, g, 256, 0, stream, ids, D, table, pos, T, H, V, S,
                                    pos_offset));
    else ZB_CUDA_OK(launch_pass(embedding_bwd_kernel<GT, false>, g, 256, 0, stream, ids, D, table, pos, T, H, V, S,
                                pos_offset));
    return 0;
  };
  return grad_f32 ? launch(static_cast<float*>(dtable), static_cast<float*>(dpos))
                  : launch(static_cast<__nv_bfloat16*>(dtable), static_cast<__nv_bfloat16*>(dpos));
}

}  // extern "C"
