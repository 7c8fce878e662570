// Several column sums in one launch: out[n] += sum_t src[t, n], for the bias gradients of a block's backward pass (src: bf16
// gradients) and the weight and bias gradients of its norms (src: fp32 partial sums, one row per CTA of the norm kernel).
//
// Each of these sums reads a few megabytes that are still in L2, takes longer to launch than to read, and alone its strips of
// columns make too few CTAs (768 columns: 24).  Together they fill the GPU: a cluster of eight CTAs takes 64 columns of one
// matrix, each CTA an eighth of the rows with four 16-byte requests per thread in flight, and the eight partial sums are
// added through distributed shared memory, in their order, so results do not depend on timing.
// The four bias and four norm gradients of a BERT block (3072 tokens, 768 / 3072 wide): six launches 28 us, one launch 7.
#include "../common/host.h"
#include "../common/ptx.cuh"
#include "norm_common.cuh"

namespace zb {

constexpr int COLSUM_MAX = 8, COLSUM_COLS = 64, COLSUM_RANKS = 8;
struct ColSumItem {
  const void* src;
  void* out;
  int rows, cols, ld;
  int src_f32, out_f32;
  int strip_end;   // strips of this item and those before it
};
struct ColSumItems {
  ColSumItem item[COLSUM_MAX];
  int late;   // nothing that the kernel before this one writes is read here (chain_late in ptx.cuh)
};

__global__ void __cluster_dims__(COLSUM_RANKS, 1, 1) __launch_bounds__(256)
column_sums_kernel(const __grid_constant__ ColSumItems p) {
  chain_trigger();
  if (!p.late) chain_wait();
  __shared__ float warp_sum[8][COLSUM_COLS], cta_sum[COLSUM_COLS];
  const int strip = blockIdx.x / COLSUM_RANKS, rank = blockIdx.x % COLSUM_RANKS;
  int i = 0;
  while (strip >= p.item[i].strip_end) ++i;
  const ColSumItem it = p.item[i];
  const int col0 = (strip - (i > 0 ? p.item[i - 1].strip_end : 0)) * COLSUM_COLS;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int chunk = (it.rows + COLSUM_RANKS - 1) / COLSUM_RANKS;
  const int row_end = min(it.rows, (rank + 1) * chunk);
  float s[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
  // 16 bytes per lane: a row's 64 columns are 8 lanes of bf16 or 16 of fp32
  auto walk = [&](const char* base, size_t pitch, int step, auto add) {
    int r = rank * chunk + int(threadIdx.x) / (256 / step);
    for (; r + 3 * step < row_end; r += 4 * step) {
      uint4 u[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) u[k] = ld_v4(base + size_t(r + k * step) * pitch);
#pragma unroll
      for (int k = 0; k < 4; ++k) add(u[k]);
    }
    for (; r < row_end; r += step) add(ld_v4(base + size_t(r) * pitch));
  };
  if (it.src_f32) {
    const int col = col0 + (threadIdx.x & 15) * 4;
    if (col < it.cols) {
      walk(reinterpret_cast<const char*>(static_cast<const float*>(it.src) + col), size_t(it.ld) * 4, 16, [&](const uint4& u) {
        s[0] += __uint_as_float(u.x); s[1] += __uint_as_float(u.y); s[2] += __uint_as_float(u.z); s[3] += __uint_as_float(u.w);
      });
    }
#pragma unroll
    for (int j = 0; j < 4; ++j) s[j] += __shfl_xor_sync(0xffffffffu, s[j], 16);
    if (lane < 16) {
#pragma unroll
      for (int j = 0; j < 4; ++j) warp_sum[warp][lane * 4 + j] = s[j];
    }
  } else {
    const int col = col0 + (threadIdx.x & 7) * 8;
    if (col < it.cols) {
      walk(reinterpret_cast<const char*>(static_cast<const __nv_bfloat16*>(it.src) + col), size_t(it.ld) * 2, 32, [&](const uint4& u) {
        float f[8];
        unpack8(u, f);
#pragma unroll
        for (int j = 0; j < 8; ++j) s[j] += f[j];
      });
    }
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      s[j] += __shfl_xor_sync(0xffffffffu, s[j], 8);
      s[j] += __shfl_xor_sync(0xffffffffu, s[j], 16);
    }
    if (lane < 8) {
#pragma unroll
      for (int j = 0; j < 8; ++j) warp_sum[warp][lane * 8 + j] = s[j];
    }
  }
  __syncthreads();
  if (threadIdx.x < COLSUM_COLS) {
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < 8; ++w) t += warp_sum[w][threadIdx.x];
    cta_sum[threadIdx.x] = t;
  }
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
  if (threadIdx.x < COLSUM_COLS / COLSUM_RANKS) {   // each CTA finishes eight of the columns
    const int c = rank * (COLSUM_COLS / COLSUM_RANKS) + int(threadIdx.x);
    float t = 0.f;
#pragma unroll
    for (int q = 0; q < COLSUM_RANKS; ++q) {
      uint32_t a;
      float v;
      asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"(smem_u32(&cta_sum[c])), "r"(q));
      asm volatile("ld.shared::cluster.f32 %0, [%1];" : "=f"(v) : "r"(a) : "memory");
      t += v;
    }
    if (col0 + c < it.cols) {
      if (it.out_f32) {
        float* o = static_cast<float*>(it.out) + col0 + c;
        *o += t;
      } else {
        __nv_bfloat16* o = static_cast<__nv_bfloat16*>(it.out) + col0 + c;
        *o = __float2bfloat16(__bfloat162float(*o) + t);
      }
    }
  }
  // nobody leaves while its sums are read
  asm volatile("barrier.cluster.arrive.release;\nbarrier.cluster.wait.acquire;" ::: "memory");
  if (p.late) chain_wait();
}

}  // namespace zb

// n <= 8 sums.  desc: per sum src, out, rows, cols, row distance in elements, 1 if src is fp32 (else bf16), 1 if out is.  Rows
// of src start on 16-byte boundaries and cols is a multiple of 8 (bf16) or 4 (fp32).  Returns 1, with nothing done, otherwise.
// late: the kernel in front of this one in the stream writes none of the sources (see chain_late in ptx.cuh).
extern "C" int zb_column_sums(const long* desc, int n, int late, cudaStream_t stream) {
  using namespace zb;
  if (n <= 0) return 0;
  if (n > COLSUM_MAX) ZB_FAIL(-1, "column_sums: %d sums (at most %d)", n, COLSUM_MAX);
  ColSumItems p = {};
  p.late = late;
  int strips = 0, used = 0;
  for (int i = 0; i < n; ++i, desc += 7) {
    ColSumItem& it = p.item[used];
    it.src = reinterpret_cast<const void*>(desc[0]);
    it.out = reinterpret_cast<void*>(desc[1]);
    it.rows = int(desc[2]); it.cols = int(desc[3]); it.ld = int(desc[4]);
    it.src_f32 = int(desc[5]); it.out_f32 = int(desc[6]);
    const int per16 = it.src_f32 ? 4 : 8;
    if ((desc[0] & 15) || it.cols % per16 || it.ld % per16) return 1;
    if (it.rows <= 0 || it.cols <= 0) continue;
    strips += (it.cols + COLSUM_COLS - 1) / COLSUM_COLS;
    it.strip_end = strips;
    ++used;
  }
  if (used == 0) return 0;
  ZB_CUDA_OK(launch_pass(column_sums_kernel, dim3(strips * COLSUM_RANKS), 256, 0, stream, p));
  return 0;
}
