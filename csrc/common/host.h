// Host-side helpers shared by every launcher: TMA tensor-map encoding through the
// driver entry point (no link-time dependency on libcuda), device attributes, and the
// error-return convention (0 = ok, negative = host-side failure, see zb_last_error()).
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>
#include <stdio.h>
#include <string.h>

namespace zb {

inline char* last_error_buf() {
  static thread_local char buf[512];
  return buf;
}
#define ZB_FAIL(code, ...)                                   \
  do {                                                       \
    snprintf(zb::last_error_buf(), 512, __VA_ARGS__);        \
    return (code);                                           \
  } while (0)
#define ZB_CUDA_OK(expr)                                                              \
  do {                                                                                \
    cudaError_t e_ = (expr);                                                          \
    if (e_ != cudaSuccess) ZB_FAIL(-2, "%s: %s", #expr, cudaGetErrorString(e_));      \
  } while (0)

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*,
                                  const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                                  CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (!fn) {
    void* p = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) ==
            cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFn>(p);
  }
  return fn;
}

// 2-D bf16 tensor, row-major: `rows` x `cols`, row stride `ld` elements; box = box_cols x
// box_rows with 128-byte swizzle (box_cols must be 64). Returns 0 on success.
inline int make_tmap_2d_bf16(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols,
                             uint64_t ld, uint32_t box_rows, uint32_t box_cols) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) ZB_FAIL(-3, "cuTensorMapEncodeTiled entry point not available");
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) ZB_FAIL(-4, "TMA base not 16-byte aligned");
  if ((ld * 2) % 16 != 0) ZB_FAIL(-4, "TMA row stride (%llu elements) not a multiple of 16 bytes",
                                  (unsigned long long)ld);
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base), dims, strides,
                  box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) ZB_FAIL(-5, "cuTensorMapEncodeTiled failed with %d", int(r));
  return 0;
}

// 2-D output tensor (bf16 or fp32, row stride `ld` elements) read and written in boxes of `row_bytes` (128 or 64) x `box_rows`
// rows, swizzled over `row_bytes`.
inline int make_tmap_2d_out(CUtensorMap* out, const void* base, uint64_t rows, uint64_t cols, uint64_t ld, bool f32,
                            uint32_t box_rows, uint32_t row_bytes = 128) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) ZB_FAIL(-3, "cuTensorMapEncodeTiled entry point not available");
  const uint64_t es = f32 ? 4 : 2;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * es};
  cuuint32_t box[2] = {cuuint32_t(row_bytes / es), box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUresult r = fn(out, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, const_cast<void*>(base),
                  dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  row_bytes == 64 ? CU_TENSOR_MAP_SWIZZLE_64B : CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) ZB_FAIL(-5, "cuTensorMapEncodeTiled failed with %d", int(r));
  return 0;
}

// General N-d bf16 tensor map (innermost dimension first), 128-byte swizzle.
inline int make_tmap_nd_bf16(CUtensorMap* out, const void* base, int rank, const uint64_t* dims,
                             const uint64_t* strides_bytes /* rank-1 */, const uint32_t* box) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) ZB_FAIL(-3, "cuTensorMapEncodeTiled entry point not available");
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0) ZB_FAIL(-4, "TMA base not 16-byte aligned");
  cuuint64_t d[5];
  cuuint64_t s[4];
  cuuint32_t b[5], e[5];
  for (int i = 0; i < rank; ++i) {
    d[i] = dims[i];
    b[i] = box[i];
    e[i] = 1;
    if (i < rank - 1) {
      s[i] = strides_bytes[i];
      if (s[i] % 16 != 0) ZB_FAIL(-4, "TMA stride %d not a multiple of 16 bytes", i);
    }
  }
  CUresult r = fn(out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, rank, const_cast<void*>(base), d, s, b, e,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                  CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) ZB_FAIL(-5, "cuTensorMapEncodeTiled failed with %d", int(r));
  return 0;
}

// Launch that may begin while the kernel before it in the stream is still running; `kern` calls chain_wait (ptx.cuh).  For
// the kernels fed by TMA: barrier set-up, tensor-memory allocation and the launch itself go under the tail of the
// kernel before.  Steps: BERT 11.13 -> 10.11 ms, ViT 14.72 -> 13.61, offloaded OPT 42.6 -> 39.7; one block forward of the 1B
// model 417 -> 399 us.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_chained(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t stream,
                                  int cluster_x, Args&&... args) {
  cudaLaunchConfig_t cfg = {};
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[0].val.programmaticStreamSerializationAllowed = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim.x = cluster_x;
  attr[1].val.clusterDim.y = 1;
  attr[1].val.clusterDim.z = 1;
  cfg.gridDim = grid;
  cfg.blockDim = dim3(threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = stream;
  cfg.attrs = attr;
  cfg.numAttrs = cluster_x > 0 ? 2 : 1;   // 0: what the kernel itself declares
  return cudaLaunchKernelEx(&cfg, kern, static_cast<KArgs>(args)...);
}

// The same for the passes over memory (norms, activations, RoPE, column sums, loss): `kern` starts with chain_trigger and
// chain_wait and reads its inputs with coherent loads.  A plain launch leaves about 2 us between two kernels, and a
// block's backward has eleven of these.  Steps: BERT 10.22 -> 9.80 ms, ViT 13.69 -> 13.21, GPT of 512 21.1 -> 20.2; the large
// models, whose clock follows their power, gain nothing.
template <typename... KArgs, typename... Args>
inline cudaError_t launch_pass(void (*kern)(KArgs...), dim3 grid, int threads, size_t smem, cudaStream_t stream, Args&&... args) {
  return launch_chained(kern, grid, threads, smem, stream, 0, static_cast<Args&&>(args)...);
}

inline int num_sms() {
  static int n[64] = {0};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) dev = 0;
  if (n[dev] == 0) cudaDeviceGetAttribute(&n[dev], cudaDevAttrMultiProcessorCount, dev);
  return n[dev] > 0 ? n[dev] : 148;
}

}  // namespace zb
