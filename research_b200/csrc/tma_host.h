// Host-side construction of 2-D bf16 TMA tensor maps (128-byte swizzle). The driver entry
// point is fetched at run time so the libraries do not link against libcuda.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <mutex>
#include <stdint.h>

namespace rb {

typedef CUresult (*EncodeTiledFnT)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                   const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFnT tma_encode_fn() {
  static EncodeTiledFnT fn = nullptr;
  static std::once_flag once;
  std::call_once(once, [] {
    void* f = nullptr;
    cudaDriverEntryPointQueryResult q;
    if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &f, cudaEnableDefault, &q) == cudaSuccess &&
        q == cudaDriverEntryPointSuccess)
      fn = reinterpret_cast<EncodeTiledFnT>(f);
  });
  return fn;
}

// The encoder needs the device's context to be current in the calling thread, which a thread that has made no runtime call of its own
// yet does not have (autograd's, whose allocations may all come from the cache): selecting the thread's device makes it so.
inline CUresult tma_encode_2d(EncodeTiledFnT fn, CUtensorMap* out, CUtensorMapDataType type, void* base, const cuuint64_t* dims,
                              const cuuint64_t* strides, const cuuint32_t* box, CUtensorMapL2promotion promotion,
                              CUtensorMapSwizzle swizzle = CU_TENSOR_MAP_SWIZZLE_128B) {
  const cuuint32_t estr[2] = {1, 1};
  for (int attempt = 0;; ++attempt) {
    const CUresult r = fn(out, type, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE, swizzle, promotion,
                          CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    int device = 0;
    if (r == CUDA_SUCCESS || attempt > 0 || cudaGetDevice(&device) != cudaSuccess || cudaSetDevice(device) != cudaSuccess) return r;
  }
}

// rows x cols matrix, cols contiguous, leading dimension ld (elements); box = box_rows x 64 columns.
inline int tma_map_2d_bf16(CUtensorMap* out, const void* base, unsigned long long rows, unsigned long long cols,
                           unsigned long long ld, unsigned box_rows) {
  EncodeTiledFnT fn = tma_encode_fn();
  if (fn == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld * 2) % 16 != 0) return -2;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {64, box_rows};
  const CUresult r = tma_encode_2d(fn, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, const_cast<void*>(base), dims, strides, box,
                                   CU_TENSOR_MAP_L2_PROMOTION_L2_256B);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// bf16 output matrix, boxes of box_rows x box_cols, rows of a box back to back in shared memory.
inline int tma_map_2d_plain(CUtensorMap* out, void* base, unsigned long long rows, unsigned long long cols, unsigned long long ld, unsigned box_rows,
                            unsigned box_cols) {
  EncodeTiledFnT fn = tma_encode_fn();
  if (fn == nullptr) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld * 2) % 16 != 0) return -2;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * 2};
  cuuint32_t box[2] = {box_cols, box_rows};
  const CUresult r = tma_encode_2d(fn, out, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, dims, strides, box, CU_TENSOR_MAP_L2_PROMOTION_NONE,
                                   CU_TENSOR_MAP_SWIZZLE_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// Output matrix, bf16 or fp32: boxes of box_rows x 128 bytes (64 or 32 columns).
inline int tma_map_2d_out(CUtensorMap* out, void* base, unsigned long long rows, unsigned long long cols, unsigned long long ld, int f32,
                          unsigned box_rows) {
  EncodeTiledFnT fn = tma_encode_fn();
  if (fn == nullptr) return -1;
  const unsigned es = f32 ? 4 : 2;
  if ((reinterpret_cast<uintptr_t>(base) & 15) != 0 || (ld * es) % 16 != 0) return -2;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * es};
  cuuint32_t box[2] = {128 / es, box_rows};
  const CUresult r = tma_encode_2d(fn, out, f32 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT32 : CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, base, dims, strides, box,
                                   CU_TENSOR_MAP_L2_PROMOTION_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

}  // namespace rb
