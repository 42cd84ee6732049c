// Host-side TMA descriptor (CUtensorMap) construction without linking libcuda:
// the driver entry point is fetched through the runtime.
#pragma once
#include <cuda.h>
#include <cudaTypedefs.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace ronn {

typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                  const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                  CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeTiledFn encode_tiled_fn() {
  static EncodeTiledFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeTiledFn>(p);
  return fn;
}

typedef CUresult (*EncodeIm2colFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                                   const int*, const int*, cuuint32_t, cuuint32_t, const cuuint32_t*, CUtensorMapInterleave,
                                   CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline EncodeIm2colFn encode_im2col_fn() {
  static EncodeIm2colFn fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult q;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeIm2col", &p, cudaEnableDefault, &q) != cudaSuccess ||
      q != cudaDriverEntryPointSuccess)
    return nullptr;
  fn = reinterpret_cast<EncodeIm2colFn>(p);
  return fn;
}

// Whether the descriptor holds the window positions of an im2col tensor: they run from the lower corner to (size - 1 + upper
// corner), both stored in 8 bits, in steps of up to 8.
inline bool im2col_fits(int H, int W, int Ho, int Wo, int stride, int pad_h, int pad_w) {
  const int lower[2] = {-pad_w, -pad_h};
  const int upper[2] = {-pad_w + (Wo - 1) * stride - (W - 1), -pad_h + (Ho - 1) * stride - (H - 1)};
  for (int i = 0; i < 2; ++i)
    if (lower[i] < -128 || upper[i] < -128 || upper[i] > 127) return false;
  return stride >= 1 && stride <= 8;
}

// NHWC tensor of 2-byte elements for im2col loads: a load starts at a filter window's top-left position (w, h of image n)
// and takes `channels` channels at one filter tap of `pixels` consecutive output positions, in (w, h, n) order; the
// windows are `stride` apart, Wo x Ho of them per image, the first at (-pad_w, -pad_h).  Positions outside the tensor, the
// images past the last one included, read zero.  channels x 2 bytes is 128 or 32 and sets the swizzle.  The strides of W, H
// and N are in elements; neighbouring positions may overlap (w_stride < C).  Returns 0 on success, -2 for a geometry the
// descriptor cannot hold.
inline int make_tmap_im2col(CUtensorMap* map, const void* base, int N, int H, int W, int C, uint64_t w_stride, uint64_t h_stride,
                            uint64_t n_stride, int Ho, int Wo, int stride, int pad_h, int pad_w, int channels, int pixels) {
  EncodeIm2colFn fn = encode_im2col_fn();
  if (!fn) return -1;
  if (!im2col_fits(H, W, Ho, Wo, stride, pad_h, pad_w) || (reinterpret_cast<uintptr_t>(base) & 15) || (w_stride & 7) ||
      (h_stride & 7) || (n_stride & 7) || channels > C)
    return -2;
  const int lower[2] = {-pad_w, -pad_h};
  const int upper[2] = {-pad_w + (Wo - 1) * stride - (W - 1), -pad_h + (Ho - 1) * stride - (H - 1)};
  cuuint64_t dims[4] = {cuuint64_t(C), cuuint64_t(W), cuuint64_t(H), cuuint64_t(N)};
  cuuint64_t strides[3] = {w_stride * 2, h_stride * 2, n_stride * 2};
  cuuint32_t estr[4] = {1, cuuint32_t(stride), cuuint32_t(stride), 1};
  CUresult r = fn(map, CU_TENSOR_MAP_DATA_TYPE_UINT16, 4, const_cast<void*>(base), dims, strides, lower, upper,
                  cuuint32_t(channels), cuuint32_t(pixels), estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  channels == 64 ? CU_TENSOR_MAP_SWIZZLE_128B : CU_TENSOR_MAP_SWIZZLE_32B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

// 2-D row-major tensor [rows, cols] of 1- or 2-byte elements with leading dimension ld (elements); box = [box_rows, box_cols];
// 128-byte swizzle (box_cols * elem_size must be 128).  Returns 0 on success.
inline int make_tmap_2d(CUtensorMap* map, const void* base, uint64_t rows, uint64_t cols, uint64_t ld,
                        uint32_t box_rows, uint32_t box_cols, int elem_size) {
  EncodeTiledFn fn = encode_tiled_fn();
  if (!fn) return -1;
  if ((reinterpret_cast<uintptr_t>(base) & 15) || ((ld * elem_size) & 15) || box_cols * elem_size != 128 ||
      box_rows == 0 || box_rows > 256)
    return -2;
  cuuint64_t dims[2] = {cols, rows};
  cuuint64_t strides[1] = {ld * uint64_t(elem_size)};
  cuuint32_t box[2] = {box_cols, box_rows};
  cuuint32_t estr[2] = {1, 1};
  CUtensorMapDataType dt = elem_size == 2 ? CU_TENSOR_MAP_DATA_TYPE_UINT16 : CU_TENSOR_MAP_DATA_TYPE_UINT8;
  CUresult r = fn(map, dt, 2, const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                  CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_128B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return r == CUDA_SUCCESS ? 0 : -3;
}

}  // namespace ronn
