// Epilogue shared by the dense GEMM and the implicit-GEMM convolution: bias, activation, residual, store.
#pragma once
#include "common.cuh"

namespace ronn {

// Second launch bound of a kernel that runs `per_sm` CTAs per SM: 0 (no bound) for one.
constexpr int min_blocks(int per_sm) { return per_sm > 1 ? per_sm : 0; }

// CTAs of a kernel that one SM of the current device holds by registers (whole groups of 8 per thread) and shared memory, or a
// negative error.  cudaOccupancyMaxActiveBlocksPerMultiprocessor answers 1 for every kernel that uses TMEM.
template <class Kernel>
int resident_ctas(Kernel kern, int threads, int dyn_smem) {
  cudaFuncAttributes a;
  int dev = 0, regs = 0, smem = 0, reserved = 0;
  if (cudaFuncGetAttributes(&a, kern) != cudaSuccess || cudaGetDevice(&dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&regs, cudaDevAttrMaxRegistersPerMultiprocessor, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&smem, cudaDevAttrMaxSharedMemoryPerMultiprocessor, dev) != cudaSuccess ||
      cudaDeviceGetAttribute(&reserved, cudaDevAttrReservedSharedMemoryPerBlock, dev) != cudaSuccess)
    return -12;
  const int by_regs = regs / ((a.numRegs + 7) / 8 * 8 * threads), by_smem = smem / (dyn_smem + int(a.sharedSizeBytes) + reserved);
  return by_regs < by_smem ? by_regs : by_smem;
}

struct DenseEpilogue {
  void* C;
  const void* bias;        // [N] in the operand dtype, or null
  const void* residual;    // [M, ldc] in the operand dtype, or null
  int M, N, ldc;
  int m0, n0;
  int act;                 // 0 none, 1 relu, 2 gelu(tanh)
  int out_fp32;
  int res_first;           // 1: add the residual before the activation (convolution blocks), 0: after it

  // `stage` (optional): 32 x 80 bytes of shared memory owned by the calling warp.  With it, and when the whole warp
  // calls with the same `col`, 16-bit results leave as 64 contiguous bytes per row from 4 lanes (8 rows per store
  // instruction) instead of 32 rows of 16 bytes, which halves the number of write transactions and fills every sector.
  // EARLY: the residual row is fetched before the bias and the activation, which hides its latency and costs 16 registers.  Forms
  // that run two CTAs per SM cannot pay them (102 registers per thread) and hide it behind the other CTA: with the early fetch the
  // shallow 128-wide GEMM and the 64-wide gather convolution went from 96 to 132 registers and ran one CTA per SM (norm + 1 x 32000
  // x 64: 6.9 -> 9.9 us).
  template <class T, bool EARLY = true>
  __device__ __forceinline__ void run(int row, int col, uint32_t (&r)[32], uint8_t* stage = nullptr) const {
    const int gm = m0 + row;
    const int gn = n0 + col;
    if (gn >= N) return;                         // uniform across the warp
    // re-shaping the stores through shared memory pays for bandwidth-bound results; a decode-sized GEMM (a few row
    // tiles) is a latency chain and keeps the direct stores
    const bool staged = stage != nullptr && M >= 1024 && !out_fp32 && (gn + 32 <= N) && ((ldc & 7) == 0);
    const bool ragged = stage != nullptr && !out_fp32 && (ldc & 7) != 0;
    if (gm >= M && !staged && !ragged) return;
    if (gm >= M) {                               // staged paths: rows past the end only take part in the exchange
      __syncwarp();
      if (staged) store_staged<T>(stage, gm - (threadIdx.x & 31), gn);
      else store_ragged<T>(stage, gm - (threadIdx.x & 31), gn);
      return;
    }
    float v[32];
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
    const bool full = (gn + 32 <= N) && ((ldc & 7) == 0);
    Vec8 rp[EARLY ? 4 : 1];
    if (EARLY && residual && full) {
      const T* res = reinterpret_cast<const T*>(residual) + size_t(gm) * ldc + gn;
#pragma unroll
      for (int j = 0; j < (EARLY ? 4 : 0); ++j) rp[j] = *reinterpret_cast<const Vec8*>(res + j * 8);
    }
    auto add_residual = [&]() {
      if (full) {
        const T* res = reinterpret_cast<const T*>(residual) + size_t(gm) * ldc + gn;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float f[8];
          unpack8<T>(EARLY ? rp[EARLY ? j : 0] : *reinterpret_cast<const Vec8*>(res + j * 8), f);
#pragma unroll
          for (int i = 0; i < 8; ++i) v[j * 8 + i] += f[i];
        }
      } else {
        const T* res = reinterpret_cast<const T*>(residual) + size_t(gm) * ldc + gn;
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (gn + i < N) v[i] += Cvt<T>::to_f(res[i]);
      }
    };
    if (bias) {
      const T* b = reinterpret_cast<const T*>(bias) + gn;
      if (gn + 32 <= N && (reinterpret_cast<uintptr_t>(b) & 15) == 0) {      // four 16-byte loads instead of 32 of two bytes
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float f[8];
          unpack8<T>(*reinterpret_cast<const Vec8*>(b + j * 8), f);
#pragma unroll
          for (int i = 0; i < 8; ++i) v[j * 8 + i] += f[i];
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (gn + i < N) v[i] += Cvt<T>::to_f(b[i]);
      }
    }
    if (residual && res_first) add_residual();
    if (act == 1) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = fmaxf(v[i], 0.f);
    } else if (act == 2) {
#pragma unroll
      for (int i = 0; i < 32; ++i) v[i] = gelu_tanh_f(v[i]);
    }
    if (residual && !res_first) add_residual();
    if (out_fp32) {
      float* out = reinterpret_cast<float*>(C) + size_t(gm) * ldc + gn;
      if (full && (ldc & 3) == 0) {
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<float4*>(out + j * 4) = make_float4(v[j * 4], v[j * 4 + 1], v[j * 4 + 2], v[j * 4 + 3]);
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (gn + i < N) out[i] = v[i];
      }
    } else if (staged || ragged) {
      uint8_t* mine = stage + (threadIdx.x & 31) * 80;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        float f[8];
#pragma unroll
        for (int i = 0; i < 8; ++i) f[i] = v[j * 8 + i];
        *reinterpret_cast<Vec8*>(mine + j * 16) = pack8<T>(f);
      }
      __syncwarp();
      if (staged) store_staged<T>(stage, gm - (threadIdx.x & 31), gn);
      else store_ragged<T>(stage, gm - (threadIdx.x & 31), gn);
    } else {
      T* out = reinterpret_cast<T*>(C) + size_t(gm) * ldc + gn;
      if (full) {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          float f[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) f[i] = v[j * 8 + i];
          *reinterpret_cast<Vec8*>(out + j * 8) = pack8<T>(f);
        }
      } else {
#pragma unroll
        for (int i = 0; i < 32; ++i)
          if (gn + i < N) out[i] = Cvt<T>::from_f(v[i]);
      }
    }
  }

  // second half of the staged store: lane l writes 16-byte piece (l % 4) of rows (l / 4) + 8 i
  template <class T>
  __device__ __forceinline__ void store_staged(const uint8_t* stage, int base_row, int gn) const {
    const int lane = threadIdx.x & 31;
    const int piece = lane & 3;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int rr = (lane >> 2) + 8 * i;
      if (base_row + rr < M) {
        const Vec8 pk = *reinterpret_cast<const Vec8*>(stage + rr * 80 + piece * 16);
        *reinterpret_cast<Vec8*>(reinterpret_cast<T*>(C) + size_t(base_row + rr) * ldc + gn + piece * 8) = pk;
      }
    }
    __syncwarp();                                // the stage is free for the warp's next chunk
  }

  // The same for rows that do not start on 16-byte boundaries (ldc not a multiple of 8): lane l writes column gn + l,
  // so a store instruction covers one run of 64 bytes of one row.  Stored from the accumulator layout (lane = row) each
  // instruction touched 32 rows, two bytes in each.
  template <class T>
  __device__ __forceinline__ void store_ragged(const uint8_t* stage, int base_row, int gn) const {
    const int lane = threadIdx.x & 31;
    const int rows = min(32, M - base_row);
    if (gn + lane < N) {
      T* dst = reinterpret_cast<T*>(C) + size_t(base_row) * ldc + gn + lane;
#pragma unroll 8
      for (int i = 0; i < rows; ++i) dst[size_t(i) * ldc] = *reinterpret_cast<const T*>(stage + i * 80 + lane * 2);
    }
    __syncwarp();
  }
};

}  // namespace ronn
