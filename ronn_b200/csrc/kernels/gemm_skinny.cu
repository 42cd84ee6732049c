// GEMM for few activation rows:  C[M,N] = act(norm(A)[M,K] * W[N,K]^T + bias) + residual, M up to a few tens.
//
// With one or a few rows a projection is a stream of its weights, and the tcgen05 kernel is bound by its own set-up:
// barriers, TMEM, a TMA ring, the accumulator hand-over.  Here every warp loads weights straight into the registers
// that the matrix instruction reads, no shared memory in between:
//
//   * mma.m16n8k16 with the activations as the 16-row operand and 8 weight rows as the 8-column operand.  The order of
//     the K index inside a product is free as long as both operands share it: lane (g, t) takes the 8 consecutive
//     values k = 32 c + 8 t .. + 7 of weight row g (one 16-byte load, 64 contiguous bytes per row and instruction) and
//     the same values of activation rows g and g + 8.  Words 0 and 1 feed one instruction, words 2 and 3 the next.
//   * The 8 warps of a CTA split K in 64-value pieces and add their sums through shared memory once per tile of 8 R
//     weight rows.  A CTA walks tiles (tile = blockIdx.x, += gridDim.x) with the next piece of the stream in flight.
//   * Weights never depend on the previous kernel of the stream: the first two pieces are requested before the
//     dependency wait, so the stream runs under the predecessor's tail.
//   * K <= 1024 (RES): a warp's share of the activations stays in registers for all tiles, and LayerNorm / RMSNorm can
//     be applied to it on the way in (every CTA normalises the rows again: 2 KB per row from L2 instead of a launch).
//
// More than 16 rows run as slices of 16 rows (blockIdx.y), which read the weights again from L2.
#include "common.cuh"

namespace ronn {

constexpr int SK_WARPS = 8;
constexpr int SK_THREADS = SK_WARPS * 32;
constexpr int SK_CH = 4;                       // 32-value pieces of K per warp and step (two neighbouring pairs)
constexpr int SK_STEP_K = SK_WARPS * SK_CH * 32;   // K values of a step of the CTA: 1024
constexpr int SK_NORM_ROWS = 8;                // rows of a call with a fused norm: with 16 the statistics and the
                                               // normalisation of both halves cost more than the norm kernel's launch

struct SkinnyArgs {
  const void* A;
  const void* W;
  void* C;
  const void* bias;        // [N] or null
  const void* residual;    // [M, ldc] or null
  const void* gamma;       // [K] (NORM != 0)
  const void* beta;        // [K] or null
  float eps;
  int M, N, K;
  long lda, ldw, ldc;
  int act, out_fp32;
};

template <class T>
__device__ __forceinline__ void mma_16x8x16(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                            uint32_t b1);
template <>
__device__ __forceinline__ void mma_16x8x16<__nv_bfloat16>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                           uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
template <>
__device__ __forceinline__ void mma_16x8x16<__half>(float (&d)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3,
                                                    uint32_t b0, uint32_t b1) {
  asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
               : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
               : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// streamed once: no reason to keep the line in L1
__device__ __forceinline__ uint4 ld_stream16(const void* p) {
  uint4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.u32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w)
               : "l"(p));
  return v;
}

// MH: 8-row halves of the activation operand that hold rows (1: M <= 8, 2: up to 16 rows per CTA).
// R: groups of 8 weight rows per tile.  RES: K <= 1024, the activations stay in registers.  NORM (RES only): 0 none,
// 1 LayerNorm, 2 RMSNorm over the K values of a row, rounded to T as the stand-alone norm kernel stores it.
template <class T, int MH, int R, bool RES, int NORM>
__global__ void __launch_bounds__(SK_THREADS, 2) gemm_skinny_kernel(const SkinnyArgs p) {
  static_assert(RES || (NORM == 0 && R == 1), "the streamed form has no norm and one row group");
  constexpr int COLS = 8 * R;
  __shared__ float2 red[2][SK_WARPS][MH * 8][COLS / 2 + 1];
  __shared__ float stat[2][SK_WARPS][16];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int g = lane >> 2, t = lane & 3;
  const T* const W = static_cast<const T*>(p.W);
  const int tiles = (p.N + COLS - 1) / COLS;
  const int nb = RES ? 1 : (p.K + SK_STEP_K - 1) / SK_STEP_K;
  const int own = (tiles - int(blockIdx.x) + int(gridDim.x) - 1) / int(gridDim.x);   // tiles of this CTA, >= 1
  const int items = own * nb;
  const int m0 = int(blockIdx.y) * 16;

  // first K value of this lane's piece c in step b: 64-value pairs go round the warps
  auto k_of = [&](int b, int c) { return b * SK_STEP_K + (c >> 1) * (SK_WARPS * 64) + warp * 64 + (c & 1) * 32 + t * 8; };
  auto load_w = [&](uint4 (&w)[R][SK_CH], int item) {
    const int tile = int(blockIdx.x) + (RES ? item : item / nb) * int(gridDim.x);
    const int b = RES ? 0 : item % nb;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int n = tile * COLS + r * 8 + g;
      const T* row = W + long(n) * p.ldw;
#pragma unroll
      for (int c = 0; c < SK_CH; ++c) {
        const int k = k_of(b, c);
        w[r][c] = (item < items && n < p.N && k < p.K) ? ld_stream16(row + k) : make_uint4(0, 0, 0, 0);
      }
    }
  };
  const T* arow[MH];
  bool alive[MH];
#pragma unroll
  for (int h = 0; h < MH; ++h) {
    const int m = m0 + g + 8 * h;
    alive[h] = m < p.M;
    arow[h] = static_cast<const T*>(p.A) + long(alive[h] ? m : 0) * p.lda;
  }
  auto load_a = [&](uint4 (&a)[SK_CH][MH], int b) {
#pragma unroll
    for (int c = 0; c < SK_CH; ++c) {
      const int k = k_of(b, c);
#pragma unroll
      for (int h = 0; h < MH; ++h)
        a[c][h] = (alive[h] && k < p.K) ? *reinterpret_cast<const uint4*>(arow[h] + k) : make_uint4(0, 0, 0, 0);
    }
  };

  uint4 w0[R][SK_CH], w1[R][SK_CH];
  load_w(w0, 0);
  load_w(w1, 1);
  uint4 gm[NORM ? SK_CH : 1], bt[NORM ? SK_CH : 1];
  if constexpr (NORM != 0) {
#pragma unroll
    for (int c = 0; c < SK_CH; ++c) {
      const int k = k_of(0, c);
      gm[c] = k < p.K ? *reinterpret_cast<const uint4*>(static_cast<const T*>(p.gamma) + k) : make_uint4(0, 0, 0, 0);
      bt[c] = (p.beta && k < p.K) ? *reinterpret_cast<const uint4*>(static_cast<const T*>(p.beta) + k) : make_uint4(0, 0, 0, 0);
    }
  }
  pdl_wait();
  pdl_trigger();
  uint4 a0[SK_CH][MH], a1[RES ? 1 : SK_CH][MH];
  load_a(a0, 0);

  if constexpr (NORM != 0) {
    // sum over the row of f(x): lanes t of a row, then the 8 warps
    auto row_sum = [&](float (&s)[MH], int slot) {
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        s[h] += __shfl_xor_sync(0xffffffffu, s[h], 1);
        s[h] += __shfl_xor_sync(0xffffffffu, s[h], 2);
        if (t == 0) stat[slot][warp][g + 8 * h] = s[h];
      }
      __syncthreads();
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        s[h] = 0.f;
#pragma unroll
        for (int w = 0; w < SK_WARPS; ++w) s[h] += stat[slot][w][g + 8 * h];
      }
    };
    float mean[MH], inv[MH], s[MH];
#pragma unroll
    for (int h = 0; h < MH; ++h) mean[h] = s[h] = 0.f;
    if (NORM == 1) {
#pragma unroll
      for (int c = 0; c < SK_CH; ++c)
#pragma unroll
        for (int h = 0; h < MH; ++h) {
          float f[8];
          unpack8<T>(*reinterpret_cast<const Vec8*>(&a0[c][h]), f);
#pragma unroll
          for (int i = 0; i < 8; ++i) s[h] += f[i];
        }
      row_sum(s, 0);
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        mean[h] = s[h] / float(p.K);
        s[h] = 0.f;
      }
    }
#pragma unroll
    for (int c = 0; c < SK_CH; ++c)
      if (k_of(0, c) < p.K) {
#pragma unroll
        for (int h = 0; h < MH; ++h) {
          float f[8];
          unpack8<T>(*reinterpret_cast<const Vec8*>(&a0[c][h]), f);
#pragma unroll
          for (int i = 0; i < 8; ++i) s[h] += (f[i] - mean[h]) * (f[i] - mean[h]);
        }
      }
    row_sum(s, 1);
#pragma unroll
    for (int h = 0; h < MH; ++h) inv[h] = rsqrtf(s[h] / float(p.K) + p.eps);
#pragma unroll
    for (int c = 0; c < SK_CH; ++c) {
      float ga[8], be[8];
      unpack8<T>(*reinterpret_cast<const Vec8*>(&gm[c]), ga);
      unpack8<T>(*reinterpret_cast<const Vec8*>(&bt[c]), be);
#pragma unroll
      for (int h = 0; h < MH; ++h) {
        float f[8];
        unpack8<T>(*reinterpret_cast<const Vec8*>(&a0[c][h]), f);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          f[i] = (f[i] - mean[h]) * inv[h] * ga[i];
          if (p.beta) f[i] += be[i];
        }
        const Vec8 v = pack8<T>(f);
        a0[c][h] = *reinterpret_cast<const uint4*>(&v);
      }
    }
  }

  float acc[R][4];
  int seen = 0;                                  // tiles finished: parity of the exchange buffer
  auto step = [&](const uint4 (&w)[R][SK_CH], const uint4 (&a)[SK_CH][MH], int item) {
    const int b = RES ? 0 : item % nb;
    if (b == 0) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < 4; ++i) acc[r][i] = 0.f;
    }
#pragma unroll
    for (int c = 0; c < SK_CH; ++c) {
      const uint4 lo = a[c][0];
      const uint4 hi = MH == 2 ? a[c][MH - 1] : make_uint4(0, 0, 0, 0);
#pragma unroll
      for (int r = 0; r < R; ++r) mma_16x8x16<T>(acc[r], lo.x, hi.x, lo.y, hi.y, w[r][c].x, w[r][c].y);
#pragma unroll
      for (int r = 0; r < R; ++r) mma_16x8x16<T>(acc[r], lo.z, hi.z, lo.w, hi.w, w[r][c].z, w[r][c].w);
    }
  };
  // sums of the 8 warps -> bias, activation, residual, store.  Two exchange buffers: the barrier of the next tile
  // separates the readers of this one from the writers of the one after.
  auto finish = [&](int item) {
    const int n0 = (int(blockIdx.x) + (RES ? item : item / nb) * int(gridDim.x)) * COLS;
    auto& buf = red[seen & 1];
    ++seen;
#pragma unroll
    for (int r = 0; r < R; ++r) {
      buf[warp][g][r * 4 + t] = make_float2(acc[r][0], acc[r][1]);
      if (MH == 2) buf[warp][g + 8 * (MH - 1)][r * 4 + t] = make_float2(acc[r][2], acc[r][3]);
    }
    __syncthreads();
    constexpr int OUT = MH * 8 * COLS;
#pragma unroll
    for (int o = threadIdx.x; o < OUT; o += SK_THREADS) {
      const int row = o / COLS, col = o - row * COLS;
      const int m = m0 + row, n = n0 + col;
      if (m < p.M && n < p.N) {
        const float add = p.bias ? Cvt<T>::to_f(static_cast<const T*>(p.bias)[n]) : 0.f;
        const float res = p.residual ? Cvt<T>::to_f(static_cast<const T*>(p.residual)[long(m) * p.ldc + n]) : 0.f;
        float v = 0.f;
#pragma unroll
        for (int w = 0; w < SK_WARPS; ++w) v += reinterpret_cast<const float*>(&buf[w][row][0])[col];
        v += add;
        if (p.act == 1) v = fmaxf(v, 0.f);
        else if (p.act == 2) v = gelu_tanh_f(v);
        v += res;
        if (p.out_fp32) static_cast<float*>(p.C)[long(m) * p.ldc + n] = v;
        else static_cast<T*>(p.C)[long(m) * p.ldc + n] = Cvt<T>::from_f(v);
      }
    }
  };

  for (int i = 0; i < items; i += 2) {
    if constexpr (RES) {
      step(w0, a0, i);
      load_w(w0, i + 2);
      finish(i);
      if (i + 1 < items) {
        step(w1, a0, i + 1);
        load_w(w1, i + 3);
        finish(i + 1);
      }
    } else {
      load_a(a1, (i + 1) % nb);
      step(w0, a0, i);
      load_w(w0, i + 2);
      if (i % nb == nb - 1) finish(i);
      if (i + 1 < items) {
        load_a(a0, (i + 2) % nb);
        step(w1, a1, i + 1);
        load_w(w1, i + 3);
        if ((i + 1) % nb == nb - 1) finish(i + 1);
      }
    }
  }
}

template <class T, int MH, int R, bool RES, int NORM>
static int launch_skinny(const SkinnyArgs& a, cudaStream_t stream) {
  const int tiles = (a.N + 8 * R - 1) / (8 * R);
  const int resident = 2 * device_sm_count();
  const int slices = (a.M + 15) / 16;
  const dim3 grid(unsigned(tiles < resident ? tiles : resident), unsigned(slices));
  const cudaError_t err = launch(gemm_skinny_kernel<T, MH, R, RES, NORM>, grid, dim3(SK_THREADS), 0, stream, a);
  return (err == cudaSuccess && cudaGetLastError() == cudaSuccess) ? 0 : -11;
}

// Two row groups per tile (twice the bytes in flight, half the exchanges) once one group per tile would give every CTA
// of a full grid several tiles anyway.
static bool wide_tiles(int N) { return (N + 7) / 8 > 4 * device_sm_count(); }

template <class T, int NORM>
static int dispatch_skinny(const SkinnyArgs& a, cudaStream_t stream) {
  const bool one = a.M <= 8;
  if constexpr (NORM != 0) {
    if (!one || a.K > SK_STEP_K) return -2;
    return wide_tiles(a.N) ? launch_skinny<T, 1, 2, true, NORM>(a, stream) : launch_skinny<T, 1, 1, true, NORM>(a, stream);
  } else {
    if (a.K > SK_STEP_K) return one ? launch_skinny<T, 1, 1, false, 0>(a, stream) : launch_skinny<T, 2, 1, false, 0>(a, stream);
    if (one) return wide_tiles(a.N) ? launch_skinny<T, 1, 2, true, 0>(a, stream) : launch_skinny<T, 1, 1, true, 0>(a, stream);
    return wide_tiles(a.N) ? launch_skinny<T, 2, 2, true, 0>(a, stream) : launch_skinny<T, 2, 1, true, 0>(a, stream);
  }
}

// Whether the skinny kernel takes a plain projection of this size from the tcgen05 kernel.
//
// Up to 16 rows it reads the weights once and wins (N 10 to 50257, K 64 to 8192), but for 9 to 16 rows against matrices of
// 64 Mi values and more that the other kernel holds in one wave: 12 x 8192 x 8192 40 / 37 us, 16 x 16384 x 4096 37 / 28.
// What it still loses there: 16 x 32000 x 4096 69 / 51, 8 x 16384 x 8192 63 / 52, 12 x 32000 x 1536 35 / 29, 16 x 16384 x 1536 20 /
// 17, 1 x 50257 x 1536 51 / 44, 1 x 50257 x 256 11.9 / 10.5.
// K of up to 128 gives one or two of the 8 warps weights to read: the vocabulary of a very narrow model, behind its norm kernel,
// is left to tcgen05 (1 to 8 x 50257 x 64 11.2 / 8.7 with the norm, x 32000 x 128 8.8 / 8.1; x 16384 x 64 stays, 5.6 / 7.0).
//
// Beyond that every further 16 rows read the weights again, and the two are compared by what they cost, in microseconds of a
// chain inside a CUDA graph, weights from DRAM (1390 sizes: M 17 to 96, N 10 to 50257, K 64 to 8192, bf16):
//   skinny   1.1 + waves of CTAs x (0.6 + 0.24 per 8 weight rows of a CTA) + 0.46 per million weights and slice
//   tcgen05  3.15 + 0.23 per K block + 0.23 per million weights, and when the tiles are more than the SMs
//            5.6 per further wave of two tiles per SM + 0.36 per K block and wave
// Where it names the skinny kernel the other is at most 9 % faster; where it names the other, 15 sizes of N 3072 and more and
// K 512 to 1536 would be 5 to 24 % faster here (40 x 3072 x 1024 7.8 / 9.2, 17 x 50257 x 1024 35 / 43).  By weights and slices alone (a line at 12 Mi values) short K went to the wrong side: 96 x 16384 x 64 19.7 / 5.2 us, 64 x 3072
// x 1024 10.1 / 7.5, and long K stayed on it: 64 x 1024 x 4096 11.9 / 18.7.
//   us, skinny / tcgen05   N 3072 K 1024   N 1024 K 1024   N 768 K 768   N 1024 K 4096   N 8192 K 256
//   M  1                     3.6 / 10.7      2.0 / 7.1      1.9 / 6.1      5.3 / 18.6      3.0 / 5.2
//     16                     3.8 / 10.1      2.4 / 7.0      2.1 / 6.0      6.2 / 18.5      3.3 / 5.1
//     32                     6.0 / 9.4       2.8 / 7.0      2.5 / 6.0      7.0 / 18.5      5.5 / 5.0
//     48                     8.2 / 8.8       4.5 / 7.2      2.5 / 6.1     11.5 / 18.6      7.5 / 5.0
//     64                    10.1 / 7.5       4.7 / 7.0      4.1 / 6.0     11.9 / 18.7      9.7 / 5.0
//     96                    14.3 / 7.7       6.6 / 7.0      4.3 / 6.2     16.7 / 18.7     13.8 / 5.0
int pick_bn(int M, int N);                     // gemm_umma.cu: tile width of the tcgen05 kernel for few rows
bool skinny_rule(int M, int N, int K) {
  if (M > 96 || (K <= 128 && N > 24576)) return false;
  if (M <= 8) return true;
  const int sms = device_sm_count(), bn = pick_bn(M, N);
  const int tiles = (N + bn - 1) / bn;
  const float mega = float(N) * float(K) * 1e-6f;
  if (M <= 16) return tiles > sms || mega < 67.1f;
  const int slices = (M + 15) / 16, groups = K <= SK_STEP_K && wide_tiles(N) ? 2 : 1;
  const int sk_tiles = (N + 8 * groups - 1) / (8 * groups), grid = sk_tiles < 2 * sms ? sk_tiles : 2 * sms;
  const int waves = (grid * slices + 2 * sms - 1) / (2 * sms), own = (sk_tiles + grid - 1) / grid;
  // past the register-resident limit a step is 1024 values of K, whole or not
  const float padded = K <= SK_STEP_K ? 1.f : float((K + SK_STEP_K - 1) / SK_STEP_K * SK_STEP_K) / float(K);
  const float skinny = 1.1f + float(waves) * (0.6f + 0.24f * float(own * groups)) + 0.46f * float(slices) * mega * padded;
  const float kb = float((K + 63) / 64);
  float umma = 3.15f + 0.23f * kb + 0.23f * mega;
  if (tiles > sms) {
    const float w = float((tiles + 2 * sms - 1) / (2 * sms));
    umma += 5.6f * (w - 1.f) + 0.36f * kb * w;
  }
  return skinny < umma;
}

}  // namespace ronn

using namespace ronn;

// Whether a projection whose result a norm reads next is faster as one skinny GEMM followed by the norm kernel than as four
// K slices on tcgen05 whose reduction applies the norm: where a plain GEMM takes the skinny kernel and its CTAs run as one
// wave, or up to 16 rows against 8 Mi weights.  Measured, us with the norm, skinny / slices: 16 x 1024 x 4096 8.3 / 10.2, 32 x
// 1024 x 4096 9.5 / 10.2, 48 x 768 x 2048 7.0 / 8.5, 64 x 512 x 8192 13.1 / 14.1; past one wave 48 x 1024 x 2048 9.3 / 8.3,
// 80 x 512 x 4096 11.4 / 10.4, 32 x 2048 x 2048 10.7 / 8.8; not skinny at all (few unsliced tiles): 128 x 256 x 2048 13.4 / 9.2.
extern "C" int ronn_skinny_down_ok(int M, int N, int K) {
  if (M <= 0 || N <= 0 || K <= 0 || !skinny_rule(M, N, K)) return 0;
  return long((M + 15) / 16) * ((N + 7) / 8) <= 2 * device_sm_count() || (M <= 16 && long(N) * K <= (8l << 20));
}

// out[M,N] = act(norm(A)[M,K] W[N,K]^T + bias) + residual for few rows.  norm: 0 none, 1 LayerNorm, 2 RMSNorm over K
// (K <= 1024; gamma, and for LayerNorm optionally beta).  dtype 0 bf16, 1 fp16; act 0 none, 1 relu, 2 gelu(tanh).
// K, lda and ldw multiples of 8; A, W, gamma and beta 16-byte aligned.  M at most 16 x 65535.
extern "C" int ronn_gemm_skinny(const void* A, const void* W, void* C, const void* bias, const void* residual,
                                const void* gamma, const void* beta, float eps, int norm, int M, int N, int K, long lda,
                                long ldw, long ldc, int dtype, int act, int out_fp32, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || M > 16 * 65535) return -1;
  if ((K & 7) || (lda & 7) || (ldw & 7)) return -2;
  if ((reinterpret_cast<uintptr_t>(A) | reinterpret_cast<uintptr_t>(W)) & 15) return -22;
  if (norm < 0 || norm > 2 || (norm && (K > SK_STEP_K || !gamma))) return -2;
  if (norm && M > SK_NORM_ROWS) return -2;
  if (norm && ((reinterpret_cast<uintptr_t>(gamma) | reinterpret_cast<uintptr_t>(beta)) & 15)) return -22;
  const SkinnyArgs a{A, W, C, bias, residual, gamma, beta, eps, M, N, K, lda, ldw, ldc, act, out_fp32};
#define RONN_SK(T) (norm == 0 ? dispatch_skinny<T, 0>(a, stream) : norm == 1 ? dispatch_skinny<T, 1>(a, stream) : dispatch_skinny<T, 2>(a, stream))
  if (dtype == 0) return RONN_SK(__nv_bfloat16);
  if (dtype == 1) return RONN_SK(__half);
  return -1;
#undef RONN_SK
}
