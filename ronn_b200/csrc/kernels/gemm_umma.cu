// Dense bf16/fp16 GEMM on tcgen05 tensor cores:  C[M,N] = act(A[M,K] * W[N,K]^T + bias) + residual.
//
// A is row-major activations, W is stored K-major ("[N,K]", the transposed form of an ONNX MatMul
// weight), so both operands are K-major UMMA tiles loaded by TMA with the 128-byte swizzle.  The
// accumulator lives in TMEM; the epilogue applies bias, activation (none / ReLU / tanh-GELU) and an
// optional residual add and writes bf16/fp16 or fp32.
//
// Replaces the reference's library matmul (crates/ronn-core/src/ops/matrix.rs:27-60) and its two
// never-compiled templates: the scalar fused matmul+bias and the one-wmma-tile-per-warp GEMM
// (crates/ronn-providers/src/gpu/cuda_kernels.rs:319-347, 479-534).
#include <stdlib.h>

#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "tma_desc.cuh"
#include "umma_pair.cuh"
#include "umma_persistent.cuh"

namespace ronn {

// Tile list of a dense (optionally split-K) GEMM for the persistent mainloop.  Tiles are numbered with the
// M index fastest so that CTAs running side by side share the same weight tile in L2.
template <int BN, class T, bool EARLY>
struct DenseProblem {
  static constexpr bool kForceStage = false;
  const CUtensorMap* map_a;
  const CUtensorMap* map_b;
  DenseEpilogue e;
  int m_tiles, n_tiles, num_kb, splitk, kb_per;

  __device__ __forceinline__ int num_tiles() const { return m_tiles * n_tiles * splitk; }
  __device__ __forceinline__ void tile(int t, int& m0, int& n0, int& kb0, int& nkb) const {
    const int per_z = m_tiles * n_tiles;
    const int z = t / per_z, r = t - z * per_z;
    m0 = (r % m_tiles) * PG_BM;
    n0 = (r / m_tiles) * BN;
    kb0 = z * kb_per;
    nkb = min(kb_per, num_kb - kb0);
  }
  __device__ __forceinline__ void load_a(uint8_t* smem, uint64_t* bar, int k_elem, int m0) const {
    tma_load_2d(smem, map_a, bar, k_elem, m0);
  }
  __device__ __forceinline__ void load_b(uint8_t* smem, uint64_t* bar, int k_elem, int n0) const {
    tma_load_2d(smem, map_b, bar, k_elem, n0);
  }
  __device__ __forceinline__ void epilogue(int t, int m0, int n0, int row, int col, uint32_t (&r)[32], uint8_t* stage) const {
    DenseEpilogue ep = e;
    ep.m0 = m0;
    ep.n0 = n0;
    if (splitk > 1)     // raw fp32 partial sums go to slice z of the workspace
      ep.C = reinterpret_cast<float*>(e.C) + size_t(t / (m_tiles * n_tiles)) * size_t(e.M) * size_t(e.ldc);
    ep.run<T, EARLY>(row, col, r, stage);
  }
};

template <int BN, int STAGES, class T, int KA>
__global__ void __launch_bounds__(PG_THREADS, min_blocks(PGemmSmem<BN, STAGES, false, KA>::PER_SM))
gemm_dense_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                  DenseEpilogue epi, int K, int splitk, uint32_t idesc, uint32_t* status) {
  extern __shared__ uint8_t dyn_smem[];
  using Problem = DenseProblem<BN, T, PGemmSmem<BN, STAGES, false, KA>::PER_SM == 1>;
  Problem prob;
  prob.map_a = &map_a;
  prob.map_b = &map_b;
  prob.e = epi;
  prob.m_tiles = (epi.M + PG_BM - 1) / PG_BM;
  prob.n_tiles = (epi.N + BN - 1) / BN;
  prob.num_kb = (K + 63) / 64;
  prob.splitk = splitk;
  prob.kb_per = (prob.num_kb + splitk - 1) / splitk;
  gemm_persistent<BN, STAGES, 0, Problem, KA>(dyn_smem, prob, 64, idesc, status);
}

static int sm_count() { return device_sm_count(); }

// The same problem on CTA pairs: tiles of 256 x BN, M index fastest.
template <int BN, class T>
struct DensePairProblem {
  static constexpr bool kConstB = true;
  const CUtensorMap* map_a;
  const CUtensorMap* map_b;
  PairOut out;
  int m_tiles, n_tiles, num_kb;

  __device__ __forceinline__ float row_scale(int) const { return 1.f; }
  __device__ __forceinline__ int num_tiles() const { return m_tiles * n_tiles; }
  __device__ __forceinline__ void tile(int t, int& m0, int& n0) const {
    const int n = t / m_tiles;
    m0 = (t - n * m_tiles) * 256;
    n0 = n * BN;
  }
  __device__ __forceinline__ void load_a(uint8_t* smem, uint32_t bar, int k, int m) const { tma_load_2d_pair(smem, map_a, bar, k, m); }
  __device__ __forceinline__ void load_b(uint8_t* smem, uint32_t bar, int k, int n) const { tma_load_2d_pair(smem, map_b, bar, k, n); }
};

template <int BN, int STAGES, class T>
__global__ void __launch_bounds__(PP_THREADS)
gemm_pair_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                 const __grid_constant__ CUtensorMap map_c, const __grid_constant__ CUtensorMap map_r, DenseEpilogue epi,
                 int by_tma, int K, uint32_t idesc, uint32_t* status) {
  extern __shared__ uint8_t dyn_smem[];
  DensePairProblem<BN, T> prob{&map_a, &map_b, {&map_c, &map_r, epi, by_tma}, (epi.M + 255) / 256, (epi.N + BN - 1) / BN, (K + 63) / 64};
  gemm_pair<BN, STAGES, 0, T>(dyn_smem, prob, idesc, status);
}

template <int BN, int STAGES, class T>
static int launch_pair(const CUtensorMap& ma, const CUtensorMap& mb, DenseEpilogue epi, int M, int N, int K, int is_bf16,
                       uint32_t* status, cudaStream_t stream) {
  using L = PairSmem<BN, STAGES>;
  auto kern = gemm_pair_kernel<BN, STAGES, T>;
  static bool configured[MAX_DEVICES] = {false};
  if (first_use_on_device(configured)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::DYN_SMEM) != cudaSuccess) return -10;
  }
  CUtensorMap mc = ma, mr = ma;
  const int by_tma = pair_out_maps(epi, 2, &mc, &mr);
  const int tiles = ((N + BN - 1) / BN) * ((M + 255) / 256), pairs = sm_count() / 2;
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(2 * unsigned(tiles < pairs ? tiles : pairs));
  cfg.blockDim = dim3(PP_THREADS);
  cfg.dynamicSmemBytes = size_t(L::DYN_SMEM);
  cfg.stream = stream;
  cudaLaunchAttribute attr[2];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = 2;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
  attr[1].val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = attr;
  cfg.numAttrs = pdl_enabled() ? 2 : 1;
  prefer_max_shared(reinterpret_cast<const void*>(kern));
  const uint32_t idesc = umma_idesc(256, BN, is_bf16 ? 1u : 0u, 1u);
  const cudaError_t err = cudaLaunchKernelEx(&cfg, kern, ma, mb, mc, mr, epi, by_tma, K, idesc, status);
  return (err == cudaSuccess && cudaGetLastError() == cudaSuccess) ? 0 : -11;
}

template <int BN, int STAGES, class T, int KA = 1>
static int launch_dense(const CUtensorMap& ma, const CUtensorMap& mb, DenseEpilogue epi, int M, int N, int K,
                        int is_bf16, uint32_t* status, cudaStream_t stream, int splitk = 1) {
  using L = PGemmSmem<BN, STAGES, false, KA>;
  auto kern = gemm_dense_kernel<BN, STAGES, T, KA>;
  static bool configured[MAX_DEVICES] = {false};
  if (first_use_on_device(configured)) {
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, L::DYN_SMEM) != cudaSuccess) return -10;
  }
  const int tiles = ((N + BN - 1) / BN) * ((M + PG_BM - 1) / PG_BM) * splitk;
  const int resident = sm_count() * L::PER_SM;
  dim3 grid(tiles < resident ? tiles : resident);
  uint32_t idesc = umma_idesc(PG_BM, BN, is_bf16 ? 1u : 0u, 1u);
  cudaError_t err = launch(kern, grid, dim3(PG_THREADS), size_t(L::DYN_SMEM), stream, ma, mb, epi, K, splitk, idesc, status);
  return (err == cudaSuccess && cudaGetLastError() == cudaSuccess) ? 0 : -11;
}

int pick_bn(int M, int N) {
  const int mt = (M + PG_BM - 1) / PG_BM;
  // 256-wide tiles pay off once the problem is compute bound; with one or two row tiles every CTA is a latency
  // chain and narrower tiles spread the weight stream over more SMs (measured: M 256, N 50264, K 1024 takes 36 us
  // with 128-wide tiles against 110 us with 256-wide ones)
  const int cands[4] = {256, 128, 64, 32};
  for (int i = (mt <= 2 ? 1 : 0); i < 4; ++i) {
    int bn = cands[i];
    if (bn > 32 && N < bn) continue;
    int ctas = mt * ((N + bn - 1) / bn);
    if (ctas >= 120) return bn;
  }
  return 32;
}

// The kernel that a call runs: FORM_SKINNY, or the tile width with FORM_DEEP / FORM_SHALLOW (widths of two rings) or
// FORM_CTA_PAIR.
constexpr int FORM_SKINNY = 0x8000, FORM_CTA_PAIR = 0x4000, FORM_SHALLOW = 0x2000, FORM_DEEP = 0x1000;

// What a call costs in each form, in microseconds of a chain inside a CUDA graph:
//   start + K blocks x block + epilogue + (waves - 1) x max(K blocks x block + gap, epilogue + drain)
// `start` (dependency, set-up, first loads) and `block` (64 values of K) have one value while every SM has at most one tile
// and one beyond; the epilogue grows with GELU, a residual, fp32 results and rows off the 16-byte grid, and sets the pace of
// a wave when it is longer than the main loop.  Fitted to 84 000 timed forms of 12 000 calls: bf16, 1024 to 8192 rows and,
// where 128-wide tiles fill the chip, 512 to 1000; N 10 to 8193, K 64 to 4096; plain, ReLU, GELU, residual, both, fp32
// results, odd row lengths.  Mean error of a form 4 to 7 %.  The form it names takes 0.6 % longer than the fastest on average
// and 8 % less than the rule by tile count (pick_bn); 0.7 % of the calls take more than 5 % longer than under that rule,
// odd rows of N 1025 to 4097 at K 2048 the worst (28.6 -> 34.7 us).  On 160 calls of 257, 384 and 640 rows, not fitted: none.
// What it has to weigh, us: 1024 x 64 x 1024 fp32 8.1 at 32 wide, 9.7 at 64 shallow; 1024 x 768 x 2048 12.3 at 64 deep, 14.6
// shallow; 8192 x 2304 x 64 residual 23.8 on pairs, 34.4 at 64; 8192 x 3072 x 768 GELU 43.4 / 55.0 / 52.7 on pairs / 256 / 128;
// 4662 x 50257 x 768 (odd rows) 412 / 627 on pairs / 256.
// The shallow 128-wide entry was measured while its 132 registers let one CTA run per SM where two are launched; with two it
// costs less, so the entry keeps the form from being chosen rather than choosing it wrongly.
struct FormCost {
  int form;
  float start_one, start_more, block_one, block_more, epilogue, gelu, residual, fp32, ragged, gap, drain;
};
static const FormCost form_costs[] = {
    {32 | FORM_SHALLOW, 2.00f, 3.06f, 0.31f, 0.31f, 1.57f, 0.35f, 0.48f, 0.61f, 0.f, 0.44f, 0.19f},
    {32 | FORM_DEEP, 3.21f, 3.21f, 0.25f, 0.25f, 0.93f, 0.38f, 0.27f, 0.22f, 0.71f, 0.41f, 0.17f},
    {64 | FORM_SHALLOW, 2.34f, 3.71f, 0.31f, 0.32f, 1.67f, 0.40f, 0.81f, 1.58f, 0.f, 1.55f, 0.96f},
    {64 | FORM_DEEP, 3.14f, 3.23f, 0.24f, 0.25f, 1.11f, 0.57f, 0.51f, 0.99f, 0.59f, 0.59f, 0.23f},
    {128 | FORM_SHALLOW, 2.60f, 7.31f, 0.33f, 0.72f, 2.96f, 1.35f, 0.90f, 1.75f, 0.f, 1.63f, 2.90f},
    {128 | FORM_DEEP, 4.06f, 4.07f, 0.25f, 0.27f, 1.56f, 1.22f, 1.01f, 2.03f, 1.28f, 1.03f, 1.22f},
    {256, 4.26f, 3.62f, 0.32f, 0.41f, 3.99f, 2.08f, 2.27f, 4.36f, 2.27f, 0.18f, 2.07f},
    {256 | FORM_CTA_PAIR, 4.80f, 4.01f, 0.33f, 0.34f, 2.69f, 1.51f, 0.52f, 0.f, 2.18f, 2.27f, 1.74f},
};
// ring: 1 deep, 0 shallow, -1 either.  Rows off the 16-byte grid leave through the store-staging area, which the shallow
// rings do not carry; a tile more than twice as wide as the result would run mostly empty; pairs write 16 bits.
static int pick_form(int M, int N, int K, int act, bool residual, bool out_fp32, bool ragged, int ring) {
  const int sms = sm_count();
  const float kb = float((K + 63) / 64);
  int best = 0;
  float cost = 1e30f;
  for (const FormCost& f : form_costs) {
    const int bn = f.form & 0xfff;
    const bool pair = (f.form & FORM_CTA_PAIR) != 0, shallow = (f.form & FORM_SHALLOW) != 0;
    if ((bn > 32 && N <= bn / 2) || (pair && out_fp32)) continue;
    if (bn < 256 && (ring >= 0 ? shallow == (ring == 1) : shallow && ragged)) continue;
    const long tiles = long((M + (pair ? 255 : 127)) / (pair ? 256 : 128)) * ((N + bn - 1) / bn);
    const long slots = pair ? sms / 2 : (shallow ? 2 * sms : sms);
    const bool one = tiles <= sms;
    const float epi = f.epilogue + (act == 2 ? f.gelu : 0.f) + (residual ? f.residual : 0.f) + (out_fp32 ? f.fp32 : 0.f) +
                      (ragged ? f.ragged : 0.f);
    const float main = kb * (one ? f.block_one : f.block_more);
    const float wave = main + f.gap > epi + f.drain ? main + f.gap : epi + f.drain;
    const float t = (one ? f.start_one : f.start_more) + main + epi + float((tiles + slots - 1) / slots - 1) * wave;
    if (t < cost) { cost = t; best = f.form; }
  }
  return best;
}

// Pipeline depth.  A CTA that is alone on its SM is fed by the bytes it keeps in flight, so when the whole problem
// is at most one CTA per SM the ring is twice as deep (6 / 8 / 10 stages for BN 128 / 64 / 32, one CTA per SM)
// instead of two co-resident CTAs with half the ring each.  bn | 0x1000 asks for the deep ring, bn | 0x2000 for the
// shallow one, RONN_GEMM_RING = deep | shallow for either in every call that does not say.
static int asked_ring(int bn) {
  if (bn & 0x3000) return (bn & 0x1000) ? 1 : 0;
  static int forced = -2;
  if (forced == -2) {
    const char* e = getenv("RONN_GEMM_RING");
    forced = !e ? -1 : (e[0] == 'd' ? 1 : (e[0] == 's' ? 0 : -1));
  }
  return forced;
}
static int wants_deep(int M, int N, int bn, int splitk) {
  const int tiles = ((N + bn - 1) / bn) * ((M + PG_BM - 1) / PG_BM) * splitk;
  return tiles <= sm_count() ? 1 : 0;
}

bool skinny_rule(int M, int N, int K);       // gemm_skinny.cu

// The form of a call.  A width, a pair or a ring that the caller asks for stands.
static int gemm_form(int M, int N, int K, int act, bool residual, bool out_fp32, long ldc, int bn) {
  if (bn == 0 && skinny_rule(M, N, K)) return FORM_SKINNY;
  const int ring = asked_ring(bn);
  const bool ragged = !out_fp32 && (ldc & 7);
  if (bn & FORM_CTA_PAIR) return bn & (FORM_CTA_PAIR | 0xfff);
  bn &= 0xfff;
  if (bn == 0 && (M >= 1024 || (M > 256 && pick_bn(M, N) >= 128)))
    return pick_form(M, N, K, act, residual, out_fp32, ragged, ring);
  if (bn == 0) bn = pick_bn(M, N);
  if (bn >= 256) return bn;
  return bn | ((ring >= 0 ? ring : (ragged ? 1 : wants_deep(M, N, bn, 1))) ? FORM_DEEP : FORM_SHALLOW);
}

}  // namespace ronn

using namespace ronn;

extern "C" int ronn_gemm_skinny(const void* A, const void* W, void* C, const void* bias, const void* residual,
                                const void* gamma, const void* beta, float eps, int norm, int M, int N, int K, long lda,
                                long ldw, long ldc, int dtype, int act, int out_fp32, cudaStream_t stream);

// The form that ronn_gemm runs for these arguments (see gemm_form).
extern "C" int ronn_gemm_form(int M, int N, int K, int act, int residual, int out_fp32, long ldc, int bn) {
  return gemm_form(M, N, K, act, residual != 0, out_fp32 != 0, ldc, bn);
}

// CTAs of a tile form (its code as ronn_gemm_form gives it) that one SM of the current device holds, or a negative error.
// The launch sizes its grid for PER_SM of them.
extern "C" int ronn_gemm_ctas_per_sm(int form, int dtype) {
#define RONN_RESIDENT(BN_, ST_, KA_)                                                                                 \
  return dtype == 0 ? resident_ctas(gemm_dense_kernel<BN_, ST_, __nv_bfloat16, KA_>, PG_THREADS, PGemmSmem<BN_, ST_, false, KA_>::DYN_SMEM) \
                    : resident_ctas(gemm_dense_kernel<BN_, ST_, __half, KA_>, PG_THREADS, PGemmSmem<BN_, ST_, false, KA_>::DYN_SMEM)
  switch (form) {
    case 32 | FORM_SHALLOW: RONN_RESIDENT(32, 5, 1);
    case 64 | FORM_SHALLOW: RONN_RESIDENT(64, 4, 1);
    case 128 | FORM_SHALLOW: RONN_RESIDENT(128, 3, 1);
    case 32 | FORM_DEEP: RONN_RESIDENT(32, 5, 2);
    case 64 | FORM_DEEP: RONN_RESIDENT(64, 4, 2);
    case 128 | FORM_DEEP: RONN_RESIDENT(128, 3, 2);
    case 256: RONN_RESIDENT(256, 4, 1);
    default: return -3;
  }
#undef RONN_RESIDENT
}

// dtype: 0 = bf16, 1 = fp16.  act: 0 none, 1 relu, 2 gelu.  bn: 0 = auto, else 32|64|128|256, or 256 | 0x4000 for CTA
// pairs; | 0x1000 deep ring, | 0x2000 shallow ring.
// lda/ldw/ldc in elements; K and the leading dimensions must be multiples of 8.
// Returns 0 on success, negative on configuration errors.
extern "C" int ronn_gemm(const void* A, const void* W, void* C, const void* bias, const void* residual, int M, int N,
                         int K, int lda, int ldw, int ldc, int dtype, int act, int out_fp32, int bn,
                         uint32_t* status, cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0) return -1;
  if ((K & 7) || (lda & 7) || (ldw & 7)) return -2;
  const int form = gemm_form(M, N, K, act, residual != nullptr, out_fp32 != 0, ldc, bn);
  if (form == FORM_SKINNY)
    return ronn_gemm_skinny(A, W, C, bias, residual, nullptr, nullptr, 0.f, 0, M, N, K, lda, ldw, ldc, dtype, act, out_fp32, stream);
  const bool pair = (form & FORM_CTA_PAIR) != 0, deep = (form & FORM_DEEP) != 0;
  bn = form & 0xfff;
  CUtensorMap ma, mb;
  int rc = make_tmap_2d(&ma, A, uint64_t(M), uint64_t(K), uint64_t(lda), PG_BM, 64, 2);
  if (rc) return rc - 20;
  rc = make_tmap_2d(&mb, W, uint64_t(N), uint64_t(K), uint64_t(ldw), uint32_t(pair ? bn / 2 : bn), 64, 2);
  if (rc) return rc - 30;
  DenseEpilogue e{C, bias, residual, M, N, ldc, 0, 0, act, out_fp32};
  const int bf = dtype == 0;
#define RONN_PAIR(BN_, ST_)                                                                           \
  return bf ? launch_pair<BN_, ST_, __nv_bfloat16>(ma, mb, e, M, N, K, 1, status, stream)             \
            : launch_pair<BN_, ST_, __half>(ma, mb, e, M, N, K, 0, status, stream)
  if (pair) {
    if (bn == 256) RONN_PAIR(256, 5);
    return -3;
  }
#undef RONN_PAIR
#define RONN_DISPATCH(BN_, ST_, KA_)                                                                  \
  return bf ? launch_dense<BN_, ST_, __nv_bfloat16, KA_>(ma, mb, e, M, N, K, 1, status, stream)       \
            : launch_dense<BN_, ST_, __half, KA_>(ma, mb, e, M, N, K, 0, status, stream)
  switch (deep ? -bn : bn) {
    case 256: case -256: RONN_DISPATCH(256, 4, 1);
    case 128: RONN_DISPATCH(128, 3, 1);
    case 64: RONN_DISPATCH(64, 4, 1);
    case 32: RONN_DISPATCH(32, 5, 1);
    case -128: RONN_DISPATCH(128, 3, 2);       // deep ring, one CTA per SM: two K atoms per stage
    case -64: RONN_DISPATCH(64, 4, 2);
    case -32: RONN_DISPATCH(32, 5, 2);
    default: return -3;
  }
#undef RONN_DISPATCH
}

// Split-K variant for skinny problems (decode: M <= 256).  Each of `splitk` K-slices writes an fp32 partial
// [M, N] to workspace slice z; ronn_splitk_finalize sums the slices and applies bias / residual / norm.
// The effective split count (every slice non-empty) is returned through *splitk_out.
extern "C" int ronn_gemm_splitk(const void* A, const void* W, float* workspace, int M, int N, int K, int lda, int ldw,
                                int dtype, int bn, int splitk, int* splitk_out, uint32_t* status,
                                cudaStream_t stream) {
  if (M <= 0 || N <= 0 || K <= 0 || splitk < 1) return -1;
  if ((K & 7) || (lda & 7) || (ldw & 7) || (N & 3)) return -2;
  const int num_kb = (K + 63) / 64;
  if (splitk > num_kb) splitk = num_kb;
  const int per = (num_kb + splitk - 1) / splitk;
  splitk = (num_kb + per - 1) / per;
  if (splitk_out) *splitk_out = splitk;
  int deep = asked_ring(bn);
  bn &= 0xfff;
  if (bn == 0) bn = N >= 128 ? 128 : (N >= 64 ? 64 : 32);
  if (deep < 0) deep = wants_deep(M, N, bn, splitk);
  CUtensorMap ma, mb;
  int rc = make_tmap_2d(&ma, A, uint64_t(M), uint64_t(K), uint64_t(lda), PG_BM, 64, 2);
  if (rc) return rc - 20;
  rc = make_tmap_2d(&mb, W, uint64_t(N), uint64_t(K), uint64_t(ldw), uint32_t(bn), 64, 2);
  if (rc) return rc - 30;
  DenseEpilogue e{workspace, nullptr, nullptr, M, N, N, 0, 0, 0, 1};
  const int bf = dtype == 0;
#define RONN_DISPATCH(BN_, ST_, KA_)                                                                     \
  return bf ? launch_dense<BN_, ST_, __nv_bfloat16, KA_>(ma, mb, e, M, N, K, 1, status, stream, splitk)  \
            : launch_dense<BN_, ST_, __half, KA_>(ma, mb, e, M, N, K, 0, status, stream, splitk)
  switch (deep ? -bn : bn) {
    case 256: case -256: RONN_DISPATCH(256, 4, 1);
    case 128: RONN_DISPATCH(128, 3, 1);
    case 64: RONN_DISPATCH(64, 4, 1);
    case 32: RONN_DISPATCH(32, 5, 1);
    case -128: RONN_DISPATCH(128, 3, 2);       // deep ring, one CTA per SM: two K atoms per stage
    case -64: RONN_DISPATCH(64, 4, 2);
    case -32: RONN_DISPATCH(32, 5, 2);
    default: return -3;
  }
#undef RONN_DISPATCH
}
