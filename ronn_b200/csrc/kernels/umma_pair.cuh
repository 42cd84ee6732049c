// Persistent tcgen05 GEMM main loop on CTA pairs (cta_group::2): two SMs compute one tile of 256 x BN.
//
// A one-CTA tile of 128 x 256 reads 48 KB of operands per 512 cycles of MMA, 94 bytes per cycle, and an SM takes in about
// 64 from L2: that loop waits for its operands.  In a pair every SM loads its own 128 rows of A but only half of B
// (BN / 2 rows), which the matrix instruction reads from both shared memories: 32 KB per 512 cycles.
//
// Both CTAs run the same code with the same shared-memory layout.  Cluster rank 0 leads:
//   warp 0     TMA producer, in both CTAs: own A rows and own half of B into own shared memory; the bytes of both are
//              counted on the leader's full[s], which the leader arms for the whole pair.  (A peer's bytes may be counted
//              before the leader has armed the phase; the phase still ends only with the leader's arrival.)
//   warp 1     leader only: waits full[s], issues the MMAs for the pair, commits to empty[s] and acc_full[b] of both CTAs
//   warps 2-17 epilogue, in both CTAs: drain the CTA's own 128 accumulator rows, then arrive on the leader's acc_empty[b].
//              Four warps per TMEM lane quarter, a quarter of the columns each: with two, a 128 x 256 half tile took 7.7 us
//              to drain (9.5 us with GELU) whatever its K, longer than the MMAs of a K of 768 or 1024
// Every wait is bounded as in umma_persistent.cuh, and every thread reaches the two cluster barriers (after set-up, before
// teardown), so an abandoned wait in one CTA cannot leave the other behind.
//
// Results of 16 bits on the 16-byte grid leave through the epilogue of this file: each warp owns 32 rows x 64 columns, adds
// bias and activation in registers, meets the residual in its 4 KB of shared memory (a TMA load issued before the
// accumulator is waited for) and hands the box to one TMA store of whole 128-byte lines.  Stores and residual loads from the
// accumulator layout (64 bytes of a row per warp) ran at 2.5 to 4 TB/s and made the epilogue longer than the MMAs: at 8192 x
// 2304 x 64, where there is nothing else, 18 us plain, 23 with bias, 32 with residual or GELU.
//
// Problem: kConstB (B never depends on the previous kernel in the stream: its first stages are requested before the
// dependency wait), num_tiles(), tile(t, m0, n0), num_kb, load_a(smem, bar, k, m), load_b(smem, bar, k, n) with `bar` a shared::cluster
// address, row_scale(m) (int8: factor of a row's sums), and `out`, a PairOut.
#pragma once
#include "common.cuh"
#include "gemm_epilogue.cuh"
#include "ptx_sm100.cuh"
#include "tma_desc.cuh"

namespace ronn {

constexpr int PP_EPI_WARPS = 16;
constexpr int PP_THREADS = 64 + 32 * PP_EPI_WARPS;

struct PairOut {
  const CUtensorMap* map_c;      // output [M, N], boxes of 64 columns x 32 rows
  const CUtensorMap* map_r;      // residual, the same boxes
  DenseEpilogue e;               // bias, residual, activation; also the path of results off the 16-byte grid
  int by_tma;
};

template <int BN, int STAGES>
struct PairSmem {
  static constexpr int A_BYTES = 128 * 128;
  static constexpr int B_BYTES = BN / 2 * 128;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int TILE_BYTES = STAGES * STAGE_BYTES;
  static constexpr int NUM_BARS = 2 * STAGES + 4 + PP_EPI_WARPS;
  static constexpr int OUT_STAGE = 32 * 128;                // per epilogue warp
  static constexpr int DYN_SMEM = TILE_BYTES + PP_EPI_WARPS * OUT_STAGE + NUM_BARS * 8 + 16 + 1024;
  static_assert(DYN_SMEM <= 232448, "shared memory of an SM");
  static constexpr uint32_t TMEM_COLS = 512;               // two accumulator buffers, 256 columns apart
};

__device__ __forceinline__ uint32_t map_to_rank(uint32_t smem_addr, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(smem_addr), "r"(rank));
  return r;
}
__device__ __forceinline__ void pair_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
  asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
  asm volatile("mbarrier.arrive.release.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait_cluster(uint64_t* bar, uint32_t parity) {
  uint32_t ok;
  asm volatile(
      "{\n\t.reg .pred p;\n\t"
      "mbarrier.try_wait.parity.acquire.cluster.shared::cta.b64 p, [%1], %2;\n\t"
      "selp.u32 %0, 1, 0, p;\n\t}"
      : "=r"(ok)
      : "r"(smem_u32(bar)), "r"(parity)
      : "memory");
  return ok != 0;
}
// bounded wait for arrivals of both CTAs (cluster scope)
__device__ __forceinline__ bool mbar_wait_cluster(uint64_t* bar, uint32_t parity, volatile uint32_t* abort_flag, uint32_t* status,
                                                  uint32_t code) {
  if (mbar_try_wait_cluster(bar, parity)) return true;
  const long long t0 = clock64();
  uint32_t polls = 0;
  while (true) {
    if (mbar_try_wait_cluster(bar, parity)) return true;
    if ((++polls & 31u) == 0u) {
      if (*abort_flag) return false;
      if (clock64() - t0 > WAIT_LIMIT_CYCLES) {
        *abort_flag = 1;
        if (status) atomicCAS(status, 0u, code);
        return false;
      }
    }
  }
}
// 2-D tiled load into this CTA's shared memory whose bytes are counted on a barrier of either CTA of the pair; no multicast
__device__ __forceinline__ void tma_load_2d_pair(void* smem_dst, const CUtensorMap* map, uint32_t bar, int32_t c0, int32_t c1) {
  asm volatile(
      "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
      ::"r"(smem_u32(smem_dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(bar), "r"(c0), "r"(c1)
      : "memory");
}
template <int KIND>
__device__ __forceinline__ void umma_pair(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
  if (KIND == 0)
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
  else
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// arrive on the barrier at this offset in both CTAs once the MMAs issued so far have completed
__device__ __forceinline__ void umma_commit_pair(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(
                   smem_u32(bar)),
               "h"(uint16_t(3))
               : "memory");
}

// Tensor maps of the output and the residual.  1 when the results can leave by TMA: 16 bits, rows and bases on the 16-byte
// grid, whole 8-column pieces.
inline int pair_out_maps(const DenseEpilogue& e, int elem_size, CUtensorMap* mc, CUtensorMap* mr) {
  if (e.out_fp32 || (e.N & 7) || (e.ldc & 7) || (reinterpret_cast<uintptr_t>(e.bias) & 15) || e.res_first) return 0;
  if (make_tmap_2d(mc, e.C, uint64_t(e.M), uint64_t(e.N), uint64_t(e.ldc), 32, 64, elem_size) != 0) return 0;
  if (e.residual && make_tmap_2d(mr, e.residual, uint64_t(e.M), uint64_t(e.N), uint64_t(e.ldc), 32, 64, elem_size) != 0) return 0;
  return 1;
}

// KIND 0: 16-bit operands (64 values per 128-byte row), 1: int8 (128).
template <int BN, int STAGES, int KIND, class T, class Problem>
__device__ __forceinline__ void gemm_pair(uint8_t* dyn_smem, Problem& prob, uint32_t idesc, uint32_t* status) {
  using L = PairSmem<BN, STAGES>;
  constexpr int K_ELEMS = KIND == 0 ? 64 : 128;
  uint8_t* tiles = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(dyn_smem) + 1023) & ~uintptr_t(1023));
  uint8_t* out_stage = tiles + L::TILE_BYTES;                              // 1024-byte aligned: stages are multiples of 16 KB
  uint64_t* full = reinterpret_cast<uint64_t*>(out_stage + PP_EPI_WARPS * L::OUT_STAGE);     // the leader's is the one in use
  uint64_t* empty = full + STAGES;
  uint64_t* acc_full = empty + STAGES;
  uint64_t* acc_empty = acc_full + 2;                                      // the leader's is the one in use
  uint64_t* res_full = acc_empty + 2;                                      // one per epilogue warp
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(res_full + PP_EPI_WARPS);
  volatile uint32_t* abort = tmem_slot + 1;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const uint32_t rank = blockIdx.x & 1;                                    // cluster dimension 2 along x
  const int pair = blockIdx.x >> 1, pairs = gridDim.x >> 1;

  if (threadIdx.x == 0) {
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    for (int b = 0; b < 2; ++b) {
      mbar_init(&acc_full[b], 1);
      mbar_init(&acc_empty[b], 2 * PP_EPI_WARPS);
    }
    for (int w = 0; w < PP_EPI_WARPS; ++w) mbar_init(&res_full[w], 1);
    *abort = 0;
    mbar_fence_init();
    fence_proxy_async_smem();
  }
  __syncwarp();
  if (warp == 1) {
    asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(L::TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
  }
  tc_fence_before_sync();
  __syncthreads();
  pair_sync();                                   // both CTAs' barriers are initialised
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int ntiles = prob.num_tiles(), nkb = prob.num_kb;

  if (warp == 0) {
    if (lane == 0) {
      int pre = 0;
      if (Problem::kConstB && pair < ntiles) {
        int m0, n0;
        prob.tile(pair, m0, n0);
        pre = nkb < STAGES ? nkb : STAGES;
        for (int s = 0; s < pre; ++s) {
          if (rank == 0) mbar_expect_tx(&full[s], 2 * L::STAGE_BYTES);
          prob.load_b(tiles + s * L::STAGE_BYTES + L::A_BYTES, map_to_rank(smem_u32(&full[s]), 0), s * K_ELEMS, n0 + int(rank) * (BN / 2));
        }
      }
      pdl_wait();
      pdl_trigger();
      uint32_t it = 0;
      bool ok = true;
      for (int t = pair; t < ntiles && ok; t += pairs) {
        int m0, n0;
        prob.tile(t, m0, n0);
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int s = it % STAGES;
          uint8_t* sa = tiles + s * L::STAGE_BYTES;
          const uint32_t bar = map_to_rank(smem_u32(&full[s]), 0);
          if (it >= uint32_t(pre)) {
            if (!mbar_wait_cluster(&empty[s], ((it / STAGES) & 1) ^ 1, abort, status, STATUS_WAIT_SLOT)) { ok = false; break; }
            if (rank == 0) mbar_expect_tx(&full[s], 2 * L::STAGE_BYTES);
            prob.load_b(sa + L::A_BYTES, bar, kb * K_ELEMS, n0 + int(rank) * (BN / 2));
          }
          prob.load_a(sa, bar, kb * K_ELEMS, m0 + int(rank) * 128);
        }
      }
    }
    __syncwarp();
    pdl_trigger();
  } else if (warp == 1) {
    if (lane == 0 && rank == 0) {
      uint32_t it = 0, j = 0;
      bool ok = true;
      for (int t = pair; t < ntiles && ok; t += pairs, ++j) {
        const uint32_t buf = j & 1;
        if (!mbar_wait_cluster(&acc_empty[buf], ((j >> 1) & 1) ^ 1, abort, status, STATUS_WAIT_EPI)) break;
        tc_fence_after_sync();
        const uint32_t tmem_d = tmem_base + buf * 256u;
        bool ready = false;
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          const int s = it % STAGES;
          if (!ready && !mbar_wait_cluster(&full[s], (it / STAGES) & 1, abort, status, STATUS_WAIT_TMA)) { ok = false; break; }
          tc_fence_after_sync();
          ready = kb + 1 < nkb && mbar_try_wait_cluster(&full[(it + 1) % STAGES], ((it + 1) / STAGES) & 1);
          const uint32_t sa = smem_u32(tiles + s * L::STAGE_BYTES);
          const uint64_t adesc = umma_desc_k128(sa), bdesc = umma_desc_k128(sa + L::A_BYTES);
#pragma unroll
          for (int k = 0; k < 4; ++k) umma_pair<KIND>(tmem_d, adesc + 2 * k, bdesc + 2 * k, idesc, (kb | k) != 0);
          umma_commit_pair(&empty[s]);
        }
        if (ok) umma_commit_pair(&acc_full[buf]);
      }
    }
    __syncwarp();
    pdl_trigger();
  } else {
    const int q = warp & 3;                      // TMEM lane quarter of this warp
    const int part = (warp - 2) >> 2;            // which quarter of the columns this warp drains
    uint8_t* stage_w = out_stage + (warp - 2) * L::OUT_STAGE;
    uint64_t* my_res = res_full + (warp - 2);
    const PairOut& out = prob.out;
    const bool has_res = out.e.residual != nullptr;
    pdl_wait();
    uint32_t j = 0;
    for (int t = pair; t < ntiles; t += pairs, ++j) {
      int m0, n0;
      prob.tile(t, m0, n0);
      m0 += int(rank) * 128;
      constexpr int PART = BN / 4;
      static_assert(PART == 64, "a warp owns one box of 64 columns");
      const int c0 = part * PART;
      const int gn = n0 + c0, gm0 = m0 + q * 32;           // first column and row of the warp's box
      const uint32_t buf = j & 1;
      Vec8 bias_v[8];
      if (out.by_tma) {
        if (lane == 0) {
          tma_store_wait_read();                             // the box of the previous tile has left the stage
          if (has_res) {
            mbar_expect_tx(my_res, L::OUT_STAGE);
            tma_load_2d(stage_w, out.map_r, my_res, gn, gm0);
          }
        }
        __syncwarp();
        if (out.e.bias) {
#pragma unroll
          for (int g = 0; g < 8; ++g)
            if (gn + g * 8 < out.e.N) bias_v[g] = *reinterpret_cast<const Vec8*>(static_cast<const T*>(out.e.bias) + gn + g * 8);
        }
      }
      bool ok = mbar_wait_cluster(&acc_full[buf], (j >> 1) & 1, abort, status, STATUS_WAIT_ACCUM);
      if (out.by_tma && has_res) ok = mbar_wait(my_res, j & 1, abort, status, STATUS_WAIT_TMA) && ok;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t free_bar = map_to_rank(smem_u32(&acc_empty[buf]), 0);
      const int row = q * 32 + lane;
      const uint32_t tacc = tmem_base + (uint32_t(q * 32) << 16) + buf * 256u + uint32_t(c0);
      const float rs = KIND == 1 ? prob.row_scale(m0 + row) : 1.f;
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        uint32_t r[32];
        tmem_ld_32x32(tacc + uint32_t(h * 32), r);
        tmem_ld_wait();
        if (h == 1) {                            // the last load of this buffer has landed
          tc_fence_before_sync();
          __syncwarp();
          if (lane == 0) mbar_arrive_cluster(free_bar);
        }
        if (KIND == 1) {
#pragma unroll
          for (int i = 0; i < 32; ++i) r[i] = __float_as_uint(float(int(r[i])) * rs);
        }
        if (!out.by_tma) {
          DenseEpilogue ep = out.e;
          ep.m0 = m0;
          ep.n0 = n0;
          ep.run<T>(row, c0 + h * 32, r, stage_w);
          continue;
        }
#pragma unroll
        for (int g = 0; g < 4; ++g) {            // 16-byte piece h * 4 + g of the row
          float v[8];
#pragma unroll
          for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[g * 8 + i]);
          if (out.e.bias) {
            float f[8];
            unpack8<T>(bias_v[h * 4 + g], f);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] += f[i];
          }
          if (out.e.act == 1) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = fmaxf(v[i], 0.f);
          } else if (out.e.act == 2) {
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] = gelu_tanh_f(v[i]);
          }
          Vec8* piece = reinterpret_cast<Vec8*>(stage_w + lane * 128 + ((uint32_t(h * 4 + g) ^ uint32_t(lane & 7)) << 4));
          if (has_res) {
            float f[8];
            unpack8<T>(*piece, f);
#pragma unroll
            for (int i = 0; i < 8; ++i) v[i] += f[i];
          }
          *piece = pack8<T>(v);
        }
      }
      if (out.by_tma) {
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0 && gn < out.e.N && gm0 < out.e.M) tma_store_2d(out.map_c, stage_w, gn, gm0);
      }
    }
    if (lane == 0) tma_store_wait();
    pdl_trigger();
  }
  if (*abort) {
    const long long t0 = clock64();
    while (clock64() - t0 < 400000ll) { __nanosleep(1000); }
  }
  tc_fence_before_sync();
  __syncthreads();
  pair_sync();                                   // no MMA of the leader reads, and no arrival targets, a CTA that has left
  if (warp == 1) {
    tc_fence_after_sync();
    asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(L::TMEM_COLS) : "memory");
  }
}

}  // namespace ronn
