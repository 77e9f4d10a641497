// Split-K variant of the tcgen05 GEMM for outputs with few tiles (a few hundred tokens, narrow layers): 128 x BN output
// tiles (BN = 64 or 128), one tile per cluster of S CTAs, each CTA reducing its own slice of K.
//
// The 128 x 256 and 256 x 256 kernels give such a GEMM 8 to 50 CTAs on 148 SMs, each walking all of K alone: it is bound
// by the latency of that chain, not by the tensor cores or by reading the weights. Here the K loop is cut over the CTAs
// of a cluster (S <= 8, any number), the partial tiles meet through distributed shared memory, and two CTAs share an SM,
// so that loads of one cover the epilogue of the other:
//   mainloop : warp 0 TMA producer, warp 1 MMA issuer (128 x BN x 16), one accumulator of BN TMEM columns
//   exchange : warps 2-5 write the fp32 accumulator into their CTA's shared memory (over the ring, 16-byte chunks
//              XOR-swizzled by row), cluster barrier
//   epilogue : CTA r of the cluster owns rows [128 r / S, 128 (r+1) / S): its 192 threads add the S partial sums of an
//              element in the order of the slices (the result repeats bit for bit) and hand four columns at a time to
//              the epilogue functor, neighbouring threads on neighbouring columns, so that global accesses are whole
//              row segments without a staging pass.
// No TMA load uses cluster multicast.
#pragma once
#include "gemm_core.cuh"

namespace b200 {
namespace gemm {

// A CTA's ring: 96 KB where two CTAs share an SM; twice that (DEEP) where the grid leaves each CTA an SM of its own, since
// a single chain of K blocks runs at the latency of its loads over the blocks in flight.
template <int BN, bool DEEP>
struct SmemCluster {
  static constexpr int STAGES = (BN == 64 ? 4 : 3) * (DEEP ? 2 : 1);
  static constexpr int A_BYTES = BM * BK * 2;
  static constexpr int B_BYTES = BN * BK * 2;
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int RING_BYTES = STAGES * STAGE_BYTES;
  static constexpr int BAR_BYTES = 256;
  static constexpr int BYTES = RING_BYTES + BAR_BYTES + 1024;
  static_assert(BM * BN * 4 <= RING_BYTES, "the partial tile lies over the ring");
};
constexpr int CLUSTER_MAX_SLICES = 8;

__device__ __forceinline__ uint32_t cluster_nctas() {
  uint32_t r;
  asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
  return r;
}

// Epi concept: Params; SPLIT_B (the tile's B rows are BN/2 rows at n and BN/2 rows b_half_stride below them);
// items<BN>() work items per row; item<BN>(p, row, n0, N, it, get) with get(chunk) = the four accumulator columns
// 4 * chunk .. 4 * chunk + 3 of the row. AHEAD > 0: operands from global memory, Pre, are loaded for that many of a thread's
// items at a time by load<BN>(p, row, n0, it, pre) - the first of them while the main loop runs - and item takes one more argument.
template <int BN, bool DEEP, bool A_MN, bool B_MN, class Epi>
__global__ void __launch_bounds__(NUM_THREADS, DEEP ? 1 : 2)
    gemm_cluster_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N,
                        int K, int fmt, typename Epi::Params ep, unsigned int* err_word, int b_half_stride, int b_early) {
  using S = SmemCluster<BN, DEEP>;
  constexpr int STAGES = S::STAGES;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::RING_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* done_bar = empty_bar + STAGES;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done_bar + 1);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const int n_slices = (int)cluster_nctas();
  const int slice = (int)cluster_ctarank();

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    mbar_init(done_bar, 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, BN);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  const int m_tiles = (M + BM - 1) / BM;
  const int tile = (int)blockIdx.x / n_slices;
  const int m0 = (tile % m_tiles) * BM;          // row tiles fastest: CTAs side by side read the same weights
  const int n_blk = tile / m_tiles;
  const int n0 = n_blk * BN;
  const int num_kb = (K + BK - 1) / BK;
  const int kb0 = (int)((long long)num_kb * slice / n_slices);
  const int kb1 = (int)((long long)num_kb * (slice + 1) / n_slices);

  auto load_b = [&](int kb, uint32_t st) {
    uint8_t* sB = smem + st * S::STAGE_BYTES + S::A_BYTES;
    if constexpr (B_MN) {
#pragma unroll
      for (int i = 0; i < BN / 64; ++i) tma_load_2d(sB + i * (BK * 128), &tmB, &full_bar[st], n0 + i * 64, kb * BK);
    } else if constexpr (Epi::SPLIT_B) {
      tma_load_2d(sB, &tmB, &full_bar[st], kb * BK, n_blk * (BN / 2));
      tma_load_2d(sB + (BN / 2) * 128, &tmB, &full_bar[st], kb * BK, b_half_stride + n_blk * (BN / 2));
    } else {
      tma_load_2d(sB, &tmB, &full_bar[st], kb * BK, n0);
    }
  };
  // B of the ring's first round in front of pdl_wait, where the caller says that the kernel before this one does not write
  // it (a layer's weights): those bytes then arrive while that kernel drains. A grid starts early only when every CTA of the
  // one before it is past its own wait, so whatever ran before THAT one is complete and visible here. Steps of 512 and of 777
  // tokens 1.4 and 1.0 % shorter, a forward pass over 93 tokens 1.8 %.
  const int early = b_early ? min(kb1 - kb0, STAGES) : 0;
  if (warp == 0) {
    if (elect_one()) {
      for (int i = 0; i < early; ++i) {
        mbar_arrive_expect_tx(&full_bar[i], S::STAGE_BYTES);
        load_b(kb0 + i, i);
      }
    }
    __syncwarp();
  }
  pdl_wait();
  pdl_trigger();

  constexpr int IPR = Epi::template items<BN>(), AHEAD = Epi::AHEAD > 0 ? Epi::AHEAD : 1;
  const int r0 = BM * slice / n_slices, r1 = min(BM * (slice + 1) / n_slices, M - m0);
  const int n_items = max(r1 - r0, 0) * IPR, col0 = Epi::SPLIT_B ? n_blk * (BN / 2) : n0;
  typename Epi::Pre pre[AHEAD];
  auto load_ahead = [&](int first) {
#pragma unroll
    for (int u = 0; u < AHEAD; ++u) {
      const int i = first + u * NUM_THREADS;
      if (i < n_items) Epi::template load<BN>(ep, m0 + r0 + i / IPR, col0, i % IPR, pre[u]);
    }
  };
  if (Epi::AHEAD > 0 && warp >= 2) load_ahead(threadIdx.x);

  if (warp == 0) {
    if (elect_one()) {
      uint32_t st = 0, ph = 1u;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_bounded(&empty_bar[st], ph, abort_flag, err_word, ERR_WAIT_EMPTY)) break;
        uint8_t* sA = smem + st * S::STAGE_BYTES;
        if (kb - kb0 >= early) {
          mbar_arrive_expect_tx(&full_bar[st], S::STAGE_BYTES);
          load_b(kb, st);
        }
        if constexpr (!A_MN) {
          tma_load_2d(sA, &tmA, &full_bar[st], kb * BK, m0);
        } else {
#pragma unroll
          for (int i = 0; i < BM / 64; ++i) tma_load_2d(sA + i * (BK * 128), &tmA, &full_bar[st], m0 + i * 64, kb * BK);
        }
        if (++st == STAGES) {
          st = 0;
          ph ^= 1u;
        }
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    const uint32_t idesc = make_idesc_f16(fmt, BM, BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
    constexpr DescCfg dc = default_desc_cfg<BN, A_MN, B_MN>();
    const uint64_t da0 = make_smem_desc_sw128(smem_u32(smem), dc.a_lbo, dc.a_sbo);
    const uint64_t db0 = make_smem_desc_sw128(smem_u32(smem) + S::A_BYTES, dc.b_lbo, dc.b_sbo);
    if (elect_one()) {
      uint32_t st = 0, ph = 0u;
      for (int kb = kb0; kb < kb1; ++kb) {
        if (!mbar_wait_bounded(&full_bar[st], ph, abort_flag, err_word, ERR_WAIT_FULL)) break;
        tc_fence_after_sync();
        const uint64_t off = static_cast<uint64_t>((st * S::STAGE_BYTES) >> 4);
#pragma unroll
        for (int k = 0; k < BK / UMMA_K; ++k)
          umma_f16_ss(tmem_base, da0 + off + static_cast<uint64_t>((k * dc.a_kadv) >> 4),
                      db0 + off + static_cast<uint64_t>((k * dc.b_kadv) >> 4), idesc, (kb != kb0 || k != 0) ? 1u : 0u);
        umma_commit(&empty_bar[st]);
        if (kb + 1 == kb1) umma_commit(done_bar);
        if (++st == STAGES) {
          st = 0;
          ph ^= 1u;
        }
      }
    }
    __syncwarp();
  } else {
    // accumulator -> shared memory. done_bar means every MMA has read its stage, so the ring is free.
    const int quad = warp & 3;
    const int row = quad * 32 + lane;
    int ok = mbar_wait_bounded(done_bar, 0, abort_flag, err_word, ERR_WAIT_TMEM_FULL) ? 1 : 0;
    if (__all_sync(0xffffffffu, ok)) {
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quad * 32) << 16);
#pragma unroll
      for (int c = 0; c < BN / 32; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j)
          *reinterpret_cast<uint4*>(smem + row * (BN * 4) + (((c * 8 + j) ^ (row & 15)) << 4)) =
              make_uint4(r[4 * j], r[4 * j + 1], r[4 * j + 2], r[4 * j + 3]);
      }
    }
  }
  __syncwarp();
  tc_fence_before_sync();
  if (n_slices > 1) cluster_sync_all(); else __syncthreads();

  {
    const uint32_t part = smem_u32(smem);
    auto sum_of = [&](int row) {
      return [=](int chunk) {
        const uint32_t off = part + row * (BN * 4) + ((chunk ^ (row & 15)) << 4);
        float4 a;
        if (n_slices == 1) {
          a = *reinterpret_cast<const float4*>(smem + (off - part));
        } else {
          float4 v[CLUSTER_MAX_SLICES];
#pragma unroll
          for (int s = 0; s < CLUSTER_MAX_SLICES; ++s)
            if (s < n_slices) v[s] = ld_cluster_f32x4(mapa_shared(off, s));
          a = v[0];
#pragma unroll
          for (int s = 1; s < CLUSTER_MAX_SLICES; ++s)
            if (s < n_slices) { a.x += v[s].x; a.y += v[s].y; a.z += v[s].z; a.w += v[s].w; }
        }
        return a;
      };
    };
    if constexpr (Epi::AHEAD > 0) {
      if (warp < 2) load_ahead(threadIdx.x);
      for (int first = threadIdx.x; first < n_items; first += AHEAD * NUM_THREADS) {
        if (first != (int)threadIdx.x) load_ahead(first);
#pragma unroll
        for (int u = 0; u < AHEAD; ++u) {
          const int i = first + u * NUM_THREADS, row = r0 + i / IPR;
          if (i < n_items) Epi::template item<BN>(ep, m0 + row, col0, N, i % IPR, sum_of(row), pre[u]);
        }
      }
    } else {
      for (int i = threadIdx.x; i < n_items; i += NUM_THREADS) {
        const int row = r0 + i / IPR;
        Epi::template item<BN>(ep, m0 + row, col0, N, i % IPR, sum_of(row));
      }
    }
  }

  __syncwarp();
  if (*abort_flag) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  __syncwarp();
  if (n_slices > 1) cluster_sync_all(); else __syncthreads();   // no CTA leaves while a peer still reads its partial tile
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, BN);
  }
}

}  // namespace gemm
}  // namespace b200
