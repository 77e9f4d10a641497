// Two-SM variant of the tcgen05 GEMM mainloop: a cluster of two CTAs works on one 256 x 256 output tile with
// tcgen05.mma.cta_group::2. Each CTA TMA-loads its own 128 rows of A and its own 128-row half of B (no multicast:
// the pair MMA reads both halves), so every SM fills and reads half the B bytes of the one-SM kernel - which is what
// the shared-memory pipe was saturated by - and the ring holds 6 stages instead of 4.
//
//   rank 0 (leader): TMA producer, MMA issuer (256 x 256 x 16 per instruction), 4 epilogue warps for rows 0-127
//   rank 1         : TMA producer,                                              4 epilogue warps for rows 128-255
// Barriers: "full" lives in the leader (both CTAs' TMA bytes are credited there); "empty" and "accumulator full" are
// per CTA and are released by tcgen05.commit multicast to both; "accumulator empty" lives in the leader and is
// arrived on by all 8 epilogue warps (the peer's through its cluster address). Epilogue functors are the same as for
// the one-SM kernel (gemm_core.cuh).
//
// Split-K (k_splits > 1, epilogues with SPLIT_K only): a work unit is (slice of the K loop, tile), slice-major, so
// the pairs that run side by side work on the same K window of neighbouring tiles. The slices of one tile are added
// into C in the order of their index: slice s of a tile waits until a counter in global memory says that slice s - 1
// has been added (8 counters per tile, one per epilogue warp of the pair, because each warp owns its own rows), adds,
// and releases the counter; the last slice sets it back to zero for the next launch. The order of the additions is
// therefore fixed and the result repeats bit for bit, which atomic adds did not give. Units are handed out in
// increasing order and all CTAs of the grid are resident, so the unit a slice waits for is always running or done.
//
// Grouped (GROUPED; the experts of a layer in ONE launch): the rows of A and C are cut into consecutive groups whose lengths
// are on the device, and group e meets rows [e * b_rows, (e + 1) * b_rows) of B. Each CTA turns the lengths into tile
// offsets itself, so the host need not know them; a tile belongs to one group, its rows past the group's end are computed
// from the next group's rows and not stored. One launch fills its last round with tiles of every group (6124 tokens, two of 8
// experts each, 2048 -> 5632 -> 2048: a down projection of one expert is 48 tiles for 74 pairs), and no read-back of the
// lengths stands between the router and the experts: a collection batch of six such layers 9.13 / 8.13 ms.
#pragma once
#include "gemm_core.cuh"

namespace b200 {
namespace gemm {

constexpr int PAIR_BM = 256;  // rows per tile pair
constexpr int PAIR_BN = 256;
constexpr int PAIR_HALF_N = 128;

constexpr int MAX_GROUPS = 128;

struct GroupArgs {
  const long long* counts;   // [n] rows of each group
  int n;
  int b_rows;                // rows of B per group
};

template <int STAGES>
struct SmemPair {
  static constexpr int A_BYTES = BM * BK * 2;           // 128 x 64
  static constexpr int B_BYTES = PAIR_HALF_N * BK * 2;  // 128 x 64
  static constexpr int STAGE_BYTES = A_BYTES + B_BYTES;
  static constexpr int RING_BYTES = STAGES * STAGE_BYTES;
  static constexpr int BAR_BYTES = 256;
  static constexpr int GROUP_BYTES = 2 * (MAX_GROUPS + 1) * 4;   // first tile and first row of each group
  static constexpr int bytes(int epi_bytes, bool grouped = false) {
    return RING_BYTES + BAR_BYTES + epi_bytes + (grouped ? GROUP_BYTES : 0) + 1024;
  }
};

// An epilogue of 8 warps gives each quadrant of TMEM two of them: the second takes the tile's columns from 128 on. For
// epilogues whose arithmetic on 4 warps outlasts the main loop.
template <class Epi>
constexpr int pair_threads() {
  return 64 + 32 * Epi::WARPS;
}

template <int STAGES, bool A_MN, bool B_MN, class Epi, bool GROUPED = false>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(pair_threads<Epi>(), 1)
    gemm_pair_kernel(const __grid_constant__ CUtensorMap tmA, const __grid_constant__ CUtensorMap tmB, int M, int N,
                     int K, int fmt, typename Epi::Params ep, unsigned int* err_word, int k_splits,
                     unsigned int* split_sync, int b_half_stride, GroupArgs grp) {
  using S = SmemPair<STAGES>;
  extern __shared__ uint8_t smem_raw[];
  uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
  uint64_t* full_bar = reinterpret_cast<uint64_t*>(smem + S::RING_BYTES);
  uint64_t* empty_bar = full_bar + STAGES;
  uint64_t* tfull_bar = empty_bar + STAGES;
  uint64_t* tempty_bar = tfull_bar + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(tempty_bar + 2);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
  uint8_t* epi_smem = smem + S::RING_BYTES + S::BAR_BYTES;

  const int warp = threadIdx.x >> 5;
  const int lane = threadIdx.x & 31;
  const uint32_t cta = cluster_ctarank();  // 0 = leader
  constexpr uint32_t TMEM_COLS = 2 * PAIR_BN;

  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmA);
    tma_prefetch_desc(&tmB);
    for (int s = 0; s < STAGES; ++s) {
      mbar_init(&full_bar[s], 1);
      mbar_init(&empty_bar[s], 1);
    }
    for (int a = 0; a < 2; ++a) {
      mbar_init(&tfull_bar[a], 1);
      mbar_init(&tempty_bar[a], 2 * Epi::WARPS);
    }
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc_pair(tmem_slot, TMEM_COLS);
    tmem_relinquish_pair();
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // both CTAs' barriers exist before any remote arrive / pair TMA
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  const int n_tiles = (N + PAIR_BN - 1) / PAIR_BN;
  int* g_tile = reinterpret_cast<int*>(epi_smem + Epi::SMEM_BYTES);   // GROUPED: row tiles in front of each group
  int* g_row = g_tile + MAX_GROUPS + 1;                               //          and rows
  int m_tiles = (M + PAIR_BM - 1) / PAIR_BM;
  if constexpr (GROUPED) {
    if (warp == 0) {
      int tiles = 0, rows = 0;
      if (lane == 0) g_tile[0] = g_row[0] = 0;
      for (int e0 = 0; e0 < grp.n; e0 += 32) {
        const int e = e0 + lane;
        int r = e < grp.n ? (int)grp.counts[e] : 0;
        int t = (r + PAIR_BM - 1) / PAIR_BM;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int ur = __shfl_up_sync(0xffffffffu, r, o), ut = __shfl_up_sync(0xffffffffu, t, o);
          if (lane >= o) {
            r += ur;
            t += ut;
          }
        }
        if (e < grp.n) {
          g_tile[e + 1] = tiles + t;
          g_row[e + 1] = rows + r;
        }
        tiles += __shfl_sync(0xffffffffu, t, 31);
        rows += __shfl_sync(0xffffffffu, r, 31);
      }
    }
    __syncthreads();
    m_tiles = g_tile[grp.n];
  }
  const int num_tiles = m_tiles * n_tiles;
  const int num_kb = (K + BK - 1) / BK;
  // split-K: a work unit is (slice of the K loop, tile), slice-major. k_splits = 1: one unit per tile.
  const int num_units = num_tiles * k_splits;
  auto unit_range = [&](int unit, int& tile, int& kb0, int& kb1) {
    const int sp = unit / num_tiles;
    tile = unit - sp * num_tiles;
    kb0 = (int)((long long)num_kb * sp / k_splits);
    kb1 = (int)((long long)num_kb * (sp + 1) / k_splits);
  };
  const int pair_id = blockIdx.x >> 1;
  const int num_pairs = gridDim.x >> 1;
  constexpr int GROUP_M = 8;
  // First row and column block of a tile, the first row of B that its columns count from, and the end of its rows. `e`:
  // the group of the caller's tile before this one (tiles are visited in increasing order), 0 at first.
  auto locate = [&](int tile, int& e, int& row, int& n_blk, int& b_row, int& row_end) {
    int mt = m_tiles, base = 0;
    row_end = M;
    b_row = 0;
    if constexpr (GROUPED) {
      while (tile >= g_tile[e + 1] * n_tiles) ++e;
      tile -= g_tile[e] * n_tiles;
      mt = g_tile[e + 1] - g_tile[e];
      base = g_row[e];
      row_end = g_row[e + 1];
      b_row = e * grp.b_rows;
    }
    const int per_group = GROUP_M * n_tiles;
    const int g = tile / per_group;
    const int first_m = g * GROUP_M;
    const int gsz = min(GROUP_M, mt - first_m);
    const int r = tile - g * per_group;
    row = base + (first_m + (r % gsz)) * PAIR_BM;
    n_blk = r / gsz;
  };

  if (warp == 0) {
    // ------------------------------------------------------------ TMA producer (both CTAs)
    if (elect_one()) {
      uint32_t it = 0, s = 0, ph = 1u;
      bool ok = true;
      int e = 0;
      for (int unit = pair_id; ok && unit < num_units; unit += num_pairs) {
        int tile, kb0, kb1, row, n_blk, b_row, row_end;
        unit_range(unit, tile, kb0, kb1);
        locate(tile, e, row, n_blk, b_row, row_end);
        const int m0 = row + (int)cta * BM;
        // B rows of this CTA's half of the tile. b_half_stride > 0 (fused gate / up projection): the leader takes 128
        // rows of the first half of B and its peer the 128 rows that lie b_half_stride below them, so columns 0-127 of
        // the accumulator are the gate and columns 128-255 the up projection of the SAME 128 output features.
        const int n0 = b_row + (b_half_stride > 0 ? n_blk * PAIR_HALF_N + (int)cta * b_half_stride
                                                  : n_blk * PAIR_BN + (int)cta * PAIR_HALF_N);
        for (int kb = kb0; kb < kb1; ++kb, ++it) {
          if (!mbar_wait_bounded(&empty_bar[s], ph, abort_flag, err_word, ERR_WAIT_EMPTY)) {
            ok = false;
            break;
          }
          uint8_t* sA = smem + s * S::STAGE_BYTES;
          uint8_t* sB = sA + S::A_BYTES;
          if (cta == 0) mbar_arrive_expect_tx(&full_bar[s], 2 * S::STAGE_BYTES);  // both CTAs' bytes land here
          if constexpr (!A_MN) {
            tma_load_2d_pair(sA, &tmA, &full_bar[s], kb * BK, m0);
          } else {
#pragma unroll
            for (int i = 0; i < BM / 64; ++i)
              tma_load_2d_pair(sA + i * (BK * 128), &tmA, &full_bar[s], m0 + i * 64, kb * BK);
          }
          if constexpr (!B_MN) {
            tma_load_2d_pair(sB, &tmB, &full_bar[s], kb * BK, n0);
          } else {
#pragma unroll
            for (int i = 0; i < PAIR_HALF_N / 64; ++i)
              tma_load_2d_pair(sB + i * (BK * 128), &tmB, &full_bar[s], n0 + i * 64, kb * BK);
          }
          if (++s == STAGES) {
            s = 0;
            ph ^= 1u;
          }
        }
      }
      // drain: the last commits must have released every stage before this CTA's shared memory goes away
      for (uint32_t d = 0; ok && d < (uint32_t)STAGES && d < it; ++d) {
        const uint32_t j = it - 1 - d;
        if (!mbar_wait_bounded(&empty_bar[j % STAGES], (j / STAGES) & 1u, abort_flag, err_word, ERR_WAIT_EMPTY)) break;
      }
    }
    __syncwarp();
  } else if (warp == 1) {
    // ------------------------------------------------------------ MMA issuer (leader only)
    if (cta == 0) {
      const uint32_t idesc = make_idesc_f16(fmt, PAIR_BM, PAIR_BN, A_MN ? 1 : 0, B_MN ? 1 : 0);
      constexpr uint32_t a_lbo = A_MN ? BK * 128 : 16, a_kadv = A_MN ? UMMA_K * 128 : UMMA_K * 2;
      constexpr uint32_t b_lbo = B_MN ? BK * 128 : 16, b_kadv = B_MN ? UMMA_K * 128 : UMMA_K * 2;
      const uint64_t da0 = make_smem_desc_sw128(smem_u32(smem), a_lbo, 1024);
      const uint64_t db0 = make_smem_desc_sw128(smem_u32(smem) + S::A_BYTES, b_lbo, 1024);
      if (elect_one()) {
        uint32_t s = 0, ph = 0u, tl = 0;
        bool ok = true;
        for (int unit = pair_id; ok && unit < num_units; unit += num_pairs, ++tl) {
          int tile, kb0, kb1;
          unit_range(unit, tile, kb0, kb1);
          const uint32_t acc = tl & 1u;
          const uint32_t aph = (tl >> 1) & 1u;
          if (!mbar_wait_bounded(&tempty_bar[acc], aph ^ 1u, abort_flag, err_word, ERR_WAIT_TMEM_EMPTY)) break;
          tc_fence_after_sync();
          const uint32_t d_tmem = tmem_base + acc * PAIR_BN;
          for (int kb = kb0; kb < kb1; ++kb) {
            if (!mbar_wait_bounded(&full_bar[s], ph, abort_flag, err_word, ERR_WAIT_FULL)) {
              ok = false;
              break;
            }
            tc_fence_after_sync();
            const uint64_t off = static_cast<uint64_t>((s * S::STAGE_BYTES) >> 4);
#pragma unroll
            for (int k = 0; k < BK / UMMA_K; ++k)
              umma_f16_ss_pair(d_tmem, da0 + off + static_cast<uint64_t>((k * a_kadv) >> 4),
                               db0 + off + static_cast<uint64_t>((k * b_kadv) >> 4), idesc, (kb != kb0 || k != 0) ? 1u : 0u);
            umma_commit_pair(&empty_bar[s], 0x3);
            if (kb + 1 == kb1) umma_commit_pair(&tfull_bar[acc], 0x3);
            if (++s == STAGES) {
              s = 0;
              ph ^= 1u;
            }
          }
        }
      }
      __syncwarp();
    }
  } else {
    // ------------------------------------------------------------ epilogue warps (both CTAs)
    const int quad = warp & 3;
    static_assert(Epi::WARPS == NUM_EPI_WARPS || (Epi::WARPS == 2 * NUM_EPI_WARPS && !Epi::SPLIT_K && !GROUPED));
    const int col0 = Epi::WARPS == NUM_EPI_WARPS ? 0 : (warp - 2) / NUM_EPI_WARPS * PAIR_HALF_N;
    if (col0) epi_smem += Epi::SMEM_BYTES / 2;
    const uint32_t leader_tempty0 = mapa_shared(smem_u32(&tempty_bar[0]), 0);
    uint32_t tl = 0;
    int e = 0;
    for (int unit = pair_id; unit < num_units; unit += num_pairs, ++tl) {
      int tile, kb0, kb1, row, n_blk, b_row, row_end;
      unit_range(unit, tile, kb0, kb1);
      locate(tile, e, row, n_blk, b_row, row_end);
      const uint32_t acc = tl & 1u;
      const uint32_t aph = (tl >> 1) & 1u;
      if constexpr (Epi::PREFETCH)      // operands from global memory, while the main loop runs
        Epi::prefetch(ep, row + (int)cta * BM, n_blk * PAIR_BN + col0, row_end, N, quad, lane, epi_smem);
      int ok = mbar_wait_bounded(&tfull_bar[acc], aph, abort_flag, err_word, ERR_WAIT_TMEM_FULL) ? 1 : 0;
      ok = __all_sync(0xffffffffu, ok);
      if (!ok) break;
      tc_fence_after_sync();
      const uint32_t taddr = tmem_base + acc * PAIR_BN + col0 + (static_cast<uint32_t>(quad * 32) << 16);
      if constexpr (Epi::SPLIT_K) {
        if (k_splits > 1) {
          const int sp = unit / num_tiles;
          unsigned int* ctr = split_sync + (size_t)tile * 8 + cta * 4 + quad;
          if (sp > 0) {      // the slices before this one have been added
            int ok2 = 1;
            if (lane == 0) ok2 = wait_equal_bounded(ctr, (unsigned)sp, abort_flag, err_word, ERR_WAIT_AUX) ? 1 : 0;
            ok2 = __all_sync(0xffffffffu, ok2);
            if (!ok2) break;
          }
          Epi::tile(Epi::slice_params(ep, sp), taddr, row + (int)cta * BM, n_blk * PAIR_BN + col0, row_end, N, quad,
                    lane, epi_smem);
          __threadfence();
          __syncwarp();
          if (lane == 0) st_release_gpu_u32(ctr, sp + 1 == k_splits ? 0u : (unsigned)(sp + 1));
        } else {
          Epi::tile(ep, taddr, row + (int)cta * BM, n_blk * PAIR_BN + col0, row_end, N, quad, lane, epi_smem);
        }
      } else {
        Epi::tile(ep, taddr, row + (int)cta * BM, n_blk * PAIR_BN + col0, row_end, N, quad, lane, epi_smem);
      }
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive_cluster(leader_tempty0 + acc * 8);
    }
    if constexpr (Epi::PREFETCH) asm volatile("cp.async.wait_all;" ::: "memory");   // of a loop that was given up
  }

  __syncwarp();
  if (*abort_flag) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  cluster_sync_all();  // neither CTA leaves while the other may still touch its barriers
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc_pair(tmem_base, TMEM_COLS);
  }
}

}  // namespace gemm
}  // namespace b200
