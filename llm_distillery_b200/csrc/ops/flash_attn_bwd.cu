// Causal GQA flash-attention backward for sm_100a on tcgen05 tensor cores.
//
// One CTA owns one (batch, kv-head, 128-key block) and a share of the query heads of its group: K_j and V_j stay resident
// in shared memory, dK_j and dV_j accumulate in TMEM over those query heads and every query block at or after the diagonal.
// dQ is produced per (query block, key block) pair, staged in shared memory and added into an fp32 buffer by TMA
// reduce-add (whole 32-byte sectors per request), then converted to bf16 by a small kernel.
//
// Everything is computed TRANSPOSED (thread = key row, tile columns = queries), five tcgen05.mma groups per pair:
//   S^T  = K_j Q_i^T               (A K-major, B K-major)               -> TMEM
//   dP^T = V_j dO_i^T              (A K-major, B K-major)               -> TMEM
//   compute warps: P = exp2(S*c - lse), dS = P * (dP - delta) * scale; P^T goes back into TMEM over S^T, dS^T into TMEM over
//   dP^T (head dim 64) and into shared memory, both bf16
//   dV += P^T  dO_i                (A = P^T from TMEM, B = dO MN-major)
//   dK += dS^T Q_i                 (A = dS^T from TMEM (64) or shared memory K-major (128), B = Q MN-major)
//   dQ  = dS   K_j                 (A = dS^T read MN-major, B = K MN-major)
// so that P never touches shared memory and dS is read from it once (64): per pair the MMAs read 144 KB of operands there
// where the form with queries as rows read 224 KB, at 128 B per clock the busiest path of that form.
//
// Roles (512 threads): warp 0 loads (TMA: Q_i and dO_i rings; -lse and -delta of a query block, scaled, through registers);
// warp 1 issues S and dP, warp 2 dV, warp 3 dK and dQ; warps 4-7 drain dQ (each its own 32 rows: TMEM -> staging -> TMA
// reduce, no barrier between them); warps 8-15 compute, two per TMEM lane quadrant, 64 query columns each.
// Order: S of the next pair is issued while the compute warps work on this one, so they go from dS_i straight to the
// exponentials of pair i + 1 while dK_i, dP_{i+1} and dQ_i run. Head dim 64: two S buffers; P_i in the lower half of its
// buffer, dQ_i in the upper half. Head dim 128 (S, dP, dV, dK take all 512 columns): one S buffer, dQ_i over dP_i.
// The compute warps' fixed work is 16 K exponentials a pair (1024 clocks of the MUFU unit). No single path bounds the kernel
// (head dim 64, 523 us in that run: without the reads of lse and delta 490, without those, exponentials, stores of dS and reduce-adds 408):
// what remains is the chain dS_i -> dK_i -> dP_{i+1} -> dS_{i+1} with its barriers (3270 clocks a pair in all, the tensor pipe busy for 1360),
// with two compute warps per scheduler to fill it. Four of them with 32 columns each measured the same (head dim 64) or slower (128: 80
// registers a thread; 800 against 710 us).
// All three kernels of a backward pass, B200, queries as rows and one S / dP buffer / now: 8 x 2048, 32/4 heads of 64
// 638 / 521 us; 2 x 4000, 32/8 of 128 1191 / 710; 1 x 777, 14/2 of 64 122 / 33 with shared heads. The rotation of dK in the epilogue instead of a
// launch behind it: 2 x 256, 8/2 of 64 21.0 / 16.0 us, 1 x 777, 14/2 34.2 / 32.0, large ones 4 to 10 us.
// Few key blocks (short sequences, few kv heads) leave SMs idle while each CTA walks all query heads of its group: then a
// cluster of up to 8 CTAs may share the heads, and the partial dK / dV meet through distributed shared memory, added in the
// order of the CTAs' ranks (`head_split` below; results repeat bit for bit). dK and dV are as far from fp64 either way (2.3 - 3.0e-3,
// their rounding to bf16; within 0.05 % of each other). The caller has to allow it: under the reference
// loss, whose value after the next update turned the other last bits into up to 0.8 % (777 tokens), the order stays.
#include "../common/ptx.cuh"
#include "../common/host.cuh"

namespace b200 {
namespace fab {

constexpr int BM = 128;  // queries per block
constexpr int BN = 128;  // keys per block
constexpr int NTHREADS = 512;
constexpr int FIRST_DRAIN_WARP = 4;
constexpr int FIRST_COMPUTE_WARP = 8;
constexpr int NCOMPUTE_WARPS = 8;
constexpr int CP = 64;   // query columns of a tile per compute warp; two warps share a TMEM lane quadrant
// Registers a thread after setmaxnreg, of 128 at launch: the compute warps hold 64 probabilities, a drain warp whole rows of dQ
constexpr int REGS_ISSUE = 64, REGS_DRAIN = 152, REGS_COMPUTE = 144;
static_assert(REGS_ISSUE + REGS_DRAIN + 2 * REGS_COMPUTE <= 4 * 128, "registers of the block");
constexpr int SUB = 128 * 128;   // bytes of a [128 rows x 64] bf16 sub-tile with 128-byte rows

template <int D>
struct Cfg {
  static constexpr int QS = (D == 64) ? 3 : 2;     // Q ring: Q_i is read by S_i first and by dK_i last
  static constexpr int OS = (D == 64) ? 2 : 1;     // dO ring: dP_i first, dV_i last
  static constexpr int NSB = (D == 64) ? 2 : 1;    // S buffers in TMEM
  static constexpr int NDS = (D == 64) ? 2 : 1;    // dS buffers in shared memory
  static constexpr bool DS_TMEM = (D == 64);       // dK reads dS^T from TMEM (else from shared memory)
  static constexpr int KV_BYTES = BN * D * 2;   // one of K or V
  static constexpr int Q_BYTES = BM * D * 2;    // one of Q or dO
  static constexpr int P_BYTES = BM * BN * 2;
  static constexpr int OFF_K = 0;
  static constexpr int OFF_V = KV_BYTES;
  static constexpr int OFF_Q = 2 * KV_BYTES;
  static constexpr int OFF_DO = OFF_Q + QS * Q_BYTES;
  static constexpr int OFF_DS = OFF_DO + OS * Q_BYTES;
  static constexpr int OFF_DQS = OFF_DS + NDS * P_BYTES;   // dQ staging: per drain warp two [32 x 32] fp32 tiles, 128B-swizzled
  static constexpr int DQS_BYTES = 4 * 2 * 4096;
  static constexpr int OFF_STAT = OFF_DQS + DQS_BYTES;     // per Q stage: -lse (log2 units) and -delta * scale of 128 queries
  static constexpr int STAT_BYTES = 2 * BM * 4;
  static constexpr int OFF_BAR = OFF_STAT + QS * STAT_BYTES;
  static constexpr int SMEM_BYTES = OFF_BAR + 512;
  static constexpr int RED_PITCH = 2 * D + 4;              // floats per key row of the cluster's dK | dV exchange (over K, V, Q ...)
  static_assert(BN * RED_PITCH * 4 <= OFF_DQS, "the exchange may not reach the staging tiles, which the TMA may still read");
  static_assert(SMEM_BYTES <= 227 * 1024, "shared memory of one CTA");
  static constexpr uint32_t S_COL = 0;
  static constexpr uint32_t DP_COL = NSB * 128;
  static constexpr uint32_t DV_COL = DP_COL + 128;
  static constexpr uint32_t DK_COL = DV_COL + D;
  static constexpr uint32_t TMEM_COLS = 512;
  static_assert(DK_COL + D == TMEM_COLS, "TMEM budget");
  // P^T, 16 queries per 8 columns: at the start of the S buffer (64: dQ needs 64 whole columns behind it, so a warp stores
  // over scores of a warp before it), or each warp's at the start of its own columns (128)
  static constexpr uint32_t P_PART = (D == 64) ? CP / 2 : CP;
  // dQ of a pair: the upper half of its S buffer (64), or over dP (128)
  static __device__ __forceinline__ uint32_t dq_col(int buf) { return D == 64 ? S_COL + buf * 128 + 64 : DP_COL; }
};

struct BwdParams {
  const float* lse;    // [H, T]
  const float* delta;  // [H, T]
  __nv_bfloat16* dqkv; // [T, (H+2Hkv)*D]
  int B, L, H, Hkv;
  int window;          // > 0: the query at position i saw the keys j with i - window < j <= i; 0: all j <= i
  int hsplit;          // CTAs (one cluster) that share the query heads of a group
  float scale;
  const int* pos;      // [T], with the tables below [max_pos, D / 2]: dK leaves with the inverse rotary embedding; null: as it is
  const float* cs;
  const float* sn;
};

// The inverse rotary embedding of N pairs of columns (j, j + D/2), from the values rounded to bf16, with the rope kernel's
// expressions: what that kernel makes of stored gradients, bit for bit. `c`, `sg`: the pairs' entries of the tables.
template <int N>
__device__ __forceinline__ void load_table(const float* src, float (&v)[N]) {
#pragma unroll
  for (int j = 0; j < N; j += 4) {
    const float4 q = __ldg(reinterpret_cast<const float4*>(src + j));
    v[j] = q.x; v[j + 1] = q.y; v[j + 2] = q.z; v[j + 3] = q.w;
  }
}
template <int N>
__device__ __forceinline__ void unrotate(float (&a)[N], float (&b)[N], const float (&c)[N], const float (&sg)[N]) {
#pragma unroll
  for (int j = 0; j < N; ++j) {
    const float fa = __bfloat162float(__float2bfloat16(a[j])), fb = __bfloat162float(__float2bfloat16(b[j]));
    const float sk = sg[j] * -1.f;
    a[j] = __fmaf_rn(fa, c[j], -__fmul_rn(fb, sk));
    b[j] = __fmaf_rn(fb, c[j], __fmul_rn(fa, sk));
  }
}
template <int N>
__device__ __forceinline__ void store_bf16(__nv_bfloat16* dst, const float (&v)[N]) {
#pragma unroll
  for (int j = 0; j < N; j += 8)
    *reinterpret_cast<uint4*>(dst + j) = make_uint4(pack_bf16x2(v[j], v[j + 1]), pack_bf16x2(v[j + 2], v[j + 3]),
                                                    pack_bf16x2(v[j + 4], v[j + 5]), pack_bf16x2(v[j + 6], v[j + 7]));
}

template <int D>
__global__ void __launch_bounds__(NTHREADS, 1)
    flash_bwd_kernel(const __grid_constant__ CUtensorMap tmQKV, const __grid_constant__ CUtensorMap tmDO,
                     const __grid_constant__ CUtensorMap tmDQ, BwdParams p, unsigned int* err_word) {
  using C = Cfg<D>;
  constexpr int QS = C::QS, OS = C::OS, NSB = C::NSB;
  extern __shared__ __align__(1024) uint8_t smem[];
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + C::OFF_BAR);
  // Barriers that more than one pair can complete before their waiter looks are kept per buffer: a parity wait must never
  // be overtaken by two phases. Beside each: who arrives.
  uint64_t* kv_full = bars + 0;
  uint64_t* q_full = bars + 1;      // [QS] TMA bytes + the loader's statistics
  uint64_t* q_empty = bars + 4;     // [QS] dK
  uint64_t* do_full = bars + 7;     // [OS]
  uint64_t* do_empty = bars + 9;    // [OS] dP, dV
  uint64_t* s_full = bars + 11;     // [NSB]
  uint64_t* p_ready = bars + 13;    // [NSB] compute warps
  uint64_t* dv_done = bars + 15;    // [NSB]
  uint64_t* dq_full = bars + 17;    // [NSB]
  uint64_t* dq_empty = bars + 19;   // [NSB] drain warps
  uint64_t* dp_full = bars + 21;
  uint64_t* ds_ready = bars + 22;   // compute warps
  uint64_t* dk_done = bars + 23;
  uint64_t* s_read = bars + 24;     // [2][4] a quadrant's first warp has read its scores: the second may store P there
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 32);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  // blockIdx.y = key block (block 0 has the most work), blockIdx.x = (batch, kv head, share of the heads): blocks are handed
  // out x-fastest, so all the heavy key blocks of every head start first and the light ones fill the tail
  const int jb = blockIdx.y;
  const int part = blockIdx.x % p.hsplit;
  const int bh = blockIdx.x / p.hsplit;
  const int hkv = bh % p.Hkv, b = bh / p.Hkv;
  const int g = p.H / p.Hkv;
  const int h_first = hkv * g + g * part / p.hsplit, h_last = hkv * g + g * (part + 1) / p.hsplit;
  const int kv0 = jb * BN;
  // query blocks that see this key block: from the diagonal to the end, or to the last query whose window reaches back
  const int q_end = p.window > 0 ? min(p.L, kv0 + BN - 1 + p.window) : p.L;
  const int nqb = (q_end + BM - 1) / BM;
  const int i_start = kv0 / BM;
  const int nqi = nqb - i_start;
  const int n_it = (h_last - h_first) * nqi;
  const long long T = (long long)p.B * p.L;

  if ((smem_u32(smem) & 1023u) != 0u) {
    if (threadIdx.x == 0 && err_word) atomicCAS(err_word, 0u, (unsigned)ERR_BAD_ARG);
    return;
  }
  if (threadIdx.x == 0) {
    tma_prefetch_desc(&tmQKV);
    tma_prefetch_desc(&tmDO);
    tma_prefetch_desc(&tmDQ);
    mbar_init(kv_full, 1);
    for (int s = 0; s < QS; ++s) {
      mbar_init(&q_full[s], 2);
      mbar_init(&q_empty[s], 1);
    }
    for (int s = 0; s < OS; ++s) {
      mbar_init(&do_full[s], 1);
      mbar_init(&do_empty[s], 2);
    }
    for (int s = 0; s < NSB; ++s) {
      mbar_init(&s_full[s], 1);
      mbar_init(&p_ready[s], NCOMPUTE_WARPS);
      mbar_init(&dv_done[s], 1);
      mbar_init(&dq_full[s], 1);
      mbar_init(&dq_empty[s], 4);
    }
    mbar_init(dp_full, 1);
    mbar_init(ds_ready, NCOMPUTE_WARPS);
    mbar_init(dk_done, 1);
    for (int s = 0; s < 8; ++s) mbar_init(&s_read[s], 1);
    *abort_flag = 0;
    fence_mbar_init();
  }
  if (warp == 1) {
    tmem_alloc(tmem_slot, C::TMEM_COLS);
    tmem_relinquish();
  }
  tc_fence_before_sync();
  __syncthreads();
  tc_fence_after_sync();
  const uint32_t tmem_base = *tmem_slot;
  pdl_wait();
  pdl_trigger();

  const int colK = p.H * D + hkv * D;
  const int colV = (p.H + p.Hkv) * D + hkv * D;
  // Suspending waits for all: 16 warps that poll take issue slots and shared-memory cycles from the compute warps (538 against
  // 521 us a backward pass of 8 x 2048, 32/4 heads of 64).
  auto wait = [&](uint64_t* bar, uint32_t parity, unsigned int code) {
    return __all_sync(0xffffffffu, mbar_wait_bounded(bar, parity, abort_flag, err_word, code)) != 0;
  };

  if (warp < FIRST_DRAIN_WARP) {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(REGS_ISSUE));
    if (warp == 0) {
      // ---------------------------------------------------------------- loads
      if (elect_one()) {
        mbar_arrive_expect_tx(kv_full, 2 * C::KV_BYTES);
#pragma unroll
        for (int c = 0; c < D / 64; ++c) {
          tma_load_3d(smem + C::OFF_K + c * SUB, &tmQKV, kv_full, colK + c * 64, kv0, b);
          tma_load_3d(smem + C::OFF_V + c * SUB, &tmQKV, kv_full, colV + c * 64, kv0, b);
        }
      }
      __syncwarp();
      float st_l[4], st_d[4];      // statistics of the next query block: loaded one pair ahead
      auto load_stats = [&](int hq, int qb) {
        const long long row = (long long)hq * T + (long long)b * p.L;
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int qi = qb * BM + j * 32 + lane;
          const bool ok = qi < p.L;
          st_l[j] = ok ? p.lse[row + qi] : INFINITY;   // rows past the end: exp2(s - inf) = 0, P and dS vanish
          st_d[j] = ok ? p.delta[row + qi] : 0.f;
        }
      };
      int hq = h_first, qb = i_start;
      load_stats(hq, qb);
      for (int it = 0; it < n_it; ++it) {
        const int qs = it % QS, os = it % OS;
        const int hq_now = hq, q0 = qb * BM;
        if (it >= QS && !wait(&q_empty[qs], (it / QS - 1) & 1u, ERR_WAIT_EMPTY)) break;
        if (elect_one()) {
          uint8_t* sQ = smem + C::OFF_Q + qs * C::Q_BYTES;
          mbar_arrive_expect_tx(&q_full[qs], C::Q_BYTES);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sQ + c * SUB, &tmQKV, &q_full[qs], hq_now * D + c * 64, q0, b);
        }
        __syncwarp();
        float* stat = reinterpret_cast<float*>(smem + C::OFF_STAT + qs * C::STAT_BYTES);
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          stat[j * 32 + lane] = -(st_l[j] * 1.4426950408889634f);
          stat[BM + j * 32 + lane] = -(st_d[j] * p.scale);
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&q_full[qs]);
        if (++qb == nqb) {
          qb = i_start;
          ++hq;
        }
        if (it + 1 < n_it) load_stats(hq, qb);
        if (it >= OS && !wait(&do_empty[os], (it / OS - 1) & 1u, ERR_WAIT_EMPTY)) break;
        if (elect_one()) {
          uint8_t* sDO = smem + C::OFF_DO + os * C::Q_BYTES;
          mbar_arrive_expect_tx(&do_full[os], C::Q_BYTES);
#pragma unroll
          for (int c = 0; c < D / 64; ++c) tma_load_3d(sDO + c * SUB, &tmDO, &do_full[os], hq_now * D + c * 64, q0, b);
        }
        __syncwarp();
      }
    } else {
      // ---------------------------------------------------------------- MMA issuers (warp-uniform loops, one elected lane issues)
      // Base descriptors, built once: inside the loops an MMA's operands are a base plus a constant (k-step) and a
      // stage offset. The address field counts 16-byte units and never carries out of its 14 bits below 256 KB.
      const uint32_t sK = smem_u32(smem + C::OFF_K), sV = smem_u32(smem + C::OFF_V), sQ = smem_u32(smem + C::OFF_Q),
                     sDO = smem_u32(smem + C::OFF_DO), sDS = smem_u32(smem + C::OFF_DS);
      auto koff = [](int k) -> uint64_t {   // k-step inside a K-major tile: 64-column sub-tiles 16 KB apart, 32 B per step
        return static_cast<uint64_t>(((k >> 2) * SUB + (k & 3) * 32) >> 4);
      };
      auto units = [](int n, int bytes) -> uint64_t { return static_cast<uint64_t>((n * bytes) >> 4); };
      if (warp == 1) {
        const uint32_t idesc_kk = make_idesc_f16(1, BN, BM, 0, 0);
        const uint64_t kQ = make_smem_desc_sw128(sQ, 16, 1024), kDO = make_smem_desc_sw128(sDO, 16, 1024);
        const uint64_t kK = make_smem_desc_sw128(sK, 16, 1024), kV = make_smem_desc_sw128(sV, 16, 1024);
        auto issue_s = [&](int it) -> bool {
          if (!wait(&q_full[it % QS], (it / QS) & 1u, ERR_WAIT_FULL)) return false;
          if (it >= NSB) {      // the buffer held P (read by dV) and, head dim 64, dQ of pair it - NSB
            const int o = it - NSB;
            if (!wait(&dv_done[o % NSB], (o / NSB) & 1u, ERR_WAIT_AUX)) return false;
            if (D == 64 && !wait(&dq_empty[o % NSB], (o / NSB) & 1u, ERR_WAIT_AUX)) return false;
          }
          tc_fence_after_sync();
          const uint64_t q = kQ + units(it % QS, C::Q_BYTES);
          const uint32_t dst = tmem_base + C::S_COL + (it % NSB) * 128;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < D / 16; ++k) umma_f16_ss(dst, kK + koff(k), q + koff(k), idesc_kk, k != 0 ? 1u : 0u);
            umma_commit(&s_full[it % NSB]);
          }
          __syncwarp();
          return true;
        };
        bool ok = wait(kv_full, 0, ERR_WAIT_FULL) && issue_s(0);
        for (int it = 0; ok && it < n_it; ++it) {
          if (!wait(&do_full[it % OS], (it / OS) & 1u, ERR_WAIT_FULL)) break;
          if (it > 0) {   // dP of pair it - 1 has been read, and what took its columns since: dS^T by dK (64), dQ by the drain (128)
            if (D == 64 ? !wait(dk_done, (it - 1) & 1u, ERR_WAIT_AUX) : !wait(&dq_empty[0], (it - 1) & 1u, ERR_WAIT_AUX)) break;
          }
          tc_fence_after_sync();
          const uint64_t o = kDO + units(it % OS, C::Q_BYTES);
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < D / 16; ++k)
              umma_f16_ss(tmem_base + C::DP_COL, kV + koff(k), o + koff(k), idesc_kk, k != 0 ? 1u : 0u);
            umma_commit(dp_full);
            umma_commit(&do_empty[it % OS]);
          }
          __syncwarp();
          if (it + 1 < n_it && !issue_s(it + 1)) break;
        }
      } else if (warp == 2) {
        const uint32_t idesc = make_idesc_f16(1, BN, D, 0, 1);
        const uint64_t tDO = make_smem_desc_sw128(sDO, SUB, 1024);
        for (int it = 0; it < n_it; ++it) {
          const int bf = it % NSB;
          if (!wait(&p_ready[bf], (it / NSB) & 1u, ERR_WAIT_AUX)) break;
          if (!wait(&do_full[it % OS], (it / OS) & 1u, ERR_WAIT_FULL)) break;
          tc_fence_after_sync();
          const uint64_t o = tDO + units(it % OS, C::Q_BYTES);
          const uint32_t pcol = tmem_base + C::S_COL + bf * 128;
          if (elect_one()) {
#pragma unroll
            for (int k = 0; k < BM / 16; ++k)
              umma_f16_ts(tmem_base + C::DV_COL, pcol + (k / (CP / 16)) * C::P_PART + (k % (CP / 16)) * 8, o + (uint64_t)(k * 128), idesc,
                          (it != 0 || k != 0) ? 1u : 0u);
            umma_commit(&dv_done[bf]);
            umma_commit(&do_empty[it % OS]);
          }
          __syncwarp();
        }
      } else {
        const uint32_t idesc_dk = make_idesc_f16(1, BN, D, 0, 1);      // A = dS^T with queries as its K dimension
        const uint32_t idesc_dq = make_idesc_f16(1, BM, D, 1, 1);
        const uint64_t tQ = make_smem_desc_sw128(sQ, SUB, 1024), tK = make_smem_desc_sw128(sK, SUB, 1024);
        const uint64_t kDS = make_smem_desc_sw128(sDS, 16, 1024), tDS = make_smem_desc_sw128(sDS, SUB, 1024);
        bool ok = wait(kv_full, 0, ERR_WAIT_FULL);
        for (int it = 0; ok && it < n_it; ++it) {
          if (!wait(ds_ready, it & 1u, ERR_WAIT_AUX)) break;
          tc_fence_after_sync();
          const uint64_t q = tQ + units(it % QS, C::Q_BYTES);
          const uint64_t ds = units(it % C::NDS, C::P_BYTES);
          const uint32_t dq = tmem_base + C::dq_col(it % NSB);
          if (elect_one()) {
            auto dk = [&]() {
#pragma unroll
              for (int k = 0; k < BM / 16; ++k) {
                const uint32_t acc = (it != 0 || k != 0) ? 1u : 0u;
                if constexpr (C::DS_TMEM)   // a compute warp's queries lie at the start of its own columns of dP
                  umma_f16_ts(tmem_base + C::DK_COL, tmem_base + C::DP_COL + (k / (CP / 16)) * CP + (k % (CP / 16)) * 8,
                              q + (uint64_t)(k * 128), idesc_dk, acc);
                else
                  umma_f16_ss(tmem_base + C::DK_COL, kDS + ds + koff(k), q + (uint64_t)(k * 128), idesc_dk, acc);
              }
              umma_commit(dk_done);
              umma_commit(&q_empty[it % QS]);
            };
            auto dqm = [&]() {
#pragma unroll
              for (int k = 0; k < BN / 16; ++k)
                umma_f16_ss(dq, tDS + ds + (uint64_t)(k * 128), tK + (uint64_t)(k * 128), idesc_dq, k != 0 ? 1u : 0u);
              umma_commit(&dq_full[it % NSB]);
            };
            // first what the next dP waits for: dK frees dP's columns (64), dQ has to be drained from them (128)
            if constexpr (D == 64) {
              dk();
              dqm();
            } else {
              dqm();
              dk();
            }
          }
          __syncwarp();
        }
      }
    }
  } else if (warp < FIRST_COMPUTE_WARP) {
    // ------------------------------------------------------------------ dQ: TMEM -> staging -> TMA reduce-add
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_DRAIN));
    const int quad = warp & 3;
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    uint8_t* stage = smem + C::OFF_DQS + quad * 8192;
    int hq = h_first, qb = i_start;
    for (int it = 0; it < n_it; ++it) {
      const int bf = it % NSB;
      if (!wait(&dq_full[bf], (it / NSB) & 1u, ERR_WAIT_AUX)) break;
      tc_fence_after_sync();
      const uint32_t src = tmem_base + lane_addr + C::dq_col(bf);
      constexpr int NR = D / 64;                 // 64 columns a round through the staging tiles
      uint32_t v[2 * NR][32];
#pragma unroll
      for (int c = 0; c < 2 * NR; ++c) tmem_ld_32x32b_x32(src + c * 32, v[c]);
#pragma unroll
      for (int c = 0; c < 2 * NR; ++c) tmem_ld_wait_for(v[c]);
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&dq_empty[bf]);
#pragma unroll
      for (int rr = 0; rr < NR; ++rr) {
        if (lane == 0) tma_store_wait_read0();   // the reduce before this one has read the staging tiles
        __syncwarp();
        uint8_t* rowp = stage + lane * 128;
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
          for (int c = 0; c < 8; ++c)
            *reinterpret_cast<uint4*>(rowp + h * 4096 + (c ^ (lane & 7)) * 16) =
                make_uint4(v[2 * rr + h][c * 4], v[2 * rr + h][c * 4 + 1], v[2 * rr + h][c * 4 + 2], v[2 * rr + h][c * 4 + 3]);
        fence_proxy_async_smem();
        __syncwarp();
        if (lane == 0) {
          const int q0 = qb * BM + quad * 32;
          if (q0 < p.L) {
            tma_reduce_add_3d(&tmDQ, stage, hq * D + rr * 64, q0, b);
            tma_reduce_add_3d(&tmDQ, stage + 4096, hq * D + rr * 64 + 32, q0, b);
          }
          tma_store_commit();
        }
        __syncwarp();
      }
      if (++qb == nqb) {
        qb = i_start;
        ++hq;
      }
    }
    if (lane == 0) tma_store_wait_all0();
  } else {
    // ------------------------------------------------------------------ softmax, dS and the epilogue
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(REGS_COMPUTE));
    const int quad = warp & 3;
    const int cpart = (warp - FIRST_COMPUTE_WARP) >> 2;  // which CP query columns of the tile
    const int r = quad * 32 + lane;                      // key row
    const uint32_t lane_addr = static_cast<uint32_t>(quad * 32) << 16;
    const float c2 = p.scale * 1.4426950408889634f;
    const uint64_t c2p = pack_f32x2(c2, c2), scp = pack_f32x2(p.scale, p.scale);
    const uint32_t tS0 = tmem_base + lane_addr + C::S_COL + cpart * CP;
    const uint32_t tDP = tmem_base + lane_addr + C::DP_COL + cpart * CP;
    bool ok = true;
    int qb = i_start;
    for (int it = 0; it < n_it; ++it) {
      const int bf = it % NSB, qs = it % QS;
      const int q0 = qb * BM;
      if (++qb == nqb) qb = i_start;
      // tile columns lo .. hi (counted from this warp's first) are visible to this key; `masked`: not all of them to every key
      const bool masked = (kv0 + BN - 1) > q0 || (p.window > 0 && q0 + BM - p.window > kv0);
      const int lo = kv0 + r - q0 - cpart * CP;
      const int hi = p.window > 0 ? lo + p.window - 1 : 0x3fffffff;
      const float* stat = reinterpret_cast<const float*>(smem + C::OFF_STAT + qs * C::STAT_BYTES) + cpart * CP;

      // P = exp2(S * c - lse): S_it complete implies that the statistics of its queries are there
      if (!wait(&s_full[bf], (it / NSB) & 1u, ERR_WAIT_TMEM_FULL) || !wait(&q_full[qs], (it / QS) & 1u, ERR_WAIT_FULL)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      uint32_t s[CP / 32][32];
#pragma unroll
      for (int c = 0; c < CP / 32; ++c) tmem_ld_32x32b_x32(tS0 + bf * 128 + c * 32, s[c]);
#pragma unroll
      for (int c = 0; c < CP / 32; ++c) tmem_ld_wait_for(s[c]);
      if (D == 64 && cpart == 0) {
        tc_fence_before_sync();
        __syncwarp();
        if (lane == 0) mbar_arrive(&s_read[bf * 4 + quad]);
      }
#pragma unroll
      for (int c = 0; c < CP / 32; ++c) {
#pragma unroll
        for (int e = 0; e < 32; e += 4) {
          const ulonglong2 nl = *reinterpret_cast<const ulonglong2*>(stat + c * 32 + e);
          float x0, x1, x2, x3;
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s[c][e]), __uint_as_float(s[c][e + 1])), c2p, nl.x), x0, x1);
          unpack_f32x2(fma_f32x2(pack_f32x2(__uint_as_float(s[c][e + 2]), __uint_as_float(s[c][e + 3])), c2p, nl.y), x2, x3);
          s[c][e] = __float_as_uint(fast_exp2(x0));
          s[c][e + 1] = __float_as_uint(fast_exp2(x1));
          s[c][e + 2] = __float_as_uint(fast_exp2(x2));
          s[c][e + 3] = __float_as_uint(fast_exp2(x3));
        }
      }
      if (masked) {
#pragma unroll
        for (int q = 0; q < CP; ++q)
          if (q < lo || q > hi) s[q / 32][q % 32] = 0u;
      }
      uint32_t pk[CP / 32][16];
#pragma unroll
      for (int c = 0; c < CP / 32; ++c)
#pragma unroll
        for (int e = 0; e < 32; e += 2)
          pk[c][e >> 1] = pack_bf16x2(__uint_as_float(s[c][e]), __uint_as_float(s[c][e + 1]));
      if (D == 64 && cpart == 1) {   // these columns are the first warp's scores: long read by now
        if (!wait(&s_read[bf * 4 + quad], (it / NSB) & 1u, ERR_WAIT_AUX)) {
          ok = false;
          break;
        }
        tc_fence_after_sync();
      }
#pragma unroll
      for (int c = 0; c < CP / 32; ++c)
        tmem_st_32x32b_x16(tmem_base + lane_addr + C::S_COL + bf * 128 + cpart * C::P_PART + c * 16, pk[c]);
      tmem_st_wait();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(&p_ready[bf]);

      // dS = P * (dP - delta) * scale
      if (!wait(dp_full, it & 1u, ERR_WAIT_TMEM_FULL)) {
        ok = false;
        break;
      }
      // the one dS tile of head dim 128 is read by dK of the pair before until that is done; with two tiles the drain of
      // dQ_{it-2}, which S_it waited for, has shown that theirs is free
      if (C::NDS == 1 && it > 0 && !wait(dk_done, (it - 1) & 1u, ERR_WAIT_AUX)) {
        ok = false;
        break;
      }
      tc_fence_after_sync();
      uint8_t* srow = smem + C::OFF_DS + (it % C::NDS) * C::P_BYTES + cpart * SUB + r * 128;
      uint32_t dv[2][16];                                 // dP, 16 columns at a time, one load ahead
      tmem_ld_32x32b_x16(tDP, dv[0]);
#pragma unroll
      for (int c = 0; c < CP / 16; ++c) {
        tmem_ld_wait_for(dv[c & 1]);
        if (c + 1 < CP / 16) tmem_ld_32x32b_x16(tDP + (c + 1) * 16, dv[(c + 1) & 1]);
        const uint32_t(&pr)[32] = s[c / 2];
        uint32_t pd[8];
#pragma unroll
        for (int e = 0; e < 16; e += 4) {
          const ulonglong2 nd = *reinterpret_cast<const ulonglong2*>(stat + BM + c * 16 + e);
          const int q = (c & 1) * 16 + e;
          const uint64_t t0 = fma_f32x2(pack_f32x2(__uint_as_float(dv[c & 1][e]), __uint_as_float(dv[c & 1][e + 1])), scp, nd.x);
          const uint64_t t1 = fma_f32x2(pack_f32x2(__uint_as_float(dv[c & 1][e + 2]), __uint_as_float(dv[c & 1][e + 3])), scp, nd.y);
          float y0, y1, y2, y3;
          unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(pr[q]), __uint_as_float(pr[q + 1])), t0), y0, y1);
          unpack_f32x2(mul_f32x2(pack_f32x2(__uint_as_float(pr[q + 2]), __uint_as_float(pr[q + 3])), t1), y2, y3);
          pd[e >> 1] = pack_bf16x2(y0, y1);
          pd[(e >> 1) + 1] = pack_bf16x2(y2, y3);
        }
#pragma unroll
        for (int q4 = 0; q4 < 2; ++q4)
          *reinterpret_cast<uint4*>(srow + ((c * 2 + q4) ^ (r & 7)) * 16) =
              make_uint4(pd[q4 * 4], pd[q4 * 4 + 1], pd[q4 * 4 + 2], pd[q4 * 4 + 3]);
        if constexpr (C::DS_TMEM) tmem_st_32x32b_x8(tDP + c * 8, pd);
      }
      if constexpr (C::DS_TMEM) tmem_st_wait();
      fence_proxy_async_smem();
      tc_fence_before_sync();
      __syncwarp();
      if (lane == 0) mbar_arrive(ds_ready);
    }
    // epilogue: dK_j, dV_j (thread = key row): W columns of the first half of the head and their partners of the second. The
    // tables of the rotation are fetched while the last MMAs run.
    constexpr int W = D / 4;
    const int kvi = kv0 + r;
    const bool row_ok = kvi < p.L;
    const bool rotate = p.pos && row_ok && p.hsplit == 1;
    float rc[W], rs[W];
    if (rotate) {
      const size_t e = (size_t)p.pos[(long long)b * p.L + kvi] * (D / 2) + cpart * W;
      load_table(p.cs + e, rc);
      load_table(p.sn + e, rs);
    }
    if (ok && n_it > 0) {
      const int last = n_it - 1;
      ok = wait(dk_done, last & 1u, ERR_WAIT_AUX) && wait(&dv_done[last % NSB], (last / NSB) & 1u, ERR_WAIT_AUX) &&
           wait(&dq_full[last % NSB], (last / NSB) & 1u, ERR_WAIT_AUX);   // dQ's MMAs have read K: its memory may be reused
    }
    if (ok && n_it > 0) {
      tc_fence_after_sync();
      const long long width = (long long)(p.H + 2 * p.Hkv) * D;
      __nv_bfloat16* row = p.dqkv + ((long long)b * p.L + kvi) * width;
#pragma unroll
      for (int which = 0; which < 2; ++which) {          // dK, dV
        const uint32_t src = tmem_base + lane_addr + (which == 0 ? C::DK_COL : C::DV_COL) + cpart * W;
        uint32_t ra[W], rb[W];
        if constexpr (W == 32) {
          tmem_ld_32x32b_x32(src, ra);
          tmem_ld_32x32b_x32(src + D / 2, rb);
        } else {
          tmem_ld_32x32b_x16(src, ra);
          tmem_ld_32x32b_x16(src + D / 2, rb);
        }
        tmem_ld_wait_for(ra);
        tmem_ld_wait_for(rb);
        if (p.hsplit > 1) {
          float* dst = reinterpret_cast<float*>(smem) + r * C::RED_PITCH + which * D + cpart * W;
#pragma unroll
          for (int j = 0; j < W; j += 4) {
            *reinterpret_cast<uint4*>(dst + j) = make_uint4(ra[j], ra[j + 1], ra[j + 2], ra[j + 3]);
            *reinterpret_cast<uint4*>(dst + D / 2 + j) = make_uint4(rb[j], rb[j + 1], rb[j + 2], rb[j + 3]);
          }
        } else if (row_ok) {
          float fa[W], fb[W];
#pragma unroll
          for (int j = 0; j < W; ++j) {
            fa[j] = __uint_as_float(ra[j]);
            fb[j] = __uint_as_float(rb[j]);
          }
          if (which == 0 && rotate) unrotate(fa, fb, rc, rs);
          __nv_bfloat16* dst = row + (which == 0 ? colK : colV) + cpart * W;
          store_bf16(dst, fa);
          store_bf16(dst + D / 2, fb);
        }
      }
    }
  }

  __syncwarp();
  if (*abort_flag) {
    const unsigned long long t0 = globaltimer_ns();
    while (globaltimer_ns() - t0 < 200000ull) __nanosleep(1000);
  }
  tc_fence_before_sync();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after_sync();
    tmem_dealloc(tmem_base, C::TMEM_COLS);
  }
  if (p.hsplit > 1) {
    // the CTAs of the cluster each sum their share of dK | dV over all of them, in the order of the ranks
    cluster_sync_all();
    const uint32_t rank = cluster_ctarank(), n = (uint32_t)p.hsplit;
    const uint32_t base = smem_u32(smem);
    const long long width = (long long)(p.H + 2 * p.Hkv) * D;
    constexpr int IPR = D / 4;                       // items of a key row: 4 columns and their partners, of dK, then of dV
    const int rows = min(BN, p.L - kv0);
    if (!*abort_flag) {
      for (int i = (int)(rank * NTHREADS + threadIdx.x); i < rows * IPR; i += (int)(n * NTHREADS)) {
        const int row = i / IPR, which = (i - row * IPR) / (D / 8), j0 = (i - row * IPR) % (D / 8) * 4;
        float fa[4] = {0.f, 0.f, 0.f, 0.f}, fb[4] = {0.f, 0.f, 0.f, 0.f};
        const long long t = (long long)b * p.L + kv0 + row;
        const bool rotate = which == 0 && p.pos;
        float rc[4], rs[4];
        if (rotate) {
          const size_t e = (size_t)p.pos[t] * (D / 2) + j0;
          load_table(p.cs + e, rc);
          load_table(p.sn + e, rs);
        }
        const uint32_t at = base + (row * C::RED_PITCH + which * D + j0) * 4;
        for (uint32_t j = 0; j < n; ++j) {
          const float4 x = ld_cluster_f32x4(mapa_shared(at, j)), y = ld_cluster_f32x4(mapa_shared(at + D * 2, j));
          fa[0] += x.x; fa[1] += x.y; fa[2] += x.z; fa[3] += x.w;
          fb[0] += y.x; fb[1] += y.y; fb[2] += y.z; fb[3] += y.w;
        }
        if (rotate) unrotate(fa, fb, rc, rs);
        __nv_bfloat16* dst = p.dqkv + t * width + (which == 0 ? colK : colV) + j0;
        *reinterpret_cast<uint2*>(dst) = make_uint2(pack_bf16x2(fa[0], fa[1]), pack_bf16x2(fa[2], fa[3]));
        *reinterpret_cast<uint2*>(dst + D / 2) = make_uint2(pack_bf16x2(fb[0], fb[1]), pack_bf16x2(fb[2], fb[3]));
      }
    }
    cluster_sync_all();    // nobody's shared memory goes away while a peer reads it
  }
}

// delta[h, t] = sum_d dout[t, h*D + d] * out[t, h*D + d]; one group of D/8 lanes per (t, h). Also zeroes the fp32 dQ
// accumulator: a memset of its own costs a launch and keeps the kernels on both sides of it from overlapping (16 384
// tokens of 32 heads of 64: 35 + 29 us apart, 42 together).
// Bound by HBM: 8 bytes an element. A thread takes 8 elements (they lie in the order of the threads, so only the lane that
// stores a sum needs its token and head), and zeroes two pieces of 16 bytes that lie in runs over the warp. Inside a training
// step of 16 384 x 2048: 51 us (every lane its own 64-bit division, 32 bytes zeroed a lane: 56).
template <int D>
__global__ void __launch_bounds__(256) delta_kernel(const __nv_bfloat16* __restrict__ dout, const __nv_bfloat16* __restrict__ out,
                                                    float* __restrict__ delta, float* __restrict__ dq_acc, long long T, int H) {
  pdl_wait();
  pdl_trigger();
  constexpr int LPG = D / 8;  // lanes per (t,h)
  const long long total = T * H * LPG, gid = blockIdx.x * 256ll + threadIdx.x;
  float s = 0.f;
  const bool ok = gid < total;
  if (ok) {
    const uint4 a = reinterpret_cast<const uint4*>(dout)[gid];
    const uint4 b = reinterpret_cast<const uint4*>(out)[gid];
    const __nv_bfloat162* pa = reinterpret_cast<const __nv_bfloat162*>(&a);
    const __nv_bfloat162* pb = reinterpret_cast<const __nv_bfloat162*>(&b);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      float2 x = __bfloat1622float2(pa[i]), y = __bfloat1622float2(pb[i]);
      s += x.x * y.x + x.y * y.y;
    }
  }
#pragma unroll
  for (int k = 0; k < 2; ++k) {
    const long long z = blockIdx.x * 512ll + k * 256 + threadIdx.x;
    if (z < 2 * total) reinterpret_cast<float4*>(dq_acc)[z] = make_float4(0.f, 0.f, 0.f, 0.f);
  }
#pragma unroll
  for (int o = LPG / 2; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  if (ok && threadIdx.x % LPG == 0) {
    const long long grp = gid / LPG;
    const long long t = grp < 0x7fffffffll ? (uint32_t)grp / (uint32_t)H : grp / H;
    delta[(grp - t * H) * T + t] = s;
  }
}

// dqkv[t, 0:H*D] = bf16(dq_acc[t, :])
__global__ void dq_convert_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dqkv, long long T, int HD,
                                  long long width) {
  pdl_wait();
  pdl_trigger();
  const int hv = HD >> 3;
  const long long total = T * hv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total;
       i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / hv;
    const int v = (int)(i - t * hv);
    const float4 a = reinterpret_cast<const float4*>(acc + t * HD)[2 * v];
    const float4 b = reinterpret_cast<const float4*>(acc + t * HD)[2 * v + 1];
    uint4 o;
    o.x = pack_bf16x2(a.x, a.y);
    o.y = pack_bf16x2(a.z, a.w);
    o.z = pack_bf16x2(b.x, b.y);
    o.w = pack_bf16x2(b.z, b.w);
    reinterpret_cast<uint4*>(dqkv + t * width)[v] = o;
  }
}

// The same with the inverse rotary embedding of the query heads applied on the way: one thread takes the two 4-element
// vectors that the rotation pairs (i and i + D/2 of a head), rounds them to bf16 first - what the stand-alone rope
// kernel would read back - and rotates with that kernel's expressions, so the result is bit-identical to convert + rope.
// Bound by HBM: 6 bytes an element. A block takes TOKENS tokens, a thread's loads of two items are under way together, and
// the grid covers all tokens. Inside a training step of 16 384 x 2048: 44.5 us (two 8-element vectors a thread, 64-bit
// divisions, a resident grid: 56).
constexpr int TOKENS = 4;
template <int D>
__global__ void __launch_bounds__(256) dq_convert_rope_kernel(const float* __restrict__ acc, __nv_bfloat16* __restrict__ dqkv,
                                                              const int* __restrict__ pos, const float* __restrict__ cs,
                                                              const float* __restrict__ sn, long long T, int H, long long width) {
  pdl_wait();
  pdl_trigger();
  constexpr int HALF = D / 2, VPH = HALF / 4;                  // vector pairs per head
  const uint32_t vpt = H * VPH;
  const long long t0 = blockIdx.x * (long long)TOKENS;
  const uint32_t items = (uint32_t)min(T - t0, (long long)TOKENS) * vpt;
  for (uint32_t first = threadIdx.x; first < items; first += 512) {
    float4 a[2], b[2], c[2], g[2];
    long long dst[2];
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const uint32_t i = first + u * 256;
      if (i >= items) continue;
      const uint32_t t = i / vpt, r = i - t * vpt, hd = r / VPH, j = (r - hd * VPH) * 4;
      const float* src = acc + (t0 + t) * (H * D) + hd * D + j;
      a[u] = *reinterpret_cast<const float4*>(src);
      b[u] = *reinterpret_cast<const float4*>(src + HALF);
      const size_t tab = (size_t)pos[t0 + t] * HALF + j;
      c[u] = *reinterpret_cast<const float4*>(cs + tab);
      g[u] = *reinterpret_cast<const float4*>(sn + tab);
      dst[u] = (t0 + t) * width + hd * D + j;
    }
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      if (first + u * 256 >= items) continue;
      const float *pa = &a[u].x, *pb = &b[u].x, *pc = &c[u].x, *pg = &g[u].x;
      float oa[4], ob[4];
#pragma unroll
      for (int k = 0; k < 4; ++k) {
        const float fa = __bfloat162float(__float2bfloat16(pa[k]));
        const float fb = __bfloat162float(__float2bfloat16(pb[k]));
        const float sk = pg[k] * -1.f;                         // the transposed rotation
        oa[k] = __fmaf_rn(fa, pc[k], -__fmul_rn(fb, sk));
        ob[k] = __fmaf_rn(fb, pc[k], __fmul_rn(fa, sk));
      }
      *reinterpret_cast<uint2*>(dqkv + dst[u]) = make_uint2(pack_bf16x2(oa[0], oa[1]), pack_bf16x2(oa[2], oa[3]));
      *reinterpret_cast<uint2*>(dqkv + dst[u] + HALF) = make_uint2(pack_bf16x2(ob[0], ob[1]), pack_bf16x2(ob[2], ob[3]));
    }
  }
}

template <int D>
static int launch_dq_convert_rope(const float* acc, __nv_bfloat16* dqkv, const int* pos, const float* cs, const float* sn,
                                  long long T, int H, long long width, cudaStream_t st) {
  launch_pdl(dq_convert_rope_kernel<D>, (unsigned)((T + TOKENS - 1) / TOKENS), 256, 0, st, acc, dqkv, pos, cs, sn, T, H, width);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// CTAs that share the query heads of one (batch, kv head, key block). The kernel takes about as long as the longer of its
// longest CTA (the first key block: every query block of its heads) and its whole work spread over the SMs, in pairs of
// blocks with kOverhead for a CTA's start and end; the smallest split within 5 % of the best of that is taken, so a grid
// that fills the GPU keeps one CTA per key block.
static int head_split(int B, int L, int window, int H, int Hkv) {
  constexpr double kOverhead = 3.0;
  const int g = H / Hkv, nkb = ceil_div(L, BN);
  long long pairs = 0;    // of one head
  int longest = 0;
  for (int j = 0; j < nkb; ++j) {
    const long long q_end = window > 0 ? (long long)j * BN + BN - 1 + window : L;
    const int n = (int)ceil_div_ll(q_end < L ? q_end : L, BM) - j;
    pairs += n;
    longest = n > longest ? n : longest;
  }
  const double sms = sm_count();
  auto cost = [&](int hs) {
    const double chain = (double)ceil_div(g, hs) * longest + kOverhead;
    const double all = ((double)B * H * pairs + (double)B * Hkv * hs * nkb * kOverhead) / sms;
    return chain > all ? chain : all;
  };
  double best = cost(1);
  for (int hs = 2; hs <= g && hs <= 8; ++hs) best = cost(hs) < best ? cost(hs) : best;
  int hs = 1;
  while (cost(hs) > 1.05 * best) ++hs;
  return hs;
}

template <int D>
static int launch_bwd(const void* dout, const void* qkv, const void* out, const float* lse, float* delta, void* dqkv,
                      float* dq_acc, int B, int L, int window, int H, int Hkv, const int* pos,
                      const float* cos_tab, const float* sin_tab, int share_heads, cudaStream_t st) {
  using C = Cfg<D>;
  const long long width = (long long)(H + 2 * Hkv) * D;
  const long long T = (long long)B * L;
  const long long HD = (long long)H * D;
  CUtensorMap tmQKV, tmDO;
  int rc = make_tmap_3d(&tmQKV, qkv, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)width, (uint64_t)L, (uint64_t)B,
                        (uint64_t)width * 2, (uint64_t)L * width * 2, 64, 128, 1, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  rc = make_tmap_3d(&tmDO, dout, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)HD, (uint64_t)L, (uint64_t)B,
                    (uint64_t)HD * 2, (uint64_t)L * HD * 2, 64, 128, 1, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  CUtensorMap tmDQ;   // one drain warp's 32 rows at a time
  rc = make_tmap_3d(&tmDQ, dq_acc, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 4, (uint64_t)HD, (uint64_t)L, (uint64_t)B,
                    (uint64_t)HD * 4, (uint64_t)L * HD * 4, 32, 32, 1, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  {
    const long long threads = T * H * (D / 8);
    launch_pdl(delta_kernel<D>, (unsigned)((threads + 255) / 256), 256, 0, st, (const __nv_bfloat16*)dout,
                                                                      (const __nv_bfloat16*)out, delta, dq_acc, T, H);
    B200_CUDA_CHECK(cudaGetLastError());
  }
  auto kern = flash_bwd_kernel<D>;
  static bool attr = false;
  if (!attr) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, C::SMEM_BYTES));
    attr = true;
  }
  const int hs = share_heads ? head_split(B, L, window, H, Hkv) : 1;
  BwdParams p{lse, delta, (__nv_bfloat16*)dqkv, B, L, H, Hkv, window, hs, 1.0f / sqrtf((float)D), pos, cos_tab, sin_tab};
  dim3 grid(Hkv * B * hs, (L + BN - 1) / BN);
  if (hs > 1)
    launch_pdl_cluster(kern, grid, NTHREADS, C::SMEM_BYTES, st, hs, tmQKV, tmDO, tmDQ, p, device_err_word());
  else
    launch_pdl(kern, grid, NTHREADS, C::SMEM_BYTES, st, tmQKV, tmDO, tmDQ, p, device_err_word());
  B200_CUDA_CHECK(cudaGetLastError());
  if (pos) return launch_dq_convert_rope<D>(dq_acc, (__nv_bfloat16*)dqkv, pos, cos_tab, sin_tab, T, H, width, st);
  const long long blocks = (T * (HD >> 3) + 255) / 256;
  launch_pdl(dq_convert_kernel, (unsigned)(blocks < 0x7fffffffll ? blocks : 0x7fffffffll), 256, 0, st, dq_acc,
             (__nv_bfloat16*)dqkv, T, (int)HD, width);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

}  // namespace fab
}  // namespace b200

// dq_acc: fp32 scratch [T, H*D] (zeroed here); delta: fp32 scratch [H, T]. dqkv receives dQ | dK | dV.
extern "C" int b200_flash_attn_bwd(const void* dout, const void* qkv, const void* out, const float* lse, float* delta,
                                   void* dqkv, float* dq_acc, int B, int L, int window, int H, int Hkv, int D,
                                   cudaStream_t st) {
  using namespace b200;
  if (!dout || !qkv || !out || !lse || !delta || !dqkv || !dq_acc || B <= 0 || L <= 0 || window < 0 || H <= 0 ||
      Hkv <= 0 || (H % Hkv) != 0)
    return B200_ERR_ARG;
  if (window >= L) window = 0;      // causal; also keeps the sum of position and window inside 32 bits
  if (D == 64) return fab::launch_bwd<64>(dout, qkv, out, lse, delta, dqkv, dq_acc, B, L, window, H, Hkv, nullptr, nullptr, nullptr, 0, st);
  if (D == 128)
    return fab::launch_bwd<128>(dout, qkv, out, lse, delta, dqkv, dq_acc, B, L, window, H, Hkv, nullptr, nullptr, nullptr, 0, st);
  return B200_ERR_ARG;
}

// The same with the inverse rotary embedding of the query and key heads (pos int32 [B*L]; cos / sin fp32 [max_pos, D/2]; pos
// null: without): where the fp32 dQ accumulator is converted to bf16 and in the main kernel's epilogue. share_heads: the query
// heads of a group may be shared by a cluster where that is faster; the order of the additions into dK and dV then depends on
// the sizes. Without it the heads of a group are added one after the other at every size.
extern "C" int b200_flash_attn_bwd_rope(const void* dout, const void* qkv, const void* out, const float* lse,
                                        float* delta, void* dqkv, float* dq_acc, const int* pos, const float* cos_tab,
                                        const float* sin_tab, int B, int L, int window, int H, int Hkv, int D, int share_heads,
                                        cudaStream_t st) {
  using namespace b200;
  if (!dout || !qkv || !out || !lse || !delta || !dqkv || !dq_acc || (pos && (!cos_tab || !sin_tab)) || B <= 0 || L <= 0 ||
      window < 0 || H <= 0 || Hkv <= 0 || (H % Hkv) != 0)
    return B200_ERR_ARG;
  if (window >= L) window = 0;      // causal; also keeps the sum of position and window inside 32 bits
  if (D == 64) return fab::launch_bwd<64>(dout, qkv, out, lse, delta, dqkv, dq_acc, B, L, window, H, Hkv, pos, cos_tab, sin_tab, share_heads, st);
  if (D == 128)
    return fab::launch_bwd<128>(dout, qkv, out, lse, delta, dqkv, dq_acc, B, L, window, H, Hkv, pos, cos_tab, sin_tab, share_heads, st);
  return B200_ERR_ARG;
}

// The conversion pass alone (fp32 dQ accumulator -> bf16 query columns of dqkv with the inverse rotation): exported so
// that its bit-exactness against convert + rope kernel can be tested on a given accumulator.
extern "C" int b200_dq_convert_rope(const float* acc, void* dqkv, const int* pos, const float* cos_tab,
                                    const float* sin_tab, long long T, int H, int D, long long width, cudaStream_t st) {
  using namespace b200;
  if (!acc || !dqkv || !pos || !cos_tab || !sin_tab || T <= 0 || H <= 0 || (D != 64 && D != 128)) return B200_ERR_ARG;
  return D == 64 ? fab::launch_dq_convert_rope<64>(acc, (__nv_bfloat16*)dqkv, pos, cos_tab, sin_tab, T, H, width, st)
                 : fab::launch_dq_convert_rope<128>(acc, (__nv_bfloat16*)dqkv, pos, cos_tab, sin_tab, T, H, width, st);
}
