// Plain GEMM entry points on the tcgen05 mainloop (gemm_core.cuh):
//   C[M,N] = alpha * A * B^T (+ C) (+ residual)     bf16/fp16 operands, fp32 accumulate,
// with A and B each either K-major or MN-major, so forward (NT), dgrad (NN) and wgrad (TN)
// GEMMs of a linear layer all run without a transpose pass.
#include "gemm_pair.cuh"
#include "gemm_cluster.cuh"
#include <stdlib.h>
#include <atomic>
#include "../common/host.cuh"

namespace b200 {
namespace gemm {

struct StoreParams {
  void* C;
  long long ldc;               // elements
  const __nv_bfloat16* resid;  // optional residual added to the result (bf16, same shape as C), may be null
  long long ldr;
  float alpha;
  int out_f32;     // 1: C is fp32, 0: C is 16-bit (bf16 or fp16 according to fmt)
  int accumulate;  // 1: C += result
  int fmt;         // 0 fp16, 1 bf16 (16-bit output type)
};

template <int BN>
struct EpiStore {
  using Params = StoreParams;
  static constexpr bool SPLIT_K = true;   // the pair kernel may cut the K loop into slices that are added in order
  static constexpr bool PREFETCH = false;
  static constexpr int WARPS = NUM_EPI_WARPS;
  // slice 0 of a tile stores (or adds to what C held, if the caller accumulates); every later slice adds
  static __device__ __forceinline__ Params slice_params(const Params& p, int slice) {
    Params q = p;
    if (slice > 0) q.accumulate = 1;
    return q;
  }
  static constexpr int STAGE_BYTES = 32 * 256;              // per epilogue warp: 32 rows x 128 bf16 columns
  static constexpr int SMEM_BYTES = NUM_EPI_WARPS * STAGE_BYTES;

  // bf16 output without accumulation (forward and dgrad GEMMs): the warp's 32 x 128 slice goes through a swizzled
  // shared-memory stage so that each store instruction writes two whole 256-byte row segments instead of 32
  // scattered 16-byte pieces. alpha and the residual are applied in fp32 before the rounding to bf16.
  static __device__ __forceinline__ void tile_staged(const Params& p, uint32_t taddr, int m0, int n0, int M, int N,
                                                     int quad, int lane, uint8_t* epi_smem) {
    uint8_t* stage = epi_smem + quad * STAGE_BYTES;
    const int row0 = m0 + quad * 32;
    const int rows_valid = min(32, M - row0);
    const bool my_row_ok = lane < rows_valid;
    __nv_bfloat16* C = reinterpret_cast<__nv_bfloat16*>(p.C);
#pragma unroll 1
    for (int half = 0; half < BN / 128; ++half) {
#pragma unroll 1
      for (int c4 = 0; c4 < 4; ++c4) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + half * 128 + c4 * 32, r);
        tmem_ld_wait();
        const int col0 = n0 + half * 128 + c4 * 32;
        float v[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * p.alpha;
        if (p.resid && my_row_ok && col0 < N) {
          const __nv_bfloat16* rp = p.resid + (long long)(row0 + lane) * p.ldr + col0;
          if (col0 + 32 <= N && ((reinterpret_cast<uintptr_t>(rp) & 15) == 0)) {
#pragma unroll
            for (int j = 0; j < 4; ++j) {
              const uint4 q = *reinterpret_cast<const uint4*>(rp + j * 8);
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                const float2 f = __bfloat1622float2(h[t]);
                v[j * 8 + t * 2] += f.x;
                v[j * 8 + t * 2 + 1] += f.y;
              }
            }
          } else {
            const int ncols = min(32, N - col0);
#pragma unroll
            for (int j = 0; j < 32; ++j)
              if (j < ncols) v[j] += __bfloat162float(rp[j]);
          }
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 o;
          o.x = pack_bf16x2(v[j * 8 + 0], v[j * 8 + 1]);
          o.y = pack_bf16x2(v[j * 8 + 2], v[j * 8 + 3]);
          o.z = pack_bf16x2(v[j * 8 + 4], v[j * 8 + 5]);
          o.w = pack_bf16x2(v[j * 8 + 6], v[j * 8 + 7]);
          const int chunk = c4 * 4 + j;
          *reinterpret_cast<uint4*>(stage + lane * 256 + ((chunk ^ (lane & 15)) << 4)) = o;
        }
      }
      __syncwarp();
      const int chunk = lane & 15;
      const int col = n0 + half * 128 + chunk * 8;
#pragma unroll 4
      for (int j = 0; j < 16; ++j) {
        const int row = 2 * j + (lane >> 4);
        const uint4 o = *reinterpret_cast<const uint4*>(stage + row * 256 + ((chunk ^ (row & 15)) << 4));
        if (row < rows_valid && col < N) *reinterpret_cast<uint4*>(C + (long long)(row0 + row) * p.ldc + col) = o;
      }
      __syncwarp();
    }
  }

  // fp32 output (weight gradients, with or without accumulation): 64 columns of the warp's 32 rows at a time go
  // through the same swizzled stage, so that one instruction reads-modifies-writes 256 contiguous bytes of two rows
  // (whole sectors) instead of 16 bytes of 32 different rows.
  static __device__ __forceinline__ void tile_staged_f32(const Params& p, uint32_t taddr, int m0, int n0, int M, int N,
                                                         int quad, int lane, uint8_t* epi_smem) {
    uint8_t* stage = epi_smem + quad * STAGE_BYTES;
    const int row0 = m0 + quad * 32;
    const int rows_valid = min(32, M - row0);
    float* C = reinterpret_cast<float*>(p.C);
#pragma unroll 1
    for (int g = 0; g < BN / 64; ++g) {
#pragma unroll
      for (int c2 = 0; c2 < 2; ++c2) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + g * 64 + c2 * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 8; ++j) {
          const float4 o = make_float4(__uint_as_float(r[4 * j]) * p.alpha, __uint_as_float(r[4 * j + 1]) * p.alpha,
                                       __uint_as_float(r[4 * j + 2]) * p.alpha, __uint_as_float(r[4 * j + 3]) * p.alpha);
          const int chunk = c2 * 8 + j;
          *reinterpret_cast<float4*>(stage + lane * 256 + ((chunk ^ (lane & 15)) << 4)) = o;
        }
      }
      __syncwarp();
      const int chunk = lane & 15;
      const int col = n0 + g * 64 + chunk * 4;
#pragma unroll 4
      for (int j = 0; j < 16; ++j) {
        const int row = 2 * j + (lane >> 4);
        float4 o = *reinterpret_cast<const float4*>(stage + row * 256 + ((chunk ^ (row & 15)) << 4));
        if (row < rows_valid && col < N) {
          float* cp = C + (long long)(row0 + row) * p.ldc + col;
          if (p.accumulate) {
            // a reduction, not a load + add + store: the L2 round trip of the load made short K slices epilogue-bound.
            // The order of the additions into one element is still fixed: the slices of a tile take turns (the
            // counter protocol of the pair kernel, with a fence before each hand-over) and nothing else adds to C.
            asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" ::"l"(cp), "f"(o.x), "f"(o.y), "f"(o.z), "f"(o.w)
                         : "memory");
          } else {
            *reinterpret_cast<float4*>(cp) = o;
          }
        }
      }
      __syncwarp();
    }
  }

  static __device__ __forceinline__ void tile(const Params& p, uint32_t taddr, int m0, int n0, int M, int N, int quad,
                                              int lane, uint8_t* epi_smem) {
    if (!p.out_f32 && p.fmt == 1 && !p.accumulate && !(N & 7) && !(p.ldc & 7) &&
        !(reinterpret_cast<uintptr_t>(p.C) & 15)) {
      tile_staged(p, taddr, m0, n0, M, N, quad, lane, epi_smem);
      return;
    }
    if (p.out_f32 && !p.resid && !(N & 3) && !(p.ldc & 3) && !(reinterpret_cast<uintptr_t>(p.C) & 15)) {
      tile_staged_f32(p, taddr, m0, n0, M, N, quad, lane, epi_smem);
      return;
    }
    const int row = m0 + quad * 32 + lane;
    const bool row_ok = row < M;
#pragma unroll 1
    for (int c = 0; c < BN / 32; ++c) {
      uint32_t r[32];
      __syncwarp();  // lanes may have diverged in the previous chunk; tcgen05.ld is warp-collective
      tmem_ld_32x32b_x32(taddr + c * 32, r);
      tmem_ld_wait();
      const int col0 = n0 + c * 32;
      if (!row_ok || col0 >= N) continue;
      float v[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) v[j] = __uint_as_float(r[j]) * p.alpha;
      const int ncols = min(32, N - col0);
      if (p.resid) {
        const __nv_bfloat16* rp = p.resid + (long long)row * p.ldr + col0;
        if (ncols == 32 && ((reinterpret_cast<uintptr_t>(rp) & 15) == 0)) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            uint4 q = *reinterpret_cast<const uint4*>(rp + j * 8);
            const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
            for (int t = 0; t < 4; ++t) {
              float2 f = __bfloat1622float2(h[t]);
              v[j * 8 + t * 2] += f.x;
              v[j * 8 + t * 2 + 1] += f.y;
            }
          }
        } else {
          for (int j = 0; j < ncols; ++j) v[j] += __bfloat162float(rp[j]);
        }
      }
      if (p.out_f32) {
        float* cp = reinterpret_cast<float*>(p.C) + (long long)row * p.ldc + col0;
        if (ncols == 32 && ((reinterpret_cast<uintptr_t>(cp) & 15) == 0)) {
#pragma unroll
          for (int j = 0; j < 8; ++j) {
            float4 o = make_float4(v[j * 4], v[j * 4 + 1], v[j * 4 + 2], v[j * 4 + 3]);
            if (p.accumulate) {
              float4 old = *reinterpret_cast<float4*>(cp + j * 4);
              o.x += old.x; o.y += old.y; o.z += old.z; o.w += old.w;
            }
            *reinterpret_cast<float4*>(cp + j * 4) = o;
          }
        } else {
          for (int j = 0; j < ncols; ++j) cp[j] = p.accumulate ? cp[j] + v[j] : v[j];
        }
      } else if (p.fmt == 1) {
        __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)row * p.ldc + col0;
        if (ncols == 32 && ((reinterpret_cast<uintptr_t>(cp) & 15) == 0)) {
#pragma unroll
          for (int j = 0; j < 4; ++j) {
            if (p.accumulate) {
              uint4 q = *reinterpret_cast<const uint4*>(cp + j * 8);
              const __nv_bfloat162* h = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
              for (int t = 0; t < 4; ++t) {
                float2 f = __bfloat1622float2(h[t]);
                v[j * 8 + t * 2] += f.x;
                v[j * 8 + t * 2 + 1] += f.y;
              }
            }
            uint4 o;
            o.x = pack_bf16x2(v[j * 8 + 0], v[j * 8 + 1]);
            o.y = pack_bf16x2(v[j * 8 + 2], v[j * 8 + 3]);
            o.z = pack_bf16x2(v[j * 8 + 4], v[j * 8 + 5]);
            o.w = pack_bf16x2(v[j * 8 + 6], v[j * 8 + 7]);
            *reinterpret_cast<uint4*>(cp + j * 8) = o;
          }
        } else {
          for (int j = 0; j < ncols; ++j) {
            float x = v[j] + (p.accumulate ? __bfloat162float(cp[j]) : 0.f);
            cp[j] = __float2bfloat16(x);
          }
        }
      } else {
        __half* cp = reinterpret_cast<__half*>(p.C) + (long long)row * p.ldc + col0;
        for (int j = 0; j < ncols; ++j) {
          float x = v[j] + (p.accumulate ? __half2float(cp[j]) : 0.f);
          cp[j] = __float2half(x);
        }
      }
    }
  }
};

// Fused gate / up projection + SwiGLU on the CTA-pair kernel. The accumulator of a tile holds, for 256 rows, the gate
// (columns 0-127) and the up projection (columns 128-255) of the same 128 features (the B halves come from rows
// j*128 and f + j*128 of the fused weight, gemm_pair.cuh). The epilogue writes three things per row: gate and up,
// rounded to bf16, into gu [M, 2f] (the backward pass reads them; without one, two thirds of the output and of the epilogue
// go: 16384 x 2048 -> 5632 510 us, then 475), and act = silu(gate) * up computed from the ROUNDED
// values, so that it equals what the stand-alone SwiGLU kernel makes of gu bit for bit. Each leaves through the
// swizzled stage as 256-byte row segments.
struct SwigluParams {
  __nv_bfloat16* gu;    // [M, 2f]; null: not written
  long long ld_gu;
  __nv_bfloat16* act;   // [M, f]
  long long ld_act;
  int f;
};

struct EpiSwiglu {
  using Params = SwigluParams;
  static constexpr bool SPLIT_K = false;
  static constexpr bool PREFETCH = false;
  static constexpr int WARPS = NUM_EPI_WARPS;
  static constexpr int STAGE_BYTES = 32 * 256;
  static constexpr int SMEM_BYTES = NUM_EPI_WARPS * STAGE_BYTES;

  static __device__ __forceinline__ void flush(uint8_t* stage, __nv_bfloat16* dst, long long ld, int row0, int rows_valid,
                                               int col0, int f, int lane) {
    __syncwarp();
    const int chunk = lane & 15;
    const int col = col0 + chunk * 8;
#pragma unroll 4
    for (int j = 0; j < 16; ++j) {
      const int row = 2 * j + (lane >> 4);
      const uint4 o = *reinterpret_cast<const uint4*>(stage + row * 256 + ((chunk ^ (row & 15)) << 4));
      if (row < rows_valid && col < f) *reinterpret_cast<uint4*>(dst + (long long)(row0 + row) * ld + col) = o;
    }
    __syncwarp();
  }

  static __device__ __forceinline__ void tile(const Params& p, uint32_t taddr, int m0, int n0, int M, int N, int quad,
                                              int lane, uint8_t* epi_smem) {
    uint8_t* stage = epi_smem + quad * STAGE_BYTES;
    const int row0 = m0 + quad * 32;
    const int rows_valid = min(32, M - row0);
    const int col0 = (n0 / PAIR_BN) * PAIR_HALF_N;       // first of the tile's 128 features
    // gate, then up: rounded copies into gu
#pragma unroll 1
    for (int half = p.gu ? 0 : 2; half < 2; ++half) {
#pragma unroll 1
      for (int c4 = 0; c4 < 4; ++c4) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + half * 128 + c4 * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          uint4 o;
          o.x = pack_bf16x2(__uint_as_float(r[j * 8 + 0]), __uint_as_float(r[j * 8 + 1]));
          o.y = pack_bf16x2(__uint_as_float(r[j * 8 + 2]), __uint_as_float(r[j * 8 + 3]));
          o.z = pack_bf16x2(__uint_as_float(r[j * 8 + 4]), __uint_as_float(r[j * 8 + 5]));
          o.w = pack_bf16x2(__uint_as_float(r[j * 8 + 6]), __uint_as_float(r[j * 8 + 7]));
          const int chunk = c4 * 4 + j;
          *reinterpret_cast<uint4*>(stage + lane * 256 + ((chunk ^ (lane & 15)) << 4)) = o;
        }
      }
      flush(stage, p.gu + (half ? p.f : 0), p.ld_gu, row0, rows_valid, col0, p.f, lane);
    }
    // act = silu(gate) * up from the rounded values
#pragma unroll 1
    for (int c4 = 0; c4 < 4; ++c4) {
      uint32_t g[32], u[32];
      tmem_ld_32x32b_x32(taddr + c4 * 32, g);
      tmem_ld_32x32b_x32(taddr + 128 + c4 * 32, u);
      tmem_ld_wait();
      float a[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) {
        const float gj = __bfloat162float(__float2bfloat16(__uint_as_float(g[j])));
        const float uj = __bfloat162float(__float2bfloat16(__uint_as_float(u[j])));
        a[j] = __fdividef(gj, 1.f + __expf(-gj)) * uj;
      }
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        uint4 o;
        o.x = pack_bf16x2(a[j * 8 + 0], a[j * 8 + 1]);
        o.y = pack_bf16x2(a[j * 8 + 2], a[j * 8 + 3]);
        o.z = pack_bf16x2(a[j * 8 + 4], a[j * 8 + 5]);
        o.w = pack_bf16x2(a[j * 8 + 6], a[j * 8 + 7]);
        const int chunk = c4 * 4 + j;
        *reinterpret_cast<uint4*>(stage + lane * 256 + ((chunk ^ (lane & 15)) << 4)) = o;
      }
    }
    flush(stage, p.act, p.ld_act, row0, rows_valid, col0, p.f, lane);
  }
};

// Rotary embedding in the epilogue of the fused q/k/v projection. A head of d = 64 is two 32-column chunks of the
// accumulator, a head of d = 128 four; the rotation pairs column i with i + d/2, i.e. chunk c with chunk c + 1 (d = 64)
// or c + 2 (d = 128) of the same 128-column half. Each lane owns one row, fetches the cos / sin entries of that row's
// position, rounds the two chunks to bf16 first (what the stand-alone kernel reads back from memory) and rotates with
// the same expressions, so the result is bit-identical to GEMM + rope kernel. Columns from n_rot on (the value heads)
// are stored unrotated.
struct RopeParams {
  __nv_bfloat16* C;     // [M, N]
  long long ldc;
  const int* pos;       // [M]
  const float* cs;      // [max_pos, d/2]
  const float* sn;
  int d;                // 64 or 128
  int n_rot;            // first n_rot columns are rotated ((H + Hkv) * d)
};

template <int D>
struct EpiRope {
  using Params = RopeParams;
  static constexpr bool SPLIT_K = false;
  static constexpr bool PREFETCH = false;
  static constexpr int WARPS = NUM_EPI_WARPS;
  static constexpr int STAGE_BYTES = 32 * 256;
  static constexpr int SMEM_BYTES = NUM_EPI_WARPS * STAGE_BYTES;

  static __device__ __forceinline__ void put(uint8_t* stage, int lane, int c4, const float (&v)[32]) {
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      uint4 o;
      o.x = pack_bf16x2(v[j * 8 + 0], v[j * 8 + 1]);
      o.y = pack_bf16x2(v[j * 8 + 2], v[j * 8 + 3]);
      o.z = pack_bf16x2(v[j * 8 + 4], v[j * 8 + 5]);
      o.w = pack_bf16x2(v[j * 8 + 6], v[j * 8 + 7]);
      const int chunk = c4 * 4 + j;
      *reinterpret_cast<uint4*>(stage + lane * 256 + ((chunk ^ (lane & 15)) << 4)) = o;
    }
  }

  static __device__ __forceinline__ void tile(const Params& p, uint32_t taddr, int m0, int n0, int M, int N, int quad,
                                              int lane, uint8_t* epi_smem) {
    uint8_t* stage = epi_smem + quad * STAGE_BYTES;
    const int row0 = m0 + quad * 32;
    const int rows_valid = min(32, M - row0);
    constexpr int half_d = D >> 1;
    const long long tpos = lane < rows_valid ? (long long)p.pos[row0 + lane] : 0;
    // heads of 64: all pairs of a row take the same 32 entries, fetched once for the tile (once per pair: 16384 x 2560 x 2048
    // 130 us, now 116)
    float cc[32], ss[32];
    auto entries = [&](int j0) {
      const float* cp = p.cs + tpos * half_d + j0;
      const float* sp = p.sn + tpos * half_d + j0;
#pragma unroll
      for (int j = 0; j < 32; j += 4) {
        const float4 c4 = *reinterpret_cast<const float4*>(cp + j), s4 = *reinterpret_cast<const float4*>(sp + j);
        cc[j] = c4.x; cc[j + 1] = c4.y; cc[j + 2] = c4.z; cc[j + 3] = c4.w;
        ss[j] = s4.x; ss[j + 1] = s4.y; ss[j + 2] = s4.z; ss[j + 3] = s4.w;
      }
    };
    if (D == 64 && n0 < p.n_rot) entries(0);
#pragma unroll 1
    for (int half = 0; half < 2; ++half) {
      const int colh = n0 + half * 128;
      if (colh >= N) break;                               // N is a multiple of 128
#pragma unroll 1
      for (int k = 0; k < 2; ++k) {
        // d = 64: pair (0,1) then (2,3); d = 128: pair (0,2) then (1,3)
        const int ca = D == 64 ? 2 * k : k;
        const int cb = ca + (D == 64 ? 1 : 2);
        uint32_t ra[32], rb[32];
        tmem_ld_32x32b_x32(taddr + half * 128 + ca * 32, ra);
        tmem_ld_32x32b_x32(taddr + half * 128 + cb * 32, rb);
        const bool rotate = colh + ca * 32 < p.n_rot;
        if (D == 128 && rotate) entries(k * 32);
        tmem_ld_wait_for(ra);
        tmem_ld_wait_for(rb);
        float a[32], b[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) {
          a[j] = __bfloat162float(__float2bfloat16(__uint_as_float(ra[j])));
          b[j] = __bfloat162float(__float2bfloat16(__uint_as_float(rb[j])));
        }
        if (rotate) {
#pragma unroll
          for (int j = 0; j < 32; ++j) {
            const float fa = a[j], fb = b[j];
            a[j] = __fmaf_rn(fa, cc[j], -__fmul_rn(fb, ss[j]));
            b[j] = __fmaf_rn(fb, cc[j], __fmul_rn(fa, ss[j]));
          }
        }
        put(stage, lane, ca, a);
        put(stage, lane, cb, b);
      }
      EpiSwiglu::flush(stage, p.C, p.ldc, row0, rows_valid, colh, N, lane);
    }
  }
};

template <int D>
static int launch_rope_pair(const void* A, const void* W, int M, int N, int K, long long lda, long long ldb,
                            const RopeParams& rp, cudaStream_t stream) {
  using Epi = EpiRope<D>;
  constexpr int STAGES = 6;
  using S = SmemPair<STAGES>;
  CUtensorMap tmA, tmB;
  int rc = make_tmap_2d(&tmA, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  rc = make_tmap_2d(&tmB, W, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, BK,
                    PAIR_HALF_N, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  auto kern = gemm_pair_kernel<STAGES, false, false, Epi>;
  const int smem_bytes = S::bytes(Epi::SMEM_BYTES);
  static bool attr_set = false;
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    attr_set = true;
  }
  const int tiles = ceil_div(M, PAIR_BM) * ceil_div(N, PAIR_BN);
  const int max_pairs = sm_count() / 2;
  const int pairs = tiles < max_pairs ? tiles : max_pairs;
  launch_pdl(kern, 2 * pairs, pair_threads<Epi>(), smem_bytes, stream, tmA, tmB, M, N, K, 1, rp, device_err_word(), 1, nullptr, 0,
               gemm::GroupArgs{});
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// Backward of SwiGLU in the epilogue of the down projection's dgrad GEMM: the accumulator tile is d(act) for 256 tokens
// x 256 features. A warp takes its 32 rows in quarters of 64 columns: the matching gate and up values come by asynchronous
// copies of whole 128-byte row segments into one of two swizzled stages while it works on the quarter before (the first one's
// while the main loop still runs), every lane then works on its own row - d(act) rounded to bf16 first, so that the
// result equals GEMM + stand-alone kernel bit for bit - and overwrites the stage with d(gate) and d(up), which leave
// as whole row segments. d(act) itself is never written. With the loads in front of each half, through registers, a tile's
// epilogue took longer than its main loop: 16384 x 2048 -> 5632 379 us,
// now 321 (under the power cap 470 / 342).
struct SwigluBwdParams {
  const __nv_bfloat16* gu;   // [M, 2f] saved by the forward pass
  long long ld_gu;
  __nv_bfloat16* dgu;        // [M, 2f]
  long long ld_dgu;
  int f;
};

struct EpiSwigluBwd {
  using Params = SwigluBwdParams;
  static constexpr bool SPLIT_K = false;
  static constexpr bool PREFETCH = true;
  static constexpr int WARPS = NUM_EPI_WARPS;
  static constexpr int QUARTER = 32 * 128;               // gate or up values of a quarter
  static constexpr int STAGE_BYTES = 2 * 2 * QUARTER;    // two stages of both per epilogue warp
  static constexpr int SMEM_BYTES = NUM_EPI_WARPS * STAGE_BYTES;

  static __device__ __forceinline__ int rows_of(int m0, int M, int quad) { return min(32, M - (m0 + quad * 32)); }

  // gate and up values of quarter q into its stage, as one group of copies (empty where the quarter lies beyond N)
  static __device__ __forceinline__ void fetch(const Params& p, int q, int m0, int n0, int M, int N, int quad, int lane,
                                               uint8_t* epi_smem) {
    const int rows = rows_of(m0, M, quad), col = n0 + q * 64 + (lane & 7) * 8;
    if (n0 + q * 64 < N) {
      const uint32_t sg = smem_u32(epi_smem + quad * STAGE_BYTES + (q & 1) * 2 * QUARTER);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = 4 * j + (lane >> 3);
        if (row < rows) {
          const __nv_bfloat16* src = p.gu + (long long)(m0 + quad * 32 + row) * p.ld_gu + col;
          const uint32_t dst = sg + row * 128 + (((lane & 7) ^ (row & 7)) << 4);
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + QUARTER), "l"(src + p.f) : "memory");
        }
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  static __device__ __forceinline__ void prefetch(const Params& p, int m0, int n0, int M, int N, int quad, int lane,
                                                  uint8_t* epi_smem) {
    fetch(p, 0, m0, n0, M, N, quad, lane, epi_smem);
  }

  static __device__ __forceinline__ void tile(const Params& p, uint32_t taddr, int m0, int n0, int M, int N, int quad,
                                              int lane, uint8_t* epi_smem) {
    const int rows = rows_of(m0, M, quad), row0 = m0 + quad * 32;
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      if (q < 3) {
        fetch(p, q + 1, m0, n0, M, N, quad, lane, epi_smem);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncwarp();
      if (n0 + q * 64 >= N) continue;                    // N is a multiple of 128
      uint8_t* sg = epi_smem + quad * STAGE_BYTES + (q & 1) * 2 * QUARTER;
      uint8_t* su = sg + QUARTER;
#pragma unroll
      for (int c = 0; c < 2; ++c) {
        uint32_t r[32];
        tmem_ld_32x32b_x32(taddr + q * 64 + c * 32, r);
        tmem_ld_wait();
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int off = lane * 128 + (((c * 4 + j) ^ (lane & 7)) << 4);
          const uint4 qg = *reinterpret_cast<const uint4*>(sg + off);
          const uint4 qu = *reinterpret_cast<const uint4*>(su + off);
          const __nv_bfloat162* hg = reinterpret_cast<const __nv_bfloat162*>(&qg);
          const __nv_bfloat162* hu = reinterpret_cast<const __nv_bfloat162*>(&qu);
          float dg[8], du[8];
#pragma unroll
          for (int t2 = 0; t2 < 4; ++t2) {
            const float2 g2 = __bfloat1622float2(hg[t2]);
            const float2 u2 = __bfloat1622float2(hu[t2]);
            const float gg[2] = {g2.x, g2.y}, uu[2] = {u2.x, u2.y};
#pragma unroll
            for (int e = 0; e < 2; ++e) {
              const float d = __bfloat162float(__float2bfloat16(__uint_as_float(r[j * 8 + t2 * 2 + e])));
              const float sgm = __fdividef(1.f, 1.f + __expf(-gg[e]));
              const float silu = gg[e] * sgm;
              dg[t2 * 2 + e] = d * uu[e] * (sgm + silu * (1.f - sgm));
              du[t2 * 2 + e] = d * silu;
            }
          }
          uint4 og, ou;
          og.x = pack_bf16x2(dg[0], dg[1]); og.y = pack_bf16x2(dg[2], dg[3]);
          og.z = pack_bf16x2(dg[4], dg[5]); og.w = pack_bf16x2(dg[6], dg[7]);
          ou.x = pack_bf16x2(du[0], du[1]); ou.y = pack_bf16x2(du[2], du[3]);
          ou.z = pack_bf16x2(du[4], du[5]); ou.w = pack_bf16x2(du[6], du[7]);
          *reinterpret_cast<uint4*>(sg + off) = og;
          *reinterpret_cast<uint4*>(su + off) = ou;
        }
      }
      __syncwarp();
      __nv_bfloat16* dst = p.dgu + (long long)row0 * p.ld_dgu + n0 + q * 64 + (lane & 7) * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = 4 * j + (lane >> 3);
        const int off = row * 128 + (((lane & 7) ^ (row & 7)) << 4);
        if (row < rows) {
          *reinterpret_cast<uint4*>(dst + (long long)row * p.ld_dgu) = *reinterpret_cast<const uint4*>(sg + off);
          *reinterpret_cast<uint4*>(dst + (long long)row * p.ld_dgu + p.f) = *reinterpret_cast<const uint4*>(su + off);
        }
      }
      __syncwarp();                                      // the stage may be filled again
    }
  }
};

// bf16 output with a residual, whole groups of eight columns on 16-byte boundaries: the residual's quarters of 64 columns arrive
// like the gate values above, every lane adds its row's sums to them (scaled and added in fp32, rounded once, as EpiStore does)
// and the stage leaves as whole row segments. Loaded by each lane from its own row behind the accumulator, the residual cost
// 16384 x 2048 x 2048 100 us where it is 93 now.
struct EpiResidual {
  using Params = StoreParams;
  static constexpr bool SPLIT_K = false;
  static constexpr bool PREFETCH = true;
  static constexpr int WARPS = NUM_EPI_WARPS;
  static constexpr int QUARTER = 32 * 128;
  static constexpr int STAGE_BYTES = 2 * QUARTER;
  static constexpr int SMEM_BYTES = NUM_EPI_WARPS * STAGE_BYTES;

  static bool fits(const Params& p, int N) {
    return p.resid && !p.out_f32 && p.fmt == 1 && !p.accumulate && !(N & 7) && !(p.ldc & 7) && !(p.ldr & 7) &&
           !(reinterpret_cast<uintptr_t>(p.C) & 15) && !(reinterpret_cast<uintptr_t>(p.resid) & 15);
  }

  static __device__ __forceinline__ void fetch(const Params& p, int q, int m0, int n0, int M, int N, int quad, int lane,
                                               uint8_t* epi_smem) {
    const int row0 = m0 + quad * 32, col = n0 + q * 64 + (lane & 7) * 8;
    if (col < N) {
      const uint32_t dst = smem_u32(epi_smem + quad * STAGE_BYTES + (q & 1) * QUARTER);
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = 4 * j + (lane >> 3);
        if (row0 + row < M)
          asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst + row * 128 + (((lane & 7) ^ (row & 7)) << 4)),
                       "l"(p.resid + (long long)(row0 + row) * p.ldr + col)
                       : "memory");
      }
    }
    asm volatile("cp.async.commit_group;" ::: "memory");
  }

  static __device__ __forceinline__ void prefetch(const Params& p, int m0, int n0, int M, int N, int quad, int lane,
                                                  uint8_t* epi_smem) {
    fetch(p, 0, m0, n0, M, N, quad, lane, epi_smem);
  }

  static __device__ __forceinline__ void tile(const Params& p, uint32_t taddr, int m0, int n0, int M, int N, int quad,
                                              int lane, uint8_t* epi_smem) {
    const int row0 = m0 + quad * 32;
    __nv_bfloat16* C = reinterpret_cast<__nv_bfloat16*>(p.C);
#pragma unroll 1
    for (int q = 0; q < 4; ++q) {
      if (q < 3) {
        fetch(p, q + 1, m0, n0, M, N, quad, lane, epi_smem);
        asm volatile("cp.async.wait_group 1;" ::: "memory");
      } else {
        asm volatile("cp.async.wait_group 0;" ::: "memory");
      }
      __syncwarp();
      if (n0 + q * 64 >= N) continue;
      uint8_t* stage = epi_smem + quad * STAGE_BYTES + (q & 1) * QUARTER;
      uint32_t r[2][32];
      tmem_ld_32x32b_x32(taddr + q * 64, r[0]);
      tmem_ld_32x32b_x32(taddr + q * 64 + 32, r[1]);
      tmem_ld_wait_for(r[0]);
      tmem_ld_wait_for(r[1]);
#pragma unroll
      for (int c = 0; c < 8; ++c) {
        uint4* at = reinterpret_cast<uint4*>(stage + lane * 128 + ((c ^ (lane & 7)) << 4));
        uint4 o = *at;
        uint32_t* w = reinterpret_cast<uint32_t*>(&o);
#pragma unroll
        for (int t = 0; t < 4; ++t) {
          const float2 f = __bfloat1622float2(*reinterpret_cast<__nv_bfloat162*>(&w[t]));
          const uint32_t* v = &r[c >> 2][(c & 3) * 8 + 2 * t];
          w[t] = pack_bf16x2(__fadd_rn(__fmul_rn(__uint_as_float(v[0]), p.alpha), f.x),
                             __fadd_rn(__fmul_rn(__uint_as_float(v[1]), p.alpha), f.y));
        }
        *at = o;
      }
      __syncwarp();
      const int col = n0 + q * 64 + (lane & 7) * 8;
#pragma unroll
      for (int j = 0; j < 8; ++j) {
        const int row = 4 * j + (lane >> 3);
        if (row0 + row < M && col < N)
          *reinterpret_cast<uint4*>(C + (long long)(row0 + row) * p.ldc + col) =
              *reinterpret_cast<const uint4*>(stage + row * 128 + (((lane & 7) ^ (row & 7)) << 4));
      }
      __syncwarp();                                      // the stage may be filled again
    }
  }
};

static int launch_swiglu_bwd_pair(const void* dY, const void* Wd, int M, int f, int K, long long lda, long long ldb,
                                  const SwigluBwdParams& sp, cudaStream_t stream) {
  using Epi = EpiSwigluBwd;
  constexpr int STAGES = 5;                    // one ring stage less than the store kernel: the epilogue needs 64 KB
  using S = SmemPair<STAGES>;
  CUtensorMap tmA, tmB;
  int rc = make_tmap_2d(&tmA, dY, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  // W_d is [K = h, N = f] in memory: an MN-major B operand
  rc = make_tmap_2d(&tmB, Wd, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)f, (uint64_t)K, (uint64_t)ldb * 2, 64, BK,
                    CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  auto kern = gemm_pair_kernel<STAGES, false, true, Epi>;
  const int smem_bytes = S::bytes(Epi::SMEM_BYTES);
  static bool attr_set = false;
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    attr_set = true;
  }
  const int tiles = ceil_div(M, PAIR_BM) * ceil_div(f, PAIR_BN);
  const int max_pairs = sm_count() / 2;
  const int pairs = tiles < max_pairs ? tiles : max_pairs;
  launch_pdl(kern, 2 * pairs, pair_threads<Epi>(), smem_bytes, stream, tmA, tmB, M, f, K, 1, sp, device_err_word(), 1, nullptr, 0,
               gemm::GroupArgs{});
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

static int launch_swiglu_pair(const void* A, const void* Wgu, int M, int f, int K, long long lda, long long ldb,
                              const SwigluParams& sp, cudaStream_t stream) {
  using Epi = EpiSwiglu;
  constexpr int STAGES = 6;
  using S = SmemPair<STAGES>;
  CUtensorMap tmA, tmB;
  int rc = make_tmap_2d(&tmA, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  rc = make_tmap_2d(&tmB, Wgu, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)(2 * f), (uint64_t)ldb * 2, BK,
                    PAIR_HALF_N, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  auto kern = gemm_pair_kernel<STAGES, false, false, Epi>;
  const int smem_bytes = S::bytes(Epi::SMEM_BYTES);
  static bool attr_set = false;
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    attr_set = true;
  }
  const int N = 2 * f;
  const int tiles = ceil_div(M, PAIR_BM) * ceil_div(N, PAIR_BN);
  const int max_pairs = sm_count() / 2;
  const int pairs = tiles < max_pairs ? tiles : max_pairs;
  launch_pdl(kern, 2 * pairs, pair_threads<Epi>(), smem_bytes, stream, tmA, tmB, M, N, K, 1, sp, device_err_word(), 1, nullptr, f,
               gemm::GroupArgs{});
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

template <int BN, int STAGES, bool A_MN, bool B_MN>
static int launch_store(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb, int fmt,
                        const StoreParams& sp, const DescCfg* dc_override, cudaStream_t stream) {
  using Epi = EpiStore<BN>;
  using S = Smem<BN, STAGES>;
  CUtensorMap tmA, tmB;
  const CUtensorMapDataType dt = fmt == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  int rc;
  if (!A_MN)
    rc = make_tmap_2d(&tmA, A, dt, 2, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = make_tmap_2d(&tmA, A, dt, 2, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, 64, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  if (!B_MN)
    rc = make_tmap_2d(&tmB, B, dt, 2, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, BK, BN, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = make_tmap_2d(&tmB, B, dt, 2, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;

  auto kern = gemm_kernel<BN, STAGES, A_MN, B_MN, Epi>;
  const int smem_bytes = S::bytes(Epi::SMEM_BYTES);
  static bool attr_set = false;
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    attr_set = true;
  }
  const int tiles = ceil_div(M, BM) * ceil_div(N, BN);
  const int grid = tiles < sm_count() ? tiles : sm_count();
  DescCfg dc = dc_override ? *dc_override : default_desc_cfg<BN, A_MN, B_MN>();
  launch_pdl(kern, grid, NUM_THREADS, smem_bytes, stream, tmA, tmB, M, N, K, fmt, dc, sp, device_err_word());
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// Counters of the ordered split-K epilogue: 8 per tile (one per epilogue warp of a CTA pair), zero between launches.
constexpr int SPLIT_MAX_TILES = 1024;
constexpr int SPLIT_MAX_SLICES = 15;
constexpr int SPLIT_REGIONS = 8;
__device__ unsigned int g_split_sync[SPLIT_REGIONS * SPLIT_MAX_TILES * 8];

// B200_GEMM_KSPLITS=n forces n slices wherever split-K is possible (experiments); unset: the launcher's estimate
static int split_k_forced() {
  static int n = -1;
  if (n < 0) {
    const char* e = getenv("B200_GEMM_KSPLITS");
    n = e ? atoi(e) : 0;
  }
  return n;
}

static bool split_k_enabled() {
  static int on = -1;
  if (on < 0) {
    const char* e = getenv("B200_GEMM_SPLITK");
    on = e ? (atoi(e) != 0) : 1;
  }
  return on != 0;
}

// K slices of a split launch on `max_pairs` SM pairs: rounds of the pair grid in units of one whole tile, ceil(tiles * s /
// pairs) / s, plus 1.5 % per extra slice for its read-modify-write epilogue; split only when that buys at least 7 %.
// `rounds` (may be null) receives the cost.
static int pair_k_splits(int tiles, int num_kb, int max_pairs, double* rounds) {
  const double unsplit = (double)((tiles + max_pairs - 1) / max_pairs);
  double best = unsplit;
  int k_splits = 1;
  for (int s = 2; s <= SPLIT_MAX_SLICES && num_kb / s >= 16; ++s) {
    const double c = (double)((tiles * s + max_pairs - 1) / max_pairs) / s * (1.0 + 0.015 * (s - 1));
    if (c < best - 1e-9) { best = c; k_splits = s; }
  }
  if (best > 0.93 * unsplit) { best = unsplit; k_splits = 1; }
  if (rounds) *rounds = best;
  return k_splits;
}

// The experts of a layer in one launch (gemm_pair.cuh, GROUPED): A [M, K] and the outputs are cut into n_groups runs of rows
// whose lengths `counts` holds on the device, B is [n_groups * b_rows, K]. b_half: as in launch_swiglu_pair.
template <class Epi>
static int launch_grouped(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb,
                          const typename Epi::Params& ep, const long long* counts, int n_groups, int b_rows, int b_half,
                          cudaStream_t stream) {
  constexpr int STAGES = 6;
  using S = SmemPair<STAGES>;
  CUtensorMap tmA, tmB;
  int rc = make_tmap_2d(&tmA, A, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM,
                        CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  rc = make_tmap_2d(&tmB, B, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, 2, (uint64_t)K, (uint64_t)n_groups * b_rows,
                    (uint64_t)ldb * 2, BK, PAIR_HALF_N, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  auto kern = gemm_pair_kernel<STAGES, false, false, Epi, true>;
  const int smem_bytes = S::bytes(Epi::SMEM_BYTES, true);
  static bool attr_set = false;
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    attr_set = true;
  }
  const int most = M / PAIR_BM + (n_groups < M ? n_groups : M);      // row tiles, however the rows are spread
  const long long tiles = (long long)most * ceil_div(N, PAIR_BN);
  const int max_pairs = sm_count() / 2;
  const int pairs = tiles < max_pairs ? (int)tiles : max_pairs;
  launch_pdl(kern, 2 * pairs, pair_threads<Epi>(), smem_bytes, stream, tmA, tmB, M, N, K, 1, ep, device_err_word(), 1, nullptr, b_half,
             GroupArgs{counts, n_groups, b_rows});
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// Two-SM (cta_group::2) launch: 256 x 256 tiles, one CTA pair per tile.
template <bool A_MN, bool B_MN, class Epi = EpiStore<PAIR_BN>>
static int launch_store_pair(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb, int fmt,
                             const StoreParams& sp, cudaStream_t stream) {
  constexpr int STAGES = 6;
  using S = SmemPair<STAGES>;
  CUtensorMap tmA, tmB;
  const CUtensorMapDataType dt = fmt == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  int rc;
  if (!A_MN)
    rc = make_tmap_2d(&tmA, A, dt, 2, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = make_tmap_2d(&tmA, A, dt, 2, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, 64, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  if (!B_MN)
    rc = make_tmap_2d(&tmB, B, dt, 2, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, BK, PAIR_HALF_N,
                      CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = make_tmap_2d(&tmB, B, dt, 2, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  auto kern = gemm_pair_kernel<STAGES, A_MN, B_MN, Epi>;
  const int smem_bytes = S::bytes(Epi::SMEM_BYTES);
  static bool attr_set = false;
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, smem_bytes));
    attr_set = true;
  }
  const int tiles = ceil_div(M, PAIR_BM) * ceil_div(N, PAIR_BN);
  const int max_pairs = sm_count() / 2;
  // split-K for fp32 outputs with a long reduction and too few tiles for even waves (weight-gradient GEMMs); the
  // slices of a tile are added in a fixed order (gemm_pair.cuh)
  int k_splits = 1;
  const int num_kb = ceil_div(K, BK);
  if (sp.out_f32 && !sp.resid && !(N & 3) && !(sp.ldc & 3) && tiles <= SPLIT_MAX_TILES && split_k_enabled()) {
    const int forced = split_k_forced();
    if (forced > 0) {
      k_splits = forced;
    } else {
      k_splits = pair_k_splits(tiles, num_kb, max_pairs, nullptr);
    }
    if (k_splits > num_kb) k_splits = num_kb;
    if (k_splits > SPLIT_MAX_SLICES) k_splits = SPLIT_MAX_SLICES;
  }
  unsigned int* sync = nullptr;
  if (k_splits > 1) {
    // one of 8 counter regions in turn, so that split launches on different streams do not share counters
    static unsigned int* base[64] = {};        // the array's address on each device of this process
    static std::atomic<unsigned int> turn{0};
    int dev = 0;
    B200_CUDA_CHECK(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return B200_ERR_ARG;
    if (!base[dev]) B200_CUDA_CHECK(cudaGetSymbolAddress(reinterpret_cast<void**>(&base[dev]), g_split_sync));
    sync = base[dev] + (size_t)(turn.fetch_add(1) % SPLIT_REGIONS) * (SPLIT_MAX_TILES * 8);
  }
  const long long units = (long long)tiles * k_splits;
  const int pairs = units < max_pairs ? (int)units : max_pairs;
  launch_pdl(kern, 2 * pairs, pair_threads<Epi>(), smem_bytes, stream, tmA, tmB, M, N, K, fmt, sp, device_err_word(), k_splits, sync, 0,
               gemm::GroupArgs{});
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// ------------------------------------------------------------------------------------------- cluster split-K launches
// Epilogues of the cluster kernel (gemm_cluster.cuh): the same arithmetic as the TMEM epilogues above, on four columns
// of a row per call.
__device__ __forceinline__ uint2 pack_bf16x4(const float (&v)[4]) {
  return make_uint2(pack_bf16x2(v[0], v[1]), pack_bf16x2(v[2], v[3]));
}
__device__ __forceinline__ void unpack_bf16x4(const uint2& q, float (&f)[4]) {
  const float2 a = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.x));
  const float2 b = __bfloat1622float2(*reinterpret_cast<const __nv_bfloat162*>(&q.y));
  f[0] = a.x; f[1] = a.y; f[2] = b.x; f[3] = b.y;
}

struct ClusterStore {
  using Params = StoreParams;
  static constexpr bool SPLIT_B = false;
  static constexpr int AHEAD = 0;
  struct Pre {};
  template <int BN>
  static __device__ __forceinline__ void load(const Params&, int, int, int, Pre&) {}
  template <int BN>
  static constexpr int items() { return BN / 4; }
  template <int BN, class Get>
  static __device__ __forceinline__ void item(const Params& p, int row, int n0, int N, int it, Get get) {
    const int col = n0 + it * 4;
    if (col >= N) return;
    const int nv = min(4, N - col);
    const float4 a = get(it);
    float v[4] = {a.x * p.alpha, a.y * p.alpha, a.z * p.alpha, a.w * p.alpha};
    if (p.resid) {
      const __nv_bfloat16* rp = p.resid + (long long)row * p.ldr + col;
      if (nv == 4 && !(reinterpret_cast<uintptr_t>(rp) & 7)) {
        float r[4];
        unpack_bf16x4(*reinterpret_cast<const uint2*>(rp), r);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += r[j];
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < nv) v[j] += __bfloat162float(rp[j]);
      }
    }
    if (p.out_f32) {
      float* cp = reinterpret_cast<float*>(p.C) + (long long)row * p.ldc + col;
      if (nv == 4 && !(reinterpret_cast<uintptr_t>(cp) & 15)) {
        float4 o = make_float4(v[0], v[1], v[2], v[3]);
        if (p.accumulate) {
          const float4 c = *reinterpret_cast<const float4*>(cp);
          o.x += c.x; o.y += c.y; o.z += c.z; o.w += c.w;
        }
        *reinterpret_cast<float4*>(cp) = o;
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < nv) cp[j] = p.accumulate ? cp[j] + v[j] : v[j];
      }
    } else if (p.fmt == 1) {
      __nv_bfloat16* cp = reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)row * p.ldc + col;
      if (nv == 4 && !(reinterpret_cast<uintptr_t>(cp) & 7)) {
        if (p.accumulate) {
          float c[4];
          unpack_bf16x4(*reinterpret_cast<const uint2*>(cp), c);
#pragma unroll
          for (int j = 0; j < 4; ++j) v[j] += c[j];
        }
        *reinterpret_cast<uint2*>(cp) = pack_bf16x4(v);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j)
          if (j < nv) cp[j] = __float2bfloat16(v[j] + (p.accumulate ? __bfloat162float(cp[j]) : 0.f));
      }
    } else {
      __half* cp = reinterpret_cast<__half*>(p.C) + (long long)row * p.ldc + col;
#pragma unroll
      for (int j = 0; j < 4; ++j)
        if (j < nv) cp[j] = __float2half(v[j] + (p.accumulate ? __half2float(cp[j]) : 0.f));
    }
  }
};

// The same for what a layer's GEMMs ask for: bf16 without accumulation or fp32, no scaling, whole groups of four columns on
// their boundaries. An epilogue runs once per launch, so that the instructions of an item and of the cases it does not meet are
// fetched for it alone: 777 x 896 x 896 6.2 us with the general form, 5.4 with this; with a residual 8.5 / 7.4.
template <bool F32, bool RESID>
struct ClusterStoreWhole {
  using Params = StoreParams;
  static constexpr bool SPLIT_B = false;
  static constexpr int AHEAD = 0;
  struct Pre {};
  template <int BN>
  static __device__ __forceinline__ void load(const Params&, int, int, int, Pre&) {}
  template <int BN>
  static constexpr int items() { return BN / 4; }
  template <int BN, class Get>
  static __device__ __forceinline__ void item(const Params& p, int row, int n0, int N, int it, Get get) {
    const int col = n0 + it * 4;
    if (col >= N) return;
    const float4 a = get(it);
    if constexpr (F32) {
      float4* cp = reinterpret_cast<float4*>(reinterpret_cast<float*>(p.C) + (long long)row * p.ldc + col);
      float4 o = a;
      if (p.accumulate) {
        const float4 c = *cp;
        o.x += c.x; o.y += c.y; o.z += c.z; o.w += c.w;
      }
      *cp = o;
    } else {
      float v[4] = {a.x, a.y, a.z, a.w};
      if constexpr (RESID) {
        float r[4];
        unpack_bf16x4(*reinterpret_cast<const uint2*>(p.resid + (long long)row * p.ldr + col), r);
#pragma unroll
        for (int j = 0; j < 4; ++j) v[j] += r[j];
      }
      *reinterpret_cast<uint2*>(reinterpret_cast<__nv_bfloat16*>(p.C) + (long long)row * p.ldc + col) = pack_bf16x4(v);
    }
  }
  // what `item` takes for granted
  static bool fits(const Params& p, int N) {
    const int mask = F32 ? 15 : 7;
    return p.alpha == 1.f && (p.out_f32 != 0) == F32 && (p.resid != nullptr) == RESID && (F32 || (p.fmt == 1 && !p.accumulate)) &&
           !(N & 3) && !(p.ldc & 3) && !(reinterpret_cast<uintptr_t>(p.C) & mask) &&
           (!RESID || (!(p.ldr & 3) && !(reinterpret_cast<uintptr_t>(p.resid) & 7)));
  }
};

struct ClusterSwiglu {
  using Params = SwigluParams;
  static constexpr bool SPLIT_B = true;
  static constexpr int AHEAD = 0;
  struct Pre {};
  template <int BN>
  static __device__ __forceinline__ void load(const Params&, int, int, int, Pre&) {}
  template <int BN>
  static constexpr int items() { return BN / 8; }
  template <int BN, class Get>
  static __device__ __forceinline__ void item(const Params& p, int row, int f0, int N, int it, Get get) {
    const int col = f0 + it * 4;
    if (col >= p.f) return;
    const float4 g4 = get(it), u4 = get(it + BN / 8);
    const float g[4] = {g4.x, g4.y, g4.z, g4.w}, u[4] = {u4.x, u4.y, u4.z, u4.w};
    const uint2 qg = pack_bf16x4(g), qu = pack_bf16x4(u);
    float gr[4], ur[4], a[4];
    unpack_bf16x4(qg, gr);
    unpack_bf16x4(qu, ur);
#pragma unroll
    for (int j = 0; j < 4; ++j) a[j] = __fdividef(gr[j], 1.f + __expf(-gr[j])) * ur[j];
    if (p.gu) {
      __nv_bfloat16* gp = p.gu + (long long)row * p.ld_gu + col;
      *reinterpret_cast<uint2*>(gp) = qg;
      *reinterpret_cast<uint2*>(gp + p.f) = qu;
    }
    *reinterpret_cast<uint2*>(p.act + (long long)row * p.ld_act + col) = pack_bf16x4(a);
  }
};

template <int D>          // elements of a head; a tile holds whole heads: BN is a multiple of it
struct ClusterRope {
  using Params = RopeParams;
  static constexpr bool SPLIT_B = false;
  static constexpr int AHEAD = 0;
  struct Pre {};
  template <int BN>
  static __device__ __forceinline__ void load(const Params&, int, int, int, Pre&) {}
  template <int BN>
  static constexpr int items() { return BN / 8; }
  template <int BN, class Get>
  static __device__ __forceinline__ void item(const Params& p, int row, int n0, int N, int it, Get get) {
    constexpr int per_head = D >> 3;                       // pairs of 4-column chunks in a head
    const int head = it / per_head, w = it - head * per_head;
    const int ca = head * (D >> 2) + w, cb = ca + per_head;
    const int col = n0 + ca * 4;
    if (col >= N) return;
    const float4 a4 = get(ca), b4 = get(cb);
    const float af[4] = {a4.x, a4.y, a4.z, a4.w}, bf[4] = {b4.x, b4.y, b4.z, b4.w};
    float a[4], b[4];
    unpack_bf16x4(pack_bf16x4(af), a);
    unpack_bf16x4(pack_bf16x4(bf), b);
    if (col < p.n_rot) {
      const long long e = (long long)p.pos[row] * (D >> 1) + w * 4;
      const float4 c4 = *reinterpret_cast<const float4*>(p.cs + e);
      const float4 s4 = *reinterpret_cast<const float4*>(p.sn + e);
      const float cc[4] = {c4.x, c4.y, c4.z, c4.w}, ss[4] = {s4.x, s4.y, s4.z, s4.w};
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        const float fa = a[j], fb = b[j];
        a[j] = __fmaf_rn(fa, cc[j], -__fmul_rn(fb, ss[j]));
        b[j] = __fmaf_rn(fb, cc[j], __fmul_rn(fa, ss[j]));
      }
    }
    __nv_bfloat16* cp = p.C + (long long)row * p.ldc + col;
    *reinterpret_cast<uint2*>(cp) = pack_bf16x4(a);
    *reinterpret_cast<uint2*>(cp + (D >> 1)) = pack_bf16x4(b);
  }
};

// A tile's 21 items a thread were each a chain from the loads of gate and up to the stores; with six of them under way 777 x
// 896 -> 4864 takes 14.8 us, before 19.4. (The residual of ClusterStore fetched like that: 0 to 1 us longer, it is more code.)
struct ClusterSwigluBwd {
  using Params = SwigluBwdParams;
  static constexpr bool SPLIT_B = false;
  static constexpr int AHEAD = 6;
  struct Pre {
    uint2 g, u;
  };
  template <int BN>
  static constexpr int items() { return BN / 4; }
  template <int BN>
  static __device__ __forceinline__ void load(const Params& p, int row, int n0, int it, Pre& pre) {
    const int col = n0 + it * 4;
    if (col >= p.f) return;
    const __nv_bfloat16* gp = p.gu + (long long)row * p.ld_gu + col;
    pre.g = __ldg(reinterpret_cast<const uint2*>(gp));
    pre.u = __ldg(reinterpret_cast<const uint2*>(gp + p.f));
  }
  template <int BN, class Get>
  static __device__ __forceinline__ void item(const Params& p, int row, int n0, int N, int it, Get get, const Pre& pre) {
    const int col = n0 + it * 4;
    if (col >= p.f) return;
    float g[4], u[4], d[4], dg[4], du[4];
    unpack_bf16x4(pre.g, g);
    unpack_bf16x4(pre.u, u);
    const float4 a = get(it);
    const float af[4] = {a.x, a.y, a.z, a.w};
    unpack_bf16x4(pack_bf16x4(af), d);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      const float sgm = __fdividef(1.f, 1.f + __expf(-g[j]));
      const float silu = g[j] * sgm;
      dg[j] = d[j] * u[j] * (sgm + silu * (1.f - sgm));
      du[j] = d[j] * silu;
    }
    __nv_bfloat16* op = p.dgu + (long long)row * p.ld_dgu + col;
    *reinterpret_cast<uint2*>(op) = pack_bf16x4(dg);
    *reinterpret_cast<uint2*>(op + p.f) = pack_bf16x4(du);
  }
};

// N: columns of B's output space covered by tiles of BN (2 f for the gate / up projection, whose tiles take BN/2 gate and
// BN/2 up rows: f = b_half > 0).
template <int BN, bool DEEP, bool A_MN, bool B_MN, class Epi>
static int launch_cluster(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb, int fmt,
                          const typename Epi::Params& ep, int slices, int b_half, int b_early, cudaStream_t stream) {
  using S = SmemCluster<BN, DEEP>;
  CUtensorMap tmA, tmB;
  const CUtensorMapDataType dt = fmt == 1 ? CU_TENSOR_MAP_DATA_TYPE_BFLOAT16 : CU_TENSOR_MAP_DATA_TYPE_FLOAT16;
  int rc;
  if (!A_MN)
    rc = make_tmap_2d(&tmA, A, dt, 2, (uint64_t)K, (uint64_t)M, (uint64_t)lda * 2, BK, BM, CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = make_tmap_2d(&tmA, A, dt, 2, (uint64_t)M, (uint64_t)K, (uint64_t)lda * 2, 64, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  if (!B_MN)
    rc = make_tmap_2d(&tmB, B, dt, 2, (uint64_t)K, (uint64_t)N, (uint64_t)ldb * 2, BK, Epi::SPLIT_B ? BN / 2 : BN,
                      CU_TENSOR_MAP_SWIZZLE_128B);
  else
    rc = make_tmap_2d(&tmB, B, dt, 2, (uint64_t)N, (uint64_t)K, (uint64_t)ldb * 2, 64, BK, CU_TENSOR_MAP_SWIZZLE_128B);
  if (rc != B200_OK) return rc;
  auto kern = gemm_cluster_kernel<BN, DEEP, A_MN, B_MN, Epi>;
  static bool attr_set = false;
  if (!attr_set) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, S::BYTES));
    attr_set = true;
  }
  const long long tiles = (long long)ceil_div(M, BM) * ceil_div(N, BN);
  launch_pdl_cluster(kern, dim3((unsigned)(tiles * slices)), dim3(NUM_THREADS), S::BYTES, stream, slices, tmA, tmB, M, N, K,
                     fmt, ep, device_err_word(), b_half, b_early);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// 0 = never, 1 = whenever the shape allows, unset = heuristic (enough 256 x 256 tiles to fill the SM pairs)
static int pair_mode() {
  static int mode = -2;
  if (mode == -2) {
    const char* e = getenv("B200_GEMM_PAIR");
    mode = e ? atoi(e) : -1;
  }
  return mode;
}

static bool use_pair(int M, int N, int K) {
  const int mode = pair_mode();
  if (mode == 0 || N <= 128) return false;
  if (mode == 1) return true;
  const long long tiles = (long long)ceil_div(M, PAIR_BM) * ceil_div(N, PAIR_BN);
  return (tiles >= sm_count() / 2 && K >= 256) || (tiles >= sm_count() / 8 && K >= 4096);
}

// Which kernel takes a GEMM: the cluster kernel with tiles of 128 x bn and `slices` CTAs per tile, or (bn = 0) the
// kernels of 128 x 256 and 256 x 256 tiles. The K slices decide the order of the additions, so the choice of `slices` is a
// function of the sizes alone and is the same for the plain GEMM and for the ones with a fused epilogue. split = false
// keeps the order of additions that the large tiles have (fp32 outputs of the 256 x 256 kernel are still cut by
// pair_k_splits). Every forward pass that a loss is taken of asks for that, training or validation, and under the
// reference loss the backward pass too: that loss divides by the largest row and clips a difference of two
// cross-entropies, and turned a last bit of an activation into 0.1 to 0.7 % of its value (38 runs of five students, 200
// to 1100 tokens; the KL losses: 0.001 %), so that the loss of a conversation would depend on the batch that it is in.
//
// Times in microseconds, least squares over 296 sizes from 40 to 2048 tokens on layers of 256 to 28672 (B200, weights from
// HBM; within 5 - 9 %), then moved a little towards the choices that were measured best: the chosen form takes 0.2 % longer than
// the best one on average, with the constants of the kernel before its issuing loops were the elected lane's 2.2 % (single sizes
// 25 %). A cluster CTA costs a fixed part (launch, first loads, exchange, epilogue) and a part per K
// block, more of both when two share an SM; the 256 x 256 kernel pays per round of its SM pairs. Clusters do not pack
// onto the last SMs of the chip (294 CTAs in clusters of 3 or 6 ran as two rounds), so split tiles stop at 7/8 of the
// resident CTAs. Examples, 128 x 256 tiles of one CTA / cluster: 93 x 2048 x 5632 37.8 / 10.2, 93 x 2560 x 2048 17.2 /
// 7.4, 777 x 896 x 4864 32.7 / 18.6 in one slice, 1100 x 512 x 512 8.1 / 4.2; 2048 x 2048 x 2048 17.7, cluster 18.0.
struct TilePlan {
  int bn, slices;
  int b_early = 0;      // B may be loaded before the kernel in front of this one has completed
};
// A CTA may take the shared memory of two where the grid fits the SMs at one each; clusters only up to 3/4 of them (147
// CTAs in clusters of 3 with an SM each ran as two rounds: 37.5 us, in shared SMs 30).
static bool deep_ring(long long ctas, int slices) {
  return ctas <= (slices > 1 ? sm_count() * 3 / 4 : sm_count());
}
static TilePlan plan_tiles(int M, int N, int K, bool f32, bool split) {
  // [bn = 64, 128][deep ring, one CTA per SM, two]: fixed, per K block, split, per slice
  static const double kCost[2][3][4] = {
      {{2.66, 0.181, 1.39, -0.030}, {1.99, 0.252, 2.12, 0.002}, {2.57, 0.279, 1.52, 0.141}},
      {{3.79, 0.200, 2.15, -0.147}, {2.64, 0.366, 2.64, 0.045}, {3.47, 0.398, 2.26, 0.183}}};
  // A grid beyond the resident CTAs, in one slice: its waves one behind the other and 15 % (a CTA starts where one has ended, but
  // the last wave ends unevenly). Where a short K meets a pair grid just above whole rounds it is the shorter form: 777 x 2 * 4864 x
  // 896 (152 tiles of 256 x 256 for 74 pairs) 30.1 / 22.0 us, [9728, 896] from 450 rows 21.5 / 16.5, from 1300 28.6 / 27.4. With
  // 10 % it also took sizes that lost 2 %.
  static const int kWaves = 4;
  static const double kWave = 1.15;
  static const double kUneven = 0.2;      // slices that are no power of two: rows and clusters do not divide evenly
  const int sms = sm_count(), num_kb = ceil_div(K, BK);
  const long long pair_tiles = (long long)ceil_div(M, PAIR_BM) * ceil_div(N, PAIR_BN);
  TilePlan plan{0, 1};
  double rounds = (double)((pair_tiles + sms / 2 - 1) / (sms / 2));
  if (f32 && pair_tiles <= SPLIT_MAX_TILES && split_k_enabled()) {
    const int s = pair_k_splits((int)pair_tiles, num_kb, sms / 2, &rounds);
    if (!split && s > 1 && use_pair(M, N, K)) return plan;      // that order of additions stays
  }
  double least = 6.0 + rounds * (0.344 * num_kb + (f32 ? 2.7 : 0.76));
  for (int w = 0; w < 2; ++w) {
    const int bn = w ? 128 : 64;
    const long long tiles = (long long)ceil_div(M, BM) * ceil_div(N, bn);
    for (int s = 1; s <= (split ? CLUSTER_MAX_SLICES : 1) && s <= num_kb; ++s) {
      const long long ctas = tiles * s;
      if (ctas > (s > 1 ? 2LL * sms * 7 / 8 : 2LL * sms * kWaves)) break;
      const double* c = kCost[w][deep_ring(ctas, s) ? 0 : ctas > sms ? 2 : 1];
      double us = c[0] + c[1] * ceil_div(num_kb, s) + (s > 1 ? c[2] : 0.0) + c[3] * s + (s & (s - 1) ? kUneven : 0.0);
      const int waves = (int)((ctas + 2 * sms - 1) / (2 * sms));
      if (waves > 1) us *= kWave * waves;
      if (us < least) { least = us; plan = TilePlan{bn, s}; }
    }
  }
  return plan;
}

template <bool A_MN, bool B_MN, class Epi>
static int launch_cluster_bn(const void* A, const void* B, int M, int N, int K, long long lda, long long ldb, int fmt,
                             const typename Epi::Params& ep, TilePlan plan, int b_half, cudaStream_t stream) {
  const bool deep = deep_ring((long long)ceil_div(M, BM) * ceil_div(N, plan.bn) * plan.slices, plan.slices);
  const int s = plan.slices, e = plan.b_early;
  if (plan.bn == 64)
    return deep ? launch_cluster<64, true, A_MN, B_MN, Epi>(A, B, M, N, K, lda, ldb, fmt, ep, s, b_half, e, stream)
                : launch_cluster<64, false, A_MN, B_MN, Epi>(A, B, M, N, K, lda, ldb, fmt, ep, s, b_half, e, stream);
  return deep ? launch_cluster<128, true, A_MN, B_MN, Epi>(A, B, M, N, K, lda, ldb, fmt, ep, s, b_half, e, stream)
              : launch_cluster<128, false, A_MN, B_MN, Epi>(A, B, M, N, K, lda, ldb, fmt, ep, s, b_half, e, stream);
}

}  // namespace gemm
}  // namespace b200

extern "C" {

// Zeroes the counters of the ordered split-K epilogue on the current device. A launch leaves them at zero by itself;
// a kernel that gave up on a bounded wait may not have, so the host calls this when it has taken note of such an error.
int b200_gemm_reset_split_sync(cudaStream_t stream) {
  using namespace b200;
  using namespace b200::gemm;
  unsigned int* base = nullptr;
  B200_CUDA_CHECK(cudaGetSymbolAddress(reinterpret_cast<void**>(&base), g_split_sync));
  B200_CUDA_CHECK(cudaMemsetAsync(base, 0, sizeof(unsigned int) * SPLIT_REGIONS * SPLIT_MAX_TILES * 8, stream));
  return B200_OK;
}

// gu[M, 2f] = x[M, K] Wgu[2f, K]^T (rows 0..f-1 of Wgu: gate, f..2f-1: up) and act[M, f] = silu(gate) * up, bf16, in one
// launch. f must be a multiple of 128; row strides (elements) multiples of 8. Returns B200_ERR_ARG for shapes the fused
// kernel does not take (the caller then runs the GEMM and the SwiGLU kernel).
int b200_gemm_swiglu(const void* x, const void* Wgu, void* gu, void* act, int M, int f, int K, long long ldx,
                     long long ldw, long long ld_gu, long long ld_act, int split_k, cudaStream_t stream) {
  using namespace b200;
  using namespace b200::gemm;
  if (!x || !Wgu || !act || M <= 0 || f <= 0 || K <= 0 || (f % PAIR_HALF_N) || (ldx & 7) || (ldw & 7) ||
      (ld_gu & 7) || (ld_act & 7) || (reinterpret_cast<uintptr_t>(gu) & 15) || (reinterpret_cast<uintptr_t>(act) & 15))
    return B200_ERR_ARG;
  SwigluParams sp{reinterpret_cast<__nv_bfloat16*>(gu), ld_gu, reinterpret_cast<__nv_bfloat16*>(act), ld_act, f};
  TilePlan plan = plan_tiles(M, 2 * f, K, false, split_k & 1);
  plan.b_early = split_k & 2;
  if (plan.bn) return launch_cluster_bn<false, false, ClusterSwiglu>(x, Wgu, M, 2 * f, K, ldx, ldw, 1, sp, plan, f, stream);
  return launch_swiglu_pair(x, Wgu, M, f, K, ldx, ldw, sp, stream);
}

static bool group_args_ok(const void* x, const void* W, const long long* counts, int M, int K, int n_groups, long long rows) {
  using namespace b200::gemm;
  return x && W && counts && M > 0 && K > 0 && !(K & 7) && n_groups > 0 && n_groups <= MAX_GROUPS &&
         (long long)n_groups * rows <= 0x7fffffffLL &&
         (long long)(M / PAIR_BM + n_groups) * b200::ceil_div_ll(rows, PAIR_BN) <= 0x7fffffffLL;
}

// The two GEMMs of a layer's experts. x [M, K] holds each expert's rows one run behind the other, counts int64 [E] their
// lengths (on the device; they sum to M); Wgu [E, 2f, K], W [E, N, K], all dense. gu [M, 2f] and act [M, f] as in
// b200_gemm_swiglu, y [M, N] = x W_e^T. bf16, E <= 128, f a multiple of 128, N and K of 8; else B200_ERR_ARG.
int b200_gemm_grouped_swiglu(const void* x, const void* Wgu, const long long* counts, void* gu, void* act, int M, int f,
                             int K, int E, cudaStream_t stream) {
  using namespace b200;
  using namespace b200::gemm;
  if (!act || f <= 0 || (f % PAIR_HALF_N) || f > 0x3fffffff || !group_args_ok(x, Wgu, counts, M, K, E, 2LL * f) ||
      (reinterpret_cast<uintptr_t>(gu) & 15) || (reinterpret_cast<uintptr_t>(act) & 15))
    return B200_ERR_ARG;
  SwigluParams sp{reinterpret_cast<__nv_bfloat16*>(gu), 2LL * f, reinterpret_cast<__nv_bfloat16*>(act), f, f};
  return launch_grouped<EpiSwiglu>(x, Wgu, M, 2 * f, K, K, K, sp, counts, E, 2 * f, f, stream);
}

int b200_gemm_grouped(const void* x, const void* W, const long long* counts, void* y, int M, int N, int K, int E,
                      cudaStream_t stream) {
  using namespace b200;
  using namespace b200::gemm;
  if (!y || N <= 0 || (N & 7) || !group_args_ok(x, W, counts, M, K, E, N) || (reinterpret_cast<uintptr_t>(y) & 15))
    return B200_ERR_ARG;
  StoreParams sp{y, N, nullptr, 0, 1.f, 0, 0, 1};
  return launch_grouped<EpiStore<PAIR_BN>>(x, W, M, N, K, K, K, sp, counts, E, N, 0, stream);
}

// qkv[M, N] = x[M, K] W[N, K]^T with the rotary embedding applied to the first n_rot_heads heads of every row in the
// epilogue (pos int32 [M]; cos / sin fp32 [max_pos, d/2]). d = 64 or 128, N a multiple of 128.
int b200_gemm_rope(const void* x, const void* W, void* out, const int* pos, const float* cos_tab, const float* sin_tab,
                   int M, int N, int K, int n_rot_heads, int d, long long ldx, long long ldw, long long ldo,
                   int split_k, cudaStream_t stream) {
  using namespace b200;
  using namespace b200::gemm;
  if (!x || !W || !out || !pos || !cos_tab || !sin_tab || M <= 0 || N <= 0 || K <= 0 || (d != 64 && d != 128) ||
      (N % PAIR_HALF_N) || n_rot_heads < 0 || n_rot_heads * d > N || (ldx & 7) || (ldw & 7) || (ldo & 7) ||
      (reinterpret_cast<uintptr_t>(out) & 15))
    return B200_ERR_ARG;
  RopeParams rp{reinterpret_cast<__nv_bfloat16*>(out), ldo, pos, cos_tab, sin_tab, d, n_rot_heads * d};
  TilePlan plan = plan_tiles(M, N, K, false, split_k & 1);
  plan.b_early = split_k & 2;
  if (plan.bn) {
    if (plan.bn < d) plan.bn = d;            // a tile holds whole heads
    return d == 64 ? launch_cluster_bn<false, false, ClusterRope<64>>(x, W, M, N, K, ldx, ldw, 1, rp, plan, 0, stream)
                   : launch_cluster_bn<false, false, ClusterRope<128>>(x, W, M, N, K, ldx, ldw, 1, rp, plan, 0, stream);
  }
  return d == 64 ? launch_rope_pair<64>(x, W, M, N, K, ldx, ldw, rp, stream)
                 : launch_rope_pair<128>(x, W, M, N, K, ldx, ldw, rp, stream);
}

// dgu[M, 2f] = SwiGLU backward of (gu, d(act)) with d(act) = dy[M, K] Wd[K, f] taken straight from the accumulator
// (never written). f a multiple of 128; strides multiples of 8. B200_ERR_ARG for shapes the fused kernel does not take.
int b200_gemm_swiglu_bwd(const void* dy, const void* Wd, const void* gu, void* dgu, int M, int f, int K, long long ld_dy,
                         long long ldw, long long ld_gu, long long ld_dgu, int split_k, cudaStream_t stream) {
  using namespace b200;
  using namespace b200::gemm;
  if (!dy || !Wd || !gu || !dgu || M <= 0 || f <= 0 || K <= 0 || (f % PAIR_HALF_N) || (ld_dy & 7) || (ldw & 7) ||
      (ld_gu & 7) || (ld_dgu & 7) || (reinterpret_cast<uintptr_t>(gu) & 15) || (reinterpret_cast<uintptr_t>(dgu) & 15))
    return B200_ERR_ARG;
  SwigluBwdParams sp{reinterpret_cast<const __nv_bfloat16*>(gu), ld_gu, reinterpret_cast<__nv_bfloat16*>(dgu), ld_dgu, f};
  TilePlan plan = plan_tiles(M, f, K, false, split_k & 1);
  plan.b_early = split_k & 2;
  if (plan.bn) return launch_cluster_bn<false, true, ClusterSwigluBwd>(dy, Wd, M, f, K, ld_dy, ldw, 1, sp, plan, 0, stream);
  return launch_swiglu_bwd_pair(dy, Wd, M, f, K, ld_dy, ldw, sp, stream);
}

// C[M,N] = alpha * op(A) * op(B)^T (+ C if accumulate) (+ residual)
//   a_mn = 0: A is [M,K] with row stride lda;   a_mn = 1: A is stored [K,M] with row stride lda
//   b_mn = 0: B is [N,K] with row stride ldb;   b_mn = 1: B is stored [K,N] with row stride ldb
//   fmt: 1 = bf16 operands, 0 = fp16.  out_f32: C is fp32, else the operand type.
// Strides are in elements and must be multiples of 8 (16 bytes); base pointers 16-byte aligned.
// split_k: bit 0: K may be cut over the CTAs of a cluster (plan_tiles); bit 1: the kernel launched just before on the stream
// does not write B, so that B may be read while that kernel still runs (gemm_cluster.cuh). The same in the fused forms above.
// desc_cfg: optional 6 x uint32 override of the matrix-descriptor byte offsets (testing hook), else null.
int b200_gemm(const void* A, const void* B, void* C, int M, int N, int K, long long lda, long long ldb,
              long long ldc, int a_mn, int b_mn, int fmt, int out_f32, int accumulate, float alpha,
              const void* residual, long long ldr, const unsigned int* desc_cfg, int split_k, cudaStream_t stream) {
  using namespace b200;
  using namespace b200::gemm;
  if (!A || !B || !C || M <= 0 || N <= 0 || K <= 0) return B200_ERR_ARG;
  if ((lda & 7) || (ldb & 7)) return B200_ERR_ARG;
  StoreParams sp;
  sp.C = C;
  sp.ldc = ldc;
  sp.resid = reinterpret_cast<const __nv_bfloat16*>(residual);
  sp.ldr = ldr;
  sp.alpha = alpha;
  sp.out_f32 = out_f32;
  sp.accumulate = accumulate;
  sp.fmt = fmt;
  DescCfg dco;
  const DescCfg* dcp = nullptr;
  if (desc_cfg) {
    dco.a_lbo = desc_cfg[0]; dco.a_sbo = desc_cfg[1]; dco.a_kadv = desc_cfg[2];
    dco.b_lbo = desc_cfg[3]; dco.b_sbo = desc_cfg[4]; dco.b_kadv = desc_cfg[5];
    dcp = &dco;
  }
  if (!dcp && pair_mode() < 0) {
    TilePlan plan = plan_tiles(M, N, K, out_f32 != 0, split_k & 1);
    plan.b_early = split_k & 2;
    if (plan.bn) {
      if (!a_mn && !b_mn && ClusterStoreWhole<false, true>::fits(sp, N))
        return launch_cluster_bn<false, false, ClusterStoreWhole<false, true>>(A, B, M, N, K, lda, ldb, fmt, sp, plan, 0, stream);
      if (!a_mn && !b_mn && ClusterStoreWhole<false, false>::fits(sp, N))
        return launch_cluster_bn<false, false, ClusterStoreWhole<false, false>>(A, B, M, N, K, lda, ldb, fmt, sp, plan, 0, stream);
      if (!a_mn && b_mn && ClusterStoreWhole<false, false>::fits(sp, N))
        return launch_cluster_bn<false, true, ClusterStoreWhole<false, false>>(A, B, M, N, K, lda, ldb, fmt, sp, plan, 0, stream);
      if (a_mn && b_mn && ClusterStoreWhole<true, false>::fits(sp, N))
        return launch_cluster_bn<true, true, ClusterStoreWhole<true, false>>(A, B, M, N, K, lda, ldb, fmt, sp, plan, 0, stream);
      if (!a_mn && !b_mn)
        return launch_cluster_bn<false, false, ClusterStore>(A, B, M, N, K, lda, ldb, fmt, sp, plan, 0, stream);
      if (!a_mn && b_mn)
        return launch_cluster_bn<false, true, ClusterStore>(A, B, M, N, K, lda, ldb, fmt, sp, plan, 0, stream);
      if (a_mn && b_mn)
        return launch_cluster_bn<true, true, ClusterStore>(A, B, M, N, K, lda, ldb, fmt, sp, plan, 0, stream);
      return launch_cluster_bn<true, false, ClusterStore>(A, B, M, N, K, lda, ldb, fmt, sp, plan, 0, stream);
    }
  }
  if (!dcp && use_pair(M, N, K)) {
    if (!a_mn && !b_mn && EpiResidual::fits(sp, N))
      return launch_store_pair<false, false, EpiResidual>(A, B, M, N, K, lda, ldb, fmt, sp, stream);
    if (!a_mn && !b_mn) return launch_store_pair<false, false>(A, B, M, N, K, lda, ldb, fmt, sp, stream);
    if (!a_mn && b_mn) return launch_store_pair<false, true>(A, B, M, N, K, lda, ldb, fmt, sp, stream);
    if (a_mn && b_mn) return launch_store_pair<true, true>(A, B, M, N, K, lda, ldb, fmt, sp, stream);
    return launch_store_pair<true, false>(A, B, M, N, K, lda, ldb, fmt, sp, stream);
  }
  const bool small_n = N <= 128;
  if (!a_mn && !b_mn) {
    return small_n ? launch_store<128, 6, false, false>(A, B, M, N, K, lda, ldb, fmt, sp, dcp, stream)
                   : launch_store<256, 4, false, false>(A, B, M, N, K, lda, ldb, fmt, sp, dcp, stream);
  } else if (!a_mn && b_mn) {
    return small_n ? launch_store<128, 6, false, true>(A, B, M, N, K, lda, ldb, fmt, sp, dcp, stream)
                   : launch_store<256, 4, false, true>(A, B, M, N, K, lda, ldb, fmt, sp, dcp, stream);
  } else if (a_mn && b_mn) {
    return small_n ? launch_store<128, 6, true, true>(A, B, M, N, K, lda, ldb, fmt, sp, dcp, stream)
                   : launch_store<256, 4, true, true>(A, B, M, N, K, lda, ldb, fmt, sp, dcp, stream);
  } else {
    return small_n ? launch_store<128, 6, true, false>(A, B, M, N, K, lda, ldb, fmt, sp, dcp, stream)
                   : launch_store<256, 4, true, false>(A, B, M, N, K, lda, ldb, fmt, sp, dcp, stream);
  }
}
}
