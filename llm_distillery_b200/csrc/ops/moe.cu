// Data movement of a sparse mixture-of-experts block: the stable sort of (token, choice) pairs by expert and the weighted
// combination of a token's expert outputs.
#include "../common/ptx.cuh"
#include "../common/host.cuh"

namespace b200 {
namespace moe {

constexpr int SORT_THREADS = 1024;
constexpr int SORT_MAX_EXPERTS = 32;

// Counting sort of n expert indices (stable): order[p] = index of the pair at sorted position p, inverse[order[p]] = p,
// token[p] = order[p] / k, counts[e] = pairs of expert e. ONE block: the keys of a layer are a few thousand to a few
// hundred thousand small numbers that sit in L2, and the point is latency (the host or the experts' GEMMs wait for the counts).
// The keys come in once, coalesced, as bytes into shared memory; each thread counts its contiguous run of them per expert there,
// one scan over (expert, thread) turns the counts into positions, and the same run is walked again in order. 12248 pairs of 8
// experts: the ten launches of a library radix sort, histogram, scatter and division that this replaces took about 90 us; with
// each thread reading its run from global memory, one 8-byte key after the other, and writing all three lists from the one
// block it took 33. The block writes `inverse` alone - stores of one SM to scattered sectors take a clock each - and a second
// launch of many blocks makes the other two of it. The runs grow with the pairs and one block does not: the library takes over
// beyond SORT_MAX_PAIRS (models/moe.py has both sides' times), for which the keys still fit beside the counts.
constexpr int SORT_MAX_PAIRS = 65536;
__global__ void __launch_bounds__(SORT_THREADS, 1)
    expert_sort_kernel(const long long* __restrict__ experts, int n, int E, long long* __restrict__ inverse,
                       long long* __restrict__ counts) {
  pdl_wait();
  pdl_trigger();
  extern __shared__ int slot[];                    // [E][SORT_THREADS], then the staged keys
  __shared__ int warp_base[SORT_MAX_EXPERTS][33];  // pairs of an expert in the warps before each, then their position
  int8_t* key = reinterpret_cast<int8_t*>(slot + E * SORT_THREADS);       // -1: of no expert
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int per = (n + SORT_THREADS - 1) / SORT_THREADS;
  const int i0 = min(n, tid * per), i1 = min(n, i0 + per);
#pragma unroll 8
  for (int i = tid; i < n; i += SORT_THREADS) {
    const long long e = experts[i];
    key[i] = e >= 0 && e < E ? (int8_t)e : (int8_t)-1;
  }
  for (int e = 0; e < E; ++e) slot[e * SORT_THREADS + tid] = 0;
  __syncthreads();
  for (int i = i0; i < i1; ++i) {
    const int e = key[i];
    if (e >= 0) ++slot[e * SORT_THREADS + tid];
  }
  for (int e = 0; e < E; ++e) {                    // scan inside each warp, expert by expert
    const int mine = slot[e * SORT_THREADS + tid];
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    if (lane == 31) warp_base[e][warp] = incl;
    slot[e * SORT_THREADS + tid] = incl - mine;
  }
  __syncthreads();
  for (int e = warp; e < E; e += 32) {             // then over the warps, one warp per expert
    const int mine = warp_base[e][lane];
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    warp_base[e][lane] = incl - mine;
    if (lane == 31) {
      warp_base[e][32] = incl;
      counts[e] = incl;
    }
  }
  __syncthreads();
  int base = 0;
  for (int e = 0; e < E; ++e) {
    slot[e * SORT_THREADS + tid] += base + warp_base[e][warp];
    base += warp_base[e][32];
  }
  for (int i = i0; i < i1; ++i) {
    const int e = key[i];
    if (e >= 0) inverse[i] = slot[e * SORT_THREADS + tid]++;
  }
}

// order and token of the sorted positions; pairs of no expert have none
__global__ void __launch_bounds__(256)
    expert_scatter_kernel(const long long* __restrict__ experts, const long long* __restrict__ inverse, int n, int E, int k,
                          long long* __restrict__ order, long long* __restrict__ token) {
  pdl_wait();
  pdl_trigger();
  const int i = (int)(blockIdx.x * blockDim.x + threadIdx.x);
  if (i >= n) return;
  const long long e = experts[i];
  if (e < 0 || e >= E) return;
  const long long p = inverse[i];
  order[p] = i;
  token[p] = i / k;
}

// out[t] = (h1[t] +) scale * sum_j w[t, j] y[inverse[t k + j]], summed in fp32 in the order of the choices: one pass over
// the k rows of a token, 16 bytes per thread and row (the gather, casts, product, reduction and addition it replaces
// moved the rows eight times: 230 us per layer of 6124 tokens, two rows of 2048 each; here about 20).
__global__ void __launch_bounds__(256)
    combine_kernel(const __nv_bfloat16* __restrict__ y, const long long* __restrict__ inverse, const float* __restrict__ w,
                   const __nv_bfloat16* __restrict__ h1, __nv_bfloat16* __restrict__ out, long long T, int k, int h, float scale) {
  pdl_wait();
  pdl_trigger();
  const int hv = h >> 3;
  const long long total = T * hv;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < total; i += (long long)gridDim.x * blockDim.x) {
    const long long t = i / hv;
    const int v = (int)(i - t * hv);
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    for (int j = 0; j < k; ++j) {
      const float wj = w[t * k + j];
      const uint4 q = reinterpret_cast<const uint4*>(y + inverse[t * k + j] * h)[v];
      const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 f = __bfloat1622float2(p[c]);
        a[2 * c] = __fadd_rn(a[2 * c], __fmul_rn(f.x, wj));
        a[2 * c + 1] = __fadd_rn(a[2 * c + 1], __fmul_rn(f.y, wj));
      }
    }
    float r[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    if (h1) {
      const uint4 q = reinterpret_cast<const uint4*>(h1 + t * h)[v];
      const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 f = __bfloat1622float2(p[c]);
        r[2 * c] = f.x;
        r[2 * c + 1] = f.y;
      }
    }
#pragma unroll
    for (int c = 0; c < 8; ++c) a[c] = __fadd_rn(r[c], __fmul_rn(a[c], scale));
    uint4 o;
    o.x = pack_bf16x2(a[0], a[1]);
    o.y = pack_bf16x2(a[2], a[3]);
    o.z = pack_bf16x2(a[4], a[5]);
    o.w = pack_bf16x2(a[6], a[7]);
    reinterpret_cast<uint4*>(out + t * h)[v] = o;
  }
}

}  // namespace moe
}  // namespace b200

extern "C" {
using namespace b200;

// experts int64 [n] in [0, E), n <= 65536, E <= 32; order, inverse, token int64 [n], counts int64 [E]
int b200_expert_sort(const long long* experts, long long n, int E, int k, long long* order, long long* inverse,
                     long long* token, long long* counts, cudaStream_t st) {
  if (!experts || !order || !inverse || !token || !counts || n <= 0 || n > moe::SORT_MAX_PAIRS || E <= 0 ||
      E > moe::SORT_MAX_EXPERTS || k <= 0)
    return B200_ERR_ARG;
  const int smem = E * moe::SORT_THREADS * (int)sizeof(int) + (int)n;
  static bool attr = false;
  if (!attr) {
    B200_CUDA_CHECK(cudaFuncSetAttribute(moe::expert_sort_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         moe::SORT_MAX_EXPERTS * moe::SORT_THREADS * (int)sizeof(int) + moe::SORT_MAX_PAIRS));
    attr = true;
  }
  launch_pdl(moe::expert_sort_kernel, 1, moe::SORT_THREADS, smem, st, experts, (int)n, E, inverse, counts);
  B200_CUDA_CHECK(cudaGetLastError());
  launch_pdl(moe::expert_scatter_kernel, (unsigned)ceil_div_ll(n, 256), 256, 0, st, experts, inverse, (int)n, E, k, order, token);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// y bf16 [T k, h], inverse int64 [T k], w fp32 [T, k], h1 bf16 [T, h] or null, out bf16 [T, h]; h a multiple of 8
int b200_moe_combine(const void* y, const long long* inverse, const float* w, const void* h1, void* out, long long T, int k,
                     int h, float scale, cudaStream_t st) {
  if (!y || !inverse || !w || !out || T <= 0 || k <= 0 || h <= 0 || (h & 7) || (reinterpret_cast<uintptr_t>(y) & 15) ||
      (reinterpret_cast<uintptr_t>(h1) & 15) || (reinterpret_cast<uintptr_t>(out) & 15))
    return B200_ERR_ARG;
  long long blocks = (T * (h >> 3) + 255) / 256;
  const long long cap = (long long)sm_count() * 8;
  if (blocks > cap) blocks = cap;
  launch_pdl(moe::combine_kernel, (unsigned)blocks, 256, 0, st, (const __nv_bfloat16*)y, inverse, w, (const __nv_bfloat16*)h1,
             (__nv_bfloat16*)out, T, k, h, scale);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}
}
