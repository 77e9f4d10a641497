// Routing and data movement of a sparse mixture-of-experts block: the router with its choice of experts, the stable sort of
// (token, choice) pairs by expert and the weighted combination of a token's expert outputs.
#include "../common/ptx.cuh"
#include "../common/host.cuh"

namespace b200 {
namespace moe {

// The router of one layer: logits = x W^T rounded to bf16, probs their softmax in fp32, top_e / top_w the k largest of a token
// (of equal ones the lower index first) and their probabilities, renormalised over the k or as they are. A warp takes four
// tokens, so that an expert's weights are fetched once for them; the sums of 32 (token, expert) pairs over the lanes meet in 31
// exchanges, after which each lane holds one of them and groups of EXPERTS lanes a token's. Bound by its chain of loads of W out of L1 and by that
// of the exchanges. 6124 tokens of 2048, 8 experts: the seven library launches that this replaces (GEMM, cast, softmax, two of a
// top-k, sum, division) took 33.5 us, this 12.4
// (100 tokens 26 / 6.3). 32 experts are 32 x 4 sums a lane or fewer tokens a warp, and slower than the library (8192 tokens
// 54 us against 42): up to 16 here.
constexpr int ROUTE_WARPS = 4;
constexpr int ROUTE_TOKENS = 4;
template <int EXPERTS>
__global__ void __launch_bounds__(32 * ROUTE_WARPS)
    route_kernel(const __nv_bfloat16* __restrict__ x, const __nv_bfloat16* __restrict__ w, long long T, int h, int E, int k,
                 int renorm, float* __restrict__ probs, long long* __restrict__ top_e, float* __restrict__ top_w) {
  pdl_wait();
  pdl_trigger();
  constexpr int PER = 32 / EXPERTS, GROUPS = ROUTE_TOKENS / PER;      // tokens of 32 sums, and how many such there are
  const int lane = threadIdx.x & 31;
  const long long t0 = (blockIdx.x * (long long)ROUTE_WARPS + (threadIdx.x >> 5)) * ROUTE_TOKENS;
  if (t0 >= T) return;
  float acc[GROUPS][32];
#pragma unroll
  for (int g = 0; g < GROUPS; ++g)
#pragma unroll
    for (int i = 0; i < 32; ++i) acc[g][i] = 0.f;
  auto unpack = [](const uint4& q, float (&f)[8]) {
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 v = __bfloat1622float2(p[c]);
      f[2 * c] = v.x;
      f[2 * c + 1] = v.y;
    }
  };
  for (int v = lane; v < (h >> 3); v += 32) {
    float xf[ROUTE_TOKENS][8];
#pragma unroll
    for (int i = 0; i < ROUTE_TOKENS; ++i)
      unpack(t0 + i < T ? reinterpret_cast<const uint4*>(x + (t0 + i) * h)[v] : make_uint4(0u, 0u, 0u, 0u), xf[i]);
#pragma unroll
    for (int e0 = 0; e0 < EXPERTS; e0 += 8) {
      uint4 q[8];
#pragma unroll
      for (int e = 0; e < 8; ++e)
        q[e] = e0 + e < E ? __ldg(reinterpret_cast<const uint4*>(w + (long long)(e0 + e) * h) + v) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
      for (int e = 0; e < 8; ++e) {
        float wf[8];
        unpack(q[e], wf);
#pragma unroll
        for (int i = 0; i < ROUTE_TOKENS; ++i) {
          float& a = acc[i / PER][i % PER * EXPERTS + e0 + e];
#pragma unroll
          for (int c = 0; c < 8; ++c) a = __fmaf_rn(xf[i][c], wf[c], a);
        }
      }
    }
  }
#pragma unroll
  for (int g = 0; g < GROUPS; ++g) {
    float* a = acc[g];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {      // lane l ends up with the sum of a[l] over the lanes
      const bool upper = lane & o;
#pragma unroll
      for (int i = 0; i < o; ++i) {
        const float keep = upper ? a[i + o] : a[i], send = upper ? a[i] : a[i + o];
        a[i] = keep + __shfl_xor_sync(0xffffffffu, send, o);
      }
    }
    const long long t = t0 + g * PER + lane / EXPERTS;
    const int e = lane % EXPERTS;
    const float logit = e < E ? __bfloat162float(__float2bfloat16(a[0])) : -INFINITY;
    float m = logit;
#pragma unroll
    for (int o = EXPERTS / 2; o > 0; o >>= 1) m = fmaxf(m, __shfl_xor_sync(0xffffffffu, m, o));
    const float ex = e < E ? expf(logit - m) : 0.f;
    float sum = ex;
#pragma unroll
    for (int o = EXPERTS / 2; o > 0; o >>= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);
    const float p = __fdiv_rn(ex, sum);
    if (t < T && e < E) probs[t * E + e] = p;
    // probabilities are not negative: their bits order them
    unsigned long long key = e < E ? ((unsigned long long)(__float_as_uint(p) + 1u) << 32) | (0xffffffffu - e) : 0ull;
    float mine_w = 0.f, total = 0.f;
    int mine_e = 0;
    for (int j = 0; j < k; ++j) {
      unsigned long long best = key;
#pragma unroll
      for (int o = EXPERTS / 2; o > 0; o >>= 1) {
        const unsigned long long other = __shfl_xor_sync(0xffffffffu, best, o);
        best = other > best ? other : best;
      }
      const int be = (int)(0xffffffffu - (uint32_t)best);
      const float bp = __uint_as_float((uint32_t)(best >> 32) - 1u);
      if (e == j) {
        mine_e = be;
        mine_w = bp;
      }
      if (e == be) key = 0ull;
      total += bp;
    }
    if (t < T && e < k) {
      top_e[t * k + e] = mine_e;
      top_w[t * k + e] = renorm ? __fdiv_rn(mine_w, total) : mine_w;
    }
  }
}

constexpr int SORT_THREADS = 512;
constexpr int SORT_WARPS = SORT_THREADS / 32;
constexpr int SORT_MAX_EXPERTS = 32;

// Counting sort of n expert indices (stable): order[p] = index of the pair at sorted position p, inverse[order[p]] = p,
// token[p] = order[p] / k, counts[e] = pairs of expert e; pairs of no expert have no position. A block places SORT_THREADS pairs,
// in one launch: it counts all keys itself - those in front of its own and the rest - which is n / 512 rounds of a warp's match
// and no scratch. The keys are a few thousand small numbers in L2, and the point is latency: 12248 pairs of 8 experts took about
// 90 us in ten library launches, 27 in one block with a second launch to scatter from it, here 6.8.
// The rounds grow with the
// pairs; beyond SORT_MAX_PAIRS the library takes over (models/moe.py has both sides' times).
constexpr int SORT_MAX_PAIRS = 65536;
__global__ void __launch_bounds__(SORT_THREADS)
    expert_sort_kernel(const long long* __restrict__ experts, int n, int E, int k, long long* __restrict__ order,
                       long long* __restrict__ inverse, long long* __restrict__ token, long long* __restrict__ counts) {
  pdl_wait();
  pdl_trigger();
  __shared__ int before[SORT_WARPS][SORT_MAX_EXPERTS], all[SORT_WARPS][SORT_MAX_EXPERTS];   // keys a warp has seen, by expert
  __shared__ int mine[SORT_WARPS][SORT_MAX_EXPERTS];                                       // of the block's own pairs
  __shared__ int base[SORT_MAX_EXPERTS];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  before[warp][lane] = all[warp][lane] = mine[warp][lane] = 0;
  __syncwarp();
  auto key_at = [&](int i) {
    const long long e = i < n ? experts[i] : -1;
    return e >= 0 && e < E ? (int)e : -1;
  };
  const int rounds = (n + SORT_THREADS - 1) / SORT_THREADS;
  int own = -1, rank = 0;
  for (int r0 = 0; r0 < rounds; r0 += 4) {
    int key[4];
#pragma unroll
    for (int u = 0; u < 4; ++u) key[u] = key_at((r0 + u) * SORT_THREADS + tid);       // four loads under way
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      const int r = r0 + u;
      if (r >= rounds) break;
      const unsigned same = __match_any_sync(0xffffffffu, key[u]);
      const int below = __popc(same & ((1u << lane) - 1u));
      if (r == (int)blockIdx.x) {
        own = key[u];
        rank = below;
      }
      if (below == 0 && key[u] >= 0) {      // one lane for each expert among these keys
        const int c = __popc(same);
        all[warp][key[u]] += c;
        if (r < (int)blockIdx.x) before[warp][key[u]] += c;
        if (r == (int)blockIdx.x) mine[warp][key[u]] = c;
      }
      __syncwarp();
    }
  }
  __syncthreads();
  if (warp == 0) {
    int b = 0, a = 0;
    for (int w = 0; w < SORT_WARPS; ++w) {
      b += before[w][lane];
      a += all[w][lane];
    }
    int incl = a;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int up = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += up;
    }
    base[lane] = incl - a + b;
    if (blockIdx.x == 0 && lane < E) counts[lane] = a;
  }
  __syncthreads();
  if (own >= 0) {
    int p = base[own] + rank;
    for (int w = 0; w < warp; ++w) p += mine[w][own];
    const int i = (int)blockIdx.x * SORT_THREADS + tid;
    inverse[i] = p;
    order[p] = i;
    token[p] = i / k;
  }
}

// out[t] = (h1[t] +) scale * sum_j w[t, j] y[inverse[t k + j]], summed in fp32 in the order of the choices: one pass over
// the k rows of a token, 16 bytes per thread and row (the gather, casts, product, reduction and addition it replaces
// moved the rows eight times: 230 us per layer of 6124 tokens, two rows of 2048 each; here about 20).
// K = 2: both rows under way at once (6124 tokens of 2048 15.0 / 13.9 us); 0: any number (eight at once: 56 / 67 us).
template <int K>
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
    uint4 hq = make_uint4(0u, 0u, 0u, 0u);
    if (h1) hq = reinterpret_cast<const uint4*>(h1 + t * h)[v];
    float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    auto add = [&](const uint4& q, float wj) {
      const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&q);
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const float2 f = __bfloat1622float2(p[c]);
        a[2 * c] = __fadd_rn(a[2 * c], __fmul_rn(f.x, wj));
        a[2 * c + 1] = __fadd_rn(a[2 * c + 1], __fmul_rn(f.y, wj));
      }
    };
    if constexpr (K > 0) {
      long long row[K];
      float wj[K];
      uint4 q[K];
#pragma unroll
      for (int j = 0; j < K; ++j) {
        row[j] = inverse[t * K + j];
        wj[j] = w[t * K + j];
      }
#pragma unroll
      for (int j = 0; j < K; ++j) q[j] = reinterpret_cast<const uint4*>(y + row[j] * h)[v];
#pragma unroll
      for (int j = 0; j < K; ++j) add(q[j], wj[j]);
    } else {
      for (int j = 0; j < k; ++j) add(reinterpret_cast<const uint4*>(y + inverse[t * k + j] * h)[v], w[t * k + j]);
    }
    const __nv_bfloat162* p = reinterpret_cast<const __nv_bfloat162*>(&hq);
    float r[8];
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float2 f = __bfloat1622float2(p[c]);
      r[2 * c] = f.x;
      r[2 * c + 1] = f.y;
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
  launch_pdl(moe::expert_sort_kernel, (unsigned)ceil_div_ll(n, moe::SORT_THREADS), moe::SORT_THREADS, 0, st, experts, (int)n, E, k,
             order, inverse, token, counts);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// x bf16 [T, h], w bf16 [E, h], E <= 16, k <= E, h a multiple of 8; probs fp32 [T, E], top_e int64 [T, k], top_w fp32 [T, k]
int b200_moe_route(const void* x, const void* w, long long T, int h, int E, int k, int renorm, float* probs, long long* top_e,
                   float* top_w, cudaStream_t st) {
  if (!x || !w || !probs || !top_e || !top_w || T <= 0 || h <= 0 || (h & 7) || E <= 0 || E > 16 || k <= 0 || k > E ||
      (reinterpret_cast<uintptr_t>(x) & 15) || (reinterpret_cast<uintptr_t>(w) & 15))
    return B200_ERR_ARG;
  auto kern = E <= 8 ? moe::route_kernel<8> : moe::route_kernel<16>;
  launch_pdl(kern, (unsigned)ceil_div_ll(T, moe::ROUTE_WARPS * moe::ROUTE_TOKENS), 32 * moe::ROUTE_WARPS, 0, st,
             (const __nv_bfloat16*)x, (const __nv_bfloat16*)w, T, h, E, k, renorm, probs, top_e, top_w);
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
  auto kern = k == 2 ? moe::combine_kernel<2> : moe::combine_kernel<0>;
  launch_pdl(kern, (unsigned)blocks, 256, 0, st, (const __nv_bfloat16*)y, inverse, w, (const __nv_bfloat16*)h1,
             (__nv_bfloat16*)out, T, k, h, scale);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}
}
