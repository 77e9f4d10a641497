// Per-conversation reductions over the rows of a micro-batch, in a fixed order.
//
// A micro-batch lists the content rows of its conversations one conversation after the other, so the conversation
// index `seg[r]` is non-decreasing in r. One warp owns one conversation: it finds the conversation's row range by
// binary search, the lanes walk it with stride 32 and the lane partials meet in a butterfly. The order of the
// additions depends on the row range only, never on scheduling, so the result is bit-identical from run to run
// (an atomic scatter-add is not). The reference adds its per-conversation losses in a Python loop
// (classes/student/model.py:415-436, classes/losses.py:43-47), which is a fixed order too.
#include "../common/ptx.cuh"
#include "../common/host.cuh"

namespace b200 {
namespace seg {

__device__ __forceinline__ long long lower_bound(const long long* __restrict__ seg, long long M, long long key) {
  long long lo = 0, hi = M;
  while (lo < hi) {
    const long long mid = (lo + hi) >> 1;
    if (seg[mid] < key) lo = mid + 1; else hi = mid;
  }
  return lo;
}

// Sum (or maximum) of x[r0 .. r1 - 1] in every lane: a lane takes every 32nd element in turn, then a butterfly. Eight loads of
// a lane are under way at a time (one: 34 us for 8 conversations of 2048 rows, now 7); the order of the additions is the same.
template <bool MAX>
__device__ __forceinline__ float reduce_rows(const float* __restrict__ x, long long r0, long long r1, int lane) {
  constexpr int U = 8;
  float acc = MAX ? -INFINITY : 0.f;
  long long r = r0 + lane;
  for (; r + 32 * (U - 1) < r1; r += 32 * U) {
    float v[U];
#pragma unroll
    for (int u = 0; u < U; ++u) v[u] = x[r + 32 * u];
#pragma unroll
    for (int u = 0; u < U; ++u) acc = MAX ? fmaxf(acc, v[u]) : acc + v[u];
  }
  for (; r < r1; r += 32) acc = MAX ? fmaxf(acc, x[r]) : acc + x[r];
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const float other = __shfl_xor_sync(0xffffffffu, acc, o);
    acc = MAX ? fmaxf(acc, other) : acc + other;
  }
  return acc;
}

// op 0: sum, op 1: max (-inf for an empty conversation), op 2: number of rows
__global__ void __launch_bounds__(256) segment_reduce_kernel(const float* __restrict__ x,
                                                             const long long* __restrict__ seg,
                                                             float* __restrict__ out, long long M, int n_seg, int op) {
  pdl_wait();
  pdl_trigger();
  const int warp = (int)((blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5);
  const int lane = threadIdx.x & 31;
  if (warp >= n_seg) return;
  const long long r0 = lower_bound(seg, M, warp), r1 = lower_bound(seg, M, (long long)warp + 1);
  if (op == 2) {
    if (lane == 0) out[warp] = (float)(r1 - r0);
    return;
  }
  const float acc = op == 1 ? reduce_rows<true>(x, r0, r1, lane) : reduce_rows<false>(x, r0, r1, lane);
  if (lane == 0) out[warp] = acc;
}

// The loss of a micro-batch whose conversations each count with the mean of their rows: *loss = the sum of the means,
// count[0 .. n_seg - 1] the number of rows of each conversation. One block, a warp per conversation; the launches that this takes
// apart (sums, counts, a division, three sums) and their graph nodes cost a step of 512 tokens more host time than its layers.
constexpr int MEAN_THREADS = 512;
__global__ void __launch_bounds__(MEAN_THREADS) mean_loss_kernel(const float* __restrict__ x, const long long* __restrict__ seg,
                                                                 float* __restrict__ loss, float* __restrict__ count,
                                                                 long long M, int n_seg) {
  pdl_wait();
  pdl_trigger();
  constexpr int WARPS = MEAN_THREADS / 32;
  __shared__ float part[WARPS];
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float mine = 0.f;
  for (int s = warp; s < n_seg; s += WARPS) {
    const long long r0 = lower_bound(seg, M, s), r1 = lower_bound(seg, M, (long long)s + 1);
    const float rows = (float)(r1 - r0);
    mine += reduce_rows<false>(x, r0, r1, lane) / rows;
    if (lane == 0) count[s] = rows;
  }
  if (lane == 0) part[warp] = mine;
  __syncthreads();
  if (threadIdx.x == 0) {
    float t = 0.f;
    for (int w = 0; w < WARPS; ++w) t += part[w];
    *loss = t;
  }
}

// g[r] = dloss / rows of r's conversation
__global__ void __launch_bounds__(256) mean_loss_grad_kernel(const long long* __restrict__ seg, const float* __restrict__ count,
                                                             const float* __restrict__ dloss, float* __restrict__ g,
                                                             long long M, int n_seg) {
  pdl_wait();
  pdl_trigger();
  const long long r = blockIdx.x * (long long)blockDim.x + threadIdx.x;
  if (r >= M) return;
  const long long s = seg[r];
  g[r] = s >= 0 && s < n_seg ? *dloss / count[s] : 0.f;
}

}  // namespace seg
}  // namespace b200

extern "C" int b200_segment_reduce(const float* x, const long long* seg, float* out, long long M, int n_seg, int op,
                                   cudaStream_t st) {
  using namespace b200;
  if (!seg || !out || M < 0 || n_seg <= 0 || op < 0 || op > 2 || (op != 2 && !x)) return B200_ERR_ARG;
  const int blocks = ceil_div(n_seg * 32, 256);
  launch_pdl(seg::segment_reduce_kernel, blocks, 256, 0, st, x, seg, out, M, n_seg, op);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

// See mean_loss_kernel. seg non-decreasing in [0, n_seg).
extern "C" int b200_mean_loss(const float* rows, const long long* seg, float* loss, float* count, long long M, int n_seg,
                              cudaStream_t st) {
  using namespace b200;
  if (!rows || !seg || !loss || !count || M <= 0 || n_seg <= 0) return B200_ERR_ARG;
  launch_pdl(seg::mean_loss_kernel, 1, seg::MEAN_THREADS, 0, st, rows, seg, loss, count, M, n_seg);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

extern "C" int b200_mean_loss_grad(const long long* seg, const float* count, const float* dloss, float* g, long long M, int n_seg,
                                   cudaStream_t st) {
  using namespace b200;
  if (!seg || !count || !dloss || !g || M <= 0 || n_seg <= 0) return B200_ERR_ARG;
  launch_pdl(seg::mean_loss_grad_kernel, (unsigned)ceil_div_ll(M, 256), 256, 0, st, seg, count, dloss, g, M, n_seg);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}
