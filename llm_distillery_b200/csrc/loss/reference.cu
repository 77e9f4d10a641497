// The reference's weighted loss (utils/finetuning_utils.py:47-124) and its gradient on the [M, K] statistics of the LM head:
// two launches forward, one backward. Written with elementwise library calls it is about 250 launches a micro-batch, each
// reading or writing [M, K] or [M] tensors: at 722 rows of 200 entries launch latency, at 7000 rows of 400 some 40 passes over
// 11 MB.
//
//   row kernel           one warp per row: softmaxes of the teacher's and the student's values over the usable entries, KL,
//                        reverse KL, the values at the label's slot
//   conversation kernel  one block per conversation, fixed order of additions (results repeat bit for bit): means, maxima and
//                        weighted sums - and, since the gradient is linear in the upstream gradient of a conversation, at once
//                        the three factors that a row's gradient consists of (of its KL, its reverse KL, its label's value)
//   gradient kernel      one warp per row: d(loss) / d(zk) and d(loss) / d(lse)
// Definitions and treatment of rows without targets, labels or hits: loss/divergence.py, which stays the form for CPU tensors and
// for few rows (loss/head.py: NATIVE_REFERENCE_ROWS, with the reason). Four batches of about 7000 rows of 400 entries: 183.2 /
// 180.0 ms a step.
#include "../common/ptx.cuh"
#include "../common/host.cuh"

namespace b200 {
namespace refloss {

// per-row values kept between the kernels, [ROWS][M]
enum { R_KL, R_RKL, R_PS, R_PT, R_HIT, R_MS, R_LS, R_MT, R_LT, R_CKL, R_CRKL, R_CPICK, ROWS };
// per-conversation outputs, [OUTS][n_seg]
enum { O_CUSTOM, O_CE, O_KL, O_RKL, O_WKL, O_WRKL, O_CET, O_DIFF, OUTS };

struct RowArgs {
  const float* zk;              // [M, K] student logits / T at the teacher's ids
  const float* lse;             // [M]
  const float* u;               // [M, K] teacher log-probs
  const int* ids;               // [M, K]
  const long long* labels;      // [M], < 0: none
  const unsigned char* avoid;   // [M]
  long long M;
  int K, vocab;
  float temperature;
};

// One entry of a row: s = student log-prob, t = teacher value / T, usable or not.
struct Entry {
  float s, t;
  bool valid;
};
__device__ __forceinline__ Entry entry(const RowArgs& p, long long r, int k, float lse) {
  const long long i = r * p.K + k;
  const float t = p.u[i] / p.temperature;
  Entry e;
  e.valid = p.ids[i] < p.vocab && isfinite(t);
  e.t = t;
  e.s = p.zk[i] - lse;
  return e;
}

__global__ void __launch_bounds__(256) rows_kernel(RowArgs p, float* __restrict__ rows) {
  pdl_wait();
  pdl_trigger();
  const long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= p.M) return;
  const float lse = p.lse[r];
  const long long label = p.labels[r];
  const bool wants = label >= 0 && !p.avoid[r];
  float ms = -INFINITY, mt = -INFINITY;
  int n = 0;
  for (int k = lane; k < p.K; k += 32) {
    const Entry e = entry(p, r, k, lse);
    if (e.valid) {
      ms = fmaxf(ms, e.s);
      mt = fmaxf(mt, e.t);
      ++n;
    }
  }
  ms = warp_max(ms);
  mt = warp_max(mt);
  const bool any = __any_sync(0xffffffffu, n > 0);
  float ss = 0.f, st = 0.f;
  for (int k = lane; k < p.K; k += 32) {
    const Entry e = entry(p, r, k, lse);
    if (e.valid) {
      ss += expf(e.s - ms);
      st += expf(e.t - mt);
    }
  }
  // log-softmax: (x - max) - log(sum)
  const float ls = any ? logf(warp_sum(ss)) : 0.f, lt = any ? logf(warp_sum(st)) : 0.f;
  float kl = 0.f, rkl = 0.f, ps = 0.f, pt = 0.f;
  int hits = 0;
  for (int k = lane; k < p.K; k += 32) {
    const Entry e = entry(p, r, k, lse);
    const float t = (e.t - mt) - lt, s1 = (e.s - ms) - ls;
    if (e.valid) {
      kl += expf(t) * (t - e.s);
      rkl += expf(s1) * (s1 - t);
    }
    if (wants && p.ids[r * p.K + k] == label) {
      ps += e.valid ? e.s : -INFINITY;
      pt += e.valid ? t : -INFINITY;
      ++hits;
    }
  }
  kl = warp_sum(kl);
  rkl = warp_sum(rkl);
  ps = warp_sum(ps);
  pt = warp_sum(pt);
  const bool hit = __any_sync(0xffffffffu, hits > 0);
  if (lane == 0) {
    float* o = rows + r;
    const long long M = p.M;
    o[R_KL * M] = kl;
    o[R_RKL * M] = rkl;
    o[R_PS * M] = ps;
    o[R_PT * M] = pt;
    o[R_HIT * M] = hit ? 1.f : 0.f;
    // maximum and log of the sum apart: rounded into one number they would put its last bit, 5e-7 at 10, on every probability
    o[R_MS * M] = any ? ms : 0.f;
    o[R_LS * M] = ls;
    o[R_MT * M] = any ? mt : 0.f;
    o[R_LT * M] = lt;
  }
}

constexpr int CONVO_THREADS = 512;

// Sums (and, for index >= NSUM, maxima that keep NaN) of N values over the block in a fixed order; every thread gets them.
template <int N, int NSUM>
__device__ __forceinline__ void block_reduce(float (&v)[N], float* sh) {
  auto later = [](float a, float b) { return (b > a || b != b) ? b : a; };
#pragma unroll
  for (int i = 0; i < N; ++i)
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const float x = __shfl_xor_sync(0xffffffffu, v[i], o);
      v[i] = i < NSUM ? v[i] + x : later(v[i], x);
    }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  constexpr int W = CONVO_THREADS / 32;
  __syncthreads();
  if (lane == 0)
#pragma unroll
    for (int i = 0; i < N; ++i) sh[i * W + warp] = v[i];
  __syncthreads();
#pragma unroll
  for (int i = 0; i < N; ++i) {
    float a = sh[i * W];
    for (int w = 1; w < W; ++w) a = i < NSUM ? a + sh[i * W + w] : later(a, sh[i * W + w]);
    v[i] = a;
  }
}

__global__ void __launch_bounds__(CONVO_THREADS)
    convo_kernel(float* __restrict__ rows, const long long* __restrict__ labels, const long long* __restrict__ seg,
                 float* __restrict__ out, long long M, int n_seg, float alpha) {
  pdl_wait();
  pdl_trigger();
  __shared__ float sh[8 * (CONVO_THREADS / 32)];
  const int c = blockIdx.x;
  auto lower = [&](long long key) {
    long long lo = 0, hi = M;
    while (lo < hi) {
      const long long mid = (lo + hi) >> 1;
      if (seg[mid] < key) lo = mid + 1; else hi = mid;
    }
    return lo;
  };
  const long long r0 = lower(c), r1 = lower((long long)c + 1);
  const float n_rows = (float)(r1 - r0);
  float a[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, -INFINITY, -INFINITY};   // hits, their s and t, kl, rkl, labels | max kl, max rkl
  for (long long r = r0 + threadIdx.x; r < r1; r += CONVO_THREADS) {
    const float* o = rows + r;
    const float kl = o[R_KL * M], rkl = o[R_RKL * M];
    if (o[R_HIT * M] != 0.f) {
      a[0] += 1.f;
      a[1] += o[R_PS * M];
      a[2] += o[R_PT * M];
    }
    a[3] += kl;
    a[4] += rkl;
    a[5] += labels[r] >= 0 ? 1.f : 0.f;
    a[6] = (kl > a[6] || kl != kl) ? kl : a[6];
    a[7] = (rkl > a[7] || rkl != rkl) ? rkl : a[7];
  }
  block_reduce<8, 6>(a, sh);
  const float n_hit = fmaxf(a[0], 1.f), mean_s = a[1] / n_hit, mean_t = a[2] / n_hit;
  const float n_lab = a[5], mk = a[6], mr = a[7];
  // the cross-entropies of a row, what their difference adds to its weight and whether a gradient passes through that
  struct RowTerms { float ces, cet, d, gate; };
  auto terms = [&](long long r) {
    const float* o = rows + r;
    const bool hit = o[R_HIT * M] != 0.f, lab = labels[r] >= 0;
    RowTerms t;
    t.ces = -(hit ? o[R_PS * M] : mean_s);
    t.cet = -(hit ? o[R_PT * M] : mean_t);
    const float diff = t.ces - t.cet;
    t.d = lab ? (diff <= 0.f ? 0.f : diff) : 0.f;
    t.gate = lab && diff > 0.f ? 1.f : 0.f;
    return t;
  };
  float b[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};   // weighted kl, rkl; CE of student, teacher, difference; rows at the maxima
  float e[3] = {0.f, 0.f, 0.f};                            // d/d(max kl), d/d(max rkl), d/d(mean of the student's hits)
  for (long long r = r0 + threadIdx.x; r < r1; r += CONVO_THREADS) {
    const float* o = rows + r;
    const float kl = o[R_KL * M], rkl = o[R_RKL * M];
    const RowTerms t = terms(r);
    const float bk = kl / mk + 1.f, br = rkl / mr + 1.f;
    b[0] += kl * (powf(bk, alpha) + t.d);
    b[1] += rkl * (powf(br, alpha) + t.d);
    if (labels[r] >= 0) {
      b[2] += t.ces;
      b[3] += t.cet;
      b[4] += t.ces - t.cet;
    }
    b[5] += kl == mk ? 1.f : 0.f;
    b[6] += rkl == mr ? 1.f : 0.f;
    e[0] += kl * (alpha * powf(bk, alpha - 1.f)) * (-(kl / mk) / mk);
    e[1] += rkl * (alpha * powf(br, alpha - 1.f)) * (-(rkl / mr) / mr);
    if (o[R_HIT * M] == 0.f) e[2] -= t.gate * (kl + rkl);
  }
  block_reduce<8, 8>(b, sh);
  block_reduce<3, 3>(e, sh);
  const float half = 0.5f / n_rows;
  for (long long r = r0 + threadIdx.x; r < r1; r += CONVO_THREADS) {
    float* o = rows + r;
    const float kl = o[R_KL * M], rkl = o[R_RKL * M];
    const RowTerms t = terms(r);
    const float bk = kl / mk + 1.f, br = rkl / mr + 1.f;
    float ck = powf(bk, alpha) + t.d + kl * (alpha * powf(bk, alpha - 1.f)) / mk;
    float cr = powf(br, alpha) + t.d + rkl * (alpha * powf(br, alpha - 1.f)) / mr;
    if (kl == mk) ck += e[0] / b[5];
    if (rkl == mr) cr += e[1] / b[6];
    o[R_CKL * M] = ck * half;
    o[R_CRKL * M] = cr * half;
    o[R_CPICK * M] = o[R_HIT * M] != 0.f ? (e[2] / n_hit - t.gate * (kl + rkl)) * half : 0.f;
  }
  if (threadIdx.x == 0) {
    const float wkl = b[0] / n_rows, wrkl = b[1] / n_rows;
    out[O_CUSTOM * n_seg + c] = (wkl + wrkl) / 2.f;
    out[O_CE * n_seg + c] = b[2] / n_lab;
    out[O_KL * n_seg + c] = a[3] / n_rows;
    out[O_RKL * n_seg + c] = a[4] / n_rows;
    out[O_WKL * n_seg + c] = wkl;
    out[O_WRKL * n_seg + c] = wrkl;
    out[O_CET * n_seg + c] = b[3] / n_lab;
    out[O_DIFF * n_seg + c] = b[4] / n_lab;
  }
}

// dzk[r, k] and dlse[r] = -sum_k dzk[r, k] for the upstream gradient g[seg[r]]
__global__ void __launch_bounds__(256) grad_kernel(RowArgs p, const float* __restrict__ rows, const long long* __restrict__ seg,
                                                   const float* __restrict__ g, float* __restrict__ dzk,
                                                   float* __restrict__ dlse) {
  pdl_wait();
  pdl_trigger();
  const long long r = (blockIdx.x * (long long)blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (r >= p.M) return;
  const long long M = p.M;
  const float* o = rows + r;
  const float gc = g[seg[r]], lse = p.lse[r];
  const float rkl = o[R_RKL * M], ms = o[R_MS * M], ls = o[R_LS * M], mt = o[R_MT * M], lt = o[R_LT * M];
  const float ck = gc * o[R_CKL * M], cr = gc * o[R_CRKL * M], cp = gc * o[R_CPICK * M];
  const long long label = p.labels[r];
  const bool wants = label >= 0 && !p.avoid[r];
  float sum = 0.f;
  for (int k = lane; k < p.K; k += 32) {
    const Entry e = entry(p, r, k, lse);
    float d = 0.f;
    if (e.valid) {
      const float t = (e.t - mt) - lt, s1 = (e.s - ms) - ls;
      d = expf(s1) * (s1 - t - rkl) * cr - expf(t) * ck;
      if (wants && p.ids[r * p.K + k] == label) d += cp;
    }
    dzk[r * p.K + k] = d;
    sum += d;
  }
  sum = warp_sum(sum);
  if (lane == 0) dlse[r] = -sum;
}

static bool args_ok(const RowArgs& p) {
  return p.zk && p.lse && p.u && p.ids && p.labels && p.avoid && p.M > 0 && p.M <= 0x7fffffffLL && p.K > 0;
}

}  // namespace refloss
}  // namespace b200

extern "C" {
using namespace b200;

// rows: fp32 [12, M], kept for the gradient; out: fp32 [8, n_seg] (custom loss, CE, KL, reverse KL, weighted KL, weighted
// reverse KL, teacher CE, CE difference of each conversation). seg int64 [M], non-decreasing in [0, n_seg).
int b200_reference_loss(const float* zk, const float* lse, const float* u, const int* ids, const long long* labels,
                        const unsigned char* avoid, const long long* seg, float* rows, float* out, long long M, int K, int vocab,
                        int n_seg, float temperature, float alpha, cudaStream_t st) {
  const refloss::RowArgs p{zk, lse, u, ids, labels, avoid, M, K, vocab, temperature};
  if (!refloss::args_ok(p) || !seg || !rows || !out || n_seg <= 0) return B200_ERR_ARG;
  launch_pdl(refloss::rows_kernel, (unsigned)ceil_div_ll(M, 8), 256, 0, st, p, rows);
  B200_CUDA_CHECK(cudaGetLastError());
  launch_pdl(refloss::convo_kernel, (unsigned)n_seg, refloss::CONVO_THREADS, 0, st, rows, labels, seg, out, M, n_seg, alpha);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

int b200_reference_loss_grad(const float* zk, const float* lse, const float* u, const int* ids, const long long* labels,
                             const unsigned char* avoid, const long long* seg, const float* rows, const float* g, float* dzk,
                             float* dlse, long long M, int K, int vocab, float temperature, cudaStream_t st) {
  const refloss::RowArgs p{zk, lse, u, ids, labels, avoid, M, K, vocab, temperature};
  if (!refloss::args_ok(p) || !seg || !rows || !g || !dzk || !dlse) return B200_ERR_ARG;
  launch_pdl(refloss::grad_kernel, (unsigned)ceil_div_ll(M, 8), 256, 0, st, p, rows, seg, g, dzk, dlse);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}
}
