// Fused optimizer steps over flat parameter shards (one launch per step, fp32 master weights and
// state, bf16 model weights written in the same pass): AdamW / Adam, SGD with momentum (+ Nesterov),
// centred RMSprop, Adagrad, and a block-wise 8-bit-state AdamW. The gradient is read as fp32 and
// may be pre-scaled (1 / (grad_accum * world)) in the same pass.
#include "../common/ptx.cuh"
#include "../common/host.cuh"

namespace b200 {
namespace optim {

struct AdamArgs {
  float lr, beta1, beta2, eps, weight_decay, bias1, bias2, grad_scale;
  int decoupled;  // 1: AdamW, 0: Adam with L2 added to the gradient
};

// Bound by HBM: 30 bytes a weight. Every thread takes one group of four and the grid covers them all: blocks that walk a
// resident grid's stride keep the five arrays' streams in pages far apart, and at 48 registers only 5 of the 8 blocks an SM that
// the grid had were resident. 1.24 G weights 6.05 -> 5.32 ms (7.0 TB/s), behind large GEMMs 6.41 -> 5.76; 26 M 135 -> 125 us.
// Two or four groups a thread or streaming loads: the same or slower.
__global__ void __launch_bounds__(256) adam_kernel(float* __restrict__ master, __nv_bfloat16* __restrict__ model,
                                                  const float* __restrict__ grad, float* __restrict__ m,
                                                  float* __restrict__ v, long long n, AdamArgs a) {
  pdl_wait();
  pdl_trigger();
  const long long nv = n >> 2;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < nv;
       i += (long long)gridDim.x * blockDim.x) {
    float4 p = reinterpret_cast<float4*>(master)[i];
    float4 g = reinterpret_cast<const float4*>(grad)[i];
    float4 mm = reinterpret_cast<float4*>(m)[i];
    float4 vv = reinterpret_cast<float4*>(v)[i];
    float* pp = &p.x; float* gp = &g.x; float* mp = &mm.x; float* vp = &vv.x;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      float gj = gp[j] * a.grad_scale;
      if (a.decoupled) pp[j] *= (1.f - a.lr * a.weight_decay);
      else gj += a.weight_decay * pp[j];
      mp[j] = a.beta1 * mp[j] + (1.f - a.beta1) * gj;
      vp[j] = a.beta2 * vp[j] + (1.f - a.beta2) * gj * gj;
      const float denom = sqrtf(vp[j] / a.bias2) + a.eps;
      pp[j] -= (a.lr / a.bias1) * mp[j] / denom;
    }
    reinterpret_cast<float4*>(master)[i] = p;
    reinterpret_cast<float4*>(m)[i] = mm;
    reinterpret_cast<float4*>(v)[i] = vv;
    if (model) {
      uint2 o;
      o.x = pack_bf16x2(p.x, p.y);
      o.y = pack_bf16x2(p.z, p.w);
      reinterpret_cast<uint2*>(model)[i] = o;
    }
  }
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    for (long long i = nv << 2; i < n; ++i) {
      float gj = grad[i] * a.grad_scale, pj = master[i];
      if (a.decoupled) pj *= (1.f - a.lr * a.weight_decay);
      else gj += a.weight_decay * pj;
      m[i] = a.beta1 * m[i] + (1.f - a.beta1) * gj;
      v[i] = a.beta2 * v[i] + (1.f - a.beta2) * gj * gj;
      pj -= (a.lr / a.bias1) * m[i] / (sqrtf(v[i] / a.bias2) + a.eps);
      master[i] = pj;
      if (model) model[i] = __float2bfloat16(pj);
    }
  }
}

// kind: 0 SGD(momentum, nesterov) ; 1 RMSprop centred (alpha, eps) ; 2 Adagrad (eps)
struct SimpleArgs {
  float lr, weight_decay, momentum, alpha, eps, grad_scale;
  int kind, nesterov, first_step;
};

__global__ void __launch_bounds__(256) simple_kernel(float* __restrict__ master, __nv_bfloat16* __restrict__ model,
                                                    const float* __restrict__ grad, float* __restrict__ s0,
                                                    float* __restrict__ s1, long long n, SimpleArgs a) {
  pdl_wait();
  pdl_trigger();
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n;
       i += (long long)gridDim.x * blockDim.x) {
    float p = master[i];
    float g = grad[i] * a.grad_scale + a.weight_decay * p;
    if (a.kind == 0) {
      float buf = a.first_step ? g : a.momentum * s0[i] + g;
      s0[i] = buf;
      const float upd = a.momentum == 0.f ? g : (a.nesterov ? g + a.momentum * buf : buf);
      p -= a.lr * upd;
    } else if (a.kind == 1) {
      const float sq = a.alpha * s0[i] + (1.f - a.alpha) * g * g;
      const float ga = a.alpha * s1[i] + (1.f - a.alpha) * g;
      s0[i] = sq;
      s1[i] = ga;
      p -= a.lr * g / (sqrtf(fmaxf(sq - ga * ga, 0.f)) + a.eps);
    } else {
      const float acc = s0[i] + g * g;
      s0[i] = acc;
      p -= a.lr * g / (sqrtf(acc) + a.eps);
    }
    master[i] = p;
    if (model) model[i] = __float2bfloat16(p);
  }
}

// Block-wise 8-bit AdamW state: each block of 256 values shares one fp32 absmax per moment; m is stored as a
// signed 8-bit linear code, v as an unsigned 8-bit code of sqrt(v) (keeps small second moments resolvable).
// A warp takes a block of 256, eight values a lane in two groups of four, and the grid covers all blocks: 131 M weights take
// 645 us (1.24 G 5.9 ms, 3.7 TB/s of their 18 bytes each; the two divisions and two roots a value hold it there). A value a
// thread, with barriers around each of the two maxima, took 1112. At 76 registers, three blocks an SM: 687.
// Rounding steps are written out, so that both forms of a block round alike.
constexpr int QB = 256;
constexpr int Q_WARPS = 8;
template <bool VEC>
__global__ void __launch_bounds__(32 * Q_WARPS, 4) adam8_kernel(float* __restrict__ master, __nv_bfloat16* __restrict__ model,
                                                             const float* __restrict__ grad, int8_t* __restrict__ mq,
                                                             uint8_t* __restrict__ vq, float* __restrict__ mabs,
                                                             float* __restrict__ vabs, long long n, AdamArgs a) {
  pdl_wait();
  pdl_trigger();
  const int lane = threadIdx.x & 31;
  for (long long blk = blockIdx.x * (long long)Q_WARPS + (threadIdx.x >> 5); blk * QB < n; blk += (long long)gridDim.x * Q_WARPS) {
    const long long i0 = blk * QB + 4 * lane;            // and i0 + 128
    const bool whole = VEC && blk * QB + QB <= n;
    __align__(16) float p[8], g[8];
    float mm[8], vv[8];
    char4 cm[2];
    uchar4 cv[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long i = i0 + 128 * h;
      if (whole) {
        *reinterpret_cast<float4*>(p + 4 * h) = *reinterpret_cast<const float4*>(master + i);
        *reinterpret_cast<float4*>(g + 4 * h) = *reinterpret_cast<const float4*>(grad + i);
        cm[h] = *reinterpret_cast<const char4*>(mq + i);
        cv[h] = *reinterpret_cast<const uchar4*>(vq + i);
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const bool ok = i + j < n;
          p[4 * h + j] = ok ? master[i + j] : 0.f;
          g[4 * h + j] = ok ? grad[i + j] : 0.f;
          (&cm[h].x)[j] = ok ? mq[i + j] : 0;
          (&cv[h].x)[j] = ok ? vq[i + j] : 0;
        }
      }
    }
    const float ms = mabs[blk] / 127.f, vs = vabs[blk] / 255.f;
    float am = 0.f, av = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
      mm[j] = (float)(&cm[j >> 2].x)[j & 3] * ms;
      const float sv = (float)(&cv[j >> 2].x)[j & 3] * vs;
      vv[j] = sv * sv;
      float gj = __fmul_rn(g[j], a.grad_scale);
      if (a.decoupled) p[j] = __fmul_rn(p[j], 1.f - a.lr * a.weight_decay);
      else gj = __fmaf_rn(a.weight_decay, p[j], gj);
      mm[j] = __fmaf_rn(a.beta1, mm[j], __fmul_rn(1.f - a.beta1, gj));
      vv[j] = __fmaf_rn(a.beta2, vv[j], __fmul_rn(__fmul_rn(1.f - a.beta2, gj), gj));
      p[j] = __fsub_rn(p[j], __fdiv_rn(__fmul_rn(a.lr / a.bias1, mm[j]), __fadd_rn(__fsqrt_rn(__fdiv_rn(vv[j], a.bias2)), a.eps)));
      vv[j] = sqrtf(vv[j]);
      if (whole || i0 + (j >> 2) * 128 + (j & 3) < n) {
        am = fmaxf(am, fabsf(mm[j]));
        av = fmaxf(av, vv[j]);
      }
    }
    // new scales of the block
    am = warp_max(am);
    av = warp_max(av);
    if (lane == 0) {
      mabs[blk] = am;
      vabs[blk] = av;
    }
    const float sm = am > 0.f ? 127.f / am : 0.f;
    const float sv = av > 0.f ? 255.f / av : 0.f;
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      const long long i = i0 + 128 * h;
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        (&cm[h].x)[j] = (int8_t)__float2int_rn(mm[4 * h + j] * sm);
        (&cv[h].x)[j] = (uint8_t)min(255, __float2int_ru(vv[4 * h + j] * sv));
      }
      if (whole) {
        *reinterpret_cast<float4*>(master + i) = *reinterpret_cast<const float4*>(p + 4 * h);
        *reinterpret_cast<char4*>(mq + i) = cm[h];
        *reinterpret_cast<uchar4*>(vq + i) = cv[h];
        if (model)
          *reinterpret_cast<uint2*>(model + i) =
              make_uint2(pack_bf16x2(p[4 * h], p[4 * h + 1]), pack_bf16x2(p[4 * h + 2], p[4 * h + 3]));
      } else {
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          if (i + j >= n) continue;
          master[i + j] = p[4 * h + j];
          mq[i + j] = (&cm[h].x)[j];
          vq[i + j] = (&cv[h].x)[j];
          if (model) model[i + j] = __float2bfloat16(p[4 * h + j]);
        }
      }
    }
  }
}

// sum of squares of a flat fp32 buffer (for gradient-norm logging), atomically added into out[0].
__global__ void sumsq_kernel(const float* __restrict__ x, long long n, float scale, float* __restrict__ out) {
  pdl_wait();
  pdl_trigger();
  float s = 0.f;
  for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x) {
    const float v = x[i] * scale;
    s += v * v;
  }
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) atomicAdd(out, s);
}

}  // namespace optim
}  // namespace b200

extern "C" {
using namespace b200;
using namespace b200::optim;

static int opt_grid(long long n, int per_thread) {
  long long b = (n / per_thread + 255) / 256;
  const long long cap = (long long)sm_count() * 8;
  if (b > cap) b = cap;
  if (b < 1) b = 1;
  return (int)b;
}

// one block per so many values, no cap but the grid's own limit
static int whole_grid(long long n, int per_block) {
  const long long b = (n + per_block - 1) / per_block;
  return (int)(b < 0x7fffffffll ? b : 0x7fffffffll);
}

// step is 1-based. model may be null (no bf16 copy). All buffers hold n elements and are 16-byte aligned.
int b200_adam_step(float* master, void* model, const float* grad, float* m, float* v, long long n, float lr,
                   float beta1, float beta2, float eps, float weight_decay, int step, float grad_scale, int decoupled,
                   cudaStream_t st) {
  if (!master || !grad || !m || !v || n <= 0 || step < 1) return B200_ERR_ARG;
  AdamArgs a{lr, beta1, beta2, eps, weight_decay, 1.f - powf(beta1, (float)step), 1.f - powf(beta2, (float)step),
             grad_scale, decoupled};
  launch_pdl(adam_kernel, whole_grid(n, 4 * 256), 256, 0, st, master, (__nv_bfloat16*)model, grad, m, v, n, a);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

int b200_adam8_step(float* master, void* model, const float* grad, void* mq, void* vq, float* mabs, float* vabs,
                    long long n, float lr, float beta1, float beta2, float eps, float weight_decay, int step,
                    float grad_scale, int decoupled, cudaStream_t st) {
  if (!master || !grad || !mq || !vq || !mabs || !vabs || n <= 0 || step < 1) return B200_ERR_ARG;
  AdamArgs a{lr, beta1, beta2, eps, weight_decay, 1.f - powf(beta1, (float)step), 1.f - powf(beta2, (float)step),
             grad_scale, decoupled};
  auto off = [](const void* p, int align) { return reinterpret_cast<uintptr_t>(p) & (align - 1); };
  const bool vec = !off(master, 16) && !off(grad, 16) && !off(model, 8) && !off(mq, 4) && !off(vq, 4);
  launch_pdl(vec ? adam8_kernel<true> : adam8_kernel<false>, whole_grid(n, QB * Q_WARPS), 32 * Q_WARPS, 0, st, master,
             (__nv_bfloat16*)model, grad, (int8_t*)mq, (uint8_t*)vq, mabs, vabs, n, a);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

int b200_simple_opt_step(float* master, void* model, const float* grad, float* s0, float* s1, long long n, int kind,
                         float lr, float weight_decay, float momentum, float alpha, float eps, int nesterov,
                         int first_step, float grad_scale, cudaStream_t st) {
  if (!master || !grad || !s0 || n <= 0 || kind < 0 || kind > 2 || (kind == 1 && !s1)) return B200_ERR_ARG;
  SimpleArgs a{lr, weight_decay, momentum, alpha, eps, grad_scale, kind, nesterov, first_step};
  launch_pdl(simple_kernel, opt_grid(n, 1), 256, 0, st, master, (__nv_bfloat16*)model, grad, s0, s1, n, a);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}

int b200_sumsq(const float* x, long long n, float scale, float* out, cudaStream_t st) {
  if (!x || !out || n <= 0) return B200_ERR_ARG;
  launch_pdl(sumsq_kernel, opt_grid(n, 4), 256, 0, st, x, n, scale, out);
  B200_CUDA_CHECK(cudaGetLastError());
  return B200_OK;
}
}
