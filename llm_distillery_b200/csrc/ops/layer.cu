// One decoder layer (RMSNorm, fused q/k/v projection with rotary embedding, causal GQA flash attention, output
// projection, RMSNorm, SwiGLU MLP; optional q/k/v bias) forward and backward as ONE host call each.
//
// A layer is 7 to 9 launches forward and about 20 backward. Issued one by one from Python (argument checks, allocations,
// a foreign call each) they cost the host about 20 us apiece, more than the kernels of a batch of a few hundred tokens
// take. Here the launchers of this library are called in sequence from C++: same kernels, same order, same bits. The
// caller hands over two slabs, one for what the backward pass needs (also the scratch of an inference pass) and one for
// the backward pass's temporaries, laid out by the functions below; nothing is allocated or kept here.
#include "../common/host.cuh"

extern "C" {
int b200_rmsnorm_fwd(const void*, const void*, const void*, void*, void*, float*, int, int, float, cudaStream_t);
int b200_rmsnorm_bwd_blocks(int);
int b200_rmsnorm_bwd(const void*, const void*, const void*, const float*, const void*, void*, float*, float*, int, int, int,
                     cudaStream_t);
int b200_gemm(const void*, const void*, void*, int, int, int, long long, long long, long long, int, int, int, int, int, float,
              const void*, long long, const unsigned int*, int, cudaStream_t);
int b200_gemm_rope(const void*, const void*, void*, const int*, const float*, const float*, int, int, int, int, int, long long,
                   long long, long long, int, cudaStream_t);
int b200_gemm_swiglu(const void*, const void*, void*, void*, int, int, int, long long, long long, long long, long long, int,
                     cudaStream_t);
int b200_gemm_swiglu_bwd(const void*, const void*, const void*, void*, int, int, int, long long, long long, long long,
                         long long, int, cudaStream_t);
int b200_rope(void*, const int*, const float*, const float*, long long, int, int, long long, int, cudaStream_t);
int b200_bias_add(void*, const void*, long long, int, long long, cudaStream_t);
int b200_bias_grad(const void*, float*, long long, int, long long, int, cudaStream_t);
int b200_swiglu_fwd(const void*, void*, long long, int, cudaStream_t);
int b200_swiglu_bwd(const void*, const void*, void*, long long, int, cudaStream_t);
int b200_flash_attn_fwd(const void*, void*, float*, int, int, int, int, int, int, cudaStream_t);
int b200_flash_attn_bwd_rope(const void*, const void*, const void*, const float*, float*, void*, float*, const int*,
                             const float*, const float*, int, int, int, int, int, int, int, cudaStream_t);
}

namespace b200 {
namespace layer {

struct Dims {
  long long T, N, A;   // tokens, q/k/v width, attention width
  int B, L, window, H, Hkv, d, h, f;
  Dims(int B_, int L_, int window_, int H_, int Hkv_, int d_, int h_, int f_)
      : T((long long)B_ * L_), N((long long)(H_ + 2 * Hkv_) * d_), A((long long)H_ * d_), B(B_), L(L_), window(window_), H(H_),
        Hkv(Hkv_), d(d_), h(h_), f(f_) {}
  bool ok() const { return B > 0 && L > 0 && H > 0 && Hkv > 0 && (d == 64 || d == 128) && h > 0 && f > 0 && T <= 0x7fffffff; }
};

// A GEMM of this layer may start on its weights while the launch before it drains (bit 1 of split_k): that launch is one of
// this layer's own, which write no weights. Not for the first launch of a call: what stands in front of it may expand or
// update them.
constexpr int kWeightsEarly = 2;
// Bit 2 of a forward call's split_k: no backward pass will read its slab (or it will be filled again first), so the gate and up
// values need not be written where the activation comes with their GEMM.
constexpr int kActOnly = 4;

// Carves 256-byte aligned pieces off a slab (base null: only sizes).
struct Slab {
  uint8_t* base;
  size_t used = 0;
  explicit Slab(void* b) : base(static_cast<uint8_t*>(b)) {}
  void* take(size_t bytes) {
    void* p = base ? base + used : nullptr;
    used += (bytes + 255) & ~size_t(255);
    return p;
  }
};

struct Saved {
  float *rstd1, *rstd2, *lse;
  void *n1, *qkv, *att, *h1, *n2, *gu, *act;
  size_t bytes;
  Saved(const Dims& m, void* base) {
    Slab s(base);
    const size_t T = (size_t)m.T;
    rstd1 = (float*)s.take(T * 4);
    rstd2 = (float*)s.take(T * 4);
    lse = (float*)s.take(T * m.H * 4);
    n1 = s.take(T * m.h * 2);
    qkv = s.take(T * m.N * 2);
    att = s.take(T * m.A * 2);
    h1 = s.take(T * m.h * 2);
    n2 = s.take(T * m.h * 2);
    gu = s.take(T * m.f * 4);
    act = s.take(T * m.f * 2);
    bytes = s.used;
  }
};

struct Scratch {
  void *dgu, *dact, *dn, *dh1, *datt, *dqkv;
  float *delta, *dq_acc, *partial, *dw;
  size_t bytes;
  Scratch(const Dims& m, void* base) {
    const size_t T = (size_t)m.T;
    Slab s(base);
    dn = s.take(T * m.h * 2);                  // gradient of a normalised input, MLP then attention
    dh1 = s.take(T * m.h * 2);
    partial = (float*)s.take((size_t)b200_rmsnorm_bwd_blocks((int)T) * m.h * 4);
    dw = (float*)s.take((size_t)m.h * 4);      // weight gradient of a norm that does not train
    const size_t mark = s.used;                // the MLP's gradients are dead when the attention's begin
    dgu = s.take(T * m.f * 4);
    dact = (m.f % 128) ? s.take(T * m.f * 2) : nullptr;
    const size_t end = s.used;
    s.used = mark;
    datt = s.take(T * m.A * 2);
    dqkv = s.take(T * m.N * 2);
    delta = (float*)s.take(T * m.H * 4);
    dq_acc = (float*)s.take(T * m.A * 4);
    bytes = s.used > end ? s.used : end;
  }
};

}  // namespace layer
}  // namespace b200

using namespace b200;

extern "C" long long b200_layer_saved_bytes(int B, int L, int H, int Hkv, int d, int h, int f) {
  const layer::Dims m(B, L, 0, H, Hkv, d, h, f);
  return m.ok() ? (long long)layer::Saved(m, nullptr).bytes : -1;
}

extern "C" long long b200_layer_scratch_bytes(int B, int L, int H, int Hkv, int d, int h, int f) {
  const layer::Dims m(B, L, 0, H, Hkv, d, h, f);
  return m.ok() ? (long long)layer::Scratch(m, nullptr).bytes : -1;
}

#define RUN(expr)                      \
  do {                                 \
    const int rc_ = (expr);            \
    if (rc_ != B200_OK) return rc_;    \
    ++launches;                        \
  } while (0)

// h2[T, h] = layer(x). h2 null: stop in front of the down projection (recomputation of what the backward pass reads).
// Returns the number of launches, or a negative error code.
extern "C" int b200_layer_fwd(const void* x, const int* pos, const float* cos_tab, const float* sin_tab, const void* w_ln1,
                              const void* w_qkv, const void* w_o, const void* w_ln2, const void* w_gu, const void* w_d,
                              const void* b_qkv, void* saved, void* h2, int B, int L, int window, int H, int Hkv, int d, int h,
                              int f, float eps, int split_k, cudaStream_t st) {
  const layer::Dims m(B, L, window, H, Hkv, d, h, f);
  if (!m.ok() || !x || !saved) return B200_ERR_ARG;
  const layer::Saved s(m, saved);
  const int T = (int)m.T, N = (int)m.N, A = (int)m.A;
  int launches = 0;
  void* gu = (split_k & layer::kActOnly) ? nullptr : s.gu;
  split_k = (split_k & ~layer::kActOnly) | layer::kWeightsEarly;
  RUN(b200_rmsnorm_fwd(x, nullptr, w_ln1, s.n1, nullptr, s.rstd1, T, h, eps, st));
  if (!b_qkv && N % 128 == 0) {
    RUN(b200_gemm_rope(s.n1, w_qkv, s.qkv, pos, cos_tab, sin_tab, T, N, h, H + Hkv, d, h, h, N, split_k, st));
  } else {
    RUN(b200_gemm(s.n1, w_qkv, s.qkv, T, N, h, h, h, N, 0, 0, 1, 0, 0, 1.f, nullptr, 0, nullptr, split_k, st));
    if (b_qkv) RUN(b200_bias_add(s.qkv, b_qkv, T, N, N, st));
    RUN(b200_rope(s.qkv, pos, cos_tab, sin_tab, T, H + Hkv, d, N, 0, st));
  }
  RUN(b200_flash_attn_fwd(s.qkv, s.att, s.lse, B, L, window, H, Hkv, d, st));
  RUN(b200_gemm(s.att, w_o, s.h1, T, h, A, A, A, h, 0, 0, 1, 0, 0, 1.f, x, h, nullptr, split_k, st));
  RUN(b200_rmsnorm_fwd(s.h1, nullptr, w_ln2, s.n2, nullptr, s.rstd2, T, h, eps, st));
  if (f % 128 == 0) {
    RUN(b200_gemm_swiglu(s.n2, w_gu, gu, s.act, T, f, h, h, h, 2LL * f, f, split_k, st));
  } else {
    RUN(b200_gemm(s.n2, w_gu, s.gu, T, 2 * f, h, h, h, 2LL * f, 0, 0, 1, 0, 0, 1.f, nullptr, 0, nullptr, split_k, st));
    RUN(b200_swiglu_fwd(s.gu, s.act, T, f, st));
  }
  if (h2) RUN(b200_gemm(s.act, w_d, h2, T, h, f, f, f, h, 0, 0, 1, 0, 0, 1.f, s.h1, h, nullptr, split_k, st));
  return launches;
}

// dx[T, h] from dh2[T, h]; weight gradients into the fp32 buffers g_* (null: that weight does not train), added to what
// the buffer holds where its bit of `acc` is set (bit 0 ln1, 1 qkv, 2 o, 3 ln2, 4 gate/up, 5 down, 6 q/k/v bias).
extern "C" int b200_layer_bwd(const void* dh2, const void* x, const int* pos, const float* cos_tab, const float* sin_tab,
                              const void* w_ln1, const void* w_qkv, const void* w_o, const void* w_ln2, const void* w_gu,
                              const void* w_d, void* saved, void* scratch, void* dx, float* g_ln1, float* g_qkv, float* g_o,
                              float* g_ln2, float* g_gu, float* g_d, float* g_bqkv, int acc, int B, int L, int window, int H,
                              int Hkv, int d, int h, int f, int split_k, cudaStream_t st) {
  const layer::Dims m(B, L, window, H, Hkv, d, h, f);
  if (!m.ok() || !dh2 || !x || !saved || !scratch || !dx) return B200_ERR_ARG;
  const layer::Saved s(m, saved);
  const layer::Scratch t(m, scratch);
  const int T = (int)m.T, N = (int)m.N, A = (int)m.A;
  int launches = 0;
  auto wgrad = [&](const void* dy, int n, const void* in, int k, float* g, int bit) {     // g[n, k] (+)= dy^T in
    return b200_gemm(dy, in, g, n, k, T, n, k, k, 1, 1, 1, 1, (acc >> bit) & 1, 1.f, nullptr, 0, nullptr, split_k, st);
  };
  auto early = [&]() { return split_k | (launches > 0 ? layer::kWeightsEarly : 0); };
  auto dgrad = [&](const void* dy, int n, const void* w, int k, void* out) {              // out[T, k] = dy[T, n] w[n, k]
    return b200_gemm(dy, w, out, T, k, n, n, k, k, 0, 1, 1, 0, 0, 1.f, nullptr, 0, nullptr, early(), st);
  };
  // MLP branch
  if (g_d) RUN(wgrad(dh2, h, s.act, f, g_d, 5));
  if (f % 128 == 0) {
    RUN(b200_gemm_swiglu_bwd(dh2, w_d, s.gu, t.dgu, T, f, h, h, f, 2LL * f, 2LL * f, early(), st));
  } else {
    RUN(dgrad(dh2, h, w_d, f, t.dact));
    RUN(b200_swiglu_bwd(s.gu, t.dact, t.dgu, T, f, st));
  }
  if (g_gu) RUN(wgrad(t.dgu, 2 * f, s.n2, h, g_gu, 4));
  RUN(dgrad(t.dgu, 2 * f, w_gu, h, t.dn));
  RUN(b200_rmsnorm_bwd(t.dn, s.h1, w_ln2, s.rstd2, dh2, t.dh1, t.partial, g_ln2 ? g_ln2 : t.dw, g_ln2 ? (acc >> 3) & 1 : 0, T,
                       h, st));
  // attention branch
  if (g_o) RUN(wgrad(t.dh1, h, s.att, A, g_o, 2));
  RUN(dgrad(t.dh1, h, w_o, A, t.datt));
  RUN(b200_flash_attn_bwd_rope(t.datt, s.qkv, s.att, s.lse, t.delta, t.dqkv, t.dq_acc, pos, cos_tab, sin_tab, B, L, window, H,
                               Hkv, d, split_k & 1, st));
  if (g_bqkv) RUN(b200_bias_grad(t.dqkv, g_bqkv, T, N, N, (acc >> 6) & 1, st));
  if (g_qkv) RUN(wgrad(t.dqkv, N, s.n1, h, g_qkv, 1));
  RUN(dgrad(t.dqkv, N, w_qkv, h, t.dn));
  RUN(b200_rmsnorm_bwd(t.dn, x, w_ln1, s.rstd1, t.dh1, dx, t.partial, g_ln1 ? g_ln1 : t.dw, g_ln1 ? acc & 1 : 0, T, h, st));
  return launches + 4;     // the two norms launch a column sum besides, attention its row sums and its conversion
}

// Several layers in one call: where a batch is a few hundred tokens the host's way from one layer to the next (a foreign call,
// a graph node, allocations: 45 us) is longer than the layer's kernels take. One record per layer, addresses as integers.
struct B200StackLayer {
  unsigned long long cos_tab, sin_tab, w_ln1, w_qkv, w_o, w_ln2, w_gu, w_d, b_qkv, saved, out;
  long long window;
};
struct B200StackGrad {
  unsigned long long x, g_ln1, g_qkv, g_o, g_ln2, g_gu, g_d, g_bqkv;   // the layer's input; gradients as in b200_layer_bwd
  long long acc;
};

// out of the last layer = layers(x). Returns the number of launches, or a negative error code.
extern "C" int b200_stack_fwd(const B200StackLayer* l, int n, const void* x, const int* pos, int B, int L, int H, int Hkv, int d,
                              int h, int f, float eps, int split_k, cudaStream_t st) {
  if (!l || n <= 0 || !x) return B200_ERR_ARG;
  int launches = 0;
  for (int i = 0; i < n; ++i) {
    if (!l[i].out) return B200_ERR_ARG;
    const int rc = b200_layer_fwd(x, pos, (const float*)l[i].cos_tab, (const float*)l[i].sin_tab, (const void*)l[i].w_ln1,
                                  (const void*)l[i].w_qkv, (const void*)l[i].w_o, (const void*)l[i].w_ln2,
                                  (const void*)l[i].w_gu, (const void*)l[i].w_d, (const void*)l[i].b_qkv, (void*)l[i].saved,
                                  (void*)l[i].out, B, L, (int)l[i].window, H, Hkv, d, h, f, eps, split_k, st);
    if (rc < 0) return rc;
    launches += rc;
    x = (const void*)l[i].out;
  }
  return launches;
}

// dx = gradient of the first layer's input; dx0 and dx1 [T, h] hold the gradients between layers in turn. `done` receives how
// many layers, from the last on, have run (all of them unless an error code is returned).
extern "C" int b200_stack_bwd(const B200StackLayer* l, const B200StackGrad* g, int n, const void* dout, const int* pos,
                              void* scratch, void* dx, void* dx0, void* dx1, int B, int L, int H, int Hkv, int d, int h, int f,
                              int split_k, int* done, cudaStream_t st) {
  if (!l || !g || n <= 0 || !done || (n > 1 && (!dx0 || !dx1))) return B200_ERR_ARG;
  int launches = 0;
  *done = 0;
  for (int i = n - 1; i >= 0; --i) {
    void* to = i == 0 ? dx : (i & 1) ? dx1 : dx0;
    const int rc = b200_layer_bwd(dout, (const void*)g[i].x, pos, (const float*)l[i].cos_tab, (const float*)l[i].sin_tab,
                                  (const void*)l[i].w_ln1, (const void*)l[i].w_qkv, (const void*)l[i].w_o,
                                  (const void*)l[i].w_ln2, (const void*)l[i].w_gu, (const void*)l[i].w_d, (void*)l[i].saved,
                                  scratch, to, (float*)g[i].g_ln1, (float*)g[i].g_qkv, (float*)g[i].g_o, (float*)g[i].g_ln2,
                                  (float*)g[i].g_gu, (float*)g[i].g_d, (float*)g[i].g_bqkv, (int)g[i].acc, B, L,
                                  (int)l[i].window, H, Hkv, d, h, f, split_k, st);
    if (rc < 0) return rc;
    launches += rc;
    ++*done;
    dout = to;
  }
  return launches;
}
