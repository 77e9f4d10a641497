"""tcgen05 GEMM (all three operand layouts, epilogue options) against fp32 PyTorch matmul."""
import pytest
import torch

from llm_distillery_b200.ops import basic, _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _ref(a, b, a_mn, b_mn):
    A = (a.t() if a_mn else a).float()
    B = (b if b_mn else b.t()).float()
    return A @ B


@pytest.mark.parametrize("a_mn,b_mn", [(False, False), (False, True), (True, True), (True, False)])
@pytest.mark.parametrize("M,N,K", [(128, 256, 64), (128, 128, 128), (384, 640, 200), (1000, 1000, 1000), (2048, 2560, 2048),
                                   (130, 72, 8)])
def test_gemm_layouts(M, N, K, a_mn, b_mn):
    torch.manual_seed(M * 7 + N * 3 + K)
    if (a_mn and M % 8) or (b_mn and N % 8):
        pytest.skip("MN-major operands need a 16-byte aligned row stride")
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV).bfloat16()
    b = torch.randn((K, N) if b_mn else (N, K), device=DEV).bfloat16()
    out = basic.gemm(a, b, a_mn=a_mn, b_mn=b_mn)
    assert _lib.take_device_error() == 0
    r = _ref(a, b, a_mn, b_mn)
    tol = 1e-2 * max(1.0, r.abs().max().item())
    assert (out.float() - r).abs().max().item() <= tol


def test_gemm_epilogues():
    torch.manual_seed(5)
    a = torch.randn(300, 136, device=DEV).bfloat16()
    b = torch.randn(520, 136, device=DEV).bfloat16()
    r = a.float() @ b.float().t()
    # fp32 output, overwrite then accumulate
    c = torch.empty(300, 520, device=DEV)
    basic.gemm(a, b, out=c)
    assert torch.allclose(c, r, atol=1e-3, rtol=1e-3)
    basic.gemm(a, b, out=c, accumulate=True, alpha=0.5)
    assert torch.allclose(c, 1.5 * r, atol=2e-3, rtol=1e-3)
    # bf16 accumulate and residual
    rsd = torch.randn(300, 520, device=DEV).bfloat16()
    o = basic.gemm(a, b, residual=rsd)
    assert torch.allclose(o.float(), (r + rsd.float()), atol=0.15, rtol=2e-2)
    # fp16 operands
    o16 = basic.gemm(a.half(), b.half())
    assert torch.allclose(o16.float(), a.half().float() @ b.half().float().t(), atol=0.1, rtol=1e-2)
    # strided (row-padded) operands and output
    big = torch.randn(300, 256, device=DEV).bfloat16()
    outbig = torch.zeros(300, 1024, device=DEV, dtype=torch.bfloat16)
    basic.gemm(big[:, :136], b, out=outbig[:, 8:528])
    assert torch.allclose(outbig[:, 8:528].float(), big[:, :136].float() @ b.float().t(), atol=0.15, rtol=2e-2)
    assert outbig[:, :8].abs().max() == 0 and outbig[:, 528:].abs().max() == 0
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("a_mn,b_mn", [(True, True), (False, False)])
def test_split_k_fp32_output_overwrite_accumulate_and_strided(a_mn, b_mn):
    """Long reduction, few tiles, fp32 output: the CTA-pair kernel splits K and adds the slices of a tile in the order
    of their index, so the result repeats bit for bit."""
    torch.manual_seed(11)
    M, N, K = 1280, 1000, 8192
    a = (torch.randn((K, M) if a_mn else (M, K), device=DEV) * 0.1).bfloat16()
    b = (torch.randn((K, N) if b_mn else (N, K), device=DEV) * 0.1).bfloat16()
    r = _ref(a, b, a_mn, b_mn)
    wide = torch.full((M, N + 24), 7.0, device=DEV)          # row-padded output: the memset must respect the stride
    c = wide[:, 8:8 + N]
    basic.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=c)
    assert torch.allclose(c, r, atol=2e-2, rtol=2e-3), (c - r).abs().max()
    assert (wide[:, :8] == 7).all() and (wide[:, 8 + N:] == 7).all()
    first = c.clone()
    for _ in range(3):
        basic.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=c)
        assert torch.equal(c, first)
    basic.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=c, accumulate=True)
    assert torch.allclose(c, 2 * r, atol=4e-2, rtol=2e-3)
    assert _lib.take_device_error() == 0


def test_linear_helpers_match_autograd():
    torch.manual_seed(6)
    x = torch.randn(512, 256, device=DEV).bfloat16()
    w = torch.randn(384, 256, device=DEV).bfloat16() * 0.05
    dy = torch.randn(512, 384, device=DEV).bfloat16()
    xf, wf = x.float().requires_grad_(), w.float().requires_grad_()
    (xf @ wf.t()).backward(dy.float())
    assert torch.allclose(basic.linear_fwd(x, w).float(), (x.float() @ w.float().t()), atol=5e-2, rtol=2e-2)
    assert torch.allclose(basic.linear_dgrad(dy, w).float(), xf.grad, atol=5e-2, rtol=2e-2)
    g = torch.zeros(384, 256, device=DEV)
    basic.linear_wgrad(dy, x, out=g, accumulate=True)
    assert torch.allclose(g, wf.grad, atol=0.5, rtol=2e-2)


@pytest.mark.parametrize("T,f,K", [(1000, 1408, 512), (4096, 5632, 2048), (513, 128, 64), (2048, 1280, 200)])
def test_gate_up_gemm_with_swiglu_in_the_epilogue(T, f, K):
    """One launch writes gu = x W^T and act = silu(gate) * up; both must equal the two-kernel path bit for bit (act is
    computed from the rounded gate / up values), and nothing may be written outside the outputs."""
    torch.manual_seed(T + f)
    x = torch.randn(T, K, device=DEV).bfloat16()
    w = (torch.randn(2 * f, K, device=DEV) * 0.05).bfloat16()
    gu, act = basic.linear_swiglu_fwd(x, w)
    assert _lib.take_device_error() == 0
    gu_ref = basic.linear_fwd(x, w)
    act_ref = basic.swiglu_fwd(gu_ref)
    assert torch.equal(gu, gu_ref)
    assert torch.equal(act, act_ref)
    r = x.float() @ w.float().t()
    assert torch.allclose(gu.float(), r, atol=2e-2 * max(1.0, r.abs().max().item()), rtol=2e-2)
    want = torch.nn.functional.silu(r[:, :f]) * r[:, f:]
    assert torch.allclose(act.float(), want, atol=3e-2 * max(1.0, want.abs().max().item()), rtol=3e-2)


@pytest.mark.parametrize("T,f,h", [(1000, 1408, 512), (4096, 5632, 2048), (513, 128, 64), (2048, 1280, 200)])
def test_down_projection_dgrad_with_swiglu_backward_in_the_epilogue(T, f, h):
    """dgu from one launch equals dgrad GEMM + SwiGLU backward kernel bit for bit (d(act) is rounded to bf16 before the
    activation's derivative is applied, exactly as when it is stored in between)."""
    torch.manual_seed(T + f + 1)
    dy = torch.randn(T, h, device=DEV).bfloat16()
    w_d = (torch.randn(h, f, device=DEV) * 0.05).bfloat16()
    gu = torch.randn(T, 2 * f, device=DEV).bfloat16()
    dgu = basic.linear_dgrad_swiglu_bwd(dy, w_d, gu)
    assert _lib.take_device_error() == 0
    dact = basic.linear_dgrad(dy, w_d)
    ref = basic.swiglu_bwd(gu, dact)
    assert torch.equal(dgu, ref)
    g, u, d = gu[:, :f].float(), gu[:, f:].float(), dy.float() @ w_d.float()
    sg = torch.sigmoid(g)
    want = torch.cat([d * u * (sg + g * sg * (1 - sg)), d * g * sg], 1)
    assert torch.allclose(dgu.float(), want, atol=3e-2 * max(1.0, want.abs().max().item()), rtol=3e-2)


@pytest.mark.parametrize("T,H,Hkv,d,K", [(1000, 8, 2, 64, 512), (4096, 32, 4, 64, 2048), (2048, 8, 2, 128, 1024),
                                         (513, 2, 1, 128, 64)])
def test_qkv_gemm_with_rotary_embedding_in_the_epilogue(T, H, Hkv, d, K):
    """One launch = GEMM + rope kernel, bit for bit; the value heads (the last Hkv) are stored unrotated."""
    torch.manual_seed(T + d)
    N = (H + 2 * Hkv) * d
    x = torch.randn(T, K, device=DEV).bfloat16()
    w = (torch.randn(N, K, device=DEV) * 0.05).bfloat16()
    L = 257
    pos = (torch.arange(T, device=DEV, dtype=torch.int32) * 7) % L
    cos, sin = basic.rope_tables(L, d, 10000.0, DEV)
    got = basic.linear_rope_fwd(x, w, pos, cos, sin, H + Hkv, d)
    assert _lib.take_device_error() == 0
    plain = basic.linear_fwd(x, w)
    ref = basic.rope_(plain.clone(), pos, cos, sin, H + Hkv, d)
    assert torch.equal(got, ref)
    assert torch.equal(got[:, (H + Hkv) * d:], plain[:, (H + Hkv) * d:])
    assert not torch.equal(got[:, : H * d], plain[:, : H * d])


@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (93, 2048, 5632), (128, 128, 512), (129, 72, 200), (300, 1152, 896),
                                   (257, 896, 1024), (896, 256, 776)])
@pytest.mark.parametrize("layout", ["nt", "nn", "tn"])
def test_few_tiles_split_over_a_cluster(M, N, K, layout):
    """Outputs of few tiles: K is cut over the CTAs of a cluster and the partial tiles are added in slice order. Every
    store form against fp64, nothing outside the output, and the same bits twice. Bound: operands are exact bf16, the
    fp32 sums err by about sqrt(K) 2^-24 of the sum of |products| / sqrt(K), far below the 2^-9 of the bf16 store."""
    a_mn, b_mn = layout == "tn", layout != "nt"
    if a_mn and M % 8:
        pytest.skip("row strides are multiples of 8 elements")
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV).bfloat16()
    b = (torch.randn((K, N) if b_mn else (N, K), device=DEV) * 0.1).bfloat16()
    kw = dict(a_mn=a_mn, b_mn=b_mn, split_k=True)
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
    scale = ref.abs().max().item()
    guard = torch.full((M + 2, N + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    out = guard[1:-1, :N]
    basic.gemm(a, b, out=out, **kw)
    assert _lib.take_device_error() == 0
    assert (guard[0] == 7).all() and (guard[-1] == 7).all() and (guard[1:-1, N:] == 7).all()
    assert (out.double() - ref).abs().max().item() <= 2 ** -8 * scale
    assert torch.equal(out, basic.gemm(a, b, **kw))
    res = torch.randn(M, N, device=DEV).bfloat16()
    got = basic.gemm(a, b, residual=res, alpha=0.5, **kw)
    want = 0.5 * ref + res.double()
    assert (got.double() - want).abs().max().item() <= 2 ** -8 * want.abs().max().item()
    acc = torch.randn(M, N, device=DEV)
    want = acc.double() + ref
    basic.gemm(a, b, out=acc, accumulate=True, **kw)
    assert (acc.double() - want).abs().max().item() <= 1e-5 * (want.abs().max().item() + K ** 0.5)


@pytest.mark.parametrize("T", [1, 31, 130, 511, 777])
def test_one_slice_keeps_the_order_of_the_large_tiles(T):
    """Without ``split_k`` a row's result has the same bits in the few-tile kernel and in the one of 128 x 256 tiles
    (4096 x 896 are 64 tiles of 256 x 256, too few for the pair kernel; the next test has that one)."""
    torch.manual_seed(T)
    a = torch.randn(4096, 1400, device=DEV).bfloat16()
    b = (torch.randn(896, 1400, device=DEV) * 0.1).bfloat16()
    assert torch.equal(basic.gemm(a[:T], b), basic.gemm(a, b)[:T])
    assert torch.equal(basic.gemm(a[:T], b, out_dtype=torch.float32), basic.gemm(a, b, out_dtype=torch.float32)[:T])


@pytest.mark.parametrize("T", [1, 130, 777, 2048])
def test_one_slice_keeps_the_order_of_the_pair_kernel(T):
    """The same against the 256 x 256 kernel (8192 x 2304: 288 tiles), for the plain, rotary and SwiGLU forms. bf16 outputs
    only: that kernel cuts the K of fp32 outputs by their tile count, with or without ``split_k``."""
    torch.manual_seed(T)
    K, N, d = 1400, 2304, 128
    a = torch.randn(8192, K, device=DEV).bfloat16()
    w = (torch.randn(N, K, device=DEV) * 0.1).bfloat16()
    pos = torch.arange(8192, device=DEV, dtype=torch.int32) % 300
    cos, sin = basic.rope_tables(300, d, 10000.0, DEV)
    assert torch.equal(basic.gemm(a[:T], w), basic.gemm(a, w)[:T])
    assert torch.equal(basic.linear_rope_fwd(a[:T], w, pos[:T], cos, sin, 14, d), basic.linear_rope_fwd(a, w, pos, cos, sin, 14, d)[:T])
    for few, many in zip(basic.linear_swiglu_fwd(a[:T], w), basic.linear_swiglu_fwd(a, w)):
        assert torch.equal(few, many[:T])
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("M,N,K", [(1, 4, 64), (31, 68, 200), (93, 2048, 1024), (130, 132, 896), (777, 896, 264)])
@pytest.mark.parametrize("split", [False, True])
def test_few_tile_stores_of_both_forms(M, N, K, split):
    """Outputs whose rows start on boundaries of four columns and outputs that are off them hold the same bits: plain, with a
    residual, and fp32 stored and added."""
    g = torch.Generator("cuda").manual_seed(M + N)
    x, w = (torch.randn(n, K, device=DEV, generator=g).bfloat16() for n in (M, N))
    res = torch.randn(M, N, device=DEV, generator=g).bfloat16()

    def off(t):
        o = torch.zeros(M, N + 1, device=DEV, dtype=t.dtype)[:, :N]
        return o.copy_(t)
    for b_mn in (False, True)[:1 + (N % 8 == 0)]:
        b = w.t().contiguous() if b_mn else w
        a = basic.gemm(x, b, b_mn=b_mn, split_k=split)
        assert torch.equal(a, basic.gemm(x, b, b_mn=b_mn, out=off(a * 0), split_k=split))
        r = basic.gemm(x, b, b_mn=b_mn, residual=res, split_k=split)
        assert torch.equal(r, basic.gemm(x, b, b_mn=b_mn, residual=res, out=off(a * 0), split_k=split))
    dy, xt = torch.randn(K, 8 * M, device=DEV, generator=g).bfloat16(), torch.randn(K, N + (-N) % 8, device=DEV, generator=g).bfloat16()
    f = basic.gemm(dy, xt, a_mn=True, b_mn=True, out_dtype=torch.float32, split_k=split)
    o = torch.zeros(f.shape[0], f.shape[1] + 1, device=DEV)[:, :-1]
    assert torch.equal(f, basic.gemm(dy, xt, a_mn=True, b_mn=True, out=o, split_k=split))
    twice = basic.gemm(dy, xt, a_mn=True, b_mn=True, out=f.clone(), accumulate=True, split_k=split)
    assert torch.equal(twice, basic.gemm(dy, xt, a_mn=True, b_mn=True, out=o, accumulate=True, split_k=split))
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("T,f,h", [(5003, 1408, 520), (4737, 1152, 264), (18945, 128, 256), (4865, 1280, 2048)])
def test_swiglu_backward_epilogue_of_ragged_pair_tiles(T, f, h):
    """Rows that end inside a warp's 32 and features that end in the middle of a 256 x 256 tile: the bits of GEMM + separate
    kernel, and nothing written behind the last row."""
    g = torch.Generator("cuda").manual_seed(T)
    dy = torch.randn(T, h, device=DEV, generator=g).bfloat16()
    w_d = (torch.randn(h, f, device=DEV, generator=g) * 0.05).bfloat16()
    gu = torch.randn(T, 2 * f, device=DEV, generator=g).bfloat16()
    out = torch.full((T + 40, 2 * f), 7.0, device=DEV, dtype=torch.bfloat16)
    dgu = basic.linear_dgrad_swiglu_bwd(dy, w_d, gu, out=out[:T])
    assert torch.equal(dgu, basic.swiglu_bwd(gu, basic.linear_dgrad(dy, w_d)))
    assert (out[T:] == 7.0).all() and _lib.take_device_error() == 0


@pytest.mark.parametrize("M,N,K", [(5003, 1416, 520), (4737, 1160, 264), (18945, 200, 256), (8200, 2048, 2048)])
def test_residual_epilogue_of_ragged_pair_tiles(M, N, K):
    """Rows that end inside a warp's 32 and columns that end inside a quarter of a 256 x 256 tile: the bits of the general
    epilogue (an output off the 16-byte boundaries takes it), in place too, and nothing written outside the output."""
    g = torch.Generator("cuda").manual_seed(M)
    x, w = (torch.randn(n, K, device=DEV, generator=g).bfloat16() for n in (M, N))
    res = torch.randn(M, N, device=DEV, generator=g).bfloat16()
    plain = torch.zeros(M, N + 1, device=DEV, dtype=torch.bfloat16)[:, :N]
    basic.gemm(x, w, residual=res, alpha=0.37, out=plain)
    out = torch.full((M + 40, N + 8), 7.0, device=DEV, dtype=torch.bfloat16)
    basic.gemm(x, w, residual=res, alpha=0.37, out=out[:M, :N])
    assert torch.equal(out[:M, :N], plain) and (out[M:] == 7.0).all() and (out[:, N:] == 7.0).all()
    assert torch.equal(basic.gemm(x, w, residual=res, alpha=0.37, out=res), plain) and _lib.take_device_error() == 0


@pytest.mark.parametrize("M,N,K", [(8, 64, 64), (128, 128, 512), (136, 72, 200), (304, 1152, 896)])
@pytest.mark.parametrize("layout,dtype", [("nt", torch.float16), ("nn", torch.float16), ("tn", torch.float16),
                                          ("tt", torch.float16), ("tt", torch.bfloat16)])
def test_few_tiles_split_in_fp16_and_with_a_alone_transposed(M, N, K, layout, dtype):
    """Forms that the models do not use: fp16 operands, and A stored [K, M] beside B stored [N, K]. Bound: one rounding of
    the result, 2^-11 (fp16) or 2^-8, and the 32-bit sums, which are far below."""
    a_mn, b_mn = layout[0] == "t", layout[1] == "n"
    torch.manual_seed(M + N + K)
    a = torch.randn((K, M) if a_mn else (M, K), device=DEV).to(dtype)
    b = (torch.randn((K, N) if b_mn else (N, K), device=DEV) * 0.1).to(dtype)
    ref = (a.t() if a_mn else a).double() @ (b if b_mn else b.t()).double()
    got = basic.gemm(a, b, a_mn=a_mn, b_mn=b_mn, split_k=True)
    eps = 2 ** -11 if dtype == torch.float16 else 2 ** -8
    assert got.dtype == dtype and ((got.double() - ref).abs() <= eps * ref.abs() + 1e-5 * K ** 0.5).all()
    acc = basic.gemm(a, b, a_mn=a_mn, b_mn=b_mn, out=got.clone(), accumulate=True, split_k=True)
    want = got.double() + ref
    assert ((acc.double() - want).abs() <= eps * want.abs() + 1e-5 * K ** 0.5).all()
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("T", [1, 31, 130, 511, 777])
@pytest.mark.parametrize("split", [False, True])
def test_fused_epilogues_on_few_rows(T, split):
    """The projections with rotary embedding and SwiGLU (forward and backward) in the cluster kernel's epilogue: the
    bits of GEMM + separate kernel, for heads of 64 and 128 and for row counts off the tile."""
    torch.manual_seed(T)
    K, f = 896, 1408
    x = torch.randn(T, K, device=DEV).bfloat16()
    w = (torch.randn(2 * f, K, device=DEV) * 0.05).bfloat16()
    gu, act = basic.linear_swiglu_fwd(x, w, split_k=split)
    assert torch.equal(gu, basic.linear_fwd(x, w, split_k=split)) and torch.equal(act, basic.swiglu_fwd(gu))
    wd = (torch.randn(K, f, device=DEV) * 0.05).bfloat16()
    dact = basic.linear_dgrad(x, wd, split)
    assert torch.equal(basic.linear_dgrad_swiglu_bwd(x, wd, gu, split_k=split), basic.swiglu_bwd(gu, dact))
    for H, Hkv, d in ((14, 2, 64), (6, 1, 128)):
        wq = (torch.randn((H + 2 * Hkv) * d, K, device=DEV) * 0.05).bfloat16()
        pos = (torch.arange(T, device=DEV, dtype=torch.int32) * 5) % 300
        cos, sin = basic.rope_tables(300, d, 10000.0, DEV)
        got = basic.linear_rope_fwd(x, wq, pos, cos, sin, H + Hkv, d, split_k=split)
        assert torch.equal(got, basic.rope_(basic.linear_fwd(x, wq, split_k=split), pos, cos, sin, H + Hkv, d))
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("T", [1, 33, 600])
@pytest.mark.parametrize("form", ["fp32", "odd stride", "offset"])
def test_fused_epilogues_copy_to_outputs_they_cannot_store_to(T, form):
    """Outputs of another type, with rows off 16 bytes or from an odd base receive the values of the call without them."""
    torch.manual_seed(T)
    K, f = 320, 256
    x = torch.randn(T, K, device=DEV).bfloat16()
    w = (torch.randn(2 * f, K, device=DEV) * 0.1).bfloat16()
    wd = (torch.randn(K, f, device=DEV) * 0.1).bfloat16()

    def output(cols):
        if form == "fp32":
            return torch.zeros(T, cols, device=DEV)
        if form == "odd stride":
            return torch.zeros(T, cols + 3, device=DEV, dtype=torch.bfloat16)[:, :cols]
        return torch.zeros(T * cols + 1, device=DEV, dtype=torch.bfloat16)[1:].view(T, cols)
    gu, act = basic.linear_swiglu_fwd(x, w)
    og, oa, od = output(2 * f), output(f), output(2 * f)
    rg, ra = basic.linear_swiglu_fwd(x, w, og, oa)
    assert rg is og and ra is oa and torch.equal(og, gu.to(og.dtype)) and torch.equal(oa, act.to(oa.dtype))
    dgu = basic.linear_dgrad_swiglu_bwd(x, wd, gu)
    assert basic.linear_dgrad_swiglu_bwd(x, wd, gu, out=od) is od and torch.equal(od, dgu.to(od.dtype))
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("T,f,K,split", [(93, 1408, 512, True), (93, 1408, 512, False), (777, 384, 896, False),
                                         (5003, 1408, 520, False), (4737, 1152, 264, True)])
def test_swiglu_epilogue_without_the_gate_and_up_values(T, f, K, split):
    """Few-tile and pair kernels: the same activation, nothing written behind it."""
    g = torch.Generator("cuda").manual_seed(T)
    x, w = torch.randn(T, K, device=DEV, generator=g).bfloat16(), (torch.randn(2 * f, K, device=DEV, generator=g) * 0.05).bfloat16()
    gu, act = basic.linear_swiglu_fwd(x, w, split_k=split)
    buf = torch.full((T + 1, f), 7.0, device=DEV, dtype=torch.bfloat16)
    none, alone = basic.linear_swiglu_fwd(x, w, out_act=buf[:T], split_k=split, keep_gu=False)
    assert none is None and gu.shape == (T, 2 * f) and torch.equal(act, alone) and alone.data_ptr() == buf.data_ptr()
    assert (buf[T] == 7).all() and _lib.take_device_error() == 0


@pytest.mark.parametrize("T", [450, 777])
def test_few_tile_kernel_beyond_the_resident_grid(T):
    """Several waves of small tiles where the large ones would just miss whole rounds: the bits of the large tiles, which a call
    with more rows of output takes."""
    g = torch.Generator("cuda").manual_seed(T)
    x, w = torch.randn(8192, 896, device=DEV, generator=g).bfloat16(), (torch.randn(2 * 4864, 896, device=DEV, generator=g) * 0.1).bfloat16()
    for few, many in zip(basic.linear_swiglu_fwd(x[:T], w), basic.linear_swiglu_fwd(x, w)):
        assert torch.equal(few, many[:T])
    dy = torch.randn(T, 4 * 9728, device=DEV, generator=g).bfloat16()
    few, many = (basic.gemm(d, x[:T], a_mn=True, b_mn=True, out_dtype=torch.float32) for d in (dy[:, :9728].contiguous(), dy))
    assert torch.equal(few, many[:9728])
    both = basic.gemm(dy[:, :9728].contiguous(), x[:T], a_mn=True, b_mn=True, out=few.clone(), accumulate=True)
    assert torch.equal(both, basic.gemm(dy, x[:T], a_mn=True, b_mn=True, out=many.clone(), accumulate=True)[:9728])
    assert _lib.take_device_error() == 0
