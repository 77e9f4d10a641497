"""sm_100a flash attention (forward and backward) against the fp32 PyTorch restatement."""
import pytest
import torch

from llm_distillery_b200.ops import attention, _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"

CASES = [(1, 128, 1, 1, 64), (1, 128, 2, 1, 64), (2, 256, 4, 2, 64), (2, 384, 8, 2, 64), (1, 200, 4, 4, 64), (3, 1024, 4, 1, 64),
         (1, 128, 2, 1, 128), (2, 320, 4, 2, 128), (1, 1024, 8, 2, 128)]


@pytest.mark.parametrize("B,L,H,Hkv,d", CASES)
def test_flash_fwd(B, L, H, Hkv, d):
    torch.manual_seed(B * 1000 + L + d)
    qkv = (torch.randn(B * L, (H + 2 * Hkv) * d, device=DEV) * 1.5).bfloat16()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d)
    assert _lib.take_device_error() == 0
    ro, rl = attention.attention_reference_fwd(qkv.float(), B, L, H, Hkv, d)
    assert torch.allclose(lse, rl, atol=2e-2, rtol=1e-3), (lse - rl).abs().max()
    assert torch.allclose(out.float(), ro, atol=3e-2, rtol=3e-2), (out.float() - ro).abs().max()


@pytest.mark.parametrize("B,L,H,Hkv,d", CASES)
def test_flash_bwd(B, L, H, Hkv, d):
    torch.manual_seed(B * 77 + L + d)
    qkv = (torch.randn(B * L, (H + 2 * Hkv) * d, device=DEV)).bfloat16()
    dout = torch.randn(B * L, H * d, device=DEV).bfloat16()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d)
    dqkv = attention.attention_bwd(dout, qkv, out, lse, B, L, H, Hkv, d)
    assert _lib.take_device_error() == 0
    ro, rl = attention.attention_reference_fwd(qkv.float(), B, L, H, Hkv, d)
    ref = attention.attention_reference_bwd(dout.float(), qkv.float(), ro, rl, B, L, H, Hkv, d)
    err = (dqkv.float() - ref).abs().max().item()
    assert err <= 6e-2 * max(1.0, ref.abs().max().item()), err


@pytest.mark.parametrize("B,L,H,Hkv,d", [(2, 384, 8, 2, 64), (1, 1000, 4, 4, 128), (3, 130, 6, 3, 64)])
def test_backward_with_the_inverse_rotation_of_dq_in_the_conversion_pass(B, L, H, Hkv, d):
    """dQ is rotated back where its fp32 accumulator becomes bf16, dK by the rope kernel on the key columns only: the
    result equals attention backward + inverse rope over q and k bit for bit."""
    from llm_distillery_b200.ops import basic
    torch.manual_seed(L + d)
    qkv = torch.randn(B * L, (H + 2 * Hkv) * d, device="cuda").bfloat16()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d)
    dout = torch.randn_like(out)
    pos = torch.arange(L, dtype=torch.int32, device="cuda").repeat(B)
    cos, sin = basic.rope_tables(L, d, 10000.0, "cuda")
    got = attention.attention_bwd_unrotated(dout, qkv, out, lse, B, L, H, Hkv, d, pos, cos, sin)
    assert _lib.take_device_error() == 0
    ref = attention.attention_bwd(dout, qkv, out, lse, B, L, H, Hkv, d)
    v_cols = slice((H + Hkv) * d, None)
    # dQ accumulates through TMA reduce-add in an order that varies from run to run: compare to rounding, and the
    # untouched value columns and the rotation itself exactly on a copy of the SAME backward result
    same = ref.clone()
    basic.rope_(same, pos, cos, sin, H + Hkv, d, inverse=True)
    assert torch.allclose(got.float(), same.float(), atol=3e-2 * max(1.0, same.float().abs().max().item()), rtol=3e-2)
    assert torch.allclose(got[:, v_cols].float(), ref[:, v_cols].float(), atol=2e-2, rtol=2e-2)
    # exactness of the fused conversion: feed one accumulator through both paths
    acc = torch.randn(B * L, H * d, device="cuda")
    a = torch.zeros(B * L, (H + 2 * Hkv) * d, device="cuda", dtype=torch.bfloat16)
    a[:, : H * d] = acc.bfloat16()
    basic.rope_(a, pos, cos, sin, H, d, inverse=True)
    from llm_distillery_b200.ops import flash  # noqa: F401  (registers the entry point)
    b = torch.zeros_like(a)
    _lib.check(_lib.kernels().b200_dq_convert_rope(_lib.ptr(acc), _lib.ptr(b), _lib.ptr(pos), _lib.ptr(cos), _lib.ptr(sin),
                                                   B * L, H, d, b.stride(0), _lib.stream()), "b200_dq_convert_rope")
    assert torch.equal(a[:, : H * d], b[:, : H * d])


@pytest.mark.parametrize("B,L,H,Hkv,d,window", [(2, 300, 4, 2, 64, 128), (1, 1000, 8, 8, 128, 256)])
def test_sequences_longer_than_a_sliding_window(B, L, H, Hkv, d, window):
    """Beyond the window the flash kernels step aside for the band-masked library path: forward and backward on the
    GPU (bf16) against the same path in fp32 on the CPU; inside the window the flash kernels still run."""
    torch.manual_seed(L + window)
    qkv = torch.randn(B * L, (H + 2 * Hkv) * d, device=DEV).bfloat16()
    dout = torch.randn(B * L, H * d, device=DEV).bfloat16()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d, window)
    dqkv = attention.attention_bwd(dout, qkv, out, lse, B, L, H, Hkv, d, window)
    assert out.dtype == torch.bfloat16 and dqkv.shape == qkv.shape
    ro, _ = attention.attention_fwd(qkv.float().cpu(), B, L, H, Hkv, d, window)
    rd = attention.attention_bwd(dout.float().cpu(), qkv.float().cpu(), ro, None, B, L, H, Hkv, d, window)
    assert torch.allclose(out.float().cpu(), ro, atol=3e-2, rtol=3e-2), (out.float().cpu() - ro).abs().max()
    err = (dqkv.float().cpu() - rd).abs().max().item()
    assert err <= 6e-2 * max(1.0, rd.abs().max().item()), err
    causal, _ = attention.attention_reference_fwd(qkv.float().cpu(), B, L, H, Hkv, d)
    assert (causal - ro).abs().max() > 0.1                    # the window matters at this length
    # a chunk against the key / value cache
    kv = Hkv * d
    kc = qkv[:, H * d:H * d + kv].reshape(B, L, kv).contiguous()
    vc = qkv[:, H * d + kv:].reshape(B, L, kv).contiguous()
    n, c0 = 128, L - 128 - (L - 128) % 8
    rows = torch.cat([qkv[b * L + c0: b * L + c0 + n] for b in range(B)])
    got = attention.attention_fwd_cached(rows.contiguous(), kc, vc, B, n, c0, H, Hkv, d, window)
    want = torch.cat([ro[b * L + c0: b * L + c0 + n] for b in range(B)])
    assert torch.allclose(got.float().cpu(), want, atol=3e-2, rtol=3e-2)
    # a window that covers the sequence: the flash kernels, bit for bit what they give without one
    a, _ = attention.attention_fwd(qkv, B, L, H, Hkv, d, L)
    b, _ = attention.attention_fwd(qkv, B, L, H, Hkv, d)
    assert torch.equal(a, b) and _lib.take_device_error() == 0


@pytest.mark.parametrize("L,H,Hkv,d,window", [(65, 2, 1, 64, 1), (129, 2, 2, 128, 64), (500, 4, 1, 64, 63), (641, 2, 1, 128, 129),
                                              (777, 2, 2, 64, 776), (1100, 4, 2, 128, 500)])
def test_window_edges_against_the_band_mask(L, H, Hkv, d, window):
    """Windows of one key, at and around the tile sizes, one short of the sequence: the flash kernels (whole sequence,
    chunk behind a cache, backward) against the masked path in fp32. Bound: probabilities and outputs are rounded to
    bf16 (2^-9 each), gradients are sums of up to ``window`` such terms - 2e-2 of the largest value."""
    B = 2
    torch.manual_seed(7 * L + window)
    qkv = torch.randn(B * L, (H + 2 * Hkv) * d, device=DEV).bfloat16()
    dout = torch.randn(B * L, H * d, device=DEV).bfloat16()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d, window)
    dqkv = attention.attention_bwd(dout, qkv, out, lse, B, L, H, Hkv, d, window)
    ro, _ = attention.windowed_fwd(qkv.float(), B, L, H, Hkv, d, window)
    rd = attention.windowed_bwd(dout.float(), qkv.float(), B, L, H, Hkv, d, window)
    for got, want in ((out, ro), (dqkv, rd)):
        assert (got.float() - want).abs().max() <= 2e-2 * want.abs().max()
    kv, n = Hkv * d, L // 3
    c0 = L - n
    kc, vc = (qkv[:, (H + i * Hkv) * d:(H + i * Hkv) * d + kv].reshape(B, L, kv).contiguous() for i in (0, 1))
    rows = qkv.view(B, L, -1)[:, c0:].reshape(B * n, -1).contiguous()
    got = attention.attention_fwd_cached(rows, kc, vc, B, n, c0, H, Hkv, d, window)
    want = ro.view(B, L, -1)[:, c0:].reshape(B * n, -1)
    assert (got.float() - want).abs().max() <= 2e-2 * want.abs().max()
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("form", ["fp32", "fp16", "strided", "offset"])
@pytest.mark.parametrize("d", [64, 128])
def test_windowed_calls_take_tensors_that_the_flash_kernels_do_not(form, d):
    """Types other than bf16 (in the masked path), column slices of wider rows and bases off 16 bytes (copied), forward,
    backward and behind a cache: against the same calls in fp32 on the CPU. Bound: 2^-9 per rounding to bf16 (2^-11 for fp16, and
    TF32 is off), gradients are sums of such terms - 2e-2 of the largest value."""
    B, L, H, Hkv, window = 2, 150, 4, 2, 40
    torch.manual_seed(d)
    width = (H + 2 * Hkv) * d
    dtype = {"fp32": torch.float32, "fp16": torch.float16}.get(form, torch.bfloat16)
    qkv = torch.randn(B * L, width + 8, device=DEV).to(dtype)
    dout = torch.randn(B * L, H * d, device=DEV).to(dtype)
    if form == "strided":
        qkv = qkv[:, 8:]
    elif form == "offset":
        qkv = torch.cat([qkv.new_zeros(1), qkv[:, 8:].reshape(-1)])[1:].view(B * L, width)
        assert qkv.is_contiguous() and qkv.data_ptr() % 16
    else:
        qkv = qkv[:, 8:].contiguous()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d, window)
    dqkv = attention.attention_bwd(dout, qkv, out, lse, B, L, H, Hkv, d, window)
    kv = Hkv * d
    kc, vc = (qkv[:, (H + i * Hkv) * d:(H + i * Hkv) * d + kv].reshape(B, L, kv) for i in (0, 1))
    n = 30
    rows = qkv.reshape(B, L, -1)[:, L - n:].reshape(B * n, -1)
    got_c = attention.attention_fwd_cached(rows, kc, vc, B, n, L - n, H, Hkv, d, window)
    ro, rl = attention.attention_fwd(qkv.float().cpu(), B, L, H, Hkv, d, window)
    rd = attention.attention_bwd(dout.float().cpu(), qkv.float().cpu(), ro, rl, B, L, H, Hkv, d, window)
    rc = ro.view(B, L, -1)[:, L - n:].reshape(B * n, -1)
    for got, want in ((out, ro), (dqkv, rd), (got_c, rc)):
        assert got.dtype == dtype and (got.float().cpu() - want).abs().max() <= 2e-2 * want.abs().max()
    with pytest.raises((TypeError, _lib.NativeError)):           # without a window such tensors stay refused
        attention.attention_fwd(qkv, B, L, H, Hkv, d)


def test_windowed_backward_takes_a_gradient_of_another_type():
    B, L, H, Hkv, d, window = 1, 150, 2, 1, 64, 40
    torch.manual_seed(0)
    qkv = torch.randn(B * L, (H + 2 * Hkv) * d, device=DEV).bfloat16()
    dout = torch.randn(B * L, H * d, device=DEV).bfloat16()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d, window)
    a = attention.attention_bwd(dout.float(), qkv, out, lse, B, L, H, Hkv, d, window)
    b = attention.attention_bwd(dout, qkv, out, lse, B, L, H, Hkv, d, window)
    # query gradients of two key blocks meet by atomic adds of two terms onto zero: any order gives the same bits
    assert torch.equal(a, b) and _lib.take_device_error() == 0


@pytest.mark.parametrize("window", [300, 2 ** 31 - 1, 2 ** 31, 2 ** 32 + 7])
def test_windows_at_and_beyond_the_sequence_are_causal(window):
    """Through the kernels' own wrappers and, where it fits 32 bits, the C entries: the bits of the call without a window."""
    from llm_distillery_b200.ops import flash
    B, L, H, Hkv, d = 1, 300, 2, 1, 64
    torch.manual_seed(3)
    qkv = torch.randn(B * L, (H + 2 * Hkv) * d, device=DEV).bfloat16()
    dout = torch.randn(B * L, H * d, device=DEV).bfloat16()
    out, lse = flash.flash_attn_fwd(qkv, B, L, H, Hkv, d)
    a, al = flash.flash_attn_fwd(qkv, B, L, H, Hkv, d, window)
    assert torch.equal(a, out) and torch.equal(al, lse)
    want = flash.flash_attn_bwd(dout, qkv, out, lse, B, L, H, Hkv, d)

    def near(got):      # query gradients of three key blocks meet by atomic adds in no fixed order: a last bit of bf16
        assert torch.equal(got[:, H * d:], want[:, H * d:])
        assert (got.float() - want.float()).abs().max() <= 2 ** -7 * want.float().abs().max()
    near(flash.flash_attn_bwd(dout, qkv, out, lse, B, L, H, Hkv, d, window=window))
    kc, vc = (qkv[:, (H + i) * d:(H + 1 + i) * d].reshape(B, L, d).contiguous() for i in (0, 1))
    rows = qkv[200:].contiguous()
    assert torch.equal(flash.flash_attn_fwd_cached(rows, kc, vc, B, 100, 200, H, Hkv, d, window),
                       flash.flash_attn_fwd_cached(rows, kc, vc, B, 100, 200, H, Hkv, d))
    if window < 2 ** 31:
        lib, p = _lib.kernels(), _lib.ptr
        o2, l2, dq = torch.empty_like(out), torch.empty_like(lse), torch.empty_like(qkv)
        _lib.check(lib.b200_flash_attn_fwd(p(qkv), p(o2), p(l2), B, L, window, H, Hkv, d, _lib.stream()), "fwd")
        delta, acc = torch.empty_like(lse), torch.empty((B * L, H * d), dtype=torch.float32, device=DEV)
        _lib.check(lib.b200_flash_attn_bwd(p(dout), p(qkv), p(o2), p(l2), p(delta), p(dq), p(acc), B, L, window, H, Hkv, d,
                                           _lib.stream()), "bwd")
        assert torch.equal(o2, out)
        near(dq)
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("d", [64, 128])
@pytest.mark.parametrize("window", [None, 1, 40, 130])
def test_scores_of_any_size(d, window):
    """Scores far below zero, a head whose scores all overflow to -inf, and NaN in one key. The values of position p are
    p, so the output of a row is the mean position over its largest scores: the others are 2^13 / sqrt(d) lower, their
    probability is exactly 0. Bound: two roundings to bf16, 2^-8."""
    B, L, H = 1, 333, 2
    ks = -(2.0 ** 8) * (1 + (torch.arange(L) * 5 % 7) / 8)              # exact in bf16
    qkv = torch.empty(B * L, 3, H, d)
    qkv[:, 0, 0], qkv[:, 0, 1] = 4.0, 2.0 ** 100                          # scores of -2^10 d and less, and -inf
    qkv[:, 1, 0], qkv[:, 1, 1] = ks.view(L, 1), ks.view(L, 1) * 2.0 ** 40
    qkv[:, 2] = torch.arange(L).float().view(L, 1, 1)
    qkv = qkv.reshape(B * L, -1).bfloat16().to(DEV)
    out, _ = attention.attention_fwd(qkv, B, L, H, H, d, window)
    out = out.float().cpu().view(L, H, d)
    see = torch.tril(torch.ones(L, L, dtype=torch.bool))
    if window is not None:
        see &= ~torch.tril(see, -window)
    s = ks.double().view(1, L).expand(L, L).masked_fill(~see, -float("inf"))
    top = (s == s.amax(1, keepdim=True)).double()
    want = (top @ torch.arange(L).bfloat16().double()) / top.sum(1)
    assert ((out[:, 0].double() - want.view(L, 1)).abs() <= 2 ** -8 * want.view(L, 1)).all()
    assert out[:, 1].isnan().all()                                       # the softmax over nothing but -inf
    nan_at = 100
    qkv = torch.randn(B * L, 3 * H * d, device=DEV).bfloat16()
    qkv[nan_at, H * d:2 * H * d] = float("nan")
    out, _ = attention.attention_fwd(qkv, B, L, H, H, d, window)
    bad = out.isnan().any(1).cpu()
    assert torch.equal(bad, see[:, nan_at])                              # the rows that see the key, and no other
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("B,L,H,Hkv,d,window", [(1, 1, 8, 1, 64, None), (1, 127, 7, 1, 64, None), (1, 777, 14, 2, 64, None),
                                                (2, 129, 16, 2, 64, 100), (1, 300, 5, 1, 128, None), (1, 257, 16, 2, 128, 200),
                                                (1, 128, 24, 2, 64, None), (8, 1025, 16, 2, 64, None)])
def test_query_heads_shared_by_a_cluster(B, L, H, Hkv, d, window):
    """Groups of 5 to 12 query heads on grids that leave SMs idle: the heads of a group are shared by the CTAs of a cluster (also
    a share that is not even, and more heads than a cluster has CTAs; the last case keeps one CTA per key block). Bound: as at the window edges, 2e-2 of the largest
    gradient; key and value gradients repeat bit for bit."""
    torch.manual_seed(L + H)
    qkv = torch.randn(B * L, (H + 2 * Hkv) * d, device=DEV).bfloat16()
    dout = torch.randn(B * L, H * d, device=DEV).bfloat16()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d, window)
    from llm_distillery_b200.ops import flash
    got = flash.flash_attn_bwd(dout, qkv, out, lse, B, L, H, Hkv, d, window=window, share_heads=True)
    again = flash.flash_attn_bwd(dout, qkv, out, lse, B, L, H, Hkv, d, window=window, share_heads=True)
    if window is None:
        ro, rl = attention.attention_reference_fwd(qkv.float(), B, L, H, Hkv, d)
        want = attention.attention_reference_bwd(dout.float(), qkv.float(), ro, rl, B, L, H, Hkv, d)
    else:
        want = attention.windowed_bwd(dout.float(), qkv.float(), B, L, H, Hkv, d, window)
    for cols in (slice(0, H * d), slice(H * d, (H + Hkv) * d), slice((H + Hkv) * d, None)):
        assert (got[:, cols].float() - want[:, cols]).abs().max() <= 2e-2 * want[:, cols].abs().max() + 1e-6
    assert torch.equal(got[:, H * d:], again[:, H * d:]) and _lib.take_device_error() == 0


@pytest.mark.parametrize("B,n,c0,rows,H,Hkv,d", [(1, 1, 0, 1, 2, 1, 64), (2, 100, 0, 777, 4, 2, 64), (3, 256, 512, 1000, 2, 2, 128),
                                                 (2, 37, 100, 137, 3, 1, 64), (1, 65, 63, 4096, 8, 8, 128)])
def test_cache_append_is_the_slice_assignment(B, n, c0, rows, H, Hkv, d):
    """One launch for the keys and values of a chunk: the bits of the two slice assignments, zeros behind them up to a
    multiple of 128 rows (or the cache's end), nothing else touched."""
    torch.manual_seed(n)
    qkv = torch.randn(B * n, (H + 2 * Hkv) * d, device=DEV).bfloat16()
    caches = [torch.full((B, rows, Hkv * d), float("nan"), device=DEV, dtype=torch.bfloat16) for _ in range(4)]
    attention.cache_append(qkv, caches[0], caches[1], B, n, c0, H, Hkv, d)
    wide = torch.zeros(B * n, (H + 2 * Hkv) * d + 1, device=DEV, dtype=torch.bfloat16)
    wide[:, 1:] = qkv
    attention.cache_append(wide[:, 1:], caches[2], caches[3], B, n, c0, H, Hkv, d)        # strided rows: slice by slice
    for i, first in ((0, H * d), (1, (H + Hkv) * d)):
        want = torch.full_like(caches[i], float("nan"))
        want[:, c0:c0 + n] = qkv[:, first:first + Hkv * d].reshape(B, n, -1)
        want[:, c0 + n:(c0 + n + 127) // 128 * 128] = 0
        for got in (caches[i], caches[i + 2]):
            assert torch.equal(got.view(torch.int16), want.view(torch.int16))


@pytest.mark.parametrize("B,L,H,Hkv,d", [(1, 777, 14, 2, 64), (2, 129, 8, 8, 64), (1, 1, 2, 1, 64), (1, 300, 12, 2, 128), (4, 1100, 32, 8, 128)])
def test_key_gradients_are_rotated_back_where_they_are_written(B, L, H, Hkv, d):
    """Key and value gradients of the backward pass that undoes the rotary embedding, written by one CTA or summed over a
    cluster: the bits of the plain backward pass followed by the rope kernel (positions in any order)."""
    from llm_distillery_b200.ops import basic
    torch.manual_seed(L)
    qkv = torch.randn(B * L, (H + 2 * Hkv) * d, device=DEV).bfloat16()
    out, lse = attention.attention_fwd(qkv, B, L, H, Hkv, d)
    dout = torch.randn_like(out)
    pos = torch.randint(0, 2000, (B * L,), device=DEV, dtype=torch.int32)
    cos, sin = basic.rope_tables(2000, d, 10000.0, DEV)
    from llm_distillery_b200.ops import flash
    for share in (False, True):
        got = attention.attention_bwd_unrotated(dout, qkv, out, lse, B, L, H, Hkv, d, pos, cos, sin, share_heads=share)
        want = flash.flash_attn_bwd(dout, qkv, out, lse, B, L, H, Hkv, d, share_heads=share)
        basic.rope_(want, pos, cos, sin, H + Hkv, d, inverse=True)
        assert torch.equal(got[:, H * d:], want[:, H * d:]) and _lib.take_device_error() == 0
