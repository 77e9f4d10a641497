"""Expert sort and weighted combination against their PyTorch restatements."""
import pytest
import torch

from llm_distillery_b200.models import moe
from llm_distillery_b200.ops import _lib

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("T,k,E", [(1, 1, 1), (1, 2, 8), (511, 2, 8), (6124, 2, 8), (1025, 8, 32), (3000, 4, 33)])
def test_expert_sort_is_the_stable_sort(T, k, E):
    g = torch.Generator("cuda").manual_seed(T)
    top_e = (torch.rand(T, k, device="cuda", generator=g) ** 2 * E).long().clamp_(max=E - 1)     # uneven, some empty
    order, inverse, token, counts = moe.sorted_pairs(top_e, E)
    flat = top_e.reshape(-1)
    want = torch.argsort(flat, stable=True)
    assert torch.equal(order, want) and torch.equal(token, want // k)
    assert torch.equal(order[inverse], torch.arange(T * k, device="cuda"))
    assert torch.equal(counts, torch.bincount(flat, minlength=E))


@pytest.mark.parametrize("T,k,dtype,native", [(16384, 2, torch.int64, True), (32768, 2, torch.int64, True),
                                              (32769, 2, torch.int64, False), (4096, 8, torch.int64, True),
                                              (16384, 8, torch.int64, False),
                                              (100, 2, torch.int32, False), (100, 2, torch.uint8, False)])
def test_which_sort_takes_the_pairs(monkeypatch, T, k, dtype, native):
    """Many pairs are left to the library, whose sort is ahead there, and so are indices that the kernel would misread."""
    top_e = torch.randint(0, 32, (T, k), device="cuda", generator=torch.Generator("cuda").manual_seed(T + k)).to(dtype)
    calls, real = [], _lib.kernels()

    class Recorder:
        def __getattr__(self, name):
            calls.append(name)
            return getattr(real, name)
    monkeypatch.setattr(_lib, "kernels", Recorder)
    order, inverse, token, counts = moe.sorted_pairs(top_e, 32)
    assert ("b200_expert_sort" in calls) == native
    flat = top_e.reshape(-1)
    want = torch.argsort(flat, stable=True)
    assert torch.equal(order, want) and torch.equal(token, want // k) and torch.equal(counts, torch.bincount(flat.long(), minlength=32))
    assert torch.equal(order[inverse], torch.arange(T * k, device="cuda"))


@pytest.mark.parametrize("T,h,E,k", [(1, 8, 1, 1), (3, 264, 8, 2), (4, 256, 7, 7), (1531, 2048, 8, 2), (5, 520, 9, 4), (33, 2048, 16, 4),
                                     (2, 8, 15, 8), (257, 1024, 16, 16)])
@pytest.mark.parametrize("renorm", [True, False])
def test_route_is_the_softmax_of_the_rounded_logits(T, h, E, k, renorm):
    """Probabilities against fp64 within one rounding of the logits to bf16 either way (2^-8 of each), choices and weights against
    the probabilities: the k largest, of equal ones (experts 0 and 1 have the same weights) the lower first."""
    g = torch.Generator("cuda").manual_seed(T + E)
    x = torch.randn(T, h, device="cuda", generator=g).bfloat16()
    w = (torch.randn(E, h, device="cuda", generator=g) * 3 / h ** 0.5).bfloat16()
    if E > 1:
        w[1] = w[0]
    probs, top_e, top_w = moe.route(x, w, k, renorm)
    logits = x.double() @ w.double().t()
    want = logits.softmax(-1)
    assert ((probs.double() / want).log().abs() <= 2 ** -8 * 2 * logits.abs().amax(-1, keepdim=True) + 1e-5).all()
    assert torch.equal(top_e, probs.sort(dim=-1, descending=True, stable=True).indices[:, :k])
    top_p = probs.gather(1, top_e)
    assert torch.allclose(top_w, top_p / top_p.sum(-1, keepdim=True) if renorm else top_p, rtol=1e-6, atol=0)
    # a caller that differentiates through it keeps the library's operators
    xr = x.clone().requires_grad_()
    assert moe.route(xr, w, k, renorm)[2].requires_grad
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("T,k,h,resid,rmul", [(1, 1, 8, True, 1.0), (257, 2, 2048, True, 1.0), (33, 8, 264, False, 1.0),
                                              (100, 4, 512, True, 0.25)])
def test_combine_matches_the_gathered_sum(T, k, h, resid, rmul):
    g = torch.Generator("cuda").manual_seed(T + h)
    y = torch.randn(T * k, h, device="cuda", generator=g).bfloat16()
    inverse = torch.randperm(T * k, device="cuda", generator=g)
    w = torch.rand(T, k, device="cuda", generator=g)
    h1 = torch.randn(T, h, device="cuda", generator=g).bfloat16() if resid else None
    got = moe.combine(y, inverse, w, h1, rmul)
    want = (y[inverse].view(T, k, h).double() * w.double().unsqueeze(-1)).sum(1) * rmul
    if resid:
        want = want + h1.double()
    # fp32 sums of at most 9 terms, then one rounding to bf16 (2^-9 of the value)
    assert ((got.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-5).all()
    assert _lib.take_device_error() == 0


def test_combine_passes_on_what_is_not_finite():
    """NaN, infinities and the product of zero and infinity as the gathered sum has them."""
    T, k, h = 64, 2, 40
    torch.manual_seed(0)
    y = torch.randn(T * k, h, device="cuda").bfloat16()
    y[3, 0], y[8, 1], y[8, 2], y[20, 3], y[21, 3] = (float(v) for v in ("nan", "inf", "-inf", "inf", "-inf"))
    w = torch.rand(T, k, device="cuda")
    w[4, 0] = 0.0                                      # times the infinities of row 8
    w[30, 1] = float("nan")
    inverse = torch.arange(T * k, device="cuda")
    for h1 in (None, torch.randn(T, h, device="cuda").bfloat16()):
        got = moe.combine(y, inverse, w, h1)
        want = (y.view(T, k, h).float() * w.unsqueeze(-1)).sum(1) + (0 if h1 is None else h1.float())
        assert torch.equal(got.isnan(), want.isnan()) and torch.equal(got.isinf(), want.isinf())
        ok = want.isfinite()
        assert ((got.float() - want).abs() <= 2 ** -8 * want.abs() + 1e-5)[ok].all() and not ok.all()
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("counts,h,f", [([1], 64, 128), ([0, 257, 0, 1, 255, 256], 128, 384), ([0] * 127 + [3], 64, 128),
                                        ([5, 0, 130, 77, 1024, 512, 33, 0], 2048, 640), ([2000, 1], 264, 128), ([0, 7] * 64, 96, 256)])
def test_experts_in_one_launch_match_a_launch_each(counts, h, f):
    """Empty experts, one row, whole tiles and one row more, 128 experts, widths that are not whole tiles: the bits of the
    launches per expert (one K slice each, the same order of additions)."""
    g = torch.Generator("cuda").manual_seed(sum(counts) + h)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    x, w_gu, w_d = rnd(sum(counts), h), rnd(len(counts), 2 * f, h) * 0.1, rnd(len(counts), h, f) * 0.1
    dev = torch.tensor(counts, device="cuda")
    assert moe._grouped(x, dev, w_gu, w_d)
    for got, want in zip(moe.experts_forward(x, dev, w_gu, w_d), moe._experts_one_by_one(x, counts, w_gu, w_d)):
        assert torch.equal(got, want)
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("case", ["width", "strided", "many", "empty", "fp16", "offset"])
def test_experts_that_one_launch_does_not_take(case):
    """Operands outside the grouped launch go expert by expert: each stage against the fp64 product of what it read (one rounding
    to 16 bits, fp32 sums of at most 192 terms), rows off the 16-byte boundaries that a GEMM loads from are refused."""
    E, h, f = (129 if case == "many" else 4), 64, (192 if case == "width" else 128)
    g = torch.Generator("cuda").manual_seed(E + f)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g).bfloat16()  # noqa: E731
    w_gu, w_d = rnd(E, 2 * f, h) * 0.1, rnd(E, h, f) * 0.1
    counts = [0] * E if case == "empty" else [3, 0, 40, 7] + [0] * (E - 5) + [2] * (E > 4)
    x = rnd(sum(counts), h + 8)
    if case == "offset":
        x = torch.cat([x.new_zeros(4), x[:, 8:].reshape(-1)])[4:].view(-1, h)
    else:
        x = x[:, 8:] if case == "strided" else x[:, 8:].contiguous()
    if case == "fp16":
        x, w_gu, w_d = x.half(), w_gu.half(), w_d.half()
    dev = torch.tensor(counts, device="cuda")
    assert not moe._grouped(x, dev, w_gu, w_d)
    if case == "offset":
        with pytest.raises(_lib.NativeError):
            moe.experts_forward(x, dev, w_gu, w_d)
        return
    gu, act, y = moe.experts_forward(x, dev, w_gu, w_d)
    assert gu.shape == (sum(counts), 2 * f) and act.shape == (sum(counts), f) and y.shape == x.shape
    runs = torch.repeat_interleave(torch.arange(E, device="cuda"), dev)

    def close(got, a, b):
        a, b = a.double(), b.double()
        err = (got.double() - torch.einsum("nk,nmk->nm", a, b)).abs()
        bound = torch.einsum("nk,nmk->nm", a.abs(), b.abs())
        assert (err <= 2 ** -8 * got.double().abs() + 192 * 2 ** -24 * bound).all()
    close(gu, x, w_gu[runs])
    if case != "fp16":                       # the activation's kernel and with it the layer are bf16
        gate, up = gu.double().split(f, 1)
        want = gate * torch.sigmoid(gate) * up
        assert ((act.double() - want).abs() <= 2 ** -8 * want.abs() + 1e-6).all()
        close(y, act, w_d[runs])
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("n,E", [(1, 1), (1023, 3), (1025, 32), (40001, 5), (65535, 1), (65536, 32)])
def test_expert_sort_of_any_number_of_pairs(n, E):
    """The kernel itself up to the number of pairs that it takes, with indices out of range left out; one more is refused."""
    e = torch.randint(-1, E + 1, (n,), device="cuda", generator=torch.Generator("cuda").manual_seed(n))
    order, inverse, token = (torch.full((n,), -7, dtype=torch.int64, device="cuda") for _ in range(3))
    counts = torch.empty(E, dtype=torch.int64, device="cuda")
    p = _lib.ptr
    _lib.check(_lib.kernels().b200_expert_sort(p(e), n, E, 3, p(order), p(inverse), p(token), p(counts), _lib.stream()), "sort")
    ok = ((e >= 0) & (e < E)).nonzero()[:, 0]
    want = ok[torch.argsort(e[ok], stable=True)]
    m = want.numel()
    assert torch.equal(order[:m], want) and torch.equal(token[:m], want // 3) and (order[m:] == -7).all()
    assert torch.equal(inverse[want], torch.arange(m, device="cuda"))
    assert torch.equal(counts, torch.bincount(e[ok], minlength=E))
    rc = _lib.kernels().b200_expert_sort(p(e), 65537, E, 3, p(order), p(inverse), p(token), p(counts), _lib.stream())
    assert rc < 0 and _lib.take_device_error() == 0
