"""Fused LM head + distillation loss kernels against the full-logits PyTorch computation."""
import pytest
import torch

from llm_distillery_b200.loss import head, divergence as dv
from llm_distillery_b200.models.llama import GradSlot
from llm_distillery_b200.ops import _lib

pytestmark = pytest.mark.gpu
DEV = "cuda"


def _setup(M, h, V, K, seed=0):
    torch.manual_seed(seed)
    Hc = torch.randn(M, h, device=DEV).bfloat16()
    W = (torch.randn(V, h, device=DEV) * 0.05).bfloat16()
    tl = torch.randn(M, V, device=DEV) * 3
    u, ids = torch.log_softmax(tl, -1).topk(K, -1)
    ids32, us = head.sort_teacher_rows(ids, u.half().float())
    return Hc, W, ids32, us


@pytest.mark.parametrize("M,h,V,K,Vc,T", [(128, 64, 256, 8, 256, 1.0), (300, 256, 1000, 50, 1000, 2.0),
                                           (517, 512, 5000, 200, 4800, 1.0), (2048, 2048, 32000, 200, 32000, 2.0)])
def test_stats_forward(M, h, V, K, Vc, T):
    Hc, W, ids, u = _setup(M, h, V, K)
    lse, zk = head.lmhead_stats(Hc, W, ids, T, Vc)
    assert _lib.take_device_error() == 0
    rl, rz = head._torch_stats(Hc, W, ids, 1.0 / T, Vc)
    assert torch.allclose(lse, rl, atol=2e-3, rtol=1e-4), (lse - rl).abs().max()
    assert torch.allclose(zk, rz, atol=2e-3, rtol=1e-3), (zk - rz).abs().max()


@pytest.mark.parametrize("kind", ["kl", "rkl", "jsd", "jsd_renorm"])
@pytest.mark.parametrize("M,h,V,K,Vc,T", [(300, 256, 1000, 50, 1000, 2.0), (517, 512, 5000, 200, 4800, 1.0)])
def test_fused_loss_and_gradients(kind, M, h, V, K, Vc, T):
    Hc, W, ids, u = _setup(M, h, V, K, seed=1)
    Hr = Hc.float().requires_grad_()
    Wr = W.float().requires_grad_()
    lse, zk = head._torch_stats(Hr, Wr, ids, 1.0 / T, Vc)
    s, t = dv.student_teacher_logprobs(lse, zk, u, ids.long() < Vc, T)
    ref_rows = dv.loss_rows("jsd", s, t, jsd_renorm=True) if kind == "jsd_renorm" else dv.loss_rows(kind, s, t)
    w = torch.rand(M, device=DEV) / M
    (ref_rows * w).sum().backward()

    Hg = Hc.clone().requires_grad_()
    Wg = W.clone().requires_grad_()
    Wg.grad_slot = GradSlot(torch.zeros(V, h, device=DEV))
    rows = head.fused_distill_rows(Hg, Wg, ids, u, "jsd" if kind == "jsd_renorm" else kind, T, Vc,
                                   jsd_renorm=(kind == "jsd_renorm"))
    (rows * w).sum().backward()
    assert _lib.take_device_error() == 0
    assert torch.allclose(rows, ref_rows.detach(), atol=3e-3, rtol=3e-3), (rows - ref_rows).abs().max()
    gH, gW = Hg.grad.float(), Wg.grad_slot.buf
    assert (gH - Hr.grad).abs().max() <= 2e-2 * Hr.grad.abs().max() + 1e-6
    assert (gW - Wr.grad).abs().max() <= 2e-2 * Wr.grad.abs().max() + 1e-6
    assert gW[Vc:].abs().max() == 0 if Vc < V else True


@pytest.mark.parametrize("lens", [[1], [31, 1], [257, 3], [40, 300, 256, 1], [3] * 70])
@pytest.mark.parametrize("kind", ["kl", "rkl", "jsd", "jsd_renorm"])
def test_mean_loss_of_conversations(kind, lens):
    """The loss of a batch as one node against its rows averaged in fp64, and its gradients against those of the rows with the
    weights that the averages give them (bound: one fp32 sum of up to 300 terms, the weights rounded once)."""
    M, h, V, K, T = sum(lens), 256, 2000, 40, 2.0
    Hc, W, ids, u = _setup(M, h, V, K, seed=len(lens))
    seg = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens)).to(DEV)
    grads = []
    for whole in (True, False):
        Hg, Wg = Hc.clone().requires_grad_(), W.clone().requires_grad_()
        if whole:
            loss, logs = head.distill_head_loss(Hg, Wg, ids, u, kind=kind.removesuffix("_renorm"), temperature=T, vocab=V, seg=seg,
                                                n_seg=len(lens), jsd_renorm=kind == "jsd_renorm")
            assert all(torch.equal(v, loss) and not v.requires_grad for v in logs.values()) and "custom loss" in logs
            (loss * 0.5).backward()
        else:
            rows = head.fused_distill_rows(Hg, Wg, ids, u, kind.removesuffix("_renorm"), T, V, jsd_renorm=kind == "jsd_renorm")
            weight = (1.0 / torch.tensor(lens, dtype=torch.float64, device=DEV))[seg]
            want = (rows.detach().double() * weight).sum()
            assert abs(loss.item() - want.item()) <= 300 * 2 ** -23 * (rows.detach().double().abs() * weight).sum().item()
            (rows * (0.5 * weight).float()).sum().backward()
        grads.append((Hg.grad.float(), Wg.grad.float()))
    for a, b in zip(*grads):
        assert (a - b).abs().max() <= 2 ** -7 * b.abs().max()
    assert _lib.take_device_error() == 0


def test_reference_loss_through_fused_stats():
    M, h, V, K, Vc, T = 400, 256, 2000, 64, 2000, 1.0
    Hc, W, ids, u = _setup(M, h, V, K, seed=2)
    seg = torch.cat([torch.zeros(250, dtype=torch.long), torch.ones(150, dtype=torch.long)]).to(DEV)
    labels = torch.randint(0, V, (M,), device=DEV)
    labels[::2] = ids[::2, 5].long()
    labels[249] = -1
    labels[399] = -1
    avoid = torch.zeros(M, dtype=torch.bool, device=DEV)
    avoid[100] = True
    kw = dict(kind="reference", temperature=T, vocab=Vc, alpha=2.0, labels=labels, avoid=avoid, seg=seg, n_seg=2)
    Hr, Wr = Hc.float().cpu().requires_grad_(), W.float().cpu().requires_grad_()
    ref, _ = head.distill_head_loss(Hr, Wr, ids.cpu(), u.cpu(), **{**kw, "labels": labels.cpu(), "avoid": avoid.cpu(),
                                                                   "seg": seg.cpu()})
    ref.backward()
    Hg, Wg = Hc.clone().requires_grad_(), W.clone().requires_grad_()
    got, logs = head.distill_head_loss(Hg, Wg, ids, u, **kw)
    got.backward()
    assert _lib.take_device_error() == 0
    assert abs(got.item() - ref.item()) <= 2e-2 * abs(ref.item()) + 1e-3
    assert (Hg.grad.float().cpu() - Hr.grad).abs().max() <= 5e-2 * Hr.grad.abs().max()
    assert (Wg.grad.float().cpu() - Wr.grad).abs().max() <= 5e-2 * Wr.grad.abs().max()
    assert set(dv.LOSS_KEYS) <= set(logs)


@pytest.mark.parametrize("M,K,Vc,T,lens", [(1, 2, 5000, 1.0, [1]), (7, 3, 5000, 1.0, [2, 5]), (65, 33, 900, 2.0, [64, 1]),
                                           (700, 200, 4800, 1.0, [700]), (1601, 400, 5000, 2.0, [1, 511, 513, 576])])
def test_reference_loss_kernels_against_fp64(monkeypatch, M, K, Vc, T, lens):
    """Loss, logged values and both gradients against the PyTorch form in fp64, with rows without a target, without a label, left
    out of the cross-entropy and without a hit, and ids beyond the cropped vocabulary. Bound: sums of up to 400 fp32 terms, their
    differences and a division by the largest of them: 2e-5 of the largest value (single values differ by 1e-6 of it)."""
    g = torch.Generator().manual_seed(M)
    V = 5000
    z = torch.randn(M, V, generator=g) * 3
    ids = torch.rand(M, V, generator=g).topk(K, -1).indices.sort(-1).values
    u = (torch.randn(M, K, generator=g) * 3).log_softmax(-1)
    zk, lse = z.gather(1, ids) / T, torch.logsumexp(z[:, :Vc] / T, -1)
    labels = ids.gather(1, torch.randint(0, K, (M, 1), generator=g))[:, 0]
    labels[torch.rand(M, generator=g) < 0.4] = 3                              # mostly outside the row's ids
    labels[labels >= Vc] = 3
    seg = torch.repeat_interleave(torch.arange(len(lens)), torch.tensor(lens))
    last = torch.tensor(lens).cumsum(0) - 1
    if M > 1:
        labels[last] = -1
    avoid = torch.rand(M, generator=g) < 0.1
    if M > 10:
        u[5], u[9, 1:] = float("-inf"), float("-inf")
        labels[5] = labels[9] = -1
    grads, outs = [], []
    assert not head._native_reference_loss(zk.to(DEV), u.to(DEV), *(x.to(DEV) for x in (ids, labels, avoid, seg)))      # few rows
    monkeypatch.setattr(head, "NATIVE_REFERENCE_ROWS", 1)
    for dev, dt in ((DEV, torch.float32), ("cpu", torch.float64)):
        a, b = (x.to(dev, dt).clone().requires_grad_() for x in (lse, zk))
        args = [x.to(dev) for x in (ids.int(), labels, avoid, seg)]
        if dev == DEV:
            assert head._native_reference_loss(b, u.to(dev), *args)
            custom, logs = head._ReferenceLossFn.apply(a, b, u.to(dev), *args, len(lens), T, Vc, 2.0)
            logs = dict(zip(dv.LOSS_KEYS, logs))
        else:
            s, t = dv.student_teacher_logprobs(a, b, u.to(dt), args[0] < Vc, T)
            custom, logs = dv.reference_loss_segments(s, t, args[0].long(), *args[1:], len(lens), 2.0)
        (custom * torch.arange(1, len(lens) + 1, device=dev)).sum().backward()
        grads.append([x.grad.double().cpu() for x in (a, b)])
        outs.append({k: v.detach().double().cpu() for k, v in logs.items()})
        assert torch.equal(logs["custom loss"].isnan(), custom.isnan())
    for k in dv.LOSS_KEYS:
        x, y = outs[0][k], outs[1][k]
        assert torch.equal(x.isnan(), y.isnan()), k                           # no labelled row: 0 / 0 in both
        assert ((x - y).abs().nan_to_num(0) <= 2e-5 * y.nan_to_num(0).abs().max() + 2e-6).all(), k
    for x, y in zip(*grads):
        assert torch.equal(x.isnan(), y.isnan())
        assert (x - y).nan_to_num(0).abs().max() <= 2e-5 * y.nan_to_num(0).abs().max() + 1e-9
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("M,K", [(1, 2), (40, 33), (300, 200)])
def test_reference_loss_gradient_of_far_log_probs(M, K):
    """Values around -1000 (a temperature of 1/128) that fp32 holds exactly: the probabilities must not carry the last bit of a
    maximum of that size (3e-5). Exact differences, exponentials and sums of up to 200 terms: 200 * 2^-24, 1.2e-5, at the very
    worst; 5e-6 of the largest value stands for sums whose roundings do not all go one way."""
    g = torch.Generator().manual_seed(M)
    T, seg = 1 / 128, torch.zeros(M, dtype=torch.int64)
    ids = torch.rand(M, 500, generator=g).topk(K, -1).indices.sort(-1).values
    u = -8 - torch.randint(0, 9 * 2 ** 10, (M, K), generator=g) / 2 ** 17                      # u / T: -1024 .. -1033 in steps of 2^-10
    lse = 1000 + torch.randint(0, 2 ** 10, (M,), generator=g) / 2 ** 10
    zk = -torch.randint(0, 9 * 2 ** 10, (M, K), generator=g) / 2 ** 10                         # zk - lse: -1000 .. -1010
    labels, avoid = ids[:, 0].clone(), torch.zeros(M, dtype=torch.bool)
    grads = []
    for dev, dt in ((DEV, torch.float32), ("cpu", torch.float64)):
        a, b, t = lse.to(dev, dt).requires_grad_(), zk.to(dev, dt).requires_grad_(), u.to(dev, dt)
        args = [x.to(dev) for x in (ids.int(), labels, avoid, seg)]
        if dev == DEV:
            custom, _ = head._ReferenceLossFn.apply(a, b, t, *args, 1, T, 500, 2.0)
        else:
            custom, _ = dv.reference_loss_segments(*dv.student_teacher_logprobs(a, b, t, args[0] < 500, T), args[0].long(),
                                                   *args[1:], 1, 2.0)
        custom.sum().backward()
        grads.append([x.grad.double().cpu() for x in (a, b)])
    for x, y in zip(*grads):
        assert (x - y).abs().max() <= 5e-6 * y.abs().max()
    assert _lib.take_device_error() == 0


@pytest.mark.parametrize("M,N,h,K", [(2500, 2000, 256, 9), (2401, 1800, 264, 33), (257, 9610, 320, 64), (5000, 1284, 256, 1)])
@pytest.mark.parametrize("ld", [0, 3])
def test_dlogits_of_ragged_pair_tiles(M, N, h, K, ld):
    """256 x 256 tiles whose last columns end in either half, ids on the halves' edges and behind the vocabulary, rows of the
    result on and off 16-byte boundaries. Bound: the result's rounding to bf16 (2^-8), and of the exponential the error of its
    argument: products of bf16 summed in fp32 (below 1e-5 sqrt(h)) and three roundings of numbers up to 40."""
    g = torch.Generator("cuda").manual_seed(M)
    x, w = (torch.randn(n, h, device=DEV, generator=g).bfloat16() * s for n, s in ((M, 1.0), (N, 0.1)))
    ids = torch.stack([torch.randperm(N, device=DEV, generator=g)[:K] for _ in range(M)]).int()
    edges = torch.tensor([0, 127, 128, 255, 256, 383, 384, N - 1], device=DEV, dtype=torch.int32)[:K]
    ids[::2, :len(edges)] = edges
    ids[1::3, -1] = N + 2
    ids = ids.sort(1).values
    ok = (ids[:, 1:] != ids[:, :-1]).all(1) if K > 1 else torch.ones(M, dtype=torch.bool, device=DEV)     # rows without a repeated id
    a = torch.randn(M, K, device=DEV, generator=g)
    A, gr = torch.randn(M, device=DEV, generator=g), torch.rand(M, device=DEV, generator=g)
    z = (x.double() @ w.double().t()) * 0.5
    lse = z.logsumexp(1)
    p = torch.exp(z - lse[:, None])
    ref = torch.zeros(M, N + 8, device=DEV, dtype=torch.float64).scatter_add_(1, ids.long(), a.double())[:, :N] - A.double()[:, None] * p
    scale = gr.double()[:, None] * 0.5
    width = (N + 7) // 8 * 8 + 8 + ld
    buf = torch.full((M + 1, width), 7.0, device=DEV, dtype=torch.bfloat16)
    lse32 = lse.float()
    rc = _lib.kernels().b200_lmhead_dlogits(_lib.ptr(x), _lib.ptr(w), M, N, h, h, h, _lib.ptr(ids), _lib.ptr(a), _lib.ptr(A),
                                            _lib.ptr(lse32), _lib.ptr(gr), K, 0.5, _lib.ptr(buf), width, _lib.stream())
    err = (buf[:M, :N].double() - ref * scale).abs()
    bound = 2.0 ** -8 * (ref * scale).abs() + scale * (A.double().abs()[:, None] * p * (1e-5 * h ** 0.5 + 1e-4) + 1e-6)
    assert rc == 0 and (err <= bound)[ok].all() and ok.float().mean() > 0.3
    assert (buf[:M, N:] == 7).all() and (buf[M:] == 7).all() and _lib.take_device_error() == 0
