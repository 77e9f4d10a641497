"""Exact top-K log-prob extraction, full log-prob rows, multi-teacher merge, collector, optimizer kernels on GPU."""
import numpy as np
import pytest
import torch

from llm_distillery_b200.collect.collector import TeacherCollector
from llm_distillery_b200.data.convo import ConvoTokenized
from llm_distillery_b200.engine.optim import FlatOptimizer, FlatParams
from llm_distillery_b200.models.llama import LlamaConfig, build_model
from llm_distillery_b200.ops import _lib, topk

pytestmark = pytest.mark.gpu
DEV = "cuda"


@pytest.mark.parametrize("rows,V,Vc,K", [(7, 1000, 1000, 10), (64, 32000, 32000, 200), (33, 5000, 4096, 400),
                                          (5, 300, 300, 300), (16, 128256, 128256, 128)])
def test_topk_logprob_exact(rows, V, Vc, K):
    torch.manual_seed(rows + K)
    x = torch.randn(rows, V, device=DEV) * 4
    x[:, ::7] = x[:, 1::7][:, : x[:, ::7].shape[1]]      # plenty of exact ties
    lp, ix = topk.topk_logprob(x, Vc, K)
    assert _lib.take_device_error() == 0
    ref_lp, ref_ix = topk.topk_logprob(x.cpu(), Vc, K)
    assert torch.equal(ix.cpu(), ref_ix)                  # ties broken by lower index, like a stable sort
    assert torch.allclose(lp.float().cpu(), ref_lp.float(), atol=2e-3, rtol=1e-3)


@pytest.mark.parametrize("case", ["one bin", "masked", "all equal", "few distinct"])
def test_topk_logprob_rows_that_defeat_the_histogram(case):
    """Rows whose K-th element shares its 11-bit histogram bin with thousands of others (the candidates no longer fit
    shared memory and the kernel narrows the threshold over the row instead), rows with masked (-inf) entries, and
    rows with more equal values at the threshold than the tie list holds."""
    torch.manual_seed(5)
    rows, V, K = 9, 20000, 200
    if case == "one bin":
        x = 1.0 + 0.1 * torch.rand(rows, V, device=DEV)            # every value in [1.0, 1.1): one bin
    elif case == "masked":
        x = torch.randn(rows, V, device=DEV) * 3
        x[:, 5000:] = float("-inf")
        x[3, 150:] = float("-inf")                                  # fewer finite values than K
    elif case == "all equal":
        x = torch.full((rows, V), 0.25, device=DEV)
        x[1, 17] = 3.0
    else:
        x = torch.randint(0, 3, (rows, V), device=DEV).float()      # ~6700 ties at the threshold
    lp, ix = topk.topk_logprob(x, V, K)
    assert _lib.take_device_error() == 0
    ref_lp, ref_ix = topk.topk_logprob(x.cpu(), V, K)
    assert torch.equal(ix.cpu(), ref_ix)
    got, want = lp.float().cpu(), ref_lp.float()
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), finite)
    assert torch.allclose(got[finite], want[finite], atol=2e-3, rtol=1e-3)


@pytest.mark.parametrize("V,K", [(1, 1), (3, 2), (255, 255), (1021, 200), (4096, 513), (16383, 400), (16384, 512), (16387, 257), (32000, 513),
                                 (32001, 1024), (40000, 256), (300001, 128)])
@pytest.mark.parametrize("layout", ["plain", "off 16 bytes", "ascending", "descending"])
def test_topk_logprob_over_group_sizes(V, K, layout):
    """Both group sizes and all sort widths, rows that are no multiple of a quad or of a round, rows off 16-byte boundaries, and rows
    whose largest elements lie side by side; the same as one vocabulary shard."""
    rows, ld = 5, V + 5
    g = torch.Generator("cuda").manual_seed(V + K)
    buf = torch.full((rows, ld + 3), 1e9, device=DEV)                    # what lies beside a row must not be read as its own
    x = buf[:, 3 if layout == "off 16 bytes" else 0:][:, :V]
    x.copy_(torch.randn(rows, V, device=DEV, generator=g) * 3)
    if "scending" in layout:
        x.copy_(x.sort(-1, descending=layout == "descending").values)
    lp, ix = topk.topk_logprob(x, V, K)
    ref_lp, ref_ix = topk.topk_logprob(x.cpu(), V, K)
    assert torch.equal(ix.cpu(), ref_ix)
    # fp16 of a log-probability; exp and log in fp32 add 1e-6
    assert torch.allclose(lp.float().cpu(), ref_lp.float(), atol=2e-6, rtol=2 ** -10)
    lib = _lib.kernels()
    raw, lse = torch.empty((rows, K), device=DEV), torch.empty(rows, device=DEV)
    ids = torch.empty((rows, K), dtype=torch.int32, device=DEV)
    from llm_distillery_b200.parallel import tp  # noqa: F401  (declares the signature)
    assert lib.b200_topk_partial(_lib.ptr(x), x.stride(0), rows, V, K, 1000, _lib.ptr(raw), _lib.ptr(ids), _lib.ptr(lse),
                                 _lib.stream()) == 0
    assert torch.equal(ids - 1000, ix) and torch.equal(raw, x.gather(1, ix.long()))
    assert torch.allclose(lse, x.double().logsumexp(-1).float(), atol=2e-6, rtol=1e-6)
    assert _lib.take_device_error() == 0


def test_topk_logprob_rows_with_infinities():
    """+inf and NaN rank above all finite values, as keys; the log-sum-exp of such a row is no finite number where an inf takes
    part, and passes over NaN."""
    V, K = 20000, 200
    x = torch.randn(4, V, device=DEV) * 3
    x[1, 777], x[2, 5], x[3, :] = float("inf"), float("nan"), float("-inf")
    lp, ix = topk.topk_logprob(x, V, K)
    assert torch.equal(ix[:1].cpu(), topk.topk_logprob(x[:1].cpu(), V, K)[1])
    assert ix[1, 0] == 777 and ix[2, 0] == 5 and torch.equal(ix[3].cpu(), torch.arange(K, dtype=torch.int32))
    rest = torch.cat([x[2, :5], x[2, 6:]]).double()
    assert torch.allclose(lp[2, 1:].double(), rest.topk(K - 1).values - rest.logsumexp(-1), atol=2e-6, rtol=2 ** -10)
    assert lp[2, 0].isnan() and lp[3].isnan().all()


def test_logprob_full_and_merge():
    torch.manual_seed(0)
    x = torch.randn(50, 777, device=DEV) * 3
    full = topk.logprob_full(x, 700)
    assert torch.allclose(full.float().cpu(), torch.log_softmax(x[:, :700].cpu(), -1), atol=3e-3, rtol=2e-3)
    K = 40
    a = torch.log_softmax(torch.randn(60, 500, device=DEV) * 3, -1)
    b = torch.log_softmax(torch.randn(60, 500, device=DEV) * 3, -1)
    av, ai = a.topk(K, -1)
    bv, bi = b.topk(K, -1)
    lp, ids = topk.topk_merge(av, ai.int(), bv, bi.int())
    rlp, rids = topk.topk_merge(av.cpu(), ai.int().cpu(), bv.cpu(), bi.int().cpu())
    assert torch.allclose(lp.cpu(), rlp, atol=1e-4, rtol=1e-4)
    same = (ids.cpu() == rids).float().mean().item()
    assert same > 0.99          # order may differ only between exactly equal probabilities


def test_merge_keeps_the_mass_of_token_zero_beside_empty_slots():
    """Empty slots are (id 0, -inf); a real token 0 in both lists must come out with both probabilities."""
    ninf = float("-inf")
    a_lp = torch.tensor([[0.5, 0.2, 0.0, 0.0, 0.0, 0.0]], device=DEV).log()
    a_id = torch.tensor([[0, 7, 0, 0, 0, 0]], device=DEV, dtype=torch.int32)
    b_lp = torch.tensor([[0.3, 0.25, 0.1, 0.0, 0.0, 0.0]], device=DEV).log()
    b_id = torch.tensor([[0, 9, 7, 0, 0, 0]], device=DEV, dtype=torch.int32)
    lp, ids = topk.topk_merge(a_lp, a_id, b_lp, b_id)
    assert ids[0, :3].tolist() == [0, 7, 9]
    assert torch.allclose(lp[0, :3].exp().cpu(), torch.tensor([0.8, 0.3, 0.25]), atol=1e-5)
    assert ids[0, 3:].tolist() == [0, 0, 0] and bool((lp[0, 3:] == ninf).all())
    rlp, rids = topk.topk_merge(a_lp.cpu(), a_id.cpu(), b_lp.cpu(), b_id.cpu())
    assert rids[0, :3].tolist() == [0, 7, 9] and torch.allclose(rlp[0, :3].exp(), torch.tensor([0.8, 0.3, 0.25]), atol=1e-5)


def test_collector_matches_full_logits_path():
    torch.manual_seed(1)
    cfg = LlamaConfig(vocab_size=2048, hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                      num_attention_heads=4, num_key_value_heads=2, max_position_embeddings=256)
    model = build_model(cfg, dtype=torch.bfloat16, device=DEV, seed=3)
    rng = np.random.default_rng(0)
    convos, toks = [], []
    for i, (length, ranges) in enumerate([(100, [(2, 40), (50, 100)]), (77, [(0, 77)]), (128, [(10, 20)])]):
        t = np.zeros(128, dtype=np.int64)
        t[:length] = rng.integers(0, 2000, length)
        convos.append(ConvoTokenized(t, ranges, 128 - length, False, i))
        toks.append(t)
    tokens = np.stack(toks)
    col = TeacherCollector(model, topk=32, crop_to_size=2000, enable_topk=True)
    rows = col.collect_batch(tokens, convos)
    assert _lib.take_device_error() == 0
    with torch.no_grad():   # oracle: fp32 logits from the same bf16 hidden states and weights
        hs = model.hidden_states(torch.from_numpy(tokens).to(DEV)).float()
        logits = (hs @ model.lm_head.float().t()).reshape(3, 128, -1)[:, :, :2000]
    lp = torch.log_softmax(logits, -1).cpu()
    for r, c in zip(rows, convos):
        ci = c.content_indices()
        ci = ci[ci < c.length]
        assert r.values.shape == (len(ci), 32) and r.indices.shape == (len(ci), 32)
        ref_v, ref_i = lp[c.origin_convo_id, ci].topk(32, -1)
        agree = (torch.from_numpy(r.indices) == ref_i).float().mean().item()
        assert agree > 0.97     # only exact-tie order may differ
        assert torch.allclose(torch.from_numpy(r.values).float()[:, :4], ref_v[:, :4], atol=3e-2, rtol=2e-2)
    full = TeacherCollector(model, topk=0, crop_to_size=2000, enable_topk=False).collect_batch(tokens, convos)
    assert full[1].indices is None and full[1].values.shape == (77, 2000)


@pytest.mark.parametrize("name", ["adamw", "adam", "adamw8bit", "sgd", "rmsprop", "adagrad"])
def test_optimizer_kernels_match_torch_restatement(name):
    torch.manual_seed(2)
    w = torch.nn.Parameter(torch.randn(300, 70, device=DEV).bfloat16())
    w_cpu = torch.nn.Parameter(w.detach().float().cpu())
    fg = FlatParams([w])
    fc = FlatParams([w_cpu])
    fc.master.copy_(fg.master.cpu())
    og = FlatOptimizer(fg, name, lr=1e-2, weight_decay=0.01)
    oc = FlatOptimizer(fc, name, lr=1e-2, weight_decay=0.01)
    for _ in range(4):
        g = torch.randn(300, 70)
        w.grad_slot.buf.copy_(g.to(DEV))
        w_cpu.grad_slot.buf.copy_(g)
        og.step(grad_scale=0.5)
        oc.step(grad_scale=0.5)
    tol = 3e-2 if name == "adamw8bit" else 1e-4
    assert torch.allclose(fg.master.cpu(), fc.master, atol=tol, rtol=tol), (fg.master.cpu() - fc.master).abs().max()
    assert torch.allclose(w.detach().float().cpu(), fg.master.cpu()[: w.numel()].view(300, 70), atol=2e-2, rtol=2e-2)


@pytest.mark.parametrize("n", [1, 6, 255, 256, 260, 2047, 70001])
@pytest.mark.parametrize("decoupled", [0, 1])
def test_8bit_adam_of_aligned_and_unaligned_shards(n, decoupled):
    """Blocks cut short, and buffers off the 16-byte boundaries: the same bits on both paths, nothing written behind the last
    value, and after the first step every block's scales are the maxima of its moments ((1 - beta) g, sqrt((1 - beta2) g^2):
    three roundings each)."""
    gen = torch.Generator("cuda").manual_seed(n)
    w0, g = (torch.randn(n, device=DEV, generator=gen) for _ in range(2))
    nb = (n + 255) // 256

    def run(off):
        f = [torch.full((n + off + 8,), 7.0, device=DEV, dtype=d) for d in (torch.float32, torch.bfloat16, torch.float32)]
        c = [torch.full((n + off + 8,), 7, device=DEV, dtype=d) for d in (torch.int8, torch.uint8)]
        s = torch.zeros(2, nb, device=DEV)
        w, m, gr, mq, vq = (t[off:off + n] for t in (f[0], f[1], f[2], *c))
        w.copy_(w0), gr.copy_(g), mq.zero_(), vq.zero_()
        scales = []
        for step in (1, 2):
            _lib.check(_lib.kernels().b200_adam8_step(
                _lib.ptr(w), _lib.ptr(m), _lib.ptr(gr), _lib.ptr(mq), _lib.ptr(vq), _lib.ptr(s[0]), _lib.ptr(s[1]), n, 1e-3, 0.9,
                0.99, 1e-8, 0.01, step, 1.0, decoupled, _lib.stream()), "adam step")
            scales.append(s.clone())
        assert all((t[:off] == 7).all() and (t[off + n:] == 7).all() for t in (*f, *c))
        return w, m, mq, vq, *scales
    got, off1 = run(0), run(1)
    assert all(torch.equal(a, b) for a, b in zip(got, off1)) and _lib.take_device_error() == 0
    ge = torch.nn.functional.pad((g if decoupled else g + 0.01 * w0).double(), (0, nb * 256 - n)).view(nb, 256).abs().amax(1)
    assert torch.allclose(got[4][0].double(), 0.1 * ge, rtol=4e-7) and torch.allclose(got[4][1].double(), 0.1 * ge, rtol=4e-6)
