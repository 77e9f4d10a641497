"""The native layer calls issue the launches of ``DecoderLayerFn``: same outputs and gradients, bit for bit."""
from types import SimpleNamespace

import pytest
import torch

from llm_distillery_b200.engine.optim import FlatParams
from llm_distillery_b200.models import layer_native, llama
from llm_distillery_b200.ops import _lib, basic

pytestmark = pytest.mark.gpu


def _run(monkeypatch, native, bias, f, d, window, checkpoint, frozen, ordered):
    cfg = llama.LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=f, num_hidden_layers=2, num_attention_heads=4,
                            num_key_value_heads=2, head_dim_override=d, max_position_embeddings=512, attention_bias=bias,
                            sliding_window=window)
    model = llama.build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=3)
    model.grad_checkpointing, model.ordered_sums = checkpoint, ordered
    if frozen:
        model.layers[0].qkv_proj.requires_grad = False
        model.layers[1].input_layernorm.requires_grad = False
    FlatParams([p for p in model.parameters() if p.requires_grad])
    ids = torch.randint(0, 512, (2, 173), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    used = []
    if not native:
        monkeypatch.setattr(layer_native, "fits", lambda *a: False)
    else:
        real = layer_native.fits
        monkeypatch.setattr(layer_native, "fits", lambda *a: used.append(real(*a)) or used[-1])
    for _ in range(2):        # the second pass accumulates
        y = model.hidden_states(ids)
        g = torch.randn(y.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(2)).to(y.dtype)
        y.backward(g)
    with torch.no_grad():
        z = model.hidden_states(ids)
    monkeypatch.undo()
    assert all(used) and len(used) == (6 if native else 0)
    assert _lib.take_device_error() == 0
    return y.detach(), {n: p.grad_slot.buf.clone() for n, p in model.named_parameters() if p.requires_grad}, z


@pytest.mark.parametrize("bias,f,d,window,checkpoint,frozen", [
    (False, 640, 64, None, False, False), (True, 640, 64, None, False, False), (False, 208, 128, None, False, True),
    (False, 640, 128, 100, True, False), (True, 208, 64, None, True, True)])
def test_native_layer_equals_the_layer_of_separate_calls(monkeypatch, bias, f, d, window, checkpoint, frozen):
    for ordered in (True, False):
        a = _run(monkeypatch, True, bias, f, d, window, checkpoint, frozen, ordered)
        b = _run(monkeypatch, False, bias, f, d, window, checkpoint, frozen, ordered)
        assert torch.equal(a[0], b[0]) and torch.equal(a[2], b[2])
        assert a[1].keys() == b[1].keys()
        for name, want in b[1].items():
            # The gradients of the embedding and of the biases meet in fp32 by atomic adds in no fixed order: sums of at
            # most 700 terms, off by up to 700 2^-24 of their absolute sum. All others repeat, also behind the atomic
            # query gradients: those of 173 positions have two terms (two key blocks), the same bits in either order.
            got = a[1][name]
            if "embed" in name or name.endswith("qkv_bias"):
                assert ((got - want).norm() / want.norm()).item() < 700 * 2 ** -24, name
            else:
                assert torch.equal(got, want), name
            assert want.norm() > 0 or name == "lm_head", name


@pytest.mark.parametrize("between", ["nothing", "backward hook", "one layer"])
def test_layers_in_one_call_equal_a_call_each(monkeypatch, between):
    """All layers in one node (a few tokens, nothing between the layers) against a node per layer: outputs, gradients and those
    of a second, accumulating pass bit for bit; a hook behind each layer's backward pass is called in order."""
    cfg = llama.LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=640, num_hidden_layers=1 if between == "one layer" else 5,
                            num_attention_heads=4, num_key_value_heads=2, max_position_embeddings=512, sliding_window=100,
                            window_layers=None)
    results, calls = [], []
    for limit in (0, layer_native.STACK_MAX_TOKENS):
        model = llama.build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=3)
        FlatParams([p for p in model.parameters() if p.requires_grad])
        ids = torch.randint(0, 512, (2, 173), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
        monkeypatch.setattr(layer_native, "STACK_MAX_TOKENS", limit)
        stacks, real = [], layer_native.run_stack
        monkeypatch.setattr(layer_native, "run_stack", lambda *a: stacks.append(1) or real(*a))
        order = []
        if between == "backward hook":
            monkeypatch.setattr(llama, "LAYER_BACKWARD_DONE", [lambda w: order.append(
                [w is l.input_layernorm for l in model.layers].index(True))])
        for _ in range(2):
            y = model.hidden_states(ids)
            y.backward(torch.randn(y.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(2)).to(y.dtype))
        with torch.no_grad():
            z = model.hidden_states(ids)
        monkeypatch.undo()
        assert len(stacks) == (2 if limit else 0)              # the passes with gradients
        assert torch.equal(y, z) and _lib.take_device_error() == 0
        results.append((y.detach(), {n: p.grad_slot.buf.clone() for n, p in model.named_parameters() if "embed" not in n}))
        calls.append(order)
    assert calls[0] == calls[1] and calls[1] == ([4, 3, 2, 1, 0] * 2 if between == "backward hook" else [])
    assert torch.equal(results[0][0], results[1][0])
    for name, want in results[0][1].items():
        assert torch.equal(results[1][1][name], want), name


@pytest.mark.parametrize("layers", [1, 2, 9])
@pytest.mark.parametrize("refused", [None, 0, 3])
def test_inference_in_calls_of_several_layers_equals_a_call_each(monkeypatch, layers, refused):
    """Passes without gradients run 1, 1, 2, 4, ... layers a call, up to a layer that does not fit; the bits of a call per
    layer, with windows that differ from layer to layer, in plain and in K-cutting GEMMs."""
    cfg = llama.LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=640, num_hidden_layers=layers, num_attention_heads=4,
                            num_key_value_heads=2, max_position_embeddings=512, attention_bias=True, sliding_window=50,
                            window_layers=[i % 2 == 0 for i in range(layers)])
    model = llama.build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=3)
    ids = torch.randint(0, 512, (2, 173), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    weight = model.layers[refused].qkv_proj if refused is not None and refused < layers else None
    real, lib, calls = layer_native.fits, _lib.kernels(), []
    monkeypatch.setattr(layer_native, "fits", lambda *a: a[4][1] is not weight and real(*a))

    class Recorder:
        def __getattr__(self, name):
            fn = getattr(lib, name)
            if name != "b200_stack_fwd":
                return fn
            return lambda rows, n, *a: calls.append(n) or fn(rows, n, *a)
    monkeypatch.setattr(_lib, "kernels", Recorder)
    for ordered in (True, False):
        model.ordered_sums = ordered
        got = []
        for limit in (0, layer_native.STACK_MAX_TOKENS):
            monkeypatch.setattr(layer_native, "STACK_MAX_TOKENS", limit)
            with torch.no_grad():
                got.append(model.hidden_states(ids))
        assert torch.equal(*got)
    fit = layers if weight is None else refused
    sizes = [n for n in (1, 1, 2, 4, 8)]
    want = [min(n, fit - sum(sizes[:i])) for i, n in enumerate(sizes) if sum(sizes[:i]) < fit]
    assert calls == want * 2 and _lib.take_device_error() == 0


@pytest.mark.parametrize("embedding,layers,stacked", [(True, 0, 5), (True, 2, 3), (True, 5, 0), (False, 2, 5)])
def test_layers_that_no_gradient_reaches_stay_out_of_the_one_call(monkeypatch, embedding, layers, stacked):
    """Frozen embedding and first layers: outputs and gradients bit for bit those of a node per layer, whose backward pass ends at
    the first layer with a trained weight - and no more launches and no more memory than it takes."""
    cfg = llama.LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=640, num_hidden_layers=5, num_attention_heads=4,
                            num_key_value_heads=2, max_position_embeddings=512)
    results = []
    for limit in (0, layer_native.STACK_MAX_TOKENS):
        model = llama.build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=3)
        for w in [model.embed_tokens] * embedding + [p for l in model.layers[:layers] for p in l.parameters()]:
            w.requires_grad_(False)
        FlatParams([p for p in model.parameters() if p.requires_grad])
        ids = torch.randint(0, 512, (2, 173), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
        monkeypatch.setattr(layer_native, "STACK_MAX_TOKENS", limit)
        sizes, real = [], layer_native.run_stack
        monkeypatch.setattr(layer_native, "run_stack", lambda x, pos, stack, *a: sizes.append(len(stack)) or real(x, pos, stack, *a))
        before = torch.cuda.memory_allocated()
        y = model.hidden_states(ids)
        held = torch.cuda.memory_allocated() - before
        launches = _lib.LAUNCH_COUNT[0]
        y.backward(torch.randn(y.shape, device="cuda", generator=torch.Generator("cuda").manual_seed(2)).to(y.dtype))
        launches = _lib.LAUNCH_COUNT[0] - launches
        monkeypatch.undo()
        assert sizes == ([stacked] if limit and stacked else []) and _lib.take_device_error() == 0
        results.append((y.detach(), {n: p.grad_slot.buf.clone() for n, p in model.named_parameters()
                                     if p.requires_grad and "embed" not in n}, launches, held))
    (want_y, want, launches_each, held_each), (got_y, got, launches, held) = results
    assert torch.equal(got_y, want_y) and got.keys() == want.keys()
    for name in want:
        assert torch.equal(got[name], want[name]), name
    assert launches <= launches_each and held <= 1.25 * held_each        # the allocator rounds blocks up; two layers more are 1.6


@pytest.mark.parametrize("trained", [False, True])
def test_a_layer_directly_behind_a_kernel_that_rewrites_its_weights(trained):
    """The few-tile GEMMs of a layer ask for weights before the launch in front of them has ended: not for those that a kernel in
    front of the whole call writes (an optimizer step, an expansion of low-bit weights). 46 M elements are rewritten right in
    front of the forward and of the backward call, with other values each time; bit for bit what comes of waiting in between."""
    T, H, Hkv, d, h, f = 93, 32, 4, 64, 2048, 5632
    shapes = ((h,), ((H + 2 * Hkv) * d, h), (h, H * d), (h,), (2 * f, h), (h, f))
    g = torch.Generator("cuda").manual_seed(0)
    sizes = [torch.Size(s).numel() for s in shapes]
    versions = [torch.randn(sum(sizes), device="cuda", generator=g) * 0.02 for _ in range(3)]
    flat = torch.empty(sum(sizes), dtype=torch.bfloat16, device="cuda")
    weights = [p.view(s).requires_grad_(trained) for p, s in zip(flat.split(sizes), shapes)]
    if trained:
        for w in weights:
            w.grad_slot = SimpleNamespace(buf=torch.empty(w.shape, dtype=torch.float32, device="cuda"))
    x = torch.randn(T, h, device="cuda", generator=g).bfloat16().requires_grad_()
    dy = torch.randn(T, h, device="cuda", generator=g).bfloat16()
    pos = torch.arange(T, dtype=torch.int32, device="cuda")
    cos, sin = basic.rope_tables(T, d, 10000.0, "cuda")

    def write(v, wait):
        basic.cast_to_bf16(versions[v], flat)
        if wait:
            torch.cuda.synchronize()

    def run(v, wait):
        for w in weights if trained else []:
            w.grad_slot.fresh = True
        write(v, wait)
        y = layer_native.NativeLayerFn.apply(x, pos, cos, sin, *weights, None, (1, T, H, Hkv, d, 1e-5, False, None), (not trained, True))
        write((v + 1) % 3, wait)
        dx, = torch.autograd.grad(y, x, dy)
        return [y.detach(), dx] + ([w.grad_slot.buf.clone() for w in weights] if trained else [])
    want = [run(v, True) for v in range(3)]
    for i in range(12):
        for got, ref in zip(run(i % 3, False), want[i % 3]):
            assert torch.equal(got, ref)
    assert _lib.take_device_error() == 0
