"""The native layer calls issue the launches of ``DecoderLayerFn``: same outputs and gradients, bit for bit."""
import pytest
import torch

from llm_distillery_b200.engine.optim import FlatParams
from llm_distillery_b200.models import layer_native, llama
from llm_distillery_b200.ops import _lib

pytestmark = pytest.mark.gpu


def _run(monkeypatch, native, bias, f, d, window, checkpoint, frozen):
    cfg = llama.LlamaConfig(vocab_size=512, hidden_size=256, intermediate_size=f, num_hidden_layers=2, num_attention_heads=4,
                            num_key_value_heads=2, head_dim_override=d, max_position_embeddings=512, attention_bias=bias,
                            sliding_window=window)
    model = llama.build_model(cfg, dtype=torch.bfloat16, device="cuda", seed=3)
    model.grad_checkpointing = checkpoint
    if frozen:
        model.layers[0].qkv_proj.requires_grad = False
        model.layers[1].input_layernorm.requires_grad = False
    flat = FlatParams([p for p in model.parameters() if p.requires_grad])
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
    return y.detach(), flat.grad.clone(), z


@pytest.mark.parametrize("bias,f,d,window,checkpoint,frozen", [
    (False, 640, 64, None, False, False), (True, 640, 64, None, False, False), (False, 208, 128, None, False, True),
    (False, 640, 128, 100, True, False), (True, 208, 64, None, True, True)])
def test_native_layer_equals_the_layer_of_separate_calls(monkeypatch, bias, f, d, window, checkpoint, frozen):
    a = _run(monkeypatch, True, bias, f, d, window, checkpoint, frozen)
    b = _run(monkeypatch, False, bias, f, d, window, checkpoint, frozen)
    assert torch.equal(a[0], b[0]) and torch.equal(a[2], b[2])
    # query gradients meet in fp32 by atomic adds in no fixed order (two key blocks), and so do the bias gradients: a last
    # bit in front of a bf16 rounding, 2^-9 of single elements
    assert ((a[1] - b[1]).norm() / b[1].norm()).item() < 1e-3
