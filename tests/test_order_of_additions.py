"""Which forwards may cut the K of their GEMMs (the calls' ``split_k``), on the CPU."""
import pytest
import torch

from llm_distillery_b200.models import llama
from llm_distillery_b200.ops import basic


@pytest.mark.parametrize("experts", [False, True])
@pytest.mark.parametrize("chunk", [0, 8])
def test_expert_layers_never_split(monkeypatch, experts, chunk):
    """Behind a router a last bit can be another expert: no GEMM of a layer with experts is cut, also where the model's
    owner allows it. (A dense model's chunked forward shows that the recorder sees the cuts.)"""
    over = dict(num_local_experts=4, num_experts_per_tok=2) if experts else {}
    cfg = llama.LlamaConfig(vocab_size=64, hidden_size=32, intermediate_size=48, num_hidden_layers=2, num_attention_heads=4,
                            num_key_value_heads=2, max_position_embeddings=64, **over)
    model = llama.build_model(cfg, dtype=torch.float32, device="cpu", seed=1)
    model.ordered_sums = False
    seen, real = [], basic.gemm
    monkeypatch.setattr(basic, "gemm", lambda *a, **k: seen.append(k.get("split_k", False)) or real(*a, **k))
    ids = torch.arange(20).reshape(1, -1)
    with torch.no_grad():
        model.hidden_states_chunked(ids, chunk) if chunk else model.hidden_states(ids)
    assert seen and (any(seen) != experts)
