"""The fused projections refuse operands of different reduction lengths, as ``gemm`` does, before anything is launched."""
import pytest
import torch

from llm_distillery_b200.ops import _lib, basic


class _NoLaunch:
    def __getattr__(self, name):
        raise AssertionError(f"{name} was reached")


@pytest.mark.parametrize("T", [33, 600])
def test_different_reductions(monkeypatch, T):
    monkeypatch.setattr(basic, "_native", lambda *t: True)       # the route of a GPU call
    monkeypatch.setattr(_lib, "kernels", _NoLaunch)
    x = torch.zeros(T, 320, dtype=torch.bfloat16)
    w = torch.zeros(512, 256, dtype=torch.bfloat16)
    pos = torch.zeros(T, dtype=torch.int32)
    cos, sin = basic.rope_tables(8, 64, 10000.0, "cpu")
    for call in (lambda: basic.linear_swiglu_fwd(x, w), lambda: basic.linear_rope_fwd(x, w, pos, cos, sin, 2, 64),
                 lambda: basic.linear_dgrad_swiglu_bwd(x, w, torch.zeros(T, 512, dtype=torch.bfloat16))):
        with pytest.raises(ValueError):
            call()
