"""Which layers the native layer call takes, and what a failing call leaves behind. On the CPU: tensors that say they are on
a GPU, and a library that answers without one."""
import pytest
import torch

from llm_distillery_b200.models import layer_native

H, HKV, D, T, W, F = 4, 2, 64, 6, 256, 208


class OnGpu(torch.Tensor):
    is_cuda = True


def _t(*shape, dtype=torch.bfloat16):
    return torch.zeros(*shape, dtype=dtype).as_subclass(OnGpu)


def _case(**change):
    n = (H + 2 * HKV) * D
    c = dict(h=_t(T, W), pos=_t(T, dtype=torch.int32), cos=_t(16, D // 2, dtype=torch.float32),
             sin=_t(16, D // 2, dtype=torch.float32), ln1=_t(W), qkv=_t(n, W), o=_t(W, H * D), ln2=_t(W), gu=_t(2 * F, W),
             down=_t(W, F), b_qkv=_t(n))
    c.update(change)
    w = tuple(c[k] for k in ("ln1", "qkv", "o", "ln2", "gu", "down"))
    return layer_native.fits(c["h"], c["pos"], c["cos"], c["sin"], w, c["b_qkv"], (H, HKV, D), False)


def test_the_plain_layer_fits():
    assert _case() and _case(b_qkv=None)


N = (H + 2 * HKV) * D


@pytest.mark.parametrize("name,tensor", [
    ("sin", _t(16, D // 2, dtype=torch.float64)), ("sin", _t(D // 2, 16, dtype=torch.float32).t()), ("sin", _t(8, D // 2, dtype=torch.float32)),
    ("cos", _t(16, D // 4, dtype=torch.float32)), ("pos", _t(T, dtype=torch.int64)), ("pos", _t(T - 1, dtype=torch.int32)),
    ("pos", _t(2 * T, dtype=torch.int32)[::2]), ("qkv", _t(N - D, W)), ("qkv", _t(N, W + 8)), ("o", _t(W, H * D - D)),
    ("gu", _t(2 * F, W - 8)), ("down", _t(W, F - 8)), ("ln1", _t(W - 8)), ("ln2", _t(W + 8)), ("b_qkv", _t(N - D)),
    ("h", _t(T, W, dtype=torch.float32)), ("qkv", _t(W, N).t())])
def test_other_layers_are_left_to_the_separate_calls(name, tensor):
    assert not _case(**{name: tensor})
