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


@pytest.mark.parametrize("rc", [-2, 20])
def test_gradient_slots_are_taken_as_written_only_by_a_call_that_ran(monkeypatch, rc):
    """A backward call that fails leaves the slots fresh, as they are: the next pass must not add to what is in them."""
    class Lib:
        def __getattr__(self, name):
            if name == "b200_last_cuda_error":
                return lambda: b""
            return lambda *a: {"b200_layer_fwd": 8, "b200_layer_bwd": rc}.get(name, 64)

    class Slot:
        def __init__(self, w):
            self.buf, self.fresh = torch.zeros(w.shape), True
    monkeypatch.setattr(layer_native._lib, "kernels", Lib)
    monkeypatch.setattr(layer_native._lib, "stream", lambda: None)
    n = (H + 2 * HKV) * D
    w = [torch.zeros(s, dtype=torch.bfloat16).requires_grad_() for s in ((W,), (n, W), (W, H * D), (W,), (2 * F, W), (W, F))]
    for t in w:
        t.grad_slot = Slot(t)
    x = torch.zeros(T, W, dtype=torch.bfloat16).requires_grad_()
    tables = torch.zeros(T, dtype=torch.int32), torch.zeros(16, D // 2), torch.zeros(16, D // 2)
    y = layer_native.NativeLayerFn.apply(x, *tables, *w, None, (1, T, H, HKV, D, 1e-5, False, None), (False, False))
    if rc < 0:
        with pytest.raises(layer_native._lib.NativeError):
            y.backward(torch.zeros_like(y))
    else:
        y.backward(torch.zeros_like(y))
    assert all(t.grad_slot.fresh == (rc < 0) for t in w)


@pytest.mark.parametrize("ran", [0, 2, 3])
def test_a_failing_call_over_several_layers_marks_those_that_ran(monkeypatch, ran):
    """Three layers in one backward call: the slots of the last ``ran`` of them count as written, the others stay fresh."""
    import ctypes

    class Lib:
        def b200_stack_bwd(self, *a):
            ctypes.cast(a[-2], ctypes.POINTER(ctypes.c_int))[0] = ran
            return 60 if ran == 3 else -2

        def __getattr__(self, name):
            return (lambda: b"") if name == "b200_last_cuda_error" else (lambda *a: 64)

    class Slot:
        def __init__(self, w):
            self.buf, self.fresh = torch.zeros(w.shape), True
    monkeypatch.setattr(layer_native._lib, "kernels", Lib)
    monkeypatch.setattr(layer_native._lib, "stream", lambda: None)
    n, layers = (H + 2 * HKV) * D, []
    tables = torch.zeros(16, D // 2), torch.zeros(16, D // 2)
    for _ in range(3):
        w = tuple(torch.zeros(s, dtype=torch.bfloat16).requires_grad_() for s in ((W,), (n, W), (W, H * D), (W,), (2 * F, W), (W, F)))
        for t in w:
            t.grad_slot = Slot(t)
        layers.append((w, None, *tables, None))
    x = torch.zeros(T, W, dtype=torch.bfloat16)
    y = layer_native.run_stack(x, torch.zeros(T, dtype=torch.int32), layers, (1, T, H, HKV, D, 1e-5, False, None),
                               (False, False))
    assert y.requires_grad                                   # by the weights alone
    if ran < 3:
        with pytest.raises(layer_native._lib.NativeError):
            y.backward(torch.zeros_like(y))
    else:
        y.backward(torch.zeros_like(y))
    assert [all(t.grad_slot.fresh for t in w) for w, *_ in layers] == [i < 3 - ran for i in range(3)]
    assert not any(t.grad_slot.fresh for w, *_ in layers[3 - ran:] for t in w)


def test_what_a_hook_moves_is_read_where_it_then_lies(monkeypatch):
    """A hook in front of a layer's backward pass (weights gathered, low-bit weights expanded) may put the layer's weights and
    gradient buffers elsewhere: the call takes their addresses behind it."""
    import ctypes
    from llm_distillery_b200.models import llama
    got = []

    class Lib:
        def b200_stack_bwd(self, rows, grads, n, *a):
            rows, grads = (ctypes.cast(r, ctypes.POINTER(ctypes.c_uint64)) for r in (rows, grads))
            got.append((rows[3], grads[2]))                  # the q/k/v matrix and its gradient
            ctypes.cast(a[-2], ctypes.POINTER(ctypes.c_int))[0] = n
            return 20

        def __getattr__(self, name):
            return (lambda: b"") if name == "b200_last_cuda_error" else (lambda *a: 64)

    class Slot:
        def __init__(self, w):
            self.buf, self.fresh = torch.zeros(w.shape), True
    monkeypatch.setattr(layer_native._lib, "kernels", Lib)
    monkeypatch.setattr(layer_native._lib, "stream", lambda: None)
    n, layers = (H + 2 * HKV) * D, []
    tables = torch.zeros(16, D // 2), torch.zeros(16, D // 2)
    for _ in range(3):
        w = tuple(torch.zeros(s, dtype=torch.bfloat16).requires_grad_() for s in ((W,), (n, W), (W, H * D), (W,), (2 * F, W), (W, F)))
        for t in w:
            t.grad_slot = Slot(t)
        layers.append((w, None, *tables, None))
    held = []

    def gather(first, backward):
        w = next(ws[1] for ws, *_ in layers if ws[0] is first)
        held.append((w.data, w.grad_slot.buf))               # the old places stay taken: nothing else lands there
        w.data, w.grad_slot.buf = w.data.clone(), w.grad_slot.buf.clone()
    y = layer_native.run_stack(torch.zeros(T, W, dtype=torch.bfloat16), torch.zeros(T, dtype=torch.int32), layers,
                               (1, T, H, HKV, D, 1e-5, False, None), (False, False))
    monkeypatch.setattr(llama, "UNIT_PRE", [gather])
    y.backward(torch.zeros_like(y))
    assert got == [(ws[1].data_ptr(), ws[1].grad_slot.buf.data_ptr()) for ws, *_ in reversed(layers)]
    assert not any(t.grad_slot.fresh for ws, *_ in layers for t in ws)
