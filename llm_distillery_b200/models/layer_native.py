"""The plain decoder layer as one native call per direction (csrc/ops/layer.cu): the kernels of ``llama.DecoderLayerFn``
in the same order with the same results, issued from C++ instead of one Python call each. A 777-token step of a 0.5 B
student spends 24 x 30 launches in its layers; from Python they cost the host about 20 us apiece, more than the kernels
take.

``fits`` says which layers run here: bf16 on a GPU, heads of 64 or 128 with a full rotation, no norms or biases besides the
two RMSNorms and a q/k/v bias, and every weight either frozen or with a gradient slot to accumulate into. All others, and
CPU tensors, keep ``DecoderLayerFn``.
"""
from __future__ import annotations

import torch

from ..ops import _lib
from ..ops._lib import _F, _I, _LL, _VP

for _n in ("b200_layer_saved_bytes", "b200_layer_scratch_bytes"):
    _lib.RESTYPES[_n] = _LL
_lib.register("b200_layer_fwd", [_VP] * 13 + [_I] * 8 + [_F, _I, _VP])
_lib.register("b200_layer_bwd", [_VP] * 21 + [_I] * 10 + [_VP])
_lib.register("b200_layer_saved_bytes", [_I] * 7)
_lib.register("b200_layer_scratch_bytes", [_I] * 7)
for _n in ("b200_layer_fwd", "b200_layer_bwd", "b200_layer_saved_bytes", "b200_layer_scratch_bytes"):
    _lib.KERNELS_PER_CALL[_n] = 0          # the calls return how many kernels they launched


def tables_fit(pos, cos, sin, tokens: int, d: int) -> bool:
    if pos.dtype != torch.int32 or not pos.is_contiguous() or pos.shape != (tokens,):
        return False
    return all(t.dtype == torch.float32 and t.is_contiguous() and 2 * t.shape[1] == d and t.shape == cos.shape for t in (cos, sin))


def fits(h, pos, cos, sin, weights, b_qkv, heads, training: bool, tables: bool | None = None) -> bool:
    """``heads`` = (query heads, key heads, head size). The C calls take sizes from the activations and trust the rest, so
    what the separate calls would refuse is left to them. ``tables``: what ``tables_fit`` said of the positions and tables,
    for a caller that runs several layers on them (this check of a layer is 3 us of the host's time, with theirs 5)."""
    H, Hkv, d = heads
    T, w = h.shape
    bf16 = torch.bfloat16
    if not h.is_cuda or h.dtype != bf16 or d not in (64, 128) or w % 8 or w > 8192:
        return False
    if not (tables_fit(pos, cos, sin, T, d) if tables is None else tables):
        return False
    n, f = (H + 2 * Hkv) * d, weights[4].shape[0] // 2
    shapes = ((w,), (n, w), (w, H * d), (w,), (2 * f, w), (w, f), (n,))
    for t, shape in zip(weights if b_qkv is None else weights + (b_qkv,), shapes):
        if t.shape != shape or t.dtype != bf16 or not t.is_cuda or not t.is_contiguous():
            return False
        if training and t.requires_grad and getattr(t, "grad_slot", None) is None:
            return False
    return f % 8 == 0


def _launched(rc: int, what: str) -> None:
    if rc < 0:
        _lib.check(rc, what)
    _lib.LAUNCH_COUNT[0] += rc


def _forward(x, pos, cos, sin, weights, b_qkv, meta, split, with_output: bool):
    B, L, H, Hkv, d, eps, _, window = meta
    h, f = x.shape[1], weights[4].shape[0] // 2
    lib = _lib.kernels()
    saved = torch.empty(lib.b200_layer_saved_bytes(B, L, H, Hkv, d, h, f), dtype=torch.uint8, device=x.device)
    out = torch.empty_like(x) if with_output else None
    window = 0 if window is None or L <= window else window
    w1, wq, wo, w2, wg, wd = weights
    _launched(lib.b200_layer_fwd(x.data_ptr(), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(), w1.data_ptr(), wq.data_ptr(),
                                 wo.data_ptr(), w2.data_ptr(), wg.data_ptr(), wd.data_ptr(),
                                 0 if b_qkv is None else b_qkv.data_ptr(), saved.data_ptr(),
                                 out.data_ptr() if with_output else 0, B, L, window, H, Hkv, d, h, f, eps, int(split),
                                 _lib.stream()), "b200_layer_fwd")
    return saved, out


class NativeLayerFn(torch.autograd.Function):
    """``llama.DecoderLayerFn`` for layers that ``fits`` accepts."""

    @staticmethod
    def forward(ctx, x, pos, cos, sin, w_ln1, w_qkv, w_o, w_ln2, w_gu, w_d, b_qkv, meta, split):
        weights = (w_ln1, w_qkv, w_o, w_ln2, w_gu, w_d)
        x = x.contiguous()
        saved, out = _forward(x, pos, cos, sin, weights, b_qkv, meta, split[0], True)
        ctx.meta, ctx.split, ctx.weights, ctx.b_qkv = meta, split, weights, b_qkv
        if meta[6]:        # gradient checkpointing: keep only the layer input
            ctx.save_for_backward(x, pos, cos, sin)
        else:
            ctx.save_for_backward(x, pos, cos, sin, saved)
        return out

    @staticmethod
    def backward(ctx, dout):
        from . import llama
        weights, b_qkv, meta = ctx.weights, ctx.b_qkv, ctx.meta
        B, L, H, Hkv, d, eps, recompute, window = meta
        if llama.UNIT_PRE[0] is not None:
            llama.UNIT_PRE[0](weights[0], True)
        if llama.LAYER_WEIGHTS_PRE[0] is not None:
            llama.LAYER_WEIGHTS_PRE[0](weights[0])
        if recompute:
            x, pos, cos, sin = ctx.saved_tensors
            saved, _ = _forward(x, pos, cos, sin, weights, b_qkv, meta, ctx.split[0], False)
        else:
            x, pos, cos, sin, saved = ctx.saved_tensors
        dout = dout.contiguous()
        h, f = x.shape[1], weights[4].shape[0] // 2
        slots = [llama._slot(w) if w is not None else None for w in weights + (b_qkv,)]
        grads = [0 if s is None else s.buf.data_ptr() for s in slots]
        acc = sum(1 << i for i, s in enumerate(slots) if s is not None and not s.fresh)
        lib = _lib.kernels()
        scratch = torch.empty(lib.b200_layer_scratch_bytes(B, L, H, Hkv, d, h, f), dtype=torch.uint8, device=x.device)
        dx = torch.empty_like(x)
        window = 0 if window is None or L <= window else window
        w1, wq, wo, w2, wg, wd = weights
        _launched(lib.b200_layer_bwd(dout.data_ptr(), x.data_ptr(), pos.data_ptr(), cos.data_ptr(), sin.data_ptr(),
                                     w1.data_ptr(), wq.data_ptr(), wo.data_ptr(), w2.data_ptr(), wg.data_ptr(), wd.data_ptr(),
                                     saved.data_ptr(), scratch.data_ptr(), dx.data_ptr(), *grads, acc, B, L, window, H, Hkv,
                                     d, h, f, int(ctx.split[1]), _lib.stream()), "b200_layer_bwd")
        for s in slots:
            if s is not None:
                s.fresh = False
        if llama.LAYER_BACKWARD_DONE[0] is not None:
            llama.LAYER_BACKWARD_DONE[0](weights[0])
        return (dx,) + (None,) * 12
