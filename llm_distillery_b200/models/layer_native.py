"""The plain decoder layer as one native call per direction (csrc/ops/layer.cu): the kernels of ``llama.DecoderLayerFn``
in the same order with the same results, issued from C++ instead of one Python call each. A 777-token step of a 0.5 B
student spends 24 x 30 launches in its layers; from Python they cost the host about 20 us apiece, more than the kernels
take.

``fits`` says which layers run here: bf16 on a GPU, heads of 64 or 128 with a full rotation, no norms or biases besides the
two RMSNorms and a q/k/v bias, and every weight either frozen or with a gradient slot to accumulate into. All others, and
CPU tensors, keep ``DecoderLayerFn``.

``run_stack`` runs all layers of a training pass over few tokens in one native call per direction, when nothing has to happen
between them; ``run_inference`` those of a pass without gradients in a few.
"""
from __future__ import annotations

import ctypes

import torch

from ..ops import _lib
from ..ops._lib import _F, _I, _LL, _VP

for _n in ("b200_layer_saved_bytes", "b200_layer_scratch_bytes"):
    _lib.RESTYPES[_n] = _LL
_lib.register("b200_layer_fwd", [_VP] * 13 + [_I] * 8 + [_F, _I, _VP])
_lib.register("b200_layer_bwd", [_VP] * 21 + [_I] * 10 + [_VP])
_lib.register("b200_layer_saved_bytes", [_I] * 7)
_lib.register("b200_layer_scratch_bytes", [_I] * 7)
_lib.register("b200_stack_fwd", [_VP, _I, _VP, _VP] + [_I] * 7 + [_F, _I, _VP])
_lib.register("b200_stack_bwd", [_VP, _VP, _I] + [_VP] * 6 + [_I] * 8 + [_VP, _VP])
for _n in ("b200_layer_fwd", "b200_layer_bwd", "b200_stack_fwd", "b200_stack_bwd", "b200_layer_saved_bytes", "b200_layer_scratch_bytes"):
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


ACT_ONLY = 4       # bit of a forward call's split: nothing will read the gate and up values (csrc/ops/layer.cu)


def _forward(x, pos, cos, sin, weights, b_qkv, meta, split, with_output: bool, act_only: bool = False):
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
                                 out.data_ptr() if with_output else 0, B, L, window, H, Hkv, d, h, f, eps,
                                 int(split) | (ACT_ONLY if act_only else 0), _lib.stream()), "b200_layer_fwd")
    return saved, out


class NativeLayerFn(torch.autograd.Function):
    """``llama.DecoderLayerFn`` for layers that ``fits`` accepts. A third entry of ``split``: no gradient will be asked for."""

    @staticmethod
    def forward(ctx, x, pos, cos, sin, w_ln1, w_qkv, w_o, w_ln2, w_gu, w_d, b_qkv, meta, split):
        weights = (w_ln1, w_qkv, w_o, w_ln2, w_gu, w_d)
        x = x.contiguous()
        saved, out = _forward(x, pos, cos, sin, weights, b_qkv, meta, split[0], True, meta[6] or (len(split) > 2 and split[2]))
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


# A training pass runs as one node up to this many tokens (a step of 512 tokens and four layers: 1.58 / 1.21 ms). Beyond, a
# layer's kernels take longer than the host's way to the next layer, and a node per layer gives its activations back as the
# backward pass moves on. Up to as many tokens a pass without gradients runs in calls of 1, 2, 4, ... layers: in one call the
# kernels start only when all layers have been looked at, with a call per layer (50 us of the host) they wait for the host in
# between (93 tokens of a 1.1 B teacher: 1.32 / 1.17 ms, of which its kernels need 1.09).
STACK_MAX_TOKENS = 2048


def run_inference(x, pos, entry, count: int, meta, split: bool):
    """The first layers of a pass without gradients, as many as fit, in calls of a growing number of them. ``entry(i)``: what
    ``run_stack`` takes of layer i, or None where it does not fit. Same kernels, order and bits as a ``NativeLayerFn`` per
    layer. Returns the output and how many layers it is of."""
    B, L, H, Hkv, d, eps = meta[:6]
    (T, h), lib, x, done = x.shape, _lib.kernels(), x.contiguous(), 0
    slab = turn = None
    while done < count:
        some = []
        while done + len(some) < count and len(some) < max(1, done):
            e = entry(done + len(some))
            if e is None or (some and e[0][4].shape != some[0][0][4].shape):
                break
            some.append(e)
        if not some:
            break
        n, f = len(some), some[0][0][4].shape[0] // 2
        size = lib.b200_layer_saved_bytes(B, L, H, Hkv, d, h, f)
        if slab is None or slab.numel() < size:
            slab = torch.empty(size, dtype=torch.uint8, device=x.device)       # a layer's activations; the next one's take their place
        if n > 1 and turn is None:
            turn = torch.empty((2, T, h), dtype=x.dtype, device=x.device)      # outputs of all layers of a call but the last
        out = torch.empty_like(x)
        to = [turn[i & 1].data_ptr() for i in range(n - 1)] + [out.data_ptr()]
        _launched(lib.b200_stack_fwd(_records(some, L, [slab.data_ptr()] * n, to), n, x.data_ptr(), pos.data_ptr(), B, L, H, Hkv, d,
                                     h, f, eps, int(split) | ACT_ONLY, _lib.stream()), "b200_stack_fwd")
        x, done = out, done + n
    return x, done


def run_stack(x, pos, layers, meta, split):
    """The layers one after the other. ``layers``: (six weights, q/k/v bias or None, cos, sin, window or None) of each, all of
    which ``fits`` accepts. Same kernels, order and bits as a ``NativeLayerFn`` per layer."""
    # one weight stands for all of them in the graph: their gradients go to their slots
    anchor = next((w for ws, b, *_ in layers for w in ws + (b,) if w is not None and w.requires_grad), None)
    return NativeStackFn.apply(x, anchor, pos, layers, meta, split)


def _u64(values):
    return (ctypes.c_uint64 * len(values))(*values)


def _records(layers, L: int, saved: list[int], out: list[int]):
    """B200StackLayer (csrc/ops/layer.cu) of each layer; ``saved`` and ``out``: addresses of its slab and its output."""
    rows = []
    for (ws, b, cos, sin, window), s, o in zip(layers, saved, out):
        rows += [cos.data_ptr(), sin.data_ptr(), *(w.data_ptr() for w in ws), 0 if b is None else b.data_ptr(), s, o,
                 0 if window is None or L <= window else window]
    return _u64(rows)


class NativeStackFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, anchor, pos, layers, meta, split):
        B, L, H, Hkv, d, eps = meta[:6]
        n, (T, h), f = len(layers), x.shape, layers[0][0][4].shape[0] // 2
        lib, x = _lib.kernels(), x.contiguous()
        size = lib.b200_layer_saved_bytes(B, L, H, Hkv, d, h, f)
        saved = torch.empty(size * n, dtype=torch.uint8, device=x.device)
        between = torch.empty((n - 1, T, h), dtype=x.dtype, device=x.device)         # the outputs of all layers but the last
        out = torch.empty_like(x)
        first, bytes_ = between.data_ptr(), T * h * x.element_size()
        rows = _records(layers, L, [saved.data_ptr() + i * size for i in range(n)],
                        [first + i * bytes_ for i in range(n - 1)] + [out.data_ptr()])
        _launched(lib.b200_stack_fwd(rows, n, x.data_ptr(), pos.data_ptr(), B, L, H, Hkv, d, h, f, eps, int(split[0]),
                                     _lib.stream()), "b200_stack_fwd")
        ctx.layers, ctx.meta, ctx.split = layers, meta, split
        ctx.save_for_backward(x, pos, saved, between)
        return out

    @staticmethod
    def backward(ctx, dout):
        from . import llama
        x, pos, saved, between = ctx.saved_tensors
        B, L, H, Hkv, d, eps = ctx.meta[:6]
        n, (T, h), f = len(ctx.layers), x.shape, ctx.layers[0][0][4].shape[0] // 2
        lib, size, bytes_ = _lib.kernels(), saved.numel() // n, T * h * x.element_size()
        dout = dout.contiguous()
        scratch = torch.empty(lib.b200_layer_scratch_bytes(B, L, H, Hkv, d, h, f), dtype=torch.uint8, device=x.device)
        turn = torch.empty((2, T, h), dtype=x.dtype, device=x.device)
        dx, done = torch.empty_like(x), ctypes.c_int(0)
        hooks = llama.UNIT_PRE[0], llama.LAYER_WEIGHTS_PRE[0], llama.LAYER_BACKWARD_DONE[0]
        each = any(k is not None for k in hooks)                 # something happens between layers: one at a time
        slots = [[llama._slot(w) if w is not None else None for w in ws + (b,)] for ws, b, *_ in ctx.layers]
        for last in (range(n - 1, -1, -1) if each else (n - 1,)):
            lo, w_ln1 = last if each else 0, ctx.layers[last][0][0]
            if hooks[0] is not None:
                hooks[0](w_ln1, True)
            if hooks[1] is not None:
                hooks[1](w_ln1)
            grads, written = [], set()                 # addresses are read behind the hooks: they may have moved what lies there
            for i in range(last, lo - 1, -1):
                mine = slots[i]
                acc = sum(1 << k for k, s in enumerate(mine) if s is not None and (not s.fresh or id(s) in written))
                written.update(id(s) for s in mine)
                grads[:0] = [x.data_ptr() if i == 0 else between.data_ptr() + (i - 1) * bytes_,
                             *(0 if s is None else s.buf.data_ptr() for s in mine), acc]
            m, to = last + 1 - lo, dx if lo == 0 else turn[lo & 1]
            rows = _records(ctx.layers[lo:last + 1], L, [saved.data_ptr() + i * size for i in range(lo, last + 1)], [0] * m)
            rc = lib.b200_stack_bwd(rows, _u64(grads), m, dout.data_ptr(), pos.data_ptr(), scratch.data_ptr(), to.data_ptr(),
                                    turn[0].data_ptr(), turn[1].data_ptr(), B, L, H, Hkv, d, h, f, int(ctx.split[1]),
                                    ctypes.byref(done), _lib.stream())
            for mine in slots[last + 1 - done.value:last + 1]:   # also of a call that failed: the layers that did run
                for s in mine:
                    if s is not None:
                        s.fresh = False
            _launched(rc, "b200_stack_bwd")
            dout = to
            if hooks[2] is not None:
                hooks[2](w_ln1)
        return (dx,) + (None,) * 5
