"""A decoder layer of a training step as one autograd function, whose kernels one native call issues in each direction
(``csrc/decoder_train.cu``)."""
from __future__ import annotations

from ctypes import c_float, c_int, c_longlong

import torch

from . import _adjacent_alias, _grad_to
from . import cuda as cu

HEAD = 128              # head size of the attention kernels' backward pass
_WORDS = ("qkv", "o", "gate_up", "down", "norm1", "norm2", "g_qkv", "g_o", "g_gate_up", "g_down", "g_norm1", "g_norm2", "x", "residual",
          "y", "h", "kept", "dy", "dh", "dx", "work", "norm_scratch", "delta", "kv_acc", "cos", "sin", "slopes", "pos", "row_start", "err",
          "T", "W", "Hq", "Hk", "F", "table_rows", "pairs", "launches", "failed")
_AT = {n: i for i, n in enumerate(_WORDS)}
_PARTS = ("", "rmsnorm", "gemm", "rope", "flash_attn", "swiglu")
# the weights of a layer in the order of the function's arguments, and those whose products are one
GROUPS = (("qkv", 0, 3), ("o", 3, 4), ("gate_up", 4, 6), ("down", 6, 7), ("norm1", 7, 8), ("norm2", 8, 9))
STEPS = ("norm1", "qkv", "o", "norm2", "gate_up", "down")


def _words(tensors, **sizes):
    args = (c_longlong * len(_WORDS))()
    for name, t in tensors.items():
        args[_AT[name]] = 0 if t is None else t.data_ptr()
    for name, n in sizes.items():
        args[_AT[name]] = n
    return args


def _issue(args, backward, eps, scale):
    pairs = args[_AT["pairs"]]
    rc = cu.lib().ell_decoder_layer(args, c_int(backward), c_float(eps), c_float(scale), cu._stream())
    if pairs and not args[_AT["pairs"]]:
        cu.pairs_refused("of a layer")
    cu._check(rc, f"decoder_layer ({_PARTS[args[_AT['failed']]]})" if rc else "decoder_layer")
    cu.LAUNCHES += args[_AT["launches"]] - 1


class TrainPlan:
    """What a layer's call needs besides the rows and the weights: weights that are applied together as one (aliases), sizes, tables."""

    def __init__(self, fused, hq, hk, ff, cos, sin, pos, row_start, slopes, eps, scale):
        self.fused = fused                     # qkv, o, gate and up, down, both norms
        self.tables = {"cos": cos, "sin": sin, "pos": pos, "row_start": row_start, "slopes": slopes}
        self.sizes = {"Hq": hq, "Hk": hk, "F": ff, "table_rows": 0 if cos is None else cos.shape[0]}
        self.eps, self.scale = eps, scale


class _DecoderLayer(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, residual, plan, *weights):
        y, h = torch.empty_like(x), torch.empty_like(x)
        names = [n for n, _, _ in GROUPS]
        tensors = dict(zip(names, plan.fused), x=x, residual=residual, y=y, h=h, err=cu.err_flag(x.device), **plan.tables)
        args = _words(tensors, T=x.shape[0], W=x.shape[1], pairs=cu.gemm_pair_enabled(), **plan.sizes)
        kept = torch.empty(cu.lib().ell_decoder_layer_kept(args), dtype=torch.uint8, device=x.device)
        args[_AT["kept"]] = kept.data_ptr()
        _issue(args, 0, plan.eps, plan.scale)
        ctx.save_for_backward(x if residual is None else None, h, kept, *plan.fused, *plan.tables.values())
        ctx.meta = (residual is not None, plan.sizes, plan.eps, plan.scale)
        ctx.wrefs = weights
        return y, h

    @staticmethod
    def backward(ctx, dy, dh):
        has_residual, sizes, eps, scale = ctx.meta
        x, h, kept, *rest = ctx.saved_tensors
        T, W = h.shape
        names = [n for n, _, _ in GROUPS]
        dy, dh = dy.contiguous(), dh.contiguous()
        dx, f32, hq, hk = torch.empty_like(h), torch.float32, sizes["Hq"], sizes["Hk"]
        tensors = dict(zip(names, rest[:len(names)]), x=x, residual=h if has_residual else None, h=h, kept=kept, dy=dy, dh=dh, dx=dx,
                       err=cu.err_flag(h.device), delta=cu.scratch(T * hq, tag="fa_bwd_delta"),
                       kv_acc=cu.scratch(2 * T * hk * HEAD, tag="fa_bwd_dkv") if hq > hk else None,
                       norm_scratch=cu.scratch(cu.lib().ell_rmsnorm_bwd_scratch_elems(c_int(T), c_int(W)), tag="rmsnorm_bwd"),
                       **dict(zip(("cos", "sin", "pos", "row_start", "slopes"), rest[len(names):])))
        grads, later = [None] * len(ctx.wrefs), []
        first = _first_step(ctx, 1 + has_residual)
        for name, a, b in GROUPS:
            if STEPS.index(name) < first:
                continue
            ws = ctx.wrefs[a:b]
            target = _main_grads(ws)
            if target is None:                 # added up apart; into each main_grad, or to autograd if one is missing
                target = torch.zeros(sum(w.shape[0] for w in ws), *ws[0].shape[1:], dtype=f32, device=h.device)
                later.append((a, ws, target))
            tensors["g_" + name] = target
        args = _words(tensors, T=T, W=W, pairs=cu.gemm_pair_enabled(), **sizes)
        work = torch.empty(cu.lib().ell_decoder_layer_work(args), dtype=torch.uint8, device=h.device)
        args[_AT["work"]] = work.data_ptr()
        _issue(args, 1, eps, scale)
        for a, ws, target in later:
            to_main = all(getattr(w, "main_grad", None) is not None for w in ws)
            for i, (w, g) in enumerate(zip(ws, target.split([w.shape[0] for w in ws]))):
                grads[a + i] = _grad_to(w, g) if to_main else g.to(w.dtype)
        if first > 0:
            dx = None
        return (dx, dx if has_residual else None, None, *grads)


def _first_step(ctx, rows):
    """The step of the layer (``STEPS``) up to which the backward pass under way has to go: the first whose weights, or whose rows, it
    asks for (``torch.autograd.grad`` may ask for less than all).  What lies in front of it gets no gradients, as with a function a step."""
    nodes = [n for n, _ in ctx.next_functions]
    if any(_runs(n) for n in nodes[:rows]):
        return 0
    places = {name: any(_runs(n) for n in nodes[rows + a:rows + b]) for name, a, b in GROUPS}
    return next((i for i, name in enumerate(STEPS) if places[name]), 0)


def _runs(node):
    if node is None:
        return False
    try:
        return torch._C._will_engine_execute_node(node)
    except RuntimeError:                       # a leaf whose gradient torch.autograd.grad returns
        return True


def _main_grads(weights):
    """The fp32 ``main_grad`` of ``weights`` as one tensor, or None where they are missing or apart."""
    gs = [getattr(w, "main_grad", None) for w in weights]
    for g, w in zip(gs, weights):              # what a product is not added to
        if g is not None and w.dim() == 2 and (g.dtype != torch.float32 or not g.is_contiguous() or g.shape != w.shape):
            raise ValueError(f"main_grad {tuple(g.shape)} {g.dtype}: expected contiguous fp32 of the weight's shape {tuple(w.shape)}")
    if any(g is None or g.dtype != torch.float32 or not g.is_contiguous() or g.shape != w.shape or g.data_ptr() & 15 for g, w in zip(gs, weights)):
        return None
    return gs[0] if len(gs) == 1 else _adjacent_alias(gs)


def rows_ok(x):
    """Whether a layer's call takes the rows ``x [T, W]``."""
    return x.is_cuda and x.dtype == torch.bfloat16 and x.dim() == 2 and x.is_contiguous() and not x.data_ptr() & 15 and x.shape[0] > 0


def train_layer(x, residual, plan, weights):
    """``(y, h)`` of a layer: norm of ``x + residual``, attention, norm of its sum ``h`` with the stream, gated feed-forward ``y``.
    ``weights``: q, k, v, o, gate, up, down, both norms, whose fp32 ``main_grad`` takes their gradients."""
    return _DecoderLayer.apply(x, residual, plan, *weights)
