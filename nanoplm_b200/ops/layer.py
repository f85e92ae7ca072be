"""One plain encoder layer through a single native call each way (nanoplm_b200/csrc/layer.cpp): the same kernels in the
same order as the op-by-op path of `EncoderLayer`, without the interpreter between the launches.

`run` returns None when the call is not the plain case; the caller then goes op by op. Plain means: bf16 on a GPU, head
dimension 64, SwiGLU, no biases, dropout, convolution, hyper-connections or experts, no hooks on the parts, no tracer,
forward-mode level or function transform, no weights that are gathered on use, default kernel choices; and either
gradients are off, or every parameter is trained into a running fp32 gradient (`main_grad`) and nobody waits for single
weight gradients."""
from __future__ import annotations

import ctypes

import torch
import torch.nn.modules.module as _mod

from . import functional as F_
from . import kernels as K
from ._lib import check_rc, count_launch, lib, raw_stream, status_word

BF = torch.bfloat16
_READY = [None]
_FwdArgs, _BwdArgs = ctypes.c_longlong * 24, ctypes.c_longlong * 37


def _native():
    if _READY[0] is None:
        h = lib("layer")
        if (h.nplm_layer_args(0), h.nplm_layer_args(1)) != (_FwdArgs._length_, _BwdArgs._length_):
            raise RuntimeError("the argument arrays of csrc/layer.cpp have changed")
        fns = [("gemm_tcgen05", "nplm_gemm_bf16"), ("gemm_tcgen05", "nplm_gemm_bf16_pair"),
               ("gemm_tcgen05", "nplm_gemm_bf16_delta"), ("elementwise", "nplm_norm_fwd"),
               ("elementwise", "nplm_norm_bwd"), ("attention_ws", "nplm_fa_fwd_ws"),
               ("attention_ws", "nplm_fa_bwd_ws_mode")]
        h.nplm_layer_init((ctypes.c_void_p * len(fns))(
            *[ctypes.cast(getattr(lib(l), f), ctypes.c_void_p).value for l, f in fns]))
        h.nplm_layer_bytes.argtypes = [ctypes.c_longlong] * 4 + [ctypes.c_int] * 3
        h.nplm_layer_bytes.restype = ctypes.c_longlong
        h.nplm_layer_fwd.argtypes = [ctypes.c_void_p] + [ctypes.c_double] * 3
        h.nplm_layer_bwd.argtypes = [ctypes.c_void_p, ctypes.c_double]
        _READY[0] = h
    return _READY[0]


def _forward(x, params, geo, meta, train: bool):
    """geo: (seq_start, seq_end, pos, cos, sin); meta: (I, H, window, norm1, rms, eps1, eps2, scale).
    Returns (y, the buffer the backward pass reads)."""
    I, H, window, norm1, rms, eps1, eps2, scale = meta
    T, C = x.shape
    h = _native()
    buf = torch.empty(h.nplm_layer_bytes(T, C, I, H, norm1, train, 0), dtype=torch.uint8, device=x.device)
    y = torch.empty_like(x)
    a = _FwdArgs(T, C, I, H, window, norm1, rms, train, x.data_ptr(), *[p.data_ptr() if p is not None else 0 for p in params],
                 *[g.data_ptr() for g in geo], buf.data_ptr(), y.data_ptr(), status_word(x.device).data_ptr(), raw_stream())
    check_rc(h.nplm_layer_fwd(a, eps1, eps2, scale), "layer_fwd")
    count_launch(6 + norm1)
    return y, buf


class _LayerFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w_qkv, w_o, w_in, w_out, n1, n2, geo, meta):
        params = (w_qkv, w_o, w_in, w_out, n1, n2)
        y, buf = _forward(x, params, geo, meta, True)
        ctx.save_for_backward(x, buf, *params, *geo)
        ctx.meta = meta
        ctx.refs = params       # saved-tensor hooks may give back copies, which do not carry the running gradients
        return y

    @staticmethod
    def backward(ctx, dy):
        x, buf, *rest = ctx.saved_tensors
        params, geo = rest[:6], rest[6:]
        I, H, window, norm1, rms, _, _, scale = ctx.meta
        T, C = x.shape
        dy = dy.contiguous()
        h = _native()
        dx = torch.empty_like(x)
        scratch = torch.empty(h.nplm_layer_bytes(T, C, I, H, norm1, 1, 1), dtype=torch.uint8, device=x.device)
        grads = [p.main_grad.data_ptr() if p is not None else 0 for p in ctx.refs]
        HD = H * 64
        a = _BwdArgs(T, C, I, H, window, norm1, rms, 1, x.data_ptr(), *[p.data_ptr() if p is not None else 0 for p in params],
                     *[g.data_ptr() for g in geo], buf.data_ptr(), dy.data_ptr(), status_word(x.device).data_ptr(),
                     raw_stream(), dx.data_ptr(), scratch.data_ptr(), *grads, K.weight_grad_splits(3 * HD, C, T),
                     K.weight_grad_splits(C, HD, T), K.weight_grad_splits(2 * I, C, T), K.weight_grad_splits(C, I, T),
                     3 if K._FA_DETERMINISTIC[0] else -1)
        check_rc(h.nplm_layer_bwd(a, scale), "layer_bwd")
        count_launch(12 + norm1)
        if F_._WGRAD_READY[0] is not None:      # (set after this layer's forward)
            for p in reversed(ctx.refs[:4]):
                F_._WGRAD_READY[0](p)
        return dx, None, None, None, None, None, None, None, None


def _quiet(parts) -> bool:
    """No hooks of any kind on modules whose calls would be passed by, and no forward of an instance's own."""
    for m in parts:
        d = m.__dict__
        if (d["_forward_hooks"] or d["_forward_pre_hooks"] or d["_backward_hooks"] or d["_backward_pre_hooks"]
                or "forward" in d):
            return False
    return True


def unobserved(parts) -> bool:
    """The modules `parts` may be passed by: nobody watches their calls or the autograd Functions behind them."""
    return not F_.functions_observed() and not _mod._has_any_global_hook() and _quiet(parts)


def _ok_weight(w, rows: int, cols: int) -> bool:
    return (w.dtype == BF and w.is_cuda and w.shape == (rows, cols) and w.is_contiguous() and w.data_ptr() % 16 == 0
            and getattr(w, "_ag", None) is None)


def run(attn, mlp, norm1, norm2, x, ctx, window: int, rope: tuple):
    """attn, mlp, norm2: the layer's Attention, MLP and Norm; norm1: its Norm, or an Identity (first layer). Returns y
    or None."""
    if F_.functions_observed():     # before anything else: a tracer also sees the sizes that the checks below look at
        return None
    am, mm = attn._modules, mlp._modules
    wqkv, wo, win, wout = am["Wqkv"], am["Wo"], mm["Wi"], mm["Wo"]
    if not (x.dtype == BF and x.is_cuda and x.dim() == 2 and x.is_contiguous() and x.data_ptr() % 16 == 0
            and x.shape[0] > 0 and attn.head_dim == 64 and mlp.swiglu and not (mlp.p_drop > 0.0 and mlp.training)
            and not F_.fp8_enabled() and K._FA_IMPL[0] == "ws" and K._GEMM_PAIR_DEFAULT[0] is None
            and type(x) is torch.Tensor):
        return None
    parts = (attn, mlp, wqkv, wo, win, wout, norm1, norm2)
    if (any(l.bias is not None for l in (wqkv, wo, win, wout, norm2)) or not _quiet(parts)
            or _mod._has_any_global_hook()):
        return None
    n1 = None
    if type(norm1) is not torch.nn.Identity:
        if norm1.bias is not None or norm1.rms != norm2.rms:
            return None
        n1 = norm1.weight
    params = (*[l._parameters.get("weight") for l in (wqkv, wo, win, wout)], n1, norm2.weight)
    if any(w is None for w in params[:4]):      # (reparametrised: a weight that is formed on each call)
        return None
    C, HD, I = x.shape[1], attn.num_heads * 64, params[3].shape[-1]
    if not (C % 64 == 0 and C <= 4096 and I % 64 == 0 and _ok_weight(params[0], 3 * HD, C) and _ok_weight(params[1], C, HD)
            and _ok_weight(params[2], 2 * I, C) and _ok_weight(params[3], C, I)
            and all(n.dtype == BF and n.is_cuda and n.shape == (C,) and n.data_ptr() % 16 == 0
                    for n in params[4:] if n is not None)):
        return None
    cos, sin = rope
    pos = ctx.position_ids
    # (what is wrong here is for the op-by-op path to refuse)
    i32, f32, ss, se = torch.int32, torch.float32, ctx.seq_start, ctx.seq_end
    if not (pos.numel() == x.shape[0] and pos.dtype == i32 and ss.dtype == i32 and se.dtype == i32 and pos.is_cuda
            and ss.is_cuda and se.is_cuda and pos.is_contiguous() and ss.is_contiguous() and se.is_contiguous()
            and cos.dtype == f32 and sin.dtype == f32 and cos.is_cuda and sin.is_cuda and cos.is_contiguous()
            and sin.is_contiguous() and cos.shape[-1] == 32 and sin.shape[-1] == 32):
        return None
    geo = (ss, se, pos, cos, sin)
    meta = (I, attn.num_heads, window, int(n1 is not None), int(norm2.rms),
            norm1.eps if n1 is not None else 0.0, norm2.eps, attn.scale)
    if torch.is_grad_enabled():
        if not (x.requires_grad and F_._WGRAD_READY[0] is None and _trained(params)):
            return None
        return _LayerFn.apply(x, *params, geo, meta)
    return _forward(x, params, geo, meta, False)[0]


def _trained(params) -> bool:
    """Every parameter requires a gradient and has a running fp32 one of its shape."""
    f32 = torch.float32
    for p in params:
        if p is not None:
            g = getattr(p, "main_grad", None)
            if (g is None or not p.requires_grad or g.dtype != f32 or not g.is_cuda or g.shape != p.shape
                    or not g.is_contiguous() or g.data_ptr() % 16):
                return False
    return True
