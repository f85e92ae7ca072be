"""Plain encoder layers through a single native call each way (nanoplm_b200/csrc/layer.cpp): the same kernels in the
same order as the op-by-op path of `EncoderLayer`, without the interpreter between the launches.

`run` takes one layer, `run_stack` the layers of an encoder, several to a call and an autograd node. What is not the plain
case is left to the caller, who goes layer by layer and op by op. Plain means: bf16 on a GPU, head
dimension 64, SwiGLU, no biases, dropout, convolution, hyper-connections or experts, no hooks on the parts, no tracer,
forward-mode level or function transform, no weights that are gathered on use, default kernel choices; and either
gradients are off, or every parameter is trained into a running fp32 gradient (`main_grad`) and nobody waits for single
weight gradients. Several layers are not one node under saved-tensor hooks either: those would get all of their tensors
back at once."""
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
               ("attention_ws", "nplm_fa_bwd_ws_zeroed")]
        h.nplm_layer_init((ctypes.c_void_p * len(fns))(
            *[ctypes.cast(getattr(lib(l), f), ctypes.c_void_p).value for l, f in fns]))
        h.nplm_layer_bytes.argtypes = [ctypes.c_longlong] * 4 + [ctypes.c_int] * 3
        h.nplm_layer_bytes.restype = ctypes.c_longlong
        h.nplm_layer_fwd.argtypes = [ctypes.c_void_p] + [ctypes.c_double] * 3
        h.nplm_layer_bwd.argtypes = [ctypes.c_void_p, ctypes.c_double]
        h.nplm_layers_fwd.argtypes = h.nplm_layers_bwd.argtypes = [ctypes.c_void_p, ctypes.c_void_p, ctypes.c_int]
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


def unwatched(module) -> bool:
    """Nobody's hooks on the module's own call, no forward of the instance's own."""
    return _quiet((module,))


def unobserved(parts) -> bool:
    """The modules `parts` may be passed by: nobody watches their calls or the autograd Functions behind them."""
    return not F_.functions_observed() and not _mod._has_any_global_hook() and _quiet(parts)


def _ok_weight(w, rows: int, cols: int) -> bool:
    return (w.dtype == BF and w.is_cuda and w.shape == (rows, cols) and w.is_contiguous() and w.data_ptr() % 16 == 0
            and getattr(w, "_ag", None) is None)


def _plain_call(x, ctx, rope) -> bool:
    """What a plain call asks of everything but the layers: the activations, the batch's metadata and the switches."""
    if not (x.dtype == BF and x.is_cuda and x.dim() == 2 and x.is_contiguous() and x.data_ptr() % 16 == 0
            and x.shape[0] > 0 and not F_.fp8_enabled() and K._FA_IMPL[0] == "ws" and K._GEMM_PAIR_DEFAULT[0] is None
            and type(x) is torch.Tensor) or _mod._has_any_global_hook():
        return False
    pos = ctx.position_ids
    # (what is wrong here is for the op-by-op path to refuse)
    i32, f32, ss, se = torch.int32, torch.float32, ctx.seq_start, ctx.seq_end
    if not (pos.numel() == x.shape[0] and pos.dtype == i32 and ss.dtype == i32 and se.dtype == i32 and pos.is_cuda
            and ss.is_cuda and se.is_cuda and pos.is_contiguous() and ss.is_contiguous() and se.is_contiguous()):
        return False
    for cos, sin in rope:
        if not (cos.dtype == f32 and sin.dtype == f32 and cos.is_cuda and sin.is_cuda and cos.is_contiguous()
                and sin.is_contiguous() and cos.shape[-1] == 32 and sin.shape[-1] == 32):
            return False
    return True


def _plain_layer(attn, mlp, norm1, norm2, C: int, window: int):
    """(parameters, meta) of a layer that qualifies, else None."""
    am, mm = attn._modules, mlp._modules
    wqkv, wo, win, wout = am["Wqkv"], am["Wo"], mm["Wi"], mm["Wo"]
    if not (attn.head_dim == 64 and mlp.swiglu and not (mlp.p_drop > 0.0 and mlp.training)):
        return None
    if (any(l.bias is not None for l in (wqkv, wo, win, wout, norm2))
            or not _quiet((attn, mlp, wqkv, wo, win, wout, norm1, norm2))):
        return None
    n1 = None
    if type(norm1) is not torch.nn.Identity:
        if norm1.bias is not None or norm1.rms != norm2.rms:
            return None
        n1 = norm1.weight
    params = (*[l._parameters.get("weight") for l in (wqkv, wo, win, wout)], n1, norm2.weight)
    if any(w is None for w in params[:4]):      # (reparametrised: a weight that is formed on each call)
        return None
    HD, I = attn.num_heads * 64, params[3].shape[-1]
    if not (C % 64 == 0 and C <= 4096 and I % 64 == 0 and _ok_weight(params[0], 3 * HD, C) and _ok_weight(params[1], C, HD)
            and _ok_weight(params[2], 2 * I, C) and _ok_weight(params[3], C, I)
            and all(n.dtype == BF and n.is_cuda and n.shape == (C,) and n.data_ptr() % 16 == 0
                    for n in params[4:] if n is not None)):
        return None
    return params, (I, attn.num_heads, window, int(n1 is not None), int(norm2.rms),
                    norm1.eps if n1 is not None else 0.0, norm2.eps, attn.scale)


def run(attn, mlp, norm1, norm2, x, ctx, window: int, rope: tuple):
    """attn, mlp, norm2: the layer's Attention, MLP and Norm; norm1: its Norm, or an Identity (first layer). Returns y
    or None."""
    if F_.functions_observed():     # before anything else: a tracer also sees the sizes that the checks below look at
        return None
    if not _plain_call(x, ctx, (rope,)):
        return None
    plain = _plain_layer(attn, mlp, norm1, norm2, x.shape[1], window)
    if plain is None:
        return None
    params, meta = plain
    geo = (ctx.seq_start, ctx.seq_end, ctx.position_ids, *rope)
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


# ------------------------------------------------------------------------------------------ a run of layers
def _layer_args(xp: int, params, geo, meta, T: int, C: int, train: int, buf: int, y: int, tail) -> list:
    """One layer's argument array for a forward call (the backward call's has more after it)."""
    I, H, window, norm1, rms = meta[:5]
    return [T, C, I, H, window, norm1, rms, train, xp, *[p.data_ptr() if p is not None else 0 for p in params], *geo, buf, y,
            *tail]


class _StackFn(torch.autograd.Function):
    """Consecutive layers as one node. refs: per layer (parameters, meta, index of its rotary tables in `tables`)."""

    @staticmethod
    def forward(ctx, x, refs, geo, tables, *params):
        T, C = x.shape
        h, dev = _native(), x.device
        tail = (status_word(dev).data_ptr(), raw_stream())
        bounds = [g.data_ptr() for g in geo]
        ropes = [(c.data_ptr(), s.data_ptr()) for c, s in tables]
        y = torch.empty_like(x)
        bufs, args, floats, xp = [], [], [], x.data_ptr()
        row = (T * C * 2 + 255) // 256 * 256
        for i, (p, meta, t) in enumerate(refs):
            saved = h.nplm_layer_bytes(T, C, meta[0], meta[1], meta[3], 1, 0)
            last = i + 1 == len(refs)
            buf = torch.empty(saved if last else saved + row, dtype=torch.uint8, device=dev)
            bufs.append(buf)
            yp = y.data_ptr() if last else buf.data_ptr() + saved       # a layer's output stays behind what it saves
            args += _layer_args(xp, p, (*bounds, *ropes[t]), meta, T, C, 1, buf.data_ptr(), yp, tail)
            floats += meta[5:8]
            xp = yp
        check_rc(h.nplm_layers_fwd((ctypes.c_longlong * len(args))(*args), (ctypes.c_double * len(floats))(*floats),
                                   len(refs)), "layers_fwd")
        count_launch(sum(6 + meta[3] for _, meta, _ in refs))
        ctx.save_for_backward(x, *bufs, *geo, *[t for pair in tables for t in pair], *params)
        ctx.refs, ctx.n_tables = refs, len(tables)
        return y

    @staticmethod
    def backward(ctx, dy):
        refs = ctx.refs
        n = len(refs)
        x, *rest = ctx.saved_tensors
        bufs, geo, rest = rest[:n], rest[n:n + 3], rest[n + 3:]
        tables, params = rest[:2 * ctx.n_tables], rest[2 * ctx.n_tables:]
        T, C = x.shape
        dy = dy.contiguous()
        h, dev = _native(), x.device
        tail = (status_word(dev).data_ptr(), raw_stream())
        bounds = [g.data_ptr() for g in geo]
        ropes = [t.data_ptr() for t in tables]
        row = (T * C * 2 + 255) // 256 * 256
        scratch_bytes = max(h.nplm_layer_bytes(T, C, m[0], m[1], m[3], 1, 1) for _, m, _ in refs)
        # one layer's gradients at a time: the scratch, and the two activations' gradients in turn
        work = torch.empty(scratch_bytes + 2 * row, dtype=torch.uint8, device=dev)
        scratch = work.data_ptr()
        between = scratch + scratch_bytes           # (a multiple of 256, as every part of these buffers)
        dx = torch.empty_like(x)
        mode = 3 if K._FA_DETERMINISTIC[0] else -1
        args, floats, saved = [], [], iter(params)
        grad_at = lambda i: dy.data_ptr() if i == n else (dx.data_ptr() if i == 0 else between + (i & 1) * row)
        for i, (p, meta, t) in enumerate(refs):
            I, H, norm1 = meta[0], meta[1], meta[3]
            here = [None if q is None else next(saved) for q in p]
            xp = x.data_ptr() if i == 0 else bufs[i - 1].data_ptr() + bufs[i - 1].numel() - row
            a = _layer_args(xp, here, (*bounds, ropes[2 * t], ropes[2 * t + 1]), meta, T, C, 1, bufs[i].data_ptr(),
                            grad_at(i + 1), tail)
            HD = H * 64
            args += [*a, grad_at(i), scratch, *[q.main_grad.data_ptr() if q is not None else 0 for q in p],
                     K.weight_grad_splits(3 * HD, C, T), K.weight_grad_splits(C, HD, T),
                     K.weight_grad_splits(2 * I, C, T), K.weight_grad_splits(C, I, T), mode]
            floats += meta[5:8]
        a, f = (ctypes.c_longlong * len(args))(*args), (ctypes.c_double * len(floats))(*floats)
        size = len(args) // n
        ready = F_._WGRAD_READY[0]
        if ready is None:
            check_rc(h.nplm_layers_bwd(a, f, n), "layers_bwd")
        else:                                   # (set after the forward: told after every layer)
            for i in range(n - 1, -1, -1):
                check_rc(h.nplm_layer_bwd(ctypes.byref(a, 8 * size * i), f[3 * i + 2]), "layer_bwd")
                for q in reversed(refs[i][0][:4]):
                    ready(q)
        count_launch(sum(12 + m[3] for _, m, _ in refs))
        return (dx, *[None] * (3 + len(params)))


def _stack_inference(x, refs, geo, tables):
    T, C = x.shape
    h, dev = _native(), x.device
    tail = (status_word(dev).data_ptr(), raw_stream())
    bounds = [g.data_ptr() for g in geo]
    ropes = [(c.data_ptr(), s.data_ptr()) for c, s in tables]
    n = len(refs)
    row = (T * C * 2 + 255) // 256 * 256
    size = max(h.nplm_layer_bytes(T, C, m[0], m[1], m[3], 0, 0) for _, m, _ in refs)
    work = torch.empty(size + (2 * row if n > 1 else 0), dtype=torch.uint8, device=dev)   # one layer's tensors, two outputs
    y = torch.empty_like(x)
    buf, args, floats, xp = work.data_ptr(), [], [], x.data_ptr()
    for i, (p, meta, t) in enumerate(refs):
        yp = y.data_ptr() if i + 1 == n else buf + size + (i & 1) * row
        args += _layer_args(xp, p, (*bounds, *ropes[t]), meta, T, C, 0, buf, yp, tail)
        floats += meta[5:8]
        xp = yp
    check_rc(h.nplm_layers_fwd((ctypes.c_longlong * len(args))(*args), (ctypes.c_double * len(floats))(*floats), n),
             "layers_fwd")
    count_launch(sum(6 + m[3] for _, m, _ in refs))
    return y


def run_stack(layers, eligible, x, ctx, windows, ropes):
    """Runs layers from the first on, as long as `eligible(layer)` holds and they are plain, with their windows and (cos, sin)
    tables. Returns (output, number of layers run).

    A run is cut into calls of 1, 2, 4 and then 8 layers: the GPU works on one while the next is checked and its arguments
    are gathered (10 - 15 us a layer; all 16 layers of the default encoder in one call kept it waiting for 0.25 ms)."""
    if F_.functions_observed() or not layers:
        return x, 0
    tables, index = [], {}
    for r in ropes:
        if id(r) not in index:
            index[id(r)] = len(tables)
            tables.append(r)
    if not _plain_call(x, ctx, tables):
        return x, 0
    grad = torch.is_grad_enabled()
    if grad and not (x.requires_grad and F_._WGRAD_READY[0] is None
                     and torch._C._autograd._top_saved_tensors_default_hooks(False) is None):
        return x, 0
    C, geo = x.shape[1], (ctx.seq_start, ctx.seq_end, ctx.position_ids)
    done, size, more = 0, 1, True
    while more and done < len(layers):
        refs = []
        for i in range(done, min(done + size, len(layers))):
            layer = layers[i]
            plain = None
            if eligible(layer):
                m = layer._modules
                plain = _plain_layer(m["attn"], m["mlp"], m["attn_norm"], m["mlp_norm"], C, windows[i])
            if plain is None or (grad and not _trained(plain[0])):
                more = False
                break
            refs.append((*plain, index[id(ropes[i])]))
        if refs:
            if grad:
                x = _StackFn.apply(x, refs, geo, tables, *[p for r in refs for p in r[0] if p is not None])
            else:
                x = _stack_inference(x, refs, geo, tables)
        done += len(refs)
        size = min(2 * size, 8)
    return x, done
