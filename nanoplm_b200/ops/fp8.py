"""FP8 (e4m3) block-scaled linear layers: quantisation kernels, the tcgen05 fp8 GEMM with
per-128-K-block promotion (nanoplm_b200/csrc/fp8.cu) and the autograd function that runs forward,
data gradient and weight gradient on e4m3 operands.

Recipe ("block128"): activations and gradients are scaled per 1 x 128 along the contraction axis
of the GEMM that consumes them, weights per 128 x 128; accumulation is fp32; master weights stay
bf16 / fp32 in the optimizer. The reference has no FP8 path (it trains under a bf16
MixedPrecisionPolicy, src/nanoplm/pretraining/pure_pipeline.py:485-487).

Quantised weights are cached per parameter and re-used across the micro-steps of one optimizer
step; `invalidate_weight_cache()` is called by the engines after every parameter update.
"""
from __future__ import annotations

from ctypes import c_int

import torch

from . import kernels as _kernels
from ._lib import check_rc, count_launch, lib, ptr, status_word, stream_ptr

_BF16 = torch.bfloat16
E4M3_MAX = 448.0


class Quantized:
    """e4m3 payload (uint8 view) [rows, K] with fp32 scales stored K-block-major."""
    __slots__ = ("q", "scale", "block")

    def __init__(self, q: torch.Tensor, scale: torch.Tensor, block: bool):
        self.q, self.scale, self.block = q, scale, block

    def dequantize(self) -> torch.Tensor:
        """fp32 tensor of the represented values (test helper)."""
        rows, K = self.q.shape
        v = self.q.view(torch.float8_e4m3fn).float()
        if self.block:
            s = self.scale.view(K // 128, -1)                     # [KB, row blocks]
            s = s.repeat_interleave(128, dim=1)[:, :rows]          # [KB, rows]
        else:
            s = self.scale.view(K // 128, rows)
        return v * s.t().repeat_interleave(128, dim=1)


def quant_rows(x: torch.Tensor) -> Quantized:
    """x bf16 [R, K] (K % 128 == 0) -> e4m3 with 1 x 128 scales along K."""
    R, K = x.shape
    if x.stride(1) != 1:
        x = x.contiguous()
    q = torch.empty((R, K), dtype=torch.uint8, device=x.device)
    s = torch.empty((K // 128, R), dtype=torch.float32, device=x.device)
    rc = lib("fp8").nplm_fp8_quant_rows(ptr(x), c_int(R), c_int(K), c_int(x.stride(0)), ptr(q), ptr(s), stream_ptr())
    check_rc(rc, "fp8_quant_rows")
    count_launch()
    return Quantized(q, s, False)


def quant_tile(x: torch.Tensor, transpose: bool, block: bool) -> Quantized:
    """128 x 128 tile quantisation of x bf16 [R, K].

    transpose=False, block=True : payload [R, K], one scale per 128 x 128 tile (weights)
    transpose=True,  block=True : payload [K, R] (weights for the data-gradient GEMM)
    transpose=True,  block=False: payload [K, R] with 1 x 128 scales along R (operands of the
                                  weight-gradient GEMM, which contracts over tokens)
    """
    R, K = x.shape
    if x.stride(1) != 1:
        x = x.contiguous()
    if transpose:
        q = torch.empty((K, R), dtype=torch.uint8, device=x.device)
        rb = (R + 127) // 128
        s = torch.empty((rb, K // 128) if block else (rb, K), dtype=torch.float32, device=x.device)
    else:
        q = torch.empty((R, K), dtype=torch.uint8, device=x.device)
        s = torch.empty((K // 128, R // 128), dtype=torch.float32, device=x.device)
    rc = lib("fp8").nplm_fp8_quant_tile(ptr(x), c_int(R), c_int(K), c_int(x.stride(0)), c_int(int(transpose)),
                                        c_int(int(block)), ptr(q), ptr(s), stream_ptr())
    check_rc(rc, "fp8_quant_tile")
    count_launch()
    return Quantized(q, s, block)


def quant_dual(x: torch.Tensor) -> tuple[Quantized, Quantized]:
    """(quant_rows(x), quant_tile(x, transpose=True, block=False)) in one pass over x bf16 [R, K], both multiples
    of 128."""
    R, K = x.shape
    if x.stride(1) != 1 or x.stride(0) % 4 or x.data_ptr() % 8:
        x = x.contiguous()
    r, t = _dual_buffers(R, K, x.device)
    rc = lib("fp8").nplm_fp8_quant_dual(ptr(x), c_int(R), c_int(K), c_int(x.stride(0)), ptr(r.q), ptr(r.scale), ptr(t.q),
                                        ptr(t.scale), stream_ptr())
    check_rc(rc, "fp8_quant_dual")
    count_launch()
    return r, t


def _dual_buffers(R: int, K: int, dev) -> tuple[Quantized, Quantized]:
    """Row form and transposed row form of an operand [R, K], to be filled."""
    u8, f32 = torch.uint8, torch.float32
    return (Quantized(torch.empty((R, K), dtype=u8, device=dev), torch.empty((K // 128, R), dtype=f32, device=dev), False),
            Quantized(torch.empty((K, R), dtype=u8, device=dev), torch.empty((R // 128, K), dtype=f32, device=dev), False))


def rope_quant_dual(x: torch.Tensor, rope: tuple) -> tuple[Quantized, Quantized]:
    """quant_dual of x bf16 [R, K] with the rotary embedding rope = (pos int32 [R], cos, sin fp32 [P, 32], rope_cols) undone
    on the 64-wide heads below column rope_cols: the gradient of an un-rotated projection from that of the rotated one."""
    pos, cos, sin, cols = rope
    R, K = x.shape
    if x.stride(1) != 1 or x.stride(0) % 4 or x.data_ptr() % 8:
        x = x.contiguous()
    r, t = _dual_buffers(R, K, x.device)
    rc = lib("fp8").nplm_fp8_rope_quant_dual(ptr(x), c_int(R), c_int(K), c_int(x.stride(0)), ptr(pos), ptr(cos), ptr(sin),
                                             c_int(cols), ptr(r.q), ptr(r.scale), ptr(t.q), ptr(t.scale), stream_ptr())
    check_rc(rc, "fp8_rope_quant_dual")
    count_launch()
    return r, t


def swiglu_quant_dual(pre: torch.Tensor) -> tuple[Quantized, Quantized]:
    """quant_dual(swiglu(pre)) for pre = [value | gate] bf16 [R, 2 I] contiguous, R and I multiples of 128."""
    R, I = pre.shape[0], pre.shape[1] // 2
    r, t = _dual_buffers(R, I, pre.device)
    rc = lib("fp8").nplm_fp8_swiglu_quant_dual(ptr(pre), c_int(R), c_int(I), ptr(r.q), ptr(r.scale), ptr(t.q),
                                               ptr(t.scale), stream_ptr())
    check_rc(rc, "fp8_swiglu_quant_dual")
    count_launch()
    return r, t


def swiglu_bwd_quant_dual(pre: torch.Tensor, dh: torch.Tensor) -> tuple[Quantized, Quantized]:
    """quant_dual of the gradient of pre (bf16 [R, 2 I]) from that of h = swiglu(pre) (bf16 [R, I]), both contiguous."""
    R, I = dh.shape
    r, t = _dual_buffers(R, 2 * I, pre.device)
    rc = lib("fp8").nplm_fp8_swiglu_bwd_quant_dual(ptr(pre), ptr(dh), c_int(R), c_int(I), ptr(r.q), ptr(r.scale),
                                                   ptr(t.q), ptr(t.scale), stream_ptr())
    check_rc(rc, "fp8_swiglu_bwd_quant_dual")
    count_launch()
    return r, t


def gemm_fp8_form(a: Quantized, b: Quantized, *, residual: torch.Tensor | None = None,
                  rope: tuple | None = None) -> torch.Tensor:
    """bf16 deq(a) deq(b)^T + residual, or with the rotary embedding of rope = (pos int32 [M], cos, sin fp32 [P, 32],
    rope_cols) on the 64-wide heads below column rope_cols; b block-scaled. The bits of the product in bf16 followed by the
    separate pass."""
    M, K = a.q.shape
    N = b.q.shape[0]
    out = torch.empty((M, N), dtype=_BF16, device=a.q.device)
    pos, cos, sin, cols = rope if rope is not None else (None, None, None, 0)
    if residual is not None and (residual.dtype != _BF16 or tuple(residual.shape) != (M, N) or residual.stride(1) != 1):
        raise ValueError("the residual must be a row-major bf16 [M, N] tensor")
    if rope is not None and (pos.dtype != torch.int32 or pos.numel() != M or cos.dtype != torch.float32
                             or sin.dtype != torch.float32 or cos.shape[-1] != 32 or sin.shape[-1] != 32):
        raise ValueError("rope needs int32 positions [M] and fp32 tables [P, 32]")
    rc = lib("fp8").nplm_gemm_fp8_form(ptr(a.q), ptr(b.q), ptr(out), ptr(residual), ptr(a.scale), ptr(b.scale), c_int(M),
                                       c_int(N), c_int(K), c_int(N), c_int(residual.stride(0) if residual is not None else 0),
                                       ptr(pos), ptr(cos), ptr(sin), c_int(cols), ptr(status_word(a.q.device)),
                                       stream_ptr())
    check_rc(rc, "gemm_fp8_form")
    count_launch()
    return out


def gemm_fp8(a: Quantized, b: Quantized, *, out: torch.Tensor | None = None, out_dtype=_BF16,
             accumulate: bool = False) -> torch.Tensor:
    """C[M,N] (+)= deq(a) deq(b)^T. a: row-scaled [M,K]; b: row- or block-scaled [N,K]. With accumulate several work
    items may add to a tile, in any order; under `kernels.set_attention_deterministic` one does."""
    if a.block:
        raise ValueError("the A operand must carry 1 x 128 scales")
    M, K = a.q.shape
    N, Kb = b.q.shape
    if K != Kb:
        raise ValueError(f"inner dims differ: {K} vs {Kb}")
    if out is None:
        if accumulate:
            raise ValueError("accumulate needs an fp32 out tensor")
        out = torch.empty((M, N), dtype=out_dtype, device=a.q.device)
    mode = 0 if out.dtype == _BF16 else (2 if accumulate else 1)
    if out.dtype not in (_BF16, torch.float32) or tuple(out.shape) != (M, N) or out.stride(1) != 1:
        raise ValueError("out must be a row-major bf16 or fp32 [M, N] tensor")
    rc = lib("fp8").nplm_gemm_fp8(ptr(a.q), ptr(b.q), ptr(out), ptr(a.scale), ptr(b.scale), c_int(M), c_int(N),
                                  c_int(K), c_int(out.stride(0)), c_int(int(b.block)), c_int(mode),
                                  c_int(int(_kernels._FA_DETERMINISTIC[0])), ptr(status_word(a.q.device)),
                                  stream_ptr())
    check_rc(rc, "gemm_fp8")
    count_launch()
    return out


def gemm_fp8_ag(a: Quantized, b_payload: torch.Tensor, b_payload_ptrs, b_scale: torch.Tensor, b_scale_ptrs,
                rank: int, world: int, flags: torch.Tensor, *, out: torch.Tensor | None = None) -> torch.Tensor:
    """All-gather fused into the fp8 GEMM: C = deq(a) deq(B)^T with B's rows (e4m3 payload [N,K] and
    block scales [K/128, N/128]) sharded over `world` ranks in peer-mapped memory. b_payload /
    b_scale are this rank's full-size buffers (only its shard valid on entry, everything valid on
    return); *_ptrs are the ctypes arrays of every rank's buffer addresses. The fp8 payload moves
    half the bytes of a bf16 gather. flags: int32 [8]."""
    M, K = a.q.shape
    N = b_payload.shape[0]
    if out is None:
        out = torch.empty((M, N), dtype=_BF16, device=a.q.device)
    mode = 0 if out.dtype == _BF16 else 1
    rc = lib("fp8").nplm_gemm_fp8_ag(ptr(a.q), b_payload_ptrs, ptr(out), ptr(a.scale), b_scale_ptrs, c_int(M),
                                     c_int(N), c_int(K), c_int(out.stride(0)), c_int(mode), c_int(rank),
                                     c_int(world), ptr(flags), ptr(status_word(a.q.device)), stream_ptr())
    check_rc(rc, "gemm_fp8_ag")
    count_launch()
    return out


# ------------------------------------------------------------------------------ weight cache
_weight_cache: dict[int, tuple] = {}


def invalidate_weight_cache() -> None:
    _weight_cache.clear()


def _quantized_weight(w: torch.Tensor):
    """(W as [N,K] block-scaled, W^T as [K,N] block-scaled) for this parameter version."""
    key = id(w)
    hit = _weight_cache.get(key)
    if hit is not None and hit[0] == w.data_ptr():
        return hit[1], hit[2]
    qw = quant_tile(w.detach(), transpose=False, block=True)
    qwt = quant_tile(w.detach(), transpose=True, block=True)
    _weight_cache[key] = (w.data_ptr(), qw, qwt)
    return qw, qwt


def supported(x: torch.Tensor, w: torch.Tensor) -> bool:
    """Shapes the fp8 path covers: bf16 CUDA tensors, both weight dims multiples of 128."""
    return (x.is_cuda and x.dtype == _BF16 and w.dtype == _BF16 and w.shape[0] % 128 == 0
            and w.shape[1] % 128 == 0)


def addable(residual: torch.Tensor, x: torch.Tensor, w: torch.Tensor) -> bool:
    """Whether the product's epilogue can add `residual`: bf16 rows of the output's shape on 16-byte boundaries, and nobody
    who has to see the sum itself (a tangent of the residual alone goes through a sum, but not through the product's node)."""
    from .functional import functions_observed
    if functions_observed():
        return False
    if residual.dtype != _BF16 or not residual.is_cuda or residual.shape != (*x.shape[:-1], w.shape[0]):
        return False
    r = residual.reshape(-1, w.shape[0])
    return r.stride(1) == 1 and r.stride(0) % 8 == 0 and r.data_ptr() % 16 == 0


def _dual_rows(T: int) -> bool:
    """Token counts for which the weight gradient runs on e4m3 operands (whole 128-token scale blocks)."""
    return T % 128 == 0 and T // 128 <= 65535


def _weight_gradient(qdy_t: Quantized, qx_t: Quantized, p):
    """dW [N, K] = dY^T X from the token-contiguous payloads; into p.main_grad, or returned."""
    from .functional import _has_main_grad
    if _has_main_grad(p):
        gemm_fp8(qdy_t, qx_t, out=p.main_grad.view(p.shape), accumulate=True)
        return None
    return gemm_fp8(qdy_t, qx_t, out_dtype=torch.float32).to(p.dtype)


class _Fp8LinearFn(torch.autograd.Function):
    @staticmethod
    def forward(ctx, x, w, train, residual, rope):
        from .functional import _as_shape
        x2 = x.reshape(-1, x.shape[-1])
        qw, _ = _quantized_weight(w)
        ctx.dual = train and ctx.needs_input_grad[1] and _dual_rows(x2.shape[0])
        if ctx.dual:      # the weight gradient's form of x comes from the same pass; x itself need not be kept
            qx, qx_t = quant_dual(x2)
            ctx.save_for_backward(qx_t.q, qx_t.scale, w)
        else:
            qx = quant_rows(x2)
            ctx.save_for_backward(x2, w)
        if residual is None and rope is None:
            y = gemm_fp8(qx, qw)
        else:
            y = gemm_fp8_form(qx, qw, residual=None if residual is None else residual.reshape(-1, w.shape[0]), rope=rope)
        ctx.has_res = residual is not None
        ctx.w_ref = w
        ctx.rope = rope
        ctx.shape = x.shape
        return _as_shape(y, (*x.shape[:-1], w.shape[0]))

    @staticmethod
    def backward(ctx, dy):
        from .functional import _as_shape, _wgrad
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        dx = dw = qdy = qdy_t = None
        if ctx.rope is not None and not (ctx.dual and ctx.needs_input_grad[0]):
            pos, cos, sin, cols = ctx.rope
            dy2 = _kernels.rope_(dy2.clone(), pos, cos, sin, cols // 128, 64, backward=True)   # (q and k: two thirds)
        if ctx.dual:
            qx_t, sx_t, _ = ctx.saved_tensors
            if ctx.needs_input_grad[0]:
                qdy, qdy_t = quant_dual(dy2) if ctx.rope is None else rope_quant_dual(dy2, ctx.rope)
            else:
                qdy_t = quant_tile(dy2, transpose=True, block=False)
        elif ctx.needs_input_grad[0]:
            qdy = quant_rows(dy2)
        if ctx.needs_input_grad[0]:
            _, qwt = _quantized_weight(ctx.w_ref)
            dx = _as_shape(gemm_fp8(qdy, qwt), ctx.shape)
        if ctx.dual:
            dw = _weight_gradient(qdy_t, Quantized(qx_t, sx_t, False), ctx.w_ref)
        elif ctx.needs_input_grad[1]:
            dw = _wgrad(dy2, ctx.saved_tensors[0], ctx.w_ref)
        return dx, dw, None, (dy if ctx.has_res else None), None


def fp8_linear(x: torch.Tensor, w: torch.Tensor, residual: torch.Tensor | None = None,
               rope: tuple | None = None) -> torch.Tensor:
    """y = x W^T with e4m3 operands (no bias), plus the residual or with the rotary embedding of `gemm_fp8_form` (q and k of a
    packed QKV projection: two thirds of its columns) in the product's epilogue and its inverse in the quantisation of the
    incoming gradient."""
    from .functional import _keeps
    return _Fp8LinearFn.apply(x, w, _keeps(), residual, rope)


class _Fp8MlpFn(torch.autograd.Function):
    """SwiGLU MLP + residual on e4m3 operands as one node: the activation exists only as the quantised operands of the two
    products that read it, and so do the gradients of the pre-activations. Whole 128-token blocks, training."""

    @staticmethod
    def forward(ctx, x, w_in, w_out, residual):
        from .functional import _as_shape
        x2 = x.reshape(-1, x.shape[-1])
        qx, qx_t = quant_dual(x2)
        pre = gemm_fp8(qx, _quantized_weight(w_in)[0])
        qh, qh_t = swiglu_quant_dual(pre)
        qw = _quantized_weight(w_out)[0]
        if residual is None:
            y = gemm_fp8(qh, qw)
        else:
            y = gemm_fp8_form(qh, qw, residual=residual.reshape(-1, w_out.shape[0]))
        ctx.save_for_backward(qx_t.q, qx_t.scale, pre, qh_t.q, qh_t.scale, w_in, w_out)
        ctx.refs = (w_in, w_out)
        ctx.has_res = residual is not None
        ctx.x_shape = x.shape
        return _as_shape(y, (*x.shape[:-1], y.shape[1]))

    @staticmethod
    def backward(ctx, dy):
        from .functional import _as_shape
        qx_t, sx_t, pre, qh_t, sh_t, _, _ = ctx.saved_tensors
        w_in, w_out = ctx.refs
        dy2 = dy.reshape(-1, dy.shape[-1])
        if not dy2.is_contiguous():
            dy2 = dy2.contiguous()
        qdy, qdy_t = quant_dual(dy2)
        dh = gemm_fp8(qdy, _quantized_weight(w_out)[1])
        dw_out = _weight_gradient(qdy_t, Quantized(qh_t, sh_t, False), w_out) if ctx.needs_input_grad[2] else None
        qd, qd_t = swiglu_bwd_quant_dual(pre, dh)
        dw_in = _weight_gradient(qd_t, Quantized(qx_t, sx_t, False), w_in) if ctx.needs_input_grad[1] else None
        dx = (_as_shape(gemm_fp8(qd, _quantized_weight(w_in)[1]), ctx.x_shape) if ctx.needs_input_grad[0] else None)
        return dx, dw_in, dw_out, (dy if ctx.has_res else None)


def mlp_fused(x: torch.Tensor, w_in: torch.Tensor, w_out: torch.Tensor, residual: torch.Tensor | None = None) -> bool:
    """Whether `fp8_mlp` takes a call: both projections fit (`supported`, whole 128-column halves), whole 128-token blocks, a
    residual that the epilogue can add, and a backward pass for both weights."""
    from .functional import _keeps, functions_observed
    inter = w_out.shape[1]
    return (not functions_observed() and supported(x, w_in) and supported(x, w_out) and w_in.shape[0] == 2 * inter
            and w_in.shape[1] == x.shape[-1] and x.numel() > 0 and _dual_rows(x.numel() // x.shape[-1]) and _keeps()
            and w_in.requires_grad and w_out.requires_grad and (residual is None or addable(residual, x, w_out)))


def fp8_mlp(x, w_in, w_out, residual=None):
    """(silu(gate) * value) W_out^T + residual with [value | gate] = x W_in^T, e4m3 operands throughout."""
    return _Fp8MlpFn.apply(x, w_in, w_out, residual)
