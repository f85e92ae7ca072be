"""e4m3 products with an epilogue, and quantisation fused with SwiGLU, against the separate passes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _randn(*s, scale=1.0):
    return (torch.randn(*s, device="cuda") * scale).to(BF)


def _operands(M, N, K):
    from nanoplm_b200.ops import fp8
    return fp8.quant_rows(_randn(M, K)), fp8.quant_tile(_randn(N, K, scale=K ** -0.5), transpose=False, block=True)


# both tile widths (the wide one from 74 wide tiles), ragged last rows, half a wide tile of columns
@pytest.mark.parametrize("M,N,K", [(1, 384, 128), (130, 384, 256), (1000, 768, 128), (9601, 384, 256), (5000, 768, 1024)])
def test_residual_and_rotary_epilogues(M, N, K, cuda_status):
    """Bit for bit the product followed by the separate pass."""
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import functional as F_
    from nanoplm_b200.ops import kernels as k
    torch.manual_seed(M)
    a, b = _operands(M, N, K)
    product = fp8.gemm_fp8(a, b)
    res = _randn(M, N + 64)[:, :N]                               # (a row stride of its own)
    assert torch.equal(fp8.gemm_fp8_form(a, b, residual=res), product + res)
    rope = _rope(M)
    want = k.rope_(product.clone(), *rope, N // 192, 64)
    assert torch.equal(fp8.gemm_fp8_form(a, b, rope=(*rope, N // 3 * 2)), want)


def _rope(M):
    from nanoplm_b200.ops import functional as F_
    return (torch.randint(0, 300, (M,), device="cuda", dtype=torch.int32),
            *F_.rope_tables(300, 64, 10000.0, torch.device("cuda")))


@pytest.mark.parametrize("R,N", [(128, 384), (1152, 768), (256, 3072)])
def test_rotary_gradient_with_quantisation(R, N, cuda_status):
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import kernels as k
    torch.manual_seed(R)
    d, rope = _randn(R, N), _rope(R)
    want = fp8.quant_dual(k.rope_(d.clone(), *rope, N // 192, 64, backward=True))
    for got, ref in zip(fp8.rope_quant_dual(d, (*rope, N // 3 * 2)), want):
        assert torch.equal(got.q, ref.q) and torch.equal(got.scale, ref.scale)


@pytest.mark.parametrize("T", [256, 200])        # whole 128-token blocks, and not
@pytest.mark.parametrize("train_input", [True, False])
def test_rotary_projection_is_the_two_nodes(T, train_input, cuda_status):
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import functional as F_
    torch.manual_seed(T)
    x0, w0, dy, rope = _randn(T, 128), _randn(384, 128, scale=0.1), _randn(T, 384), _rope(T)

    def run(fused):
        fp8.invalidate_weight_cache()
        x, w = x0.clone().requires_grad_(train_input), w0.clone().requires_grad_(True)
        w.main_grad = torch.zeros(w.shape, device="cuda")
        y = fp8.fp8_linear(x, w, rope=(*rope, 256)) if fused else F_.rope_qkv(fp8.fp8_linear(x, w), *rope, 2, 64)
        y.backward(dy)
        return y.detach(), x.grad, w.main_grad

    y, dx, dw = run(True)
    y_ref, dx_ref, dw_ref = run(False)
    assert torch.equal(y, y_ref) and (dx is None or torch.equal(dx, dx_ref))
    assert (dw - dw_ref).norm() <= 1e-5 * dw_ref.norm()          # fp32 sums of the work items in any order


@pytest.mark.parametrize("R,I", [(128, 128), (384, 256), (1152, 2048)])
def test_swiglu_with_quantisation(R, I, cuda_status):
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import kernels as k
    torch.manual_seed(R)
    pre, dh = _randn(R, 2 * I, scale=3.0), _randn(R, I)
    pre[:, I // 2] = 0
    for got, want in zip((*fp8.swiglu_quant_dual(pre), *fp8.swiglu_bwd_quant_dual(pre, dh)),
                         (*fp8.quant_dual(k.swiglu_fwd(pre)), *fp8.quant_dual(k.swiglu_bwd(pre, dh)))):
        assert torch.equal(got.q, want.q) and torch.equal(got.scale, want.scale)


def test_mlp_node_is_the_composition(cuda_status):
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import functional as F_
    torch.manual_seed(0)
    T, C, I = 384, 256, 384
    x0, r0, dy = _randn(T, C), _randn(T, C), _randn(T, C)
    wi0, wo0 = _randn(2 * I, C, scale=C ** -0.5), _randn(C, I, scale=I ** -0.5)

    def run(fused):
        fp8.invalidate_weight_cache()
        x, r, wi, wo = (t.clone().requires_grad_(True) for t in (x0, r0, wi0, wo0))
        wi.main_grad, wo.main_grad = torch.zeros_like(wi, dtype=torch.float32), torch.zeros_like(wo, dtype=torch.float32)
        if fused:
            assert fp8.mlp_fused(x, wi, wo)
            y = F_.mlp_swiglu(x, wi, wo, r)
            assert "Fp8Mlp" in type(y.grad_fn).__name__
        else:
            y = fp8.fp8_linear(F_.swiglu(fp8.fp8_linear(x, wi)), wo) + r
        y.backward(dy)
        return y.detach(), x.grad, r.grad, wi.main_grad, wo.main_grad

    F_.set_fp8(True)
    try:
        (y, dx, dr, dwi, dwo), ref = run(True), run(False)
        assert torch.equal(y, ref[0]) and torch.equal(dx, ref[1]) and torch.equal(dr, ref[2])
        for a, b in ((dwi, ref[3]), (dwo, ref[4])):
            assert (a - b).norm() <= 1e-5 * b.norm()             # fp32 sums of the work items in any order
    finally:
        F_.set_fp8(False)
        fp8.invalidate_weight_cache()


def _residuals(T, C):
    base = torch.randn(T * C + 8, device="cuda").to(BF)
    return {"fp32": torch.randn(T, C, device="cuda"), "row": _randn(1, C), "off 16 bytes": base[1:T * C + 1].view(T, C),
            "odd row stride": _randn(T, C + 1)[:, :C], "columns first": _randn(C, T).t()}


@pytest.mark.parametrize("kind", ["fp32", "row", "off 16 bytes", "odd row stride", "columns first"])
def test_residuals_that_the_epilogue_cannot_add(kind, cuda_status):
    """They are added as a sum of its own, with its result type and its gradient."""
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import functional as F_
    torch.manual_seed(1)
    T, C, I = 256, 128, 256
    x, wi, wo = _randn(T, C), _randn(2 * I, C, scale=C ** -0.5), _randn(C, I, scale=I ** -0.5)
    wi.requires_grad_(True), wo.requires_grad_(True)
    r = _residuals(T, C)[kind].requires_grad_(True)
    F_.set_fp8(True)
    try:
        for call in (lambda res: F_.mlp_swiglu(x, wi, wo, res), lambda res: F_.linear(F_.mlp_swiglu(x, wi, wo), wo[:, :C], residual=res)):
            y = call(r)
            assert torch.equal(y, call(None) + r)
            (g,) = torch.autograd.grad(y.float().sum(), r)
            assert g.shape == r.shape and torch.equal(g, torch.full_like(g, T if kind == "row" else 1))
    finally:
        F_.set_fp8(False)
        fp8.invalidate_weight_cache()


def test_tangent_of_the_residual(cuda_status):
    import torch.autograd.forward_ad as fwd
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import functional as F_
    x, w, r, t = _randn(128, 128), _randn(128, 128), _randn(128, 128), _randn(128, 128)
    F_.set_fp8(True)
    try:
        with fwd.dual_level():
            y, dy = fwd.unpack_dual(F_.linear(x, w, residual=fwd.make_dual(r, t)))
            assert torch.equal(dy, t) and torch.equal(y, F_.linear(x, w) + r)
    finally:
        F_.set_fp8(False)
        fp8.invalidate_weight_cache()
