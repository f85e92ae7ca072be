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
@pytest.mark.parametrize("M,N,K", [(1, 128, 128), (130, 384, 256), (1000, 1024, 128), (9601, 384, 256), (5000, 640, 1024)])
def test_residual_and_rotary_epilogues(M, N, K, cuda_status):
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import functional as F_
    from nanoplm_b200.ops import kernels as k
    torch.manual_seed(M)
    a, b = _operands(M, N, K)
    exact = fp8.gemm_fp8(a, b, out_dtype=torch.float32)          # the sums that the epilogues start from
    wide = _randn(M, N + 64)
    res = wide[:, :N]                                            # (a row stride of its own)
    assert torch.equal(fp8.gemm_fp8_form(a, b, residual=res), (exact + res.float()).to(BF))
    cos, sin = F_.rope_tables(300, 64, 10000.0, torch.device("cuda"))
    pos = torch.randint(0, 300, (M,), device="cuda", dtype=torch.int32)
    cols = N // 128 * 64
    y = fp8.gemm_fp8_form(a, b, rope=(pos, cos, sin, cols))
    assert torch.equal(y[:, cols:], exact[:, cols:].to(BF))
    h = exact[:, :cols].double().view(M, -1, 2, 32)
    c, s = cos[pos.long()].double()[:, None], sin[pos.long()].double()[:, None]
    ref = torch.stack((h[:, :, 0] * c - h[:, :, 1] * s, h[:, :, 1] * c + h[:, :, 0] * s), 2)
    bound = ref.abs() * 2 ** -8 + h.abs().sum(2, keepdim=True) * 2 ** -22    # one bf16 rounding, three fp32 ones
    assert ((y[:, :cols].double().view(ref.shape) - ref).abs() <= bound).all()


@pytest.mark.parametrize("R,I", [(128, 128), (384, 256), (1152, 2048)])
def test_swiglu_with_quantisation(R, I, cuda_status):
    from nanoplm_b200.ops import fp8
    from nanoplm_b200.ops import kernels as k
    torch.manual_seed(R)
    pre, dh = _randn(R, 2 * I, scale=3.0), _randn(R, I)
    pre[:, I // 2] = 0
    for got, want in zip((*fp8.swiglu_quant_dual(pre), *fp8.swiglu_bwd_quant_dual(pre, dh)),
                         (*fp8.quant_dual(k.swiglu_fwd(pre)), *fp8.quant_dual(k.swiglu_bwd(pre, dh)))):
        # the scales are the maxima of the same bf16 values; those may differ in the last bit where the compiler contracts
        # the two kernels' arithmetic differently
        assert torch.allclose(got.scale, want.scale, rtol=2 ** -7, atol=0)
        assert ((got.dequantize() - want.dequantize()).norm() <= 2 ** -9 * want.dequantize().norm())


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
        for a, b in zip(run(True), run(False)):
            assert (a.float() - b.float()).norm() <= 2 ** -7 * b.float().norm()      # bf16 roundings of y, dx
    finally:
        F_.set_fp8(False)
        fp8.invalidate_weight_cache()
