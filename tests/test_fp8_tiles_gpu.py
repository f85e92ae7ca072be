"""e4m3 GEMM at the edges of its tiles, K splits and scale forms, and the two-form quantiser."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _quantised(rows, K, seed, block):
    from nanoplm_b200.ops import fp8
    g = torch.Generator(device="cuda").manual_seed(seed)
    x = torch.randn(rows, K, device="cuda", generator=g).to(BF)
    return fp8.quant_tile(x, transpose=False, block=True) if block else fp8.quant_rows(x)


@pytest.mark.parametrize("M", [1, 127, 129, 300])
@pytest.mark.parametrize("N", [8, 72, 128, 136, 256, 264, 392])
@pytest.mark.parametrize("K", [128, 640])
@pytest.mark.parametrize("block", [False, True])
def test_gemm_fp8_tile_edges(M, N, K, block, cuda_status):
    from nanoplm_b200.ops import fp8
    if block and N % 128:
        pytest.skip("block scales come in whole 128-row blocks")
    qa, qb = _quantised(M, K, 1, False), _quantised(N, K, 2, block)
    ref = qa.dequantize().double() @ qb.dequantize().double().t()
    mag = qa.dequantize().double().abs() @ qb.dequantize().double().abs().t()
    out = fp8.gemm_fp8(qa, qb, out_dtype=torch.float32)
    # the tensor core aligns the products of one 32-wide instruction before it adds them (about 2^-13 of the
    # largest); the promoted sums are fp32
    bound = mag * 2 ** -12
    assert ((out.double() - ref).abs() <= bound).all()
    assert ((fp8.gemm_fp8(qa, qb).double() - ref).abs() <= bound + ref.abs() * 2 ** -8).all()


@pytest.mark.parametrize("T", [128, 2048, 4096, 10112])
@pytest.mark.parametrize("N,K", [(128, 128), (384, 256), (1024, 1024)])
def test_fp8_weight_gradient_splits(T, N, K, cuda_status):
    """Accumulated output: the contraction is split over work items from 4096 tokens on."""
    from nanoplm_b200.ops import fp8
    qa, qb = _quantised(N, T, 3, False), _quantised(K, T, 4, False)
    ref = qa.dequantize().double() @ qb.dequantize().double().t()
    mag = qa.dequantize().double().abs() @ qb.dequantize().double().abs().t()
    acc = torch.ones(N, K, device="cuda")
    fp8.gemm_fp8(qa, qb, out=acc, accumulate=True)
    assert ((acc.double() - 1 - ref).abs() <= mag * 2 ** -12).all()


@pytest.mark.parametrize("R,K", [(128, 128), (256, 384), (1152, 1024)])
@pytest.mark.parametrize("padded", [False, True])
def test_quant_dual_equals_the_two_kernels(R, K, padded, cuda_status):
    from nanoplm_b200.ops import fp8
    g = torch.Generator(device="cuda").manual_seed(R)
    full = (torch.randn(R, K + 64, device="cuda", generator=g) * torch.logspace(-3, 3, R, device="cuda")[:, None]).to(BF)
    x = full[:, :K] if padded else full[:, :K].contiguous()
    x[3] = 0
    rows, cols = fp8.quant_dual(x)
    want_r, want_c = fp8.quant_rows(x), fp8.quant_tile(x, transpose=True, block=False)
    for got, want in ((rows, want_r), (cols, want_c)):
        assert torch.equal(got.q, want.q) and torch.equal(got.scale, want.scale)


@pytest.mark.parametrize("N", [136, 256, 264, 392])
@pytest.mark.parametrize("block", [False, True])
def test_both_tile_widths_give_the_same_bits(N, block, cuda_status):
    """300 rows run on 128-wide tiles, 9 601 on 256-wide ones (edges in rows and columns on both)."""
    from nanoplm_b200.ops import fp8
    if block and N % 128:
        pytest.skip("block scales come in whole 128-row blocks")
    g = torch.Generator(device="cuda").manual_seed(N)
    x = torch.randn(9601, 640, device="cuda", generator=g).to(BF)
    qb = _quantised(N, 640, 2, block)
    tall, short = fp8.quant_rows(x), fp8.quant_rows(x[:300].contiguous())
    for dt in (torch.float32, BF):
        a, b = fp8.gemm_fp8(tall, qb, out_dtype=dt), fp8.gemm_fp8(short, qb, out_dtype=dt)
        assert torch.equal(a[:300], b)
    ref = tall.dequantize().double() @ qb.dequantize().double().t()
    mag = tall.dequantize().double().abs() @ qb.dequantize().double().abs().t()
    assert ((fp8.gemm_fp8(tall, qb, out_dtype=torch.float32).double() - ref).abs() <= mag * 2 ** -12).all()
