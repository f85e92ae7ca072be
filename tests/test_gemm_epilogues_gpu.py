"""GEMM epilogues that read a second operand through TMA, on CTA pairs and single CTAs, at ragged sizes."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _rand(*shape, seed, scale=1.0):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return (torch.randn(*shape, device="cuda", generator=g) * scale).to(BF)


def _close(got, want, scale):
    # one bf16 rounding of the result (2^-8 relative) and fp32 sums whose order differs from the oracle's
    assert torch.allclose(got.double(), want, rtol=2 ** -7, atol=2 ** -8 * scale)


@pytest.mark.parametrize("pair", [False, True])
@pytest.mark.parametrize("M", [1, 33, 127, 129, 256, 383])
@pytest.mark.parametrize("N,Kd", [(64, 64), (192, 128), (320, 192), (576, 72)])
def test_second_operand_epilogues(M, N, Kd, pair, cuda_status):
    from nanoplm_b200.ops import kernels as K
    dy, w = _rand(M, Kd, seed=1), _rand(Kd, N, seed=2, scale=Kd ** -0.5)
    acc = dy.double() @ w.double()
    # residual add
    res = _rand(M, N, seed=3)
    _close(K.gemm(dy, w, b_mn=True, epi=K.EPI_ADD, aux=res, bn=256, pair=pair), acc + res.double(), 2.0)
    # SwiGLU backward: gradient of [value | gate]
    pre = _rand(M, 2 * N, seed=4)
    v, g = pre.double().chunk(2, dim=1)
    s = torch.sigmoid(g)
    want = torch.cat((acc * g * s, acc * v * s * (1 + g * (1 - s))), dim=1)
    _close(K.gemm(dy, w, b_mn=True, epi=K.EPI_SWIGLU_BWD, aux=pre, pair=pair), want, 2.0)


@pytest.mark.parametrize("M", [1, 33, 127, 129, 256, 383])
@pytest.mark.parametrize("N", [64, 192, 320, 576])
def test_delta_epilogue(M, N, cuda_status):
    from nanoplm_b200.ops import kernels as K
    dy, w, o = _rand(M, 96, seed=1), _rand(96, N, seed=2, scale=0.1), _rand(M, N, seed=3)
    delta = torch.full((N // 64, M), float("nan"), device="cuda")
    out = K.gemm_dgrad_delta(dy, w, o, delta)
    _close(out, dy.double() @ w.double(), 1.0)
    want = (out.double() * o.double()).view(M, N // 64, 64).sum(-1).t()
    # 64 fp32 products and sums: 64 * 2^-24 of the sum of magnitudes
    bound = (out.double() * o.double()).abs().view(M, N // 64, 64).sum(-1).t() * 64 * 2 ** -24 + 1e-12
    assert ((delta.double() - want).abs() <= bound).all()
