"""Batched transpose with a scale, and the tall stacks of the orthogonalisation that use it."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.mark.parametrize("B,R,C", [(1, 64, 64), (3, 192, 64), (2, 64, 320), (5, 256, 128)])
@pytest.mark.parametrize("scaled", [False, True])
def test_transpose_scale(B, R, C, scaled, cuda_status):
    from nanoplm_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(R + C)
    x = torch.randn(B, R, C, device="cuda", generator=g).to(BF)
    s = torch.rand(B, device="cuda", generator=g).to(BF) if scaled else None
    want = x.transpose(1, 2).contiguous()
    if scaled:
        want = want * s[:, None, None]
    assert torch.equal(K.transpose_scale(x, s), want)


@pytest.mark.parametrize("shape", [(3, 256, 128), (2, 384, 128), (2, 320, 192), (2, 200, 72)])
def test_tall_stacks_orthogonalise_like_wide_ones(shape, cuda_status):
    from nanoplm_b200.parallel.muon import orthogonalize_batched
    g = torch.Generator(device="cuda").manual_seed(shape[1])
    G = torch.randn(*shape, device="cuda", generator=g).to(BF)
    keep = G.clone()
    sq = G.float().pow(2).sum(dim=(1, 2))
    tall = orthogonalize_batched(G, sumsq=sq)
    assert torch.equal(G, keep) and tall.shape == G.shape and tall.is_contiguous()
    wide = orthogonalize_batched(keep.transpose(1, 2).contiguous(), sumsq=sq)
    assert torch.equal(tall, wide.transpose(1, 2))          # the same products on the same values
