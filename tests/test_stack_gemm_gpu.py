"""Stacks of equal products (Newton-Schulz iterations) against fp64, at the edges of their tiles."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _stack(*s, scale=1.0):
    return (torch.randn(*s, device="cuda") * scale).to(BF)


@pytest.mark.parametrize("B,m,n,k", [(1, 256, 64, 64), (3, 256, 320, 128), (2, 512, 192, 1088), (2, 768, 1024, 256)])
@pytest.mark.parametrize("b_mn", [False, True])
@pytest.mark.parametrize("residual", [False, True])
def test_stack_product(B, m, n, k, b_mn, residual, cuda_status):
    from nanoplm_b200.ops import kernels as K
    torch.manual_seed(m + n)
    a, b = _stack(B, m, k), _stack(B, k, n) if b_mn else _stack(B, n, k)
    r = _stack(B, m, n) if residual else None
    y = K.gemm_stack(a, b, b_mn=b_mn, alpha=-0.75, r=r, beta=1.5)
    ref = -0.75 * (a.double() @ (b.double() if b_mn else b.double().transpose(1, 2)))
    if residual:
        ref = ref + 1.5 * r.double()
    # one rounding to bf16 (2^-9 of the value), plus fp32 sums of k terms
    bound = ref.abs() * 2.0 ** -8 + k * 2.0 ** -23 * (a.double().abs().amax() * b.double().abs().amax())
    assert ((y.double() - ref).abs() <= bound).all()


@pytest.mark.parametrize("B,m,k", [(1, 256, 64), (5, 512, 192), (2, 1024, 128), (3, 768, 1024)])
def test_symmetric_products(B, m, k, cuda_status):
    from nanoplm_b200.ops import kernels as K
    torch.manual_seed(m)
    x = _stack(B, m, k, scale=k ** -0.5)
    A = K.gemm_stack(x, x, symmetric=True)
    assert torch.equal(A, K.gemm_stack(x, x))           # the mirrored tiles have the bits of the computed ones
    P = K.gemm_stack(A, A, alpha=2.0, r=A, beta=-4.75, symmetric=True)
    assert torch.equal(P, K.gemm_stack(A, A, alpha=2.0, r=A, beta=-4.75))
    assert torch.equal(P, P.transpose(1, 2))


# half a pair of column chunks at the right edge, and several tiles for each of the 74 pairs
@pytest.mark.parametrize("B,m,n,k", [(64, 512, 704, 64), (40, 256, 1088, 128)])
@pytest.mark.parametrize("b_mn", [False, True])
def test_stack_of_many_ragged_tiles(B, m, n, k, b_mn, cuda_status):
    """Bit for bit the products one by one: neither tiles nor buffers change the order of a sum."""
    from nanoplm_b200.ops import kernels as K
    torch.manual_seed(n)
    a, b = _stack(B, m, k), _stack(B, k, n) if b_mn else _stack(B, n, k)
    want = torch.stack([K.gemm(x, y, b_mn=b_mn) for x, y in zip(a, b)])
    for _ in range(3):
        assert torch.equal(K.gemm_stack(a, b, b_mn=b_mn), want)


def test_stack_refusals(cuda_status):
    from nanoplm_b200.ops import kernels as K
    with pytest.raises(Exception):
        K.gemm_stack(_stack(1, 128, 64), _stack(1, 64, 64))                     # half a tile of rows
    with pytest.raises(Exception):
        K.gemm_stack(_stack(1, 256, 64), _stack(1, 64, 64), symmetric=True)     # not square
    with pytest.raises(ValueError):
        K.gemm_stack(_stack(1, 256, 64), _stack(2, 64, 64))


@pytest.mark.parametrize("r,c", [(256, 512), (1024, 256), (768, 768)])
def test_orthogonal_factor_error(r, c, cuda_status):
    """The iteration is no further from the same iteration in fp64 than with its sums rounded between the products."""
    from nanoplm_b200.parallel import muon
    torch.manual_seed(r)
    G = _stack(4, r, c)
    got = muon.orthogonalize_batched(G.clone())

    def iterate(x, rounded):
        x = x.transpose(1, 2) if r > c else x
        rd = (lambda t: t.to(BF).double()) if rounded else (lambda t: t)
        x = rd(x / (x.flatten(1).norm(dim=1) * 1.01 + 1e-7)[:, None, None])
        eye = torch.eye(x.shape[1], device="cuda", dtype=torch.float64)
        for a, b, c_ in muon.NS_QUINTIC:
            A = rd(x @ x.transpose(1, 2))
            Bm = rd(rd(rd(A * c_) + b * eye) @ A)
            x = rd(rd(Bm + a * eye) @ x)
        return x.transpose(1, 2) if r > c else x

    exact = iterate(G.double(), False)
    error = lambda y: ((y.double() - exact).norm() / exact.norm()).item()
    assert error(got) <= 1.02 * error(iterate(G.double(), True))
