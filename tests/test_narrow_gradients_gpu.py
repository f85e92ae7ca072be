"""Weight gradients narrower than a tile, and coefficient parameters read in bf16 with their gradients added in place."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.mark.parametrize("N", [8, 24, 40, 72, 136])
@pytest.mark.parametrize("T,Kd", [(64, 64), (333, 192), (5000, 768)])
@pytest.mark.parametrize("main_grad", [False, True])
def test_narrow_weight_gradient(N, T, Kd, main_grad, cuda_status):
    from nanoplm_b200.ops.functional import _wgrad
    g = torch.Generator(device="cuda").manual_seed(N + T)
    dy = torch.randn(T, N, device="cuda", generator=g).to(BF)
    x = torch.randn(T, Kd, device="cuda", generator=g).to(BF)
    w = torch.nn.Parameter(torch.zeros(N, Kd, device="cuda", dtype=BF))
    want = dy.double().t() @ x.double()
    mag = dy.double().abs().t() @ x.double().abs()
    if main_grad:
        w.main_grad = torch.ones(N, Kd, device="cuda")
        assert _wgrad(dy, x, w) is None
        # fp32 sums of T products
        assert ((w.main_grad.double() - 1 - want).abs() <= mag * T * 2 ** -24 + 1e-5).all()
    else:
        got = _wgrad(dy, x, w)
        assert got.dtype == BF
        assert ((got.double() - want).abs() <= mag * T * 2 ** -24 + want.abs() * 2 ** -8 + 1e-5).all()


@pytest.mark.parametrize("n", [2, 4])
def test_coefficient_parameters_in_bf16(n, cuda_status):
    from nanoplm_b200.models.mhc import _CoefFn
    g = torch.Generator(device="cuda").manual_seed(n)
    T = 300
    pre = torch.randn(T, 2 * n + n * n, device="cuda", generator=g).to(BF)
    params = [torch.nn.Parameter(torch.randn(*s, device="cuda", generator=g).to(BF)) for s in ((n,), (n,), (n, n), (3,))]
    outs = []
    for kind in ("bf16", "fp32", "main_grad"):
        ps = [torch.nn.Parameter(p.detach().float() if kind == "fp32" else p.detach().clone()) for p in params]
        if kind == "main_grad":
            for p in ps:
                p.main_grad = torch.ones(p.shape, device="cuda")
        x = pre.clone().requires_grad_(True)
        alpha, beta, R = _CoefFn.apply(x, *ps, 5, n)
        (alpha.square().sum() + beta.square().sum() + (R * R).sum()).backward()
        grads = [(p.main_grad - 1) if kind == "main_grad" else p.grad.float() for p in ps]
        outs.append((alpha, beta, R, x.grad, grads))
    for o in outs[1:]:
        for a, b in zip(o[:4], outs[1][:4]):
            assert torch.equal(a, b)                      # the same fp32 values enter
    for a, b in zip(outs[0][4], outs[1][4]):
        assert torch.allclose(a, b, rtol=2 ** -8, atol=1e-3)        # returned in bf16
    for a, b in zip(outs[2][4], outs[1][4]):
        assert torch.allclose(a, b, rtol=1e-4, atol=1e-3)           # atomics in another order


def test_coefficient_gradients_of_the_wrong_size_are_refused(cuda_status):
    from nanoplm_b200.models.mhc import _CoefFn
    n, T = 4, 50
    ps = [torch.nn.Parameter(torch.randn(*s, device="cuda").to(BF)) for s in ((n,), (n,), (n, n), (3,))]
    for p in ps:
        p.main_grad = torch.zeros(p.shape, device="cuda")
    ps[2].main_grad = torch.zeros(n, device="cuda")
    alpha, beta, R = _CoefFn.apply(torch.randn(T, 2 * n + n * n, device="cuda").to(BF).requires_grad_(True), *ps, 5, n)
    with pytest.raises(RuntimeError):
        (alpha.sum() + beta.sum() + R.sum()).backward()


@pytest.mark.parametrize("n", [2, 4])
def test_coefficients_do_not_depend_on_how_the_parameters_are_held(n, cuda_status):
    """bf16 parameters, the same values in fp32, and bf16 with running gradients: the same bits forward and for `pre`; a
    gradient goes to one place only."""
    from nanoplm_b200.models.mhc import _CoefFn
    g = torch.Generator(device="cuda").manual_seed(10 + n)
    pre = torch.randn(200, 2 * n + n * n, device="cuda", generator=g).to(BF)
    params = [torch.randn(*s, device="cuda", generator=g).to(BF) for s in ((n,), (n,), (n, n), (3,))]
    outs = {}
    for kind in ("bf16", "fp32", "main_grad"):
        ps = [torch.nn.Parameter(p.float() if kind == "fp32" else p.clone()) for p in params]
        if kind == "main_grad":
            for p in ps:
                p.main_grad = torch.zeros(p.shape, device="cuda")
        x = pre.clone().requires_grad_(True)
        alpha, beta, R = _CoefFn.apply(x, *ps, 5, n)
        (alpha.square().sum() + beta.square().sum() + (R * R).sum()).backward()
        assert all((p.grad is None) == (kind == "main_grad") for p in ps)
        if kind == "main_grad":
            assert all(p.main_grad.abs().sum() > 0 for p in ps)
        outs[kind] = (alpha, beta, R, x.grad)
    for kind in ("bf16", "main_grad"):
        for a, b in zip(outs[kind], outs["fp32"]):
            assert torch.equal(a, b), kind


@pytest.mark.parametrize("how", ["bf16", "strided", "misaligned"])
def test_narrow_gradient_into_any_running_gradient(how, cuda_status):
    """Running gradients that the kernel cannot add to in place take the sum all the same."""
    from nanoplm_b200.ops.functional import _wgrad
    g = torch.Generator(device="cuda").manual_seed(4)
    N, Kd, T = 24, 192, 100
    dy, x = (torch.randn(T, n, device="cuda", generator=g).to(BF) for n in (N, Kd))
    w = torch.nn.Parameter(torch.zeros(N, Kd, device="cuda", dtype=BF))
    w.main_grad = {"bf16": torch.ones(N, Kd, device="cuda", dtype=BF), "strided": torch.ones(Kd, N, device="cuda").t(),
                   "misaligned": torch.ones(N * Kd + 1, device="cuda")[1:].view(N, Kd)}[how]
    assert _wgrad(dy, x, w) is None
    want = 1 + dy.double().t() @ x.double()
    got = w.main_grad.double().reshape(N, Kd)
    bound = 2 ** -8 if how == "bf16" else 2 ** -20
    assert ((got - want).abs() <= want.abs() * bound + (dy.double().abs().t() @ x.double().abs()) * T * 2 ** -24 + 1e-5).all()
