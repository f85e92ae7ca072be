"""A site's write together with the next site's read against the two calls."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# one token, fewer channels than a warp's slice and a remainder of it; outputs of the read that nobody uses
@pytest.mark.parametrize("n,T,C", [(4, 1, 64), (4, 777, 320), (2, 1300, 768)])
@pytest.mark.parametrize("use", ["all", "h", "X"])
def test_write_and_read_of_the_next_site(n, T, C, use, cuda_status):
    from nanoplm_b200.models.mhc import HyperConnection, _WriteMeanFn
    torch.manual_seed(T)
    a, b = (HyperConnection(C, n).cuda().to(BF) for _ in range(2))
    with torch.no_grad():
        for p in (*a.parameters(), *b.parameters()):
            p.add_(0.2 * torch.randn_like(p))
    X0, G, Gh = (torch.randn(*s, device="cuda").to(BF) for s in ((T, n, C), (T, n, C), (T, C)))

    def run(joined):
        X = X0.clone().requires_grad_(True)
        for p in (*a.parameters(), *b.parameters()):
            p.grad = None
        h, state = a.read(X)
        y = torch.tanh(h)
        if joined:
            X1, h, state = a.write_read(X, y, state, b)
            assert type(X1.grad_fn).__name__.startswith(_WriteMeanFn.__name__)
        else:
            X1 = a.write(X, y, state)
            h, state = b.read(X1)
        out = {"all": lambda: (b.write(X1, torch.tanh(h), state) * G).sum(), "h": lambda: (h * Gh).sum(),
               "X": lambda: (X1 * G).sum()}[use]()
        out.backward()
        return X1.detach(), h.detach(), X.grad, [p.grad for p in (*a.parameters(), *b.parameters())]

    got, want = run(True), run(False)
    assert all(torch.equal(p, q) for p, q in zip(got[:3], want[:3]))
    for p, q in zip(got[3], want[3]):          # fp32 sums over the tokens in any order, rounded to bf16
        assert (p is None) == (q is None) and (p is None or (p.float() - q.float()).norm() <= 2 ** -8 * q.float().norm())


def test_layers_joined_in_a_model(cuda_status):
    """Layers that nobody watches against the same ones called one by one (a hook on the middle one)."""
    from nanoplm_b200.config.schema import ModelConfig
    from nanoplm_b200.models.encoder import BatchContext, EncoderModel, position_ids_from_cu_seqlens
    torch.manual_seed(3)
    m = EncoderModel(ModelConfig(hidden_size=128, intermediate_size=128, num_hidden_layers=3, num_attention_heads=2,
                                 max_position_embeddings=512, mhc_streams=4, conv_kernel_size=3)).cuda().to(BF)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(1 + 0.1 * torch.randn_like(p) if p.ndim == 1 else torch.randn_like(p) * 0.1)
    cu = torch.tensor([0, 37, 90, 300], dtype=torch.int32, device="cuda")
    ctx = BatchContext(cu, position_ids_from_cu_seqlens(cu, 300), 300)
    ids, dy = torch.randint(4, 30, (300,), device="cuda", dtype=torch.int32), torch.randn(300, 128, device="cuda").to(BF)

    def run():
        m.zero_grad()
        y, _ = m.forward_hidden(ids, ctx)
        y.backward(dy)
        with torch.no_grad():
            assert torch.equal(m.forward_hidden(ids, ctx)[0], y)
        return y.detach(), {n: p.grad.float() for n, p in m.named_parameters() if p.grad is not None}

    y, grads = run()
    seen = []
    m.layers[1].register_forward_hook(lambda mod, args, out: seen.append(len(args)))
    y_ref, grads_ref = run()
    assert seen == [4, 4] and torch.equal(y, y_ref) and grads.keys() == grads_ref.keys()
    for name, g in grads_ref.items():          # (as above)
        assert (grads[name] - g).norm() <= 2 ** -8 * g.norm(), name
