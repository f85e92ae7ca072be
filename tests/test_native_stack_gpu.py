"""All layers through one native call each way, against the same layers called one by one (forced by a hook on one of
them)."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _model(C, I, layers, norm_type="layernorm"):
    from nanoplm_b200.config.schema import ModelConfig
    from nanoplm_b200.models.encoder import EncoderModel
    torch.manual_seed(layers)
    m = EncoderModel(ModelConfig(hidden_size=C, intermediate_size=I, num_hidden_layers=layers, num_attention_heads=C // 64,
                                 max_position_embeddings=512, norm_type=norm_type)).cuda().to(BF)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(1 + 0.1 * torch.randn_like(p) if p.ndim == 1 else torch.randn_like(p) * 0.05)
    return m


def _context(lens):
    from nanoplm_b200.models.encoder import BatchContext, position_ids_from_cu_seqlens
    cu = torch.tensor([0, *lens]).cumsum(0).to(torch.int32).cuda()
    return BatchContext(cu, position_ids_from_cu_seqlens(cu, sum(lens)), sum(lens))


@pytest.fixture
def calls(monkeypatch):
    from nanoplm_b200.ops import layer as native
    seen = {"stack": 0, "layer": 0}

    def count(name, f):
        def g(*a):
            seen[name] += 1
            return f(*a)
        return g

    monkeypatch.setattr(native, "_stack_inference", count("stack", native._stack_inference))
    monkeypatch.setattr(native._StackFn, "forward", staticmethod(count("stack", native._StackFn.forward)))
    monkeypatch.setattr(native, "_forward", count("layer", native._forward))
    return seen


def _run(m, ids, ctx, grad, dy=None):
    for p in m.parameters():
        p.main_grad = torch.zeros(p.shape, device="cuda")
    with torch.set_grad_enabled(grad):
        y, _ = m.forward_hidden(ids, ctx)
    if grad:
        y.backward(dy)
    return y.detach(), {n: p.main_grad for n, p in m.named_parameters()}


# runs of 1, 2, 4, 8 and the rest (outputs and gradients take turns in two places)
@pytest.mark.parametrize("layers,runs", [(1, 1), (2, 2), (5, 3), (17, 5)])
@pytest.mark.parametrize("C,I,norm_type", [(64, 64, "layernorm"), (256, 320, "rmsnorm")])
@pytest.mark.parametrize("lens", [[1], [37, 90, 300]])
def test_stack_matches_single_layers(layers, runs, C, I, norm_type, lens, calls, cuda_status):
    from nanoplm_b200.ops import kernels as K
    m, ctx = _model(C, I, layers, norm_type), _context(lens)
    ids = torch.randint(3, 28, (sum(lens),), device="cuda")
    dy = torch.randn(sum(lens), C, device="cuda").to(BF) * 0.1
    K.set_attention_deterministic(True)     # the same bits every run
    try:
        y, grads = _run(m, ids, ctx, True, dy)
        y_eval, _ = _run(m, ids, ctx, False)
        assert calls == {"stack": 2 * runs, "layer": 0}
        hook = m.layers[0].register_forward_hook(lambda *a: None)
        y_ref, grads_ref = _run(m, ids, ctx, True, dy)
        assert calls == {"stack": 2 * runs, "layer": layers}
        hook.remove()
    finally:
        K.set_attention_deterministic(False)
    assert torch.equal(y, y_ref) and torch.equal(y_eval, y_ref)
    for n in grads:
        if n.startswith("layers") and grads[n].ndim == 2:
            assert torch.equal(grads[n], grads_ref[n]), n
        else:       # norm weights and the embedding: fp32 sums over blocks in any order
            assert (grads[n] - grads_ref[n]).norm() <= 1e-4 * grads_ref[n].norm() + 1e-6, n


def test_layers_are_called_where_somebody_watches(calls, cuda_status):
    from nanoplm_b200.ops import functional as ops
    m, ctx = _model(64, 64, 3), _context([50, 20])
    ids = torch.randint(3, 28, (70,), device="cuda")
    dy = torch.randn(70, 64, device="cuda").to(BF)

    def counted(*a):
        calls.update(stack=0, layer=0)
        _, grads = _run(m, ids, ctx, *a)
        return (calls["stack"], calls["layer"]), grads

    n, want = counted(True, dy)
    assert n == (2, 0)
    with torch.autograd.graph.save_on_cpu():            # layer by layer, so that one layer's tensors come back at a time
        n, got = counted(True, dy)
    assert n == (0, 3)
    for k in (k for k in want if k.startswith("layers")):     # (the embedding's gradient goes to .grad under such hooks)
        assert (got[k] - want[k]).norm() <= 6e-3 * want[k].norm() + 1e-6, k
    m.layers[1].mlp.Wi.weight.requires_grad_(False)     # a frozen weight: that layer goes op by op, those after it one by one
    assert counted(True, dy)[0] == (1, 1)
    m.layers[1].mlp.Wi.weight.requires_grad_(True)
    m.layers[2].forward = lambda *a: type(m.layers[2]).forward(m.layers[2], *a)
    assert counted(False)[0] == (2, 1)
    del m.layers[2].__dict__["forward"]
    told = []
    for p in m.parameters():
        p.main_grad = torch.zeros(p.shape, device="cuda")
    y, _ = m.forward_hidden(ids, ctx)
    ops.set_wgrad_ready_callback(told.append)           # set after the forward: told after every layer, last layer first
    try:
        y.backward(dy)
    finally:
        ops.set_wgrad_ready_callback(None)
    names = {id(p): n for n, p in m.named_parameters()}
    assert [names[id(p)].split(".")[1] for p in told] == ["2"] * 4 + ["1"] * 4 + ["0"] * 4
