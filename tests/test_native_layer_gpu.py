"""The native launch sequence of an encoder layer against the op-by-op path (forced by a hook on one part)."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _layer(C, I, idx, norm_type="layernorm"):
    from nanoplm_b200.config.schema import ModelConfig
    from nanoplm_b200.models.encoder import EncoderLayer
    torch.manual_seed(3 + idx)
    cfg = ModelConfig(hidden_size=C, intermediate_size=I, num_hidden_layers=4, num_attention_heads=C // 64,
                      max_position_embeddings=512, norm_type=norm_type)
    layer = EncoderLayer(cfg, idx).cuda().to(BF)
    with torch.no_grad():
        for n, p in layer.named_parameters():
            p.copy_(1 + 0.1 * torch.randn_like(p) if p.ndim == 1 else torch.randn_like(p) * 0.05)
    return layer


def _context(lens):
    from nanoplm_b200.models.encoder import BatchContext, position_ids_from_cu_seqlens
    cu = torch.tensor([0, *lens]).cumsum(0).to(torch.int32).cuda()
    return BatchContext(cu, position_ids_from_cu_seqlens(cu, sum(lens)), sum(lens))


def _rope():
    from nanoplm_b200.ops import functional as ops
    return ops.rope_tables(512, 64, 10000.0, "cuda")


@pytest.mark.parametrize("C,I", [(64, 64), (128, 320), (256, 512), (512, 1024)])
@pytest.mark.parametrize("idx", [0, 1])
@pytest.mark.parametrize("lens,window", [([1], -1), ([37, 90], 64), ([300, 5, 129], -1)])
@pytest.mark.parametrize("norm_type", ["layernorm", "rmsnorm"])
def test_layer_matches_op_by_op(C, I, idx, lens, window, norm_type, cuda_status, monkeypatch):
    from nanoplm_b200.ops import layer as native
    layer, ctx, rope = _layer(C, I, idx, norm_type), _context(lens), _rope()
    g = torch.Generator(device="cuda").manual_seed(C)
    x0 = torch.randn(sum(lens), C, device="cuda", generator=g).to(BF)
    dy = torch.randn(sum(lens), C, device="cuda", generator=g).to(BF)
    calls = []
    monkeypatch.setattr(native, "_forward", (lambda f: lambda *a: (calls.append(1), f(*a))[1])(native._forward))

    def once(grad):
        for p in layer.parameters():
            p.main_grad = torch.zeros(p.shape, device="cuda")
        x = x0.clone().requires_grad_(grad)
        with torch.set_grad_enabled(grad):
            y, _ = layer(x, ctx, window, rope)
        if not grad:
            return y, None, None
        y.backward(dy)
        return y.detach(), x.grad, {n: p.main_grad for n, p in layer.named_parameters()}

    y, dx, grads = once(True)
    y_eval, _, _ = once(False)
    assert len(calls) == 2
    hook = layer.mlp.register_forward_hook(lambda *a: None)
    y_ref, dx_ref, grads_ref = once(True)
    hook.remove()
    assert len(calls) == 2                              # the observed part went op by op
    assert torch.equal(y, y_ref) and torch.equal(y_eval, y_ref)      # the same kernels on the same values
    # dQ is summed by atomics (fp32, any order) before its bf16 rounding; the first layer adds its two gradients before
    # rounding instead of after
    assert (dx.float() - dx_ref.float()).norm() <= 6e-3 * dx_ref.float().norm()
    for n in grads:
        assert (grads[n] - grads_ref[n]).norm() <= 6e-3 * grads_ref[n].norm() + 1e-6, n


def test_layer_falls_back(cuda_status, monkeypatch):
    """Calls that are not the plain case go op by op."""
    from nanoplm_b200.ops import functional as ops
    from nanoplm_b200.ops import kernels as K
    from nanoplm_b200.ops import layer as native
    layer, ctx, rope = _layer(128, 128, 1), _context([50, 20]), _rope()
    x = torch.randn(70, 128, device="cuda").to(BF).requires_grad_(True)
    monkeypatch.setattr(native, "_forward", lambda *a: pytest.fail("native path"))
    layer(x, ctx, 64, rope)                                        # no main_grad
    for p in layer.parameters():
        p.main_grad = torch.zeros(p.shape, device="cuda")
    layer(x.detach(), ctx, 64, rope)                               # the input needs no gradient
    layer.mlp.Wi.weight.requires_grad_(False)
    layer(x, ctx, 64, rope)                                        # a frozen weight
    layer.mlp.Wi.weight.requires_grad_(True)
    ops.set_wgrad_ready_callback(lambda p: None)                   # somebody waits for single gradients
    try:
        layer(x, ctx, 64, rope)
    finally:
        ops.set_wgrad_ready_callback(None)
    K.set_attention_impl("single")
    try:
        layer(x, ctx, 64, rope)
    finally:
        K.set_attention_impl("ws")


@pytest.mark.parametrize("idx", [0, 1])
@pytest.mark.parametrize("grad", [False, True])
def test_every_part_that_is_called_op_by_op_is_observed(idx, grad, cuda_status):
    """Hooks, backward hooks and a forward of the instance's own on each part in turn: they run, as op by op."""
    layer, ctx, rope = _layer(128, 128, idx), _context([50, 20]), _rope()
    for p in layer.parameters():
        p.main_grad = torch.zeros(p.shape, device="cuda")
    x = torch.randn(70, 128, device="cuda").to(BF).requires_grad_(grad)
    seen = []

    def call():
        with torch.set_grad_enabled(grad):
            y, _ = layer(x, ctx, 64, rope)
        if grad:
            y.sum().backward()

    # (the linear layers' weights and the norms' residual form are used without a call of these modules)
    called = [layer.attn, layer.mlp] + ([layer.attn_norm] if idx == 0 else [])
    for m in called:
        for add in (lambda: m.register_forward_hook(lambda *a: seen.append(1)),
                    lambda: m.register_forward_pre_hook(lambda *a: seen.append(1))):
            h = add()
            call()
            assert seen.pop() and not seen
            h.remove()
        m.forward = lambda *a, f=m.forward, **k: (seen.append(1), f(*a, **k))[1]
        call()
        del m.forward
        assert seen.pop() and not seen
        if grad:
            h = m.register_full_backward_hook(lambda *a: seen.append(1))
            call()
            assert seen.pop() and not seen
            h.remove()


@pytest.mark.parametrize("how", ["cpu", "recomputed"])
def test_saved_tensors_may_come_back_as_copies(how, cuda_status):
    """Saved-tensor hooks (offloading, recomputation) hand the backward pass other tensors than it saved."""
    from torch.utils.checkpoint import checkpoint
    layer, ctx, rope = _layer(128, 192, 1), _context([50, 20]), _rope()
    g = torch.Generator(device="cuda").manual_seed(1)
    x0, dy = (torch.randn(70, 128, device="cuda", generator=g).to(BF) for _ in range(2))
    runs = []
    for mode in (None, how):
        for p in layer.parameters():
            p.main_grad = torch.zeros(p.shape, device="cuda")
        x = x0.clone().requires_grad_(True)
        if mode is None:
            y = layer(x, ctx, 64, rope)[0]
        elif mode == "cpu":
            with torch.autograd.graph.save_on_cpu():
                y = layer(x, ctx, 64, rope)[0]
        else:
            y = checkpoint(lambda t: layer(t, ctx, 64, rope)[0], x, use_reentrant=False)
        y.backward(dy)
        runs.append((x.grad, {n: p.main_grad for n, p in layer.named_parameters()}))
    (dx, grads), (dx_h, grads_h) = runs
    # dQ is summed by atomics before its bf16 rounding
    assert (dx.float() - dx_h.float()).norm() <= 6e-3 * dx.float().norm()
    for n in grads:
        assert (grads[n] - grads_h[n]).norm() <= 6e-3 * grads[n].norm() and grads[n].norm() > 0, n


def test_refusals_of_the_op_by_op_path_stay(cuda_status):
    """Metadata of the wrong type or on the wrong device, and running gradients of the wrong shape, are errors."""
    import copy
    layer, ctx, rope = _layer(128, 128, 1), _context([50, 20]), _rope()
    x = torch.randn(70, 128, device="cuda").to(BF).requires_grad_(True)
    for p in layer.parameters():
        p.main_grad = torch.zeros(p.shape, device="cuda")
    for wrong in (lambda p: p.long(), lambda p: p.cpu(), lambda p: p[:69]):
        c = copy.copy(ctx)
        c.position_ids = wrong(ctx.position_ids)
        for grad in (False, True):
            with torch.set_grad_enabled(grad), pytest.raises(ValueError):
                layer(x, c, 64, rope)
    for cos in (rope[0].double(), rope[0].cpu(), rope[0][:, :16]):
        with torch.no_grad(), pytest.raises(ValueError):
            layer(x, ctx, 64, (cos, rope[1]))
    layer.mlp.Wi.weight.main_grad = torch.zeros(128, 256, device="cuda")
    with pytest.raises(ValueError):
        layer(x, ctx, 64, rope)[0].sum().backward()
