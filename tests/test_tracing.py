"""torch.jit.trace over the kernels' autograd Functions: a trace replays them on its new inputs, in either gradient mode.
(The kernels write through raw addresses, so of a body that ran outside its Function a tracer sees the allocations only.)"""
import ctypes

import pytest
import torch

BF = torch.bfloat16
pytestmark = pytest.mark.filterwarnings("ignore::torch.jit.TracerWarning")


class Call(torch.nn.Module):
    """fn(module, x) as a module (a tracer wants the parameters that it meets to belong to one)."""

    def __init__(self, module, fn):
        super().__init__()
        self.module, self.fn = module, fn

    def forward(self, x):
        return self.fn(self.module, x)


@pytest.mark.parametrize("act", [None, "relu", "swiglu"])
def test_trace_without_gradients_replays_the_function(act, monkeypatch):
    """On the CPU, with a stand-in for the GEMM that writes through its outputs' addresses as the kernel does."""
    from nanoplm_b200.ops import functional as F_
    from nanoplm_b200.ops import kernels as K

    def put(dst, src):
        src = src.to(dst.dtype).contiguous()
        ctypes.memmove(dst.data_ptr(), src.data_ptr(), src.numel() * src.element_size())

    def gemm(a, b, epi=K.EPI_STORE, aux=None, **_):
        pre = a.detach().float() @ b.detach().float().t()
        v, g = pre.chunk(2, dim=1)
        res = {K.EPI_RELU: pre.relu(), K.EPI_SWIGLU: v * torch.nn.functional.silu(g)}.get(epi, pre)
        out = torch.empty(res.shape, dtype=BF)
        put(out, res)
        if aux is not None:
            put(aux, pre)
        return out

    monkeypatch.setattr(K, "gemm", gemm)
    call = Call(torch.nn.Linear(8, 16, bias=False, dtype=BF),
                lambda m, x: F_._call(F_._LinearFn, x, m.weight, None, None, act, None, F_._keeps()))
    with torch.no_grad():
        traced = torch.jit.trace(call, torch.zeros(4, 8, dtype=BF), check_trace=False)
        x = torch.randn(4, 8).to(BF)
        assert torch.equal(traced(x), call(x))


def _cases():
    from nanoplm_b200.config.schema import ModelConfig
    from nanoplm_b200.models.encoder import (MLP, BatchContext, EncoderLayer, Linear, Norm,
                                             position_ids_from_cu_seqlens)
    from nanoplm_b200.ops import functional as ops
    cfg = ModelConfig(hidden_size=128, intermediate_size=192, num_hidden_layers=4, num_attention_heads=2,
                      max_position_embeddings=64)
    cu = torch.tensor([0, 37, 70], dtype=torch.int32, device="cuda")
    ctx = BatchContext(cu, position_ids_from_cu_seqlens(cu, 70), 70)
    rope = ops.rope_tables(64, 64, 10000.0, "cuda")
    torch.manual_seed(0)
    mods = {"linear": Linear(128, 64), "norm": Norm(128, 1e-5), "mlp": MLP(cfg), "layer0": EncoderLayer(cfg, 0),
            "layer1": EncoderLayer(cfg, 1)}
    for m in mods.values():
        m.cuda().to(BF)
        with torch.no_grad():
            for p in m.parameters():
                p.copy_(1 + 0.1 * torch.randn_like(p) if p.ndim == 1 else torch.randn_like(p) * 0.1)
                p.main_grad = torch.zeros(p.shape, device="cuda")
    calls = {n: Call(m, lambda m, x: m(x)) for n, m in mods.items()}
    for n in ("layer0", "layer1"):
        calls[n].fn = lambda m, x: m(x, ctx, 64, rope)[0]
    calls["relu"] = Call(mods["linear"], lambda m, x: m(x, act="relu"))
    calls["swiglu"] = Call(mods["mlp"], lambda m, x: m.Wi(x, act="swiglu"))
    return calls


@pytest.mark.gpu
@pytest.mark.parametrize("grad", [False, True])
@pytest.mark.parametrize("name", ["linear", "relu", "swiglu", "norm", "mlp", "layer0", "layer1"])
def test_traced_modules_match_eager(name, grad, cuda_status):
    call = _cases()[name]
    x0, x = (torch.randn(70, 128, device="cuda").to(BF) for _ in range(2))
    with torch.set_grad_enabled(grad):
        traced = torch.jit.trace(call, x0.requires_grad_(grad), check_trace=False)
        assert torch.equal(traced(x), call(x))
        assert torch.equal(traced(x0), call(x0))


@pytest.mark.gpu
def test_trace_without_gradients_replays_with_them(cuda_status):
    """What a backward pass needs is kept although the trace was taken without gradients."""
    calls = _cases()
    x0 = torch.randn(70, 128, device="cuda").to(BF)
    for call in (calls["relu"], calls["swiglu"], calls["mlp"]):
        with torch.no_grad():
            traced = torch.jit.trace(call, x0, check_trace=False)
        grads = []
        for f in (call, traced):
            x = x0.clone().requires_grad_(True)
            f(x).float().square().sum().backward()
            grads.append(x.grad)
        assert torch.equal(*grads)
