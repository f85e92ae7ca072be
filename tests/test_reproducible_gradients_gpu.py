"""set_attention_deterministic: the weight gradients of linear layers have the same bits every run."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.fixture
def deterministic():
    from nanoplm_b200.ops import kernels as K
    before = K._FA_DETERMINISTIC[0]
    K.set_attention_deterministic(True)
    yield
    K.set_attention_deterministic(before)


@pytest.mark.parametrize("fp8", [False, True])
@pytest.mark.parametrize("T", [1000, 1024, 10112])
@pytest.mark.parametrize("N,Kd", [(512, 512), (24, 768)])
def test_linear_weight_gradients(fp8, T, N, Kd, deterministic, cuda_status):
    from nanoplm_b200.ops import functional as F_
    from nanoplm_b200.ops.fp8 import fp8_linear
    g = torch.Generator(device="cuda").manual_seed(T)
    x = torch.randn(T, Kd, device="cuda", generator=g).to(BF)
    dy = torch.randn(T, N, device="cuda", generator=g).to(BF)
    w = torch.nn.Parameter((torch.randn(N, Kd, device="cuda", generator=g) * 0.05).to(BF))
    if fp8 and (N % 128 or Kd % 128):
        pytest.skip("not an e4m3 shape")
    grads = []
    for _ in range(6):
        w.main_grad = torch.zeros(N, Kd, device="cuda")
        (fp8_linear if fp8 else F_.linear)(x, w).backward(dy)
        grads.append(w.main_grad)
    assert all(torch.equal(grads[0], o) for o in grads[1:])


@pytest.mark.parametrize("T", [1000, 10112])
def test_layer(T, deterministic, cuda_status):
    """A whole encoder layer through its native launch sequence and op by op (a hook forces that): the same bits every
    run and on both ways; only the norms' gradients, sums over blocks in any order, may differ in their last bits."""
    from nanoplm_b200.config.schema import ModelConfig
    from nanoplm_b200.models.encoder import BatchContext, EncoderLayer, position_ids_from_cu_seqlens
    from nanoplm_b200.ops import functional as ops
    torch.manual_seed(2)
    cfg = ModelConfig(hidden_size=256, intermediate_size=512, num_hidden_layers=4, num_attention_heads=4,
                      max_position_embeddings=512)
    layer = EncoderLayer(cfg, 1).cuda().to(BF)
    with torch.no_grad():
        for p in layer.parameters():
            p.copy_(1 + 0.1 * torch.randn_like(p) if p.ndim == 1 else torch.randn_like(p) * 0.05)
    cu = torch.arange(0, T + 1, T // 8, dtype=torch.int32, device="cuda").clamp(max=T)
    cu[-1] = T
    ctx = BatchContext(cu, position_ids_from_cu_seqlens(cu, T), T)
    rope = ops.rope_tables(2048, 64, 10000.0, "cuda")
    x0, dy = (torch.randn(T, 256, device="cuda").to(BF) for _ in range(2))
    runs = []
    for k in range(6):
        if k == 3:
            layer.mlp.register_forward_hook(lambda *a: None)
        for p in layer.parameters():
            p.main_grad = torch.zeros(p.shape, device="cuda")
        x = x0.clone().requires_grad_(True)
        layer(x, ctx, 64, rope)[0].backward(dy)
        runs.append((x.grad, {n: p.main_grad for n, p in layer.named_parameters()}))
    for dx, grads in runs[1:]:
        assert torch.equal(dx, runs[0][0])
        for n, want in runs[0][1].items():
            if want.ndim == 2:
                assert torch.equal(grads[n], want), n
            else:
                assert torch.allclose(grads[n], want, rtol=1e-4, atol=1e-3), n
