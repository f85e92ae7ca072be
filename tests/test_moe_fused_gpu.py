"""Mixture-of-experts forms that replace separate passes."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# experts without a row, with less and with more than a 128-row tile; columns of less than a tile, a tile, one and a chunk
@pytest.mark.parametrize("T,E,C,I", [(5, 16, 64, 64), (700, 8, 128, 256), (1500, 8, 256, 320)])
def test_grouped_swiglu_backward(T, E, C, I, cuda_status):
    from nanoplm_b200.ops import kernels as K
    from nanoplm_b200.ops import moe as M
    torch.manual_seed(T)
    rnd = lambda *s, scale=1.0: (torch.randn(*s, device="cuda") * scale).to(BF)
    plan = M.make_plan(M.MoEComm(C, E, 2), torch.randint(0, E, (T, 2), device="cuda", dtype=torch.int32))
    dys, Wo, pre = rnd(plan.cap, C), rnd(E, C, I, scale=C ** -0.5), rnd(plan.cap, 2 * I, scale=2.0)
    got = M.gemm_grouped(dys, Wo, plan.tile_group, b_mn=True, epi=K.EPI_SWIGLU_BWD, aux=pre).float()
    off = plan.group_off.tolist()
    for e in range(E):
        rows = slice(off[e], off[e + 1])
        dh = dys[rows].float() @ Wo[e].float()
        v, g = pre[rows, :I].float(), pre[rows, I:].float()
        s = torch.sigmoid(g)
        ref = torch.cat([dh * g * s, dh * v * s * (1 + g * (1 - s))], dim=1)
        # one rounding to bf16 (2^-9), the sigmoid of the fast exponential and fp32 sums of C terms of up to |dy| |W|
        size = torch.cat([g * s, v * s * (1 + g * (1 - s))], dim=1).abs()
        sums = (dys[rows].float().abs() @ Wo[e].float().abs()).repeat(1, 2) * C * 2 ** -23
        assert ((got[rows] - ref).abs() <= ref.abs() * 2 ** -8 + size * sums + 1e-6).all()
    with pytest.raises(ValueError):
        M.gemm_grouped(dys, Wo, plan.tile_group, b_mn=True, epi=K.EPI_SWIGLU_BWD)


@pytest.mark.parametrize("lens,E,norm_type", [([1], 8, "layernorm"), ([37, 90, 300], 64, "layernorm"), ([700], 8, "rmsnorm")])
def test_skip_connection_in_the_blocks(lens, E, norm_type, cuda_status):
    """Layers whose skip connection rides in the norm's and the experts' kernels against watched ones (a pass each)."""
    from nanoplm_b200.config.schema import ModelConfig, MoEConfig
    from nanoplm_b200.models.encoder import BatchContext, EncoderModel, position_ids_from_cu_seqlens
    torch.manual_seed(E)
    m = EncoderModel(ModelConfig(hidden_size=128, intermediate_size=256, num_hidden_layers=2, num_attention_heads=2,
                                 max_position_embeddings=1024, norm_type=norm_type,
                                 moe=MoEConfig(num_experts=E, top_k=2, expert_intermediate_size=64, every_n_layers=1)))
    m = m.cuda().to(BF)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(1 + 0.1 * torch.randn_like(p) if p.ndim == 1 else torch.randn_like(p) * 0.1)
    cu = torch.tensor([0, *lens]).cumsum(0).to(torch.int32).cuda()
    ctx = BatchContext(cu, position_ids_from_cu_seqlens(cu, sum(lens)), sum(lens))
    ids = torch.randint(4, 30, (sum(lens),), device="cuda", dtype=torch.int32)
    dy = torch.randn(sum(lens), 128, device="cuda").to(BF)

    def run(grad=True):
        for p in m.parameters():
            p.main_grad = torch.zeros(p.shape, device="cuda")
        with torch.set_grad_enabled(grad):
            y, aux = m.forward_hidden(ids, ctx)
        if grad:
            torch.autograd.backward([y, aux], [dy, None])
        return y.detach(), {n: p.main_grad for n, p in m.named_parameters()}

    y, grads = run()
    assert torch.equal(run(grad=False)[0], y)
    seen = []
    for layer in m.layers:
        layer.mlp.register_forward_hook(lambda mod, args, out: seen.append(len(args)))
    y_ref, grads_ref = run()
    assert seen == [1, 1] and torch.equal(y, y_ref)
    for n, g in grads_ref.items():     # the joined sums are rounded once (2^-9) where two or three roundings were, twice over
        assert (grads[n] - g).norm() <= 2 ** -6 * g.norm(), n
