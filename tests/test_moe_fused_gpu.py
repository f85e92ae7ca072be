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
