"""Norm backward through the shared-memory ring against the other norm kernel, whose rows a table gradient keeps in fp32."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# fewer rows than warps, one row more than the ring and its two stages hold, all widths of a lane's chunks and ragged ones
@pytest.mark.parametrize("T,C", [(1, 8), (7, 264), (2369, 256), (4737, 512), (8000, 760), (5000, 1024)])
@pytest.mark.parametrize("rms", [False, True])
@pytest.mark.parametrize("skip,weighted", [(True, True), (False, True), (True, False)])
def test_bits_of_the_other_norm_kernel(T, C, rms, skip, weighted, cuda_status):
    from nanoplm_b200.ops import kernels as k
    torch.manual_seed(T)
    rnd = lambda *s: torch.randn(*s, device="cuda")
    V = max(T, 201)                                   # (larger than the vocabularies of the kernel for embeddings)
    x, dy = rnd(V, C).to(BF), rnd(T, C).to(BF)
    w = (1 + 0.1 * rnd(C)).to(BF) if weighted else None
    dres = rnd(T, C).to(BF) if skip else None
    mean, rstd = None if rms else 0.1 * rnd(T), torch.rand(T, device="cuda") + 0.5
    rows, dw_ref, dw = torch.zeros(V, C, device="cuda"), torch.zeros(C, device="cuda"), torch.zeros(C, device="cuda")
    k.norm_bwd(dy, x, w, mean, rstd, rms=rms, ids=torch.arange(T, device="cuda", dtype=torch.int32), dtable=rows, dw=dw_ref)
    dx = k.norm_bwd(dy, x[:T], w, mean, rstd, rms=rms, dres=dres, dw=dw)
    assert torch.equal(dx, (rows[:T] + dres.float() if skip else rows[:T]).to(BF))
    assert (dw - dw_ref).norm() <= 1e-5 * dw_ref.norm()     # fp32 sums of T rows in any order
