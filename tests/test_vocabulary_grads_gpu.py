"""Gradients of the embedding table and of the decoder: sums over the token rows that share a vocabulary entry, against
fp64. fp32 sums of n terms in any order are within 2 n 2^-24 of the sum of magnitudes, far below the bounds here."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _rel(a, b):
    return ((a.double() - b).norm() / b.norm().clamp(min=1e-30)).item()


# one row, fewer rows than a warp's loads, remainders; widths off the 128-channel slice; vocabularies up to the largest
@pytest.mark.parametrize("T,C,V,rms", [(1, 64, 32, False), (15, 136, 32, False), (193, 256, 31, True), (3001, 1024, 32, False),
                                       (700, 2056, 28, False), (500, 384, 200, False), (500, 384, 201, True)])
@pytest.mark.parametrize("weighted", [True, False])
def test_embedding_norm_backward(T, C, V, rms, weighted, cuda_status):
    from nanoplm_b200.ops import kernels as k
    torch.manual_seed(T + C)
    table = (torch.randn(V, C, device="cuda") * 0.02).to(BF)
    w = (1 + 0.1 * torch.randn(C, device="cuda")).to(BF) if weighted else None
    ids = torch.randint(0, V, (T,), device="cuda", dtype=torch.int32)
    dy = torch.randn(T, C, device="cuda").to(BF)
    _, mean, rstd = k.norm_fwd(table, w, 1e-5, rms=rms, ids=ids)
    dtable, dw = torch.ones(V, C, device="cuda"), torch.ones(C, device="cuda")     # (both are added to)
    k.norm_bwd(dy, table, w, mean, rstd, rms=rms, ids=ids, dtable=dtable, dw=dw if weighted else None)
    t64 = table.double().requires_grad_(True)
    w64 = (w if weighted else torch.ones(C, device="cuda")).double().requires_grad_(True)
    x = t64[ids.long()]
    if not rms:
        x = x - x.mean(-1, keepdim=True)
    (x * torch.rsqrt(x.pow(2).mean(-1, keepdim=True) + 1e-5) * w64).backward(dy.double())
    # mean and rstd are fp32: 2^-24 each, amplified by at most the row's few hundred cancelling terms
    assert _rel(dtable - 1, t64.grad) < 1e-4
    assert torch.equal(dtable[t64.grad.abs().sum(1) == 0], torch.ones_like(dtable[t64.grad.abs().sum(1) == 0]))
    if weighted:
        assert _rel(dw - 1, w64.grad) < 1e-4


@pytest.mark.parametrize("n,C,V", [(1, 64, 32), (15, 136, 29), (17, 256, 32), (449, 264, 1), (2000, 1024, 31), (333, 2048, 32)])
@pytest.mark.parametrize("offset", [0, 1])
def test_decoder_backward(n, C, V, offset, cuda_status):
    from nanoplm_b200.ops import kernels as k
    torch.manual_seed(n + C)
    h, W = torch.randn(n, C, device="cuda").to(BF), (torch.randn(V, C, device="cuda") * 0.05).to(BF)
    dl = torch.zeros(n, 32, device="cuda")
    dl[:, :V] = torch.randn(n, V, device="cuda") / n
    dl[::5] = 0
    # a running gradient may start at any fp32 of a flat buffer
    dW = torch.ones(V * C + offset, device="cuda")[offset:].view(V, C)
    db = torch.ones(V, device="cuda")
    gs = torch.full((1,), 0.5, device="cuda")
    dh = k.ce_bwd(h, W, dl, gs, dW, db)
    d = dl[:, :V].double() * 0.5
    ref_h = d @ W.double()
    assert _rel(dh, ref_h) < 2 ** -8 if ref_h.norm() > 0 else dh.abs().max() == 0      # rounded once, to bf16
    # each sum is added to the 1 that is there: 2^-24 of it on top of the sums' own rounding
    assert (dW.double() - 1 - d.t() @ h.double()).abs().max() < 1e-5
    assert (db.double() - 1 - d.sum(0)).abs().max() < 1e-5


@pytest.mark.parametrize("n", [0, 1, 31, 1024, 1025, 70001])
def test_label_count(n, cuda_status):
    from nanoplm_b200.ops import kernels as k
    labels = torch.randint(-2, 3, (n,), device="cuda", dtype=torch.int32)
    inv, loss = k.ce_count(labels)
    assert inv.item() == (1.0 / (labels >= 0).sum().clamp(min=1).float()).item() and loss.item() == 0


@pytest.mark.parametrize("C,V", [(256, 32), (1024, 31), (1032, 29), (2048, 32)])
def test_decoder_backward_of_ignored_rows(C, V, cuda_status):
    """Rows whose dlogits are all zero have a zero gradient whatever they hold."""
    from nanoplm_b200.ops import kernels as k
    n = 83
    h, W = torch.randn(n, C, device="cuda").to(BF), (torch.randn(V, C, device="cuda") * 0.05).to(BF)
    dl = torch.zeros(n, 32, device="cuda")
    dl[:, :V] = torch.randn(n, V, device="cuda") / n
    dl[::3] = 0
    bad = h.clone()
    bad[::6], bad[3::6] = float("inf"), float("nan")
    gs = torch.full((1,), 0.5, device="cuda")
    grads = []
    for x in (bad, h):
        dW, db = torch.zeros(V, C, device="cuda"), torch.zeros(V, device="cuda")
        grads.append((k.ce_bwd(x, W, dl, gs, dW, db), dW, db))
    (dh, dW, db), (dh_ref, dW_ref, db_ref) = grads
    assert torch.equal(dh, dh_ref) and dh[::3].abs().max() == 0
    # the blocks' sums are added in any order
    assert (dW - dW_ref).abs().max() < 1e-6 and (db - db_ref).abs().max() < 1e-6
