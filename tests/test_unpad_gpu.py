"""Padded batches to packed ones against the composition of tensor operations: whole numbers, the same ones."""
import pytest
import torch
import torch.nn.functional as F

pytestmark = pytest.mark.gpu


def _composed(ids, mask):
    from nanoplm_b200.models.encoder import position_ids_from_cu_seqlens
    index = torch.nonzero(mask.reshape(-1).bool(), as_tuple=False).flatten()
    cu = F.pad(torch.cumsum(mask.sum(dim=-1, dtype=torch.int32), 0, dtype=torch.int32), (1, 0))
    return ids.reshape(-1)[index], index, position_ids_from_cu_seqlens(cu, index.numel(), ids.device), cu


# one position, a block's width and around it, more rows than one block scans
@pytest.mark.parametrize("B,S", [(1, 1), (2, 255), (3, 256), (5, 257), (9, 1001), (1024, 3), (2500, 2)])
@pytest.mark.parametrize("mask_dtype", [torch.int64, torch.int32, torch.bool, torch.uint8])
@pytest.mark.parametrize("how", ["leading", "holes", "empty rows", "nothing"])
def test_unpad(B, S, mask_dtype, how, cuda_status):
    from nanoplm_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(B + S)
    at = torch.arange(S, device="cuda")[None]
    if how == "holes":
        mask = torch.rand(B, S, device="cuda", generator=g) < 0.7
    else:
        low = 0 if how == "empty rows" else 1
        mask = at < torch.randint(low, S + 1, (B, 1), device="cuda", generator=g)
        if how == "nothing":
            mask &= False
    mask = mask.to(mask_dtype)
    ids = torch.randint(0, 32, (B, S), device="cuda", generator=g,
                        dtype=torch.int32 if mask_dtype == torch.bool else torch.int64)
    assert K.unpad_takes(ids, mask)
    for got, want in zip(K.unpad(ids, mask), _composed(ids, mask)):
        assert got.dtype == want.dtype and torch.equal(got, want)


def test_unpad_leaves_other_batches(cuda_status):
    from nanoplm_b200.ops import kernels as K
    ids, mask = torch.zeros(2, 8, dtype=torch.int64, device="cuda"), torch.ones(2, 8, dtype=torch.int64, device="cuda")
    assert K.unpad_takes(ids, mask)
    assert not K.unpad_takes(ids, mask.float()) and not K.unpad_takes(ids.float(), mask)
    assert not K.unpad_takes(ids, mask[:, :4]) and not K.unpad_takes(ids[:, ::2], mask[:, ::2])
    assert not K.unpad_takes(ids[:0], mask[:0]) and not K.unpad_takes(ids.cpu(), mask.cpu())
