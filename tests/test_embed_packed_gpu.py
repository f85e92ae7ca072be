"""Embedding of raw sequences through packed batches: against the padded forward, and the pooling kernel."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


@pytest.mark.parametrize("C", [8, 64, 72, 512, 1000])
@pytest.mark.parametrize("lens", [[1], [2, 1, 33], [31, 32, 34, 257], [1023, 3]])
@pytest.mark.parametrize("drop", [0, 1])
def test_segment_mean(C, lens, drop, cuda_status):
    from nanoplm_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(C + sum(lens))
    x = torch.randn(sum(lens), C, device="cuda", generator=g).to(BF)
    cu = torch.tensor([0, *lens], dtype=torch.int32).cumsum(0, dtype=torch.int32).cuda()
    got = K.segment_mean(x, cu, drop)
    want = torch.stack([x[int(a):int(b) - drop].double().mean(0) for a, b in zip(cu[:-1], cu[1:])])
    # fp32 sums of at most 1023 terms: below 1e-5 of the largest magnitude; an empty mean is NaN
    assert torch.allclose(got.double(), want, rtol=0, atol=5e-5, equal_nan=True)


@pytest.mark.parametrize("per_token", [False, True])
@pytest.mark.parametrize("batch_size", [1, 3, 16])
def test_embed_sequences_matches_the_padded_forward(per_token, batch_size, cuda_status):
    from nanoplm_b200.config.schema import StudentConfig
    from nanoplm_b200.data.synthetic import synthetic_sequences
    from nanoplm_b200.models.student import ProtX
    torch.manual_seed(0)
    m = ProtX(StudentConfig(hidden_size=256, intermediate_size=512, num_hidden_layers=2,
                            num_attention_heads=4)).cuda().to(BF)
    m.train()
    seqs = synthetic_sequences(7, 1, 200, seed=4) + ["A"]
    got = m.embed_sequences(seqs, batch_size=batch_size, per_token=per_token)
    assert m.training and len(got) == len(seqs)
    hook = m.register_forward_hook(lambda *a: None)          # an observer sees the padded call
    want = m.embed_sequences(seqs, batch_size=batch_size, per_token=per_token)
    hook.remove()
    for a, b in zip(got, want):
        assert a.device.type == "cpu" and a.dtype == b.dtype and a.shape == b.shape
        assert a.untyped_storage().nbytes() == a.numel() * 4          # its own storage
        # the same kernels on the same packed rows; the mean's fp32 sums run in another order
        assert torch.allclose(a, b, rtol=1e-5, atol=1e-5)
    assert m.embed_sequences([]) == []
