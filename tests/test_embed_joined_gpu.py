"""Batches that embed_sequences joins have the bits that they have one by one."""
import pytest
import torch

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("per_token", [False, True])
@pytest.mark.parametrize("variant", ["plain", "conv_mhc"])
@pytest.mark.parametrize("batch_size,n,hi", [(1, 5, 40), (4, 17, 300), (16, 90, 900)])
def test_joined_batches(per_token, variant, batch_size, n, hi, cuda_status, monkeypatch):
    from nanoplm_b200.config.schema import StudentConfig
    from nanoplm_b200.data.synthetic import synthetic_sequences
    from nanoplm_b200.models import student
    torch.manual_seed(0)
    kw = dict(conv_kernel_size=7, mhc_streams=4) if variant == "conv_mhc" else {}
    m = student.ProtX(StudentConfig(hidden_size=256, intermediate_size=512, num_hidden_layers=4, num_attention_heads=4,
                                    **kw)).cuda().to(torch.bfloat16).eval()
    seqs = synthetic_sequences(n, 1, hi, seed=n) + ["A"]
    calls = []
    real = student.ProtX._embed_packed
    monkeypatch.setattr(student.ProtX, "_embed_packed", lambda self, *a: (calls.append(len(a[0])), real(self, *a))[1])
    got = m.embed_sequences(seqs, batch_size=batch_size, per_token=per_token)
    joined = len(calls)
    assert joined < -(-len(seqs) // batch_size) and max(calls) <= student._EMBED_TOKENS
    hook = m.layers[0].register_forward_hook(lambda *a: None)        # somebody may count the batches: one by one
    want = m.embed_sequences(seqs, batch_size=batch_size, per_token=per_token)
    hook.remove()
    assert len(calls) - joined == -(-len(seqs) // batch_size)
    assert len(got) == len(want) == len(seqs)
    for a, b in zip(got, want):
        assert torch.equal(a, b)
    with pytest.raises(ValueError):
        m.embed_sequences(seqs, batch_size=0)
    assert m.embed_sequences(seqs, batch_size=-1) == []
