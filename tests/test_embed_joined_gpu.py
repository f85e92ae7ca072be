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


def _student(hidden, heads, layers=3, **kw):
    from nanoplm_b200.config.schema import StudentConfig
    from nanoplm_b200.models import student
    torch.manual_seed(0)
    return student.ProtX(StudentConfig(hidden_size=hidden, intermediate_size=2 * hidden, num_hidden_layers=layers,
                                       num_attention_heads=heads, **kw)).cuda().to(torch.bfloat16).eval()


def _runs(monkeypatch):
    from nanoplm_b200.models import student
    calls, real = [], student.ProtX._embed_packed
    monkeypatch.setattr(student.ProtX, "_embed_packed", lambda self, *a: (calls.append(len(a[0])), real(self, *a))[1])
    return calls


@pytest.mark.parametrize("hidden,heads", [(128, 4), (256, 2)])           # heads of 32 and of 128
@pytest.mark.parametrize("per_token", [False, True])
def test_other_head_widths_stay_apart(hidden, heads, per_token, cuda_status, monkeypatch):
    from nanoplm_b200.data.synthetic import synthetic_sequences
    m, calls = _student(hidden, heads), _runs(monkeypatch)
    seqs = synthetic_sequences(9, 5, 60, seed=1)
    got = m.embed_sequences(seqs, batch_size=4, per_token=per_token)
    assert len(calls) == 3
    want = [e for i in range(0, 9, 4) for e in m.embed_sequences(seqs[i:i + 4], batch_size=4, per_token=per_token)]
    for a, b in zip(got, want, strict=True):
        assert torch.isfinite(a).all() and torch.equal(a, b)


@pytest.mark.parametrize("hidden,kw", [(512, {}), (1024, {}), (512, dict(conv_kernel_size=7, mhc_streams=4))])
def test_memory_of_joined_batches(hidden, kw, cuda_status, monkeypatch):
    from nanoplm_b200.data.synthetic import synthetic_sequences
    from nanoplm_b200.models import student
    m, calls = _student(hidden, hidden // 64, 2, **kw), _runs(monkeypatch)
    seqs = synthetic_sequences(110, 400, 500, seed=2)                    # 50 000 tokens
    m.embed_sequences(seqs[:2])
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    calls.clear()
    m.embed_sequences(seqs, batch_size=2)
    assert 0.8 * m._join_tokens() < max(calls) <= m._join_tokens()
    assert torch.cuda.max_memory_allocated() - before <= student._EMBED_BYTES


def test_joined_batches_that_do_not_fit(cuda_status, monkeypatch):
    from nanoplm_b200.data.synthetic import synthetic_sequences
    from nanoplm_b200.models import student
    m = _student(128, 2)
    seqs = synthetic_sequences(9, 5, 60, seed=3)
    want = m.embed_sequences(seqs, batch_size=2)
    real, sizes = student.ProtX._embed_packed, []

    def packed(self, ids, lens, device, r):
        sizes.append(len(lens))
        if len(lens) > 2:
            raise torch.OutOfMemoryError("no room")
        return real(self, ids, lens, device, r)

    monkeypatch.setattr(student.ProtX, "_embed_packed", packed)
    got = m.embed_sequences(seqs, batch_size=2)
    assert sizes[0] > 2 and sizes[1:] == [2, 2, 2, 2, 1]
    assert len(got) == 9 and all(torch.equal(a, b) for a, b in zip(got, want))
    with pytest.raises(torch.OutOfMemoryError):                          # one batch that does not fit is an error as before
        m.embed_sequences(seqs, batch_size=9)
