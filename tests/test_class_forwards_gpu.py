"""A forward that a program puts on a class of the package is called, whatever native path there is."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


def _counting(monkeypatch, cls):
    seen, real = [], cls.forward
    monkeypatch.setattr(cls, "forward", lambda self, *a, **k: (seen.append(self), real(self, *a, **k))[1])
    return seen


@pytest.mark.parametrize("streams", [1, 4])
@pytest.mark.parametrize("grad", [True, False])
def test_a_forward_put_on_the_class_is_called(streams, grad, monkeypatch, cuda_status):
    from nanoplm_b200.config.schema import ModelConfig
    from nanoplm_b200.models import encoder
    torch.manual_seed(1)
    m = encoder.EncoderModel(ModelConfig(hidden_size=64, intermediate_size=64, num_hidden_layers=3, num_attention_heads=1,
                                         max_position_embeddings=512, mhc_streams=streams)).cuda().to(BF)
    with torch.no_grad():
        for p in m.parameters():
            p.copy_(1 + 0.1 * torch.randn_like(p) if p.ndim == 1 else torch.randn_like(p) * 0.05)
            p.main_grad = torch.zeros(p.shape, device="cuda")
    cu = torch.tensor([0, 50, 70], dtype=torch.int32, device="cuda")
    ctx = encoder.BatchContext(cu, encoder.position_ids_from_cu_seqlens(cu, 70), 70)
    ids = torch.randint(3, 28, (70,), device="cuda")
    with torch.set_grad_enabled(grad):
        want, _ = m.forward_hidden(ids, ctx)
    seen = _counting(monkeypatch, encoder.EncoderLayer)
    with torch.set_grad_enabled(grad):
        got, _ = m.forward_hidden(ids, ctx)
    assert seen == list(m.layers) and torch.equal(got, want)


def test_a_forward_put_on_the_student_is_called(monkeypatch, cuda_status):
    from nanoplm_b200.config.schema import StudentConfig
    from nanoplm_b200.models.student import ProtX
    from nanoplm_b200.runtime.distill import distillation_loss
    torch.manual_seed(0)
    m = ProtX(StudentConfig(hidden_size=128, intermediate_size=256, num_hidden_layers=2, num_attention_heads=2,
                            teacher_dim=64)).cuda().to(BF)
    seqs = ["MKTAYIAKQR", "ACDEF", "GHIKLMNP"]
    ids = torch.randint(3, 20, (2, 9), device="cuda")
    batch = {"input_ids": ids, "attention_mask": torch.ones_like(ids),
             "teacher_embeddings": torch.randn(2, 9, 64, device="cuda").to(BF)}
    want, loss = m.embed_sequences(seqs, batch_size=2), distillation_loss(m, batch)
    seen = _counting(monkeypatch, ProtX)
    got = m.embed_sequences(seqs, batch_size=2)
    assert len(seen) == 2
    for a, b in zip(got, want):         # (the padded call pools in another order)
        assert (a - b).norm() <= 1e-5 * b.norm()
    assert abs(distillation_loss(m, batch).item() - loss.item()) <= 1e-5 * abs(loss.item()) and len(seen) == 3
