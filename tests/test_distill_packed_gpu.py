"""The distillation loss on packed states against the padded composition."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


@pytest.mark.parametrize("T,N,C", [(1, 1, 8), (77, 130, 64), (500, 700, 1024)])
def test_masked_mse_rows(T, N, C, cuda_status):
    from nanoplm_b200.ops import functional as ops
    g = torch.Generator(device="cuda").manual_seed(T)
    rows = torch.randperm(N, device="cuda", generator=g)[:T].sort().values
    s = torch.randn(T, C, device="cuda", generator=g).to(BF).requires_grad_(True)
    t = torch.randn(N, C, device="cuda", generator=g).to(BF)
    loss = ops.masked_mse_rows(s, t, rows)
    loss.backward()
    full = torch.zeros(N, C, device="cuda", dtype=BF).index_copy(0, rows, s.detach()).requires_grad_(True)
    mask = torch.zeros(N, dtype=torch.int64, device="cuda").index_fill(0, rows, 1)
    want = ops.masked_mse(full, t, mask)
    want.backward()
    assert torch.equal(s.grad, full.grad[rows])
    assert abs(loss.item() - want.item()) <= 1e-5 * want.item()      # fp32 sums over blocks in any order


def test_distillation_loss_skips_the_padding(cuda_status):
    from nanoplm_b200.config.schema import StudentConfig
    from nanoplm_b200.models.student import ProtX
    from nanoplm_b200.runtime.distill import DistillDataCollator, distillation_loss
    torch.manual_seed(0)
    student = ProtX(StudentConfig(hidden_size=128, intermediate_size=128, num_hidden_layers=2, num_attention_heads=2)).cuda()
    student = student.to(BF)
    b = DistillDataCollator(True, 64)([{"raw_sequence": q} for q in ("ACDEFGH", "MKV" * 15, "A")])
    batch = {k: b[k].cuda() for k in ("input_ids", "attention_mask")}
    batch["teacher_embeddings"] = torch.randn(3, 64, 1024, device="cuda").to(BF)

    def once():
        student.zero_grad()
        loss = distillation_loss(student, batch)
        loss.backward()
        return type(loss.grad_fn).__name__, loss.item(), [p.grad.float() for p in student.parameters()]

    seen = []
    _, loss, grads = once()
    hook = student.register_forward_hook(lambda m, a, out: seen.append(out["last_hidden_state"].shape))
    _, want, want_grads = once()
    hook.remove()
    assert seen == [(3, 64, 1024)]          # an observer sees the padded call
    assert abs(loss - want) <= 1e-5 * want
    for a, c in zip(grads, want_grads):     # the same kernels on the same rows; dQ and the weight gradients add in any order
        assert (a - c).norm() <= 1e-2 * c.norm() + 1e-6
