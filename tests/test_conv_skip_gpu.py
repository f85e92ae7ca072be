"""Depthwise convolution with its skip connection in the same pass, against the sum as a pass of its own."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# sequences shorter than the taps; runs with a remainder of the rows loaded ahead; a size without a kernel of its own; channels
# off the warp's 128
@pytest.mark.parametrize("ks,C,lens", [(7, 64, [1]), (7, 776, [2, 500, 1, 90, 3001]), (3, 136, [700, 5]), (1, 64, [33, 8])])
@pytest.mark.parametrize("bias", [False, True])
def test_skip_in_the_convolution(ks, C, lens, bias, cuda_status):
    from nanoplm_b200.models.conv import dwconv_varlen
    torch.manual_seed(ks)
    ends = torch.tensor(lens).cumsum(0)
    rep = torch.tensor(lens)
    se = torch.repeat_interleave(ends, rep).to(torch.int32).cuda()
    ss = torch.repeat_interleave(ends - rep, rep).to(torch.int32).cuda()
    x0, dy = (torch.randn(sum(lens), C, device="cuda").to(BF) for _ in range(2))
    w0, b0 = (0.3 * torch.randn(C, ks, device="cuda")).to(BF), torch.randn(C, device="cuda").to(BF) if bias else None

    def run(skip):
        x, w = x0.clone().requires_grad_(True), w0.clone().requires_grad_(True)
        y = dwconv_varlen(x, w, b0, ss, se, skip=True) if skip else x + dwconv_varlen(x, w, b0, ss, se)
        y.backward(dy)
        return y.detach(), x.grad, w.grad.float()

    got, want = run(True), run(False)
    assert torch.equal(got[0], want[0]) and torch.equal(got[1], want[1])
    assert (got[2] - want[2]).norm() <= 2 ** -8 * want[2].norm()     # fp32 sums in any order, rounded to bf16
