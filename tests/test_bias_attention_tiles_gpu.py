"""Relative-position-bias attention at the edges of its tiles and of its bias table, packed and padded layouts."""
import pytest
import torch

pytestmark = pytest.mark.gpu

BF = torch.bfloat16


def _check(D, H, S, start, end, seed, scale=0.5):
    from nanoplm_b200.ops import kernels as K
    T = start.numel()
    g = torch.Generator(device="cuda").manual_seed(seed)
    qkv = (torch.randn(T, 3 * H * D, device="cuda", generator=g) * 0.5).to(BF)
    table = torch.randn(H, 2 * S - 1, device="cuda", generator=g) * 2.0
    out = K.fa_bias_fwd(qkv, start, end, table, H, D, scale)
    q, k, v = qkv.double().view(T, 3, H, D).unbind(1)
    pos = torch.arange(T, device="cuda")
    ok = (pos[None, :] >= start[:, None]) & (pos[None, :] < end[:, None])
    idx = (pos[None, :] - pos[:, None] + S - 1).clamp(0, 2 * S - 2)
    for h in range(H):
        s = (q[:, h] @ k[:, h].t() * scale + table[h].double()[idx]).masked_fill(~ok, float("-inf"))
        p = torch.nan_to_num(torch.softmax(s, -1))          # a row without keys gives zeros
        want = p @ v[:, h]
        # probabilities are rounded to bf16 (2^-9 each, relative, of their share) and the result once more
        bound = (p @ v[:, h].abs()) * 2 ** -8 + want.abs() * 2 ** -8 + 1e-6
        got = out.view(T, H, D)[:, h].double()
        assert ((got - want).abs() <= bound).all(), ((got - want).abs() / bound).max().item()


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("lens", [[1], [63], [64, 1], [127, 129], [128, 128, 1], [256], [257, 3, 255], [2, 5, 600, 31, 64]])
def test_packed_layouts(D, lens, cuda_status):
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    start = torch.cat([torch.full((n,), a) for n, a in zip(lens, cu)]).to(torch.int32).cuda()
    end = torch.cat([torch.full((n,), b) for n, b in zip(lens, cu[1:])]).to(torch.int32).cuda()
    _check(D, 3, max(lens), start, end, seed=sum(lens))


@pytest.mark.parametrize("D", [64, 128])
def test_rows_without_keys_and_long_ranges(D, cuda_status):
    # a whole tile of rows without keys, then a range longer than the bias table a tile keeps on chip (2 176 keys)
    T = 128 + 2500
    start, end = torch.zeros(T, dtype=torch.int32), torch.zeros(T, dtype=torch.int32)
    start[128:], end[128:] = 128, T
    _check(D, 1, 2500, start.cuda(), end.cuda(), seed=5)


def test_many_items_per_block(cuda_status):
    lens = [300, 41, 512, 7, 260] * 8
    cu = [0]
    for n in lens:
        cu.append(cu[-1] + n)
    start = torch.cat([torch.full((n,), a) for n, a in zip(lens, cu)]).to(torch.int32).cuda()
    end = torch.cat([torch.full((n,), b) for n, b in zip(lens, cu[1:])]).to(torch.int32).cuda()
    _check(128, 16, 512, start, end, seed=9)


@pytest.mark.parametrize("D", [64, 128])
@pytest.mark.parametrize("empty", [False, True])
def test_buffers_are_given_back_in_order(D, empty, cuda_status):
    """Several items a block, among them some whose second tile has no rows (a last pair of 100) and, with `empty`, runs
    of items without keys: these wait for no product and may not run ahead of the buffers they share."""
    T, S = 20 * 256 + 100, 256
    start = torch.arange(T, dtype=torch.int32) // S * S
    end = (start + S).clamp(max=T)
    if empty:
        end[1024:3072] = start[1024:3072]
    for seed in range(3):
        _check(D, 32, S, start.cuda(), end.cuda(), seed=seed)


@pytest.mark.parametrize("D,H", [(128, 8), (64, 8)])
@pytest.mark.parametrize("lens", [[20], [61, 120, 37], [511, 300], [1000, 640]])
@pytest.mark.parametrize("qk,b", [(0.3, 0.2), (0.6, 2.0), (1.2, 4.0)])
def test_no_further_from_fp64_than_one_rounding_of_the_probabilities(D, H, lens, qk, b, cuda_status):
    """Against a softmax in fp32 whose probabilities are rounded to bf16 once, relative to the row's maximum (which is
    then exact), and whose result is rounded to bf16: the kernel may be 2 % further from fp64 (its maximum runs over blocks
    of keys, so single roundings differ)."""
    from nanoplm_b200.ops import kernels as K
    g = torch.Generator(device="cuda").manual_seed(D + len(lens))
    T, S = sum(lens), max(lens)
    cu = torch.tensor([0, *lens]).cumsum(0).tolist()
    start = torch.cat([torch.full((n,), a) for n, a in zip(lens, cu)]).to(torch.int32).cuda()
    end = torch.cat([torch.full((n,), e) for n, e in zip(lens, cu[1:])]).to(torch.int32).cuda()
    qkv = torch.randn(T, 3 * H * D, device="cuda", generator=g)
    qkv[:, :2 * H * D] *= qk
    qkv = qkv.to(BF)
    table = torch.randn(H, 2 * S - 1, device="cuda", generator=g) * b
    out = K.fa_bias_fwd(qkv, start, end, table, H, D, 1.0).view(T, H, D).double()
    err = ref_err = 0.0
    for a, e in zip(cu, cu[1:]):
        q, k, v = qkv[a:e].double().view(e - a, 3, H, D).permute(1, 2, 0, 3)
        pos = torch.arange(e - a, device="cuda")
        s = q @ k.transpose(1, 2) + table.double()[:, pos[None] - pos[:, None] + S - 1]
        want = torch.softmax(s, -1) @ v
        p = torch.exp(s - s.amax(-1, keepdim=True))
        once = ((p.to(BF).double() @ v) / p.sum(-1, keepdim=True)).to(BF).double()
        err += (out[a:e].transpose(0, 1) - want).square().sum().item()
        ref_err += (once - want).square().sum().item()
    assert err ** 0.5 <= 1.02 * ref_err ** 0.5, (err / ref_err) ** 0.5
