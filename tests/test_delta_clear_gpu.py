"""The output-projection data gradient that also clears the attention backward's sums."""
import ctypes

import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16


# one row, remainders of a 32-row and a 256-row tile, one head and heads past a tile's 256 columns, several waves
@pytest.mark.parametrize("M,N,K", [(1, 64, 64), (161, 320, 128), (257, 1024, 256), (9000, 512, 512)])
def test_clears_its_rows_and_no_others(M, N, K, cuda_status):
    from nanoplm_b200.ops import kernels as k
    from nanoplm_b200.ops._lib import check_rc, lib, ptr, status_word, stream_ptr
    torch.manual_seed(M)
    rnd = lambda *s: torch.randn(*s, device="cuda").to(BF)
    dy, w, o = rnd(M, K), rnd(K, N), rnd(M, N)
    delta_ref = torch.empty(N // 64, M, device="cuda")
    ref = k.gemm_dgrad_delta(dy, w, o, delta_ref)
    out, delta = torch.empty_like(ref), torch.empty_like(delta_ref)
    sums = torch.full((M + 2, N), 7.0, device="cuda")
    i = ctypes.c_int
    rc = lib("gemm_tcgen05").nplm_gemm_bf16_delta(ptr(dy), ptr(w), ptr(out), ptr(o), ptr(delta), ptr(sums[1:]), i(M), i(N), i(K),
                                                  i(K), i(N), i(N), i(N), i(1), ptr(status_word(dy.device)), stream_ptr())
    check_rc(rc, "gemm_bf16_delta")
    assert torch.equal(out, ref) and torch.equal(delta, delta_ref)
    assert (sums[1:M + 1] == 0).all() and (sums[0] == 7).all() and (sums[M + 1] == 7).all()
