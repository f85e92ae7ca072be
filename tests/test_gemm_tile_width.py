"""Default tile widths: one rule in two languages, and the bits of every width."""
import ctypes

import pytest
import torch

from nanoplm_b200.csrc import build
from nanoplm_b200.ops import kernels as K

EPIS = (K.EPI_STORE, K.EPI_ADD, K.EPI_ATOMIC_F32, K.EPI_GELU, K.EPI_STORE_F32, K.EPI_SWIGLU, K.EPI_ROPE, K.EPI_RELU,
        K.EPI_SWIGLU_BWD, 9)


def test_native_rule_is_the_same():
    f = ctypes.CDLL(str(build.build_host("layer.cpp"))).nplm_gemm_tile_width
    f.argtypes = [ctypes.c_longlong] * 2 + [ctypes.c_int]
    for M in (1, 127, 128, 129, 236, 1000, 1153, 2048, 2049, 4736, 4737, 9472, 9473, 18944, 18945, 55424):
        for N in (8, 64, 72, 128, 136, 192, 255, 256, 320, 512, 1024, 1536, 3072, 4096):
            for epi in EPIS:
                assert f(M, N, epi) == K.tile_width(M, N, epi), (M, N, epi)


@pytest.mark.gpu
@pytest.mark.parametrize("M,N,Kd", [(1, 64, 64), (129, 72, 200), (236, 320, 1088), (700, 512, 128)])
@pytest.mark.parametrize("epi", [K.EPI_STORE, K.EPI_ADD, K.EPI_GELU, K.EPI_RELU, K.EPI_ROPE])
@pytest.mark.parametrize("b_mn", [False, True])
def test_every_width_gives_the_same_bits(M, N, Kd, epi, b_mn, cuda_status):
    if (b_mn and (epi not in (K.EPI_STORE, K.EPI_ADD) or N % 64)) or (epi == K.EPI_ROPE and N % 64):
        pytest.skip("not a form of the kernel")
    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w = rnd(M, Kd).to(torch.bfloat16), (rnd(*((Kd, N) if b_mn else (N, Kd))) * 0.1).to(torch.bfloat16)
    kw = {}
    if epi == K.EPI_ADD:
        kw["aux"] = rnd(M, N).to(torch.bfloat16)
    if epi == K.EPI_ROPE:
        kw["rope"] = (torch.arange(M, device="cuda", dtype=torch.int32), rnd(M, 32), rnd(M, 32), N // 128 * 64)

    def run(bn):
        pre = torch.zeros(M, N, device="cuda", dtype=torch.bfloat16)
        out = K.gemm(x, w, b_mn=b_mn, epi=epi, bn=bn, **(dict(aux=pre) if epi in (K.EPI_GELU, K.EPI_RELU) else kw))
        return out, pre

    ref = run(256)
    for bn in (64, 128, None):
        got = run(bn)
        assert torch.equal(got[0], ref[0]) and torch.equal(got[1], ref[1])
