"""Which GEMMs run on CTA pairs by default: one rule in two languages, and the bits of both forms."""
import ctypes

import pytest
import torch

from nanoplm_b200.csrc import build
from nanoplm_b200.ops import kernels as K

EPIS = (K.EPI_STORE, K.EPI_ADD, K.EPI_GELU, K.EPI_RELU, K.EPI_SWIGLU, K.EPI_ROPE, K.EPI_SWIGLU_BWD, 9)


def test_native_rule_is_the_same():
    f = ctypes.CDLL(str(build.build_host("layer.cpp"))).nplm_gemm_pair_pays
    f.argtypes = [ctypes.c_longlong] * 3 + [ctypes.c_int]
    for M in (1, 127, 128, 129, 236, 1000, 4736, 4737, 6144, 8704, 17024, 40000, 55424, 10 ** 6):
        for N in (64, 256, 257, 512, 1024, 1536, 2304, 3072, 4096, 16384):
            for Kd in (64, 512, 704, 768, 1024, 4096):
                for epi in EPIS:
                    assert bool(f(M, N, Kd, epi)) == K.pair_pays(M, N, Kd, epi), (M, N, Kd, epi)


@pytest.mark.parametrize("M", [1, 64, 128, 236, 512])
@pytest.mark.parametrize("C", [256, 512, 768, 1024])
def test_few_rows_stay_on_single_ctas(M, C):
    """Pairs were up to 1.3 times slower there (1536 columns of 512, RoPE: 9.3 against 12.2 us)."""
    for N, Kd, epi in ((3 * C, C, K.EPI_ROPE), (C, C, K.EPI_ADD), (4 * C, C, K.EPI_SWIGLU), (C, 2 * C, K.EPI_ADD),
                       (C, 4 * C, K.EPI_STORE), (C, C, K.EPI_GELU)):
        assert not K.pair_pays(M, N, Kd, epi)
    assert K.pair_pays(55424, 4 * C, 1024, K.EPI_STORE)


@pytest.mark.gpu
@pytest.mark.parametrize("M", [1, 129, 700])
@pytest.mark.parametrize("epi", [K.EPI_STORE, K.EPI_ADD, K.EPI_SWIGLU, K.EPI_ROPE])
def test_both_forms_give_the_same_bits(M, epi, cuda_status):
    g = torch.Generator(device="cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=g)
    x, w = rnd(M, 256).to(torch.bfloat16), (rnd(768, 256) * 0.1).to(torch.bfloat16)
    kw = {}
    if epi == K.EPI_ADD:
        kw["aux"] = rnd(M, 768).to(torch.bfloat16)
    if epi == K.EPI_ROPE:
        kw["rope"] = (torch.arange(M, device="cuda", dtype=torch.int32), rnd(M, 32), rnd(M, 32), 512)
    single, pair, default = (K.gemm(x, w, epi=epi, pair=p, **kw) for p in (False, True, None))
    assert torch.equal(single, pair) and torch.equal(single, default)
