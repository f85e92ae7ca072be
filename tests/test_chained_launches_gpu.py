"""Kernels wait for their predecessor themselves, so their order is theirs to keep: in a captured graph, and beside another
stream's kernels."""
import pytest
import torch

pytestmark = pytest.mark.gpu
BF = torch.bfloat16
LENS = [37, 90, 300, 1, 129]


class _Step:
    """Forward and backward pass of three layers on fixed buffers; the same bits every run."""

    def __init__(self, seed, **kw):
        from nanoplm_b200.config.schema import ModelConfig
        from nanoplm_b200.models.encoder import BatchContext, EncoderModel, position_ids_from_cu_seqlens
        torch.manual_seed(seed)
        self.m = EncoderModel(ModelConfig(hidden_size=256, intermediate_size=512, num_hidden_layers=3, num_attention_heads=4,
                                          max_position_embeddings=512, **kw)).cuda().to(BF)
        with torch.no_grad():
            for p in self.m.parameters():
                p.copy_(1 + 0.1 * torch.randn_like(p) if p.ndim == 1 else torch.randn_like(p) * 0.05)
        cu = torch.tensor([0, *LENS]).cumsum(0).to(torch.int32).cuda()
        self.ctx = BatchContext(cu, position_ids_from_cu_seqlens(cu, sum(LENS)), sum(LENS))
        self.ids = torch.zeros(sum(LENS), dtype=torch.int64, device="cuda")
        self.dy = torch.zeros(sum(LENS), 256, device="cuda", dtype=BF)
        for p in self.m.parameters():
            p.main_grad = torch.zeros(p.shape, device="cuda")
        self.draw(seed)

    def draw(self, seed):
        g = torch.Generator("cuda").manual_seed(seed)
        self.ids.random_(3, 28, generator=g)
        self.dy.normal_(0, 0.1, generator=g)

    def __call__(self):
        for p in self.m.parameters():
            p.main_grad.zero_()
        y, _ = self.m.forward_hidden(self.ids, self.ctx)
        y.backward(self.dy)
        self.y = y.detach()

    def results(self):
        return {"y": self.y.clone(), **{n: p.main_grad.clone() for n, p in self.m.named_parameters()}}


def _same(got, want):
    for n in want:
        if n == "y" or ("attn.W" in n or "mlp.W" in n):
            assert torch.equal(got[n], want[n]), n
        else:       # norm, convolution and stream weights, the embedding: fp32 sums over blocks in any order
            assert (got[n] - want[n]).norm() <= 1e-4 * want[n].norm() + 1e-6, n


@pytest.fixture(autouse=True)
def _reproducible():
    from nanoplm_b200.ops import kernels as K
    K.set_attention_deterministic(True)
    yield
    K.set_attention_deterministic(False)


VARIANTS = [{}, dict(conv_kernel_size=7, mhc_streams=4)]


@pytest.mark.parametrize("kw", VARIANTS)
def test_captured_step(kw, cuda_status):
    s = _Step(1, **kw)
    side = torch.cuda.Stream()
    side.wait_stream(torch.cuda.current_stream())
    with torch.cuda.stream(side):
        s()
        s()
    torch.cuda.current_stream().wait_stream(side)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        s()
    for seed in (2, 3, 4):
        s.draw(seed)
        graph.replay()
        graph.replay()              # (a step of the same graph follows at once)
        got = s.results()
        captured = s.y
        s()
        _same(got, s.results())
        s.y = captured


@pytest.mark.parametrize("kw", VARIANTS)
def test_steps_on_two_streams(kw, cuda_status):
    a, b = _Step(5, **kw), _Step(6, **kw)
    a(), b()
    want = a.results(), b.results()
    torch.cuda.synchronize()
    streams = torch.cuda.Stream(), torch.cuda.Stream()
    for _ in range(6):
        for s, st in zip((a, b), streams):
            with torch.cuda.stream(st):
                s()
    torch.cuda.synchronize()
    _same(a.results(), want[0])
    _same(b.results(), want[1])
