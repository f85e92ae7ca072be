"""When embed_sequences may run several batches as one."""
import pytest
import torch

from nanoplm_b200.config.schema import StudentConfig
from nanoplm_b200.models import student


def _model(hidden=128, heads=2, **kw):
    return student.ProtX(StudentConfig(hidden_size=hidden, intermediate_size=2 * hidden, num_hidden_layers=2,
                                       num_attention_heads=heads, **kw)).to(torch.bfloat16).eval()


def test_heads_of_64_join():
    assert _model()._join_tokens() == student._EMBED_TOKENS
    assert _model(512, 8)._join_tokens() == student._EMBED_TOKENS


@pytest.mark.parametrize("heads", [1, 4, 8])             # 128, 32 and 16 wide: the dense form, which has no rows without keys
def test_other_heads_do_not(heads):
    assert _model(heads=heads)._join_tokens() == 0


def test_memory_bounds_the_tokens():
    wide, streams = _model(1024, 16)._join_tokens(), _model(512, 8, mhc_streams=4)._join_tokens()
    assert 0 < wide < student._EMBED_TOKENS and 0 < streams < student._EMBED_TOKENS


def _wrap(m):
    m.layers[1].mlp.forward = m.layers[1].mlp.forward


@pytest.mark.parametrize("watch", [lambda m: m.layers[0].register_forward_hook(lambda *a: None),
                                   lambda m: m.layers[1].attn.Wo.register_forward_pre_hook(lambda *a: None), _wrap,
                                   lambda m: setattr(m.layers[0].mlp.Wi.weight, "_ag", object()),
                                   lambda m: m.layers[0].float()])
def test_watched_gathered_or_fp32_layers_do_not(watch):
    m = _model()
    watch(m)
    assert m._join_tokens() == 0
