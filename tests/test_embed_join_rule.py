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


def _wrap_attention(m):
    m.layers[0].attn = torch.nn.Sequential(m.layers[0].attn)


@pytest.mark.parametrize("change", [_wrap_attention, lambda m: m.layers[0].float()])
def test_replaced_or_fp32_attention_does_not(change):
    m = _model()
    change(m)
    assert m._join_tokens() == 0
