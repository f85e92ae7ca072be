"""embed_sequences hands the model flat ids only where nobody observes the padded call."""
import pytest
import torch
from torch.nn.modules import module as nn_module


@pytest.fixture
def model():
    from nanoplm_b200.config.schema import StudentConfig
    from nanoplm_b200.models.student import ProtX
    return ProtX(StudentConfig(hidden_size=64, intermediate_size=64, num_hidden_layers=1, num_attention_heads=1)).to(
        torch.bfloat16)


@pytest.mark.parametrize("how", ["nobody", "hook", "pre_hook", "global_hook", "global_pre_hook", "instance", "subclass"])
def test_observers(how, model):
    handle = None
    if how == "hook":
        handle = model.register_forward_hook(lambda *a: None)
    elif how == "pre_hook":
        handle = model.register_forward_pre_hook(lambda *a: None)
    elif how == "global_hook":
        handle = nn_module.register_module_forward_hook(lambda *a: None)
    elif how == "global_pre_hook":
        handle = nn_module.register_module_forward_pre_hook(lambda *a: None)
    elif how == "instance":
        model.forward = lambda *a, **k: type(model).forward(model, *a, **k)
    elif how == "subclass":
        base = type(model)
        model.__class__ = type("Sub", (base,), {"forward": lambda self, *a, **k: base.forward(self, *a, **k)})
    try:
        assert model._embeds_packed(torch.device("cuda")) is (how == "nobody")
    finally:
        if handle is not None:
            handle.remove()
