"""Memory of the native layer launch sequence: without gradients it holds no more than the op-by-op path does."""
import ctypes

import pytest

from nanoplm_b200.csrc import build


@pytest.fixture(scope="module")
def layer_bytes():
    f = ctypes.CDLL(str(build.build_host("layer.cpp"))).nplm_layer_bytes
    f.argtypes, f.restype = [ctypes.c_longlong] * 4 + [ctypes.c_int] * 3, ctypes.c_longlong
    return f


@pytest.mark.parametrize("T", [1, 37, 128, 55424])
@pytest.mark.parametrize("C,I,H", [(64, 64, 1), (256, 512, 4), (512, 1024, 8), (1024, 2048, 16), (128, 1024, 2), (512, 64, 8)])
@pytest.mark.parametrize("norm1", [0, 1])
def test_inference_buffer(T, C, I, H, norm1, layer_bytes):
    # op by op, with dead tensors freed: the attention holds its input, qkv and its output, the MLP x1, h2 and hs
    HD = H * 64
    attention = norm1 * C * 2 + 3 * HD * 2 + HD * 2 + H * 4
    mlp = C * 2 + C * 2 + I * 2
    assert layer_bytes(T, C, I, H, norm1, 0, 0) <= T * (C * 2 + max(attention, mlp - C * 2)) + 5 * 256
    assert layer_bytes(T, C, I, H, norm1, 1, 0) >= T * (norm1 * C + 4 * HD + 2 * C + 3 * I) * 2 + T * H * 4
