"""The native host side, without a GPU: it leaves to the Python code, untouched, every call that code refuses or prepares."""
import ctypes

import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200.attention import AttentionError, Unsupported, attention, attention_backward, attention_decode, attention_decode_append
from dashmag_b200.contract import AttentionMask, AttentionOptions
from dashmag_b200.rope import Rope, attention_decode_append_rope
from dashmag_b200.sample import SampleOptions, sample

NONE, OPTIONS = AttentionMask.none(), AttentionOptions()


def tensors(dtype=torch.bfloat16, device="cpu"):
    q, k = torch.zeros(1, 4, 2, 64, dtype=dtype, device=device), torch.zeros(1, 4, 1, 64, dtype=dtype, device=device)
    return q, k, k.clone()


@pytest.mark.parametrize("bad", ["cpu", "meta", "numpy", "none", "few"])
def test_everything_but_plain_cuda_tensors_is_left_alone(bad):
    b = _lib.binding()
    q, k, v = tensors(device="meta") if bad == "meta" else tensors()
    if bad == "numpy":
        q, k, v = (x.float().numpy() for x in (q, k, v))
    if bad == "none":
        q = None
    more = () if bad == "few" else (OPTIONS,)
    assert b.forward(q, k, v, NONE, *more) is None
    assert b.backward(q, k, v, q, q, q, NONE, *more) is None
    assert b.decode(q, k, v, None, *more) is None
    assert b.decode_append(q, k, v, k, v, None, *more) is None
    assert b.decode_append_rope(None, q, k, v, k, v, None, *more) is None
    assert b.sample(q, *((SampleOptions(),) if more else ())) is None


def test_refusals_are_the_python_side_s():
    q, k, v = tensors()
    with pytest.raises(Unsupported):
        attention(q, k, v)
    with pytest.raises(AttentionError, match="query is"):
        attention(q[0], k, v)
    with pytest.raises(AttentionError, match="output"):
        attention_backward(q, k, v, q[:, :2], q[..., 0], q)
    with pytest.raises(AttentionError, match=r"query is \[B, Hq, D\]"):
        attention_decode(q, k, v)
    with pytest.raises(ValueError, match="the lengths are needed"):
        attention_decode_append(q[0], k[0], v[0], k, v, None)
    with pytest.raises(AttentionError, match="the lengths are needed"):
        attention_decode_append_rope(Rope(64, 10000.0, 8, torch.bfloat16, device="cpu"), q[0], k[0], v[0], k, v, None)
    with pytest.raises(AttentionError, match="logits must be"):
        sample(q)


def test_the_binding_calls_the_library_that_is_loaded():
    b = _lib.binding()
    with pytest.raises(TypeError):
        b.use(1, 2)
    with pytest.raises(ValueError):
        b.use(*[0] * len(_lib.BOUND))
    for name in _lib.BOUND:
        assert ctypes.cast(getattr(_lib.lib(), name), ctypes.c_void_p).value
