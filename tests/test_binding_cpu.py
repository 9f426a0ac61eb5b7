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


@pytest.mark.parametrize("what", ["missing", "another torch", "not an extension"])
def test_without_a_native_host_side_the_python_side_makes_the_calls(what, monkeypatch, tmp_path):
    monkeypatch.setattr(_lib, "_binding", None)
    if what == "another torch":
        monkeypatch.setattr(torch, "__version__", "2.0.0")
    else:
        path = tmp_path / "_binding.so"
        if what == "not an extension":
            path.write_bytes(b"no library")
        monkeypatch.setattr(_lib, "BINDING_PATH", path)
    with pytest.warns(RuntimeWarning, match="the Python side"):
        b = _lib.binding()
    assert _lib.binding() is b and b.forward(1, 2) is None
    q, k, v = tensors()
    with pytest.raises(Unsupported):
        attention(q, k, v)


def test_another_torch_builds_the_binding_anew(monkeypatch, tmp_path):
    from dashmag_b200 import build

    commands = []
    monkeypatch.setattr(build, "BINDING", tmp_path / "_binding.so")
    monkeypatch.setattr(build, "OBJ", tmp_path)

    class Done:
        returncode = 0

    def compiler(cmd, **kwargs):
        commands.append(cmd)
        (tmp_path / "_binding.so").write_bytes(b"")
        return Done

    monkeypatch.setattr(build.subprocess, "run", compiler)
    for version, made in (("2.0.0", 1), ("2.0.0", 1), ("2.0.1", 2), ("2.0.1", 2)):
        monkeypatch.setattr(torch, "__version__", version)
        build.build_binding("g++")
        assert len(commands) == made
