"""The parameter structs as the Python side fills them, without a GPU: tensors of the wrong rank are refused by name, and the
packed formats lay every field where the struct has it."""
import ctypes
import struct

import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A


@pytest.mark.parametrize("which", ["output", "grad"])
@pytest.mark.parametrize("shape", [(), (4,), (1, 4, 128), (1, 1, 4, 2, 64), (1, 2, 2, 64)], ids=str)
def test_the_backward_refuses_other_shapes(which, shape):
    q, lse = torch.empty(1, 4, 2, 64, device="meta"), torch.empty(1, 4, 2, device="meta")
    other = torch.empty(shape, device="meta")
    output, grad = (other, q) if which == "output" else (q, other)
    with pytest.raises(A.AttentionError, match=f"attention_backward: {which}"):
        A.attention_backward(q, q, q, output, lse, grad)


@pytest.mark.parametrize("kind,fmt", [(_lib.Params, _lib.PARAMS_FORMAT), (_lib.DecodeParams, _lib.DECODE_PARAMS_FORMAT)], ids=["training", "decode"])
def test_the_formats_are_the_structs(kind, fmt):
    flat = []   # (type, byte offset) of every scalar of the struct
    for name, t in kind._fields_:
        at = getattr(kind, name).offset
        element, n = (t._type_, t._length_) if issubclass(t, ctypes.Array) else (t, 1)
        flat += [(element, at + i * ctypes.sizeof(element)) for i in range(n)]
    codes = {ctypes.c_int32: "i", ctypes.c_int64: "q", ctypes.c_float: "f", ctypes.c_void_p: "P"}
    want = "@" + "".join(codes[t] for t, _ in flat)
    assert struct.calcsize(fmt.format) <= ctypes.sizeof(kind)
    values = [float(i + 1) if t is ctypes.c_float else i + 1 for i, (t, _) in enumerate(flat)]
    p, raw = kind(), ctypes.create_string_buffer(ctypes.sizeof(kind))
    _lib.fill(p, fmt, *values)
    struct.pack_into(want, raw, 0, *values)
    assert bytes(p)[:fmt.size] == raw.raw[:fmt.size]
    for (t, at), value in zip(flat, values):
        assert t.from_buffer(p, at).value == value
    # A value no field holds goes the slow way, field by field, and leaves the others where they are.
    big = list(values)
    big[0] = 2 ** 40 + 7
    _lib.fill(p, fmt, *big)
    assert flat[0][0].from_buffer(p, 0).value == 7
    assert all(t.from_buffer(p, at).value == value for (t, at), value in list(zip(flat, values))[1:])
