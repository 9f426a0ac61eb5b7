"""The decoding step into an output that starts at any element of a buffer (the C ABI asks for no alignment of it): steps that clusters
take where it is aligned to eight bytes, and chunks and merge where it is not - the same sums but for their order, and nothing written
beside the output."""
import ctypes

import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,hq,hkv,d", [(1, 4096, 32, 8, 128), (3, 1000, 8, 2, 64), (12, 1500, 16, 4, 256), (2, 300, 8, 2, 128)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("append", [False, True])
def test_any_element(b, s, hq, hkv, d, dtype, append):
    g = torch.Generator(device="cuda").manual_seed(s)
    rnd = lambda *shape: torch.randn(shape, generator=g, device="cuda").to(dtype)
    q, k, v, kn, vn = rnd(b, hq, d), rnd(b, s, hkv, d), rnd(b, s, hkv, d), rnd(b, hkv, d), rnd(b, hkv, d)
    lengths = torch.randint(1, s, (b,), generator=g, device="cuda", dtype=torch.int32)
    lib = _lib.lib()
    p, _ = A.make_decode_params(q, k, v, lengths, AttentionOptions())
    ws = torch.empty(max(lib.dash_attn_decode_workspace(ctypes.byref(p)), 256), dtype=torch.uint8, device="cuda")
    at = lambda x: ctypes.c_void_p(x.data_ptr())
    stream = ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)
    n, first, launches = b * hq * d, None, []
    for shift in (0, 4, 1, 2, 3, 7):
        buffer = torch.full((n + 16,), 7.0, dtype=dtype, device="cuda")
        out = ctypes.c_void_p(buffer.data_ptr() + 2 * shift)
        before = _lib.probe("kernel_launches")
        if append:
            rc = lib.dash_attn_decode_append(ctypes.byref(p), at(q), at(kn), at(vn), at(k), at(v), out, at(ws), ws.numel(), stream)
        else:
            rc = lib.dash_attn_decode(ctypes.byref(p), at(q), at(k), at(v), out, at(ws), ws.numel(), stream)
        assert rc == _lib.OK, _lib.last_error()
        launches.append(_lib.probe("kernel_launches") - before)
        got = buffer[shift:shift + n]
        assert (buffer[:shift] == 7).all() and (buffer[shift + n:] == 7).all()
        if first is None:
            first = got.double()
        # Two orders of the same f32 sums, each rounded once: at most a unit in the last place apart.
        unit = 2.0 ** -7 if dtype == torch.bfloat16 else 2.0 ** -10
        assert ((got.double() - first).abs() <= unit * first.abs() + 1e-5).all(), shift
    assert launches == ([1, 1] if s > 512 else [2, 2]) + [2] * 4
