"""The forward with a tile's keys split over blocks (few queries, many keys): against the f64 oracle, where parts see no
key (padding, causality, a window), with one query and with ragged tiles; and without scratch, unsplit, for the same call."""
import ctypes

import numpy as np
import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions
from oracle import attention_oracle as oracle
from test_random_shapes_gpu import SWEEP

pytestmark = pytest.mark.gpu

# The output's rounding is up to 2^-8 of its largest value (2^-9 of the power of two below it), and the weights' - each
# rounded to the dtype before P V - up to 2^-9 of a row that one key dominates (2.42e-3 of 0.526 = 4.602e-3 measured, unsplit).
OUTPUT = 2.0 ** -8 + 2.0 ** -9

C, N = AttentionOptions.causal_(), AttentionOptions()
# b, hq, hkv, tq, tk, d, options, padded tail of the last sequence
CASES = [(1, 8, 2, 1, 1500, 128, C, 0), (2, 8, 2, 37, 3001, 128, C, 2500), (1, 4, 4, 300, 2000, 128, N, 0), (1, 8, 1, 130, 2222, 64, C, 0),
         (2, 3, 1, 200, 1100, 64, N, 1037), (1, 8, 2, 129, 1700, 256, C, 0), (2, 2, 2, 150, 1500, 256, N, 700),
         (1, 8, 2, 100, 4000, 128, C.with_window(900, 0), 0), (1, 4, 2, 1500, 1700, 128, C, 0), (1, 4, 2, 1700, 1600, 128, C, 0),
         (2, 4, 2, 64, 1200, 128, C, 1200)]


@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
@pytest.mark.parametrize("i", range(len(CASES)))
def test_split_forward(i, dtype):
    b, hq, hkv, tq, tk, d, options, tail = CASES[i]
    host = [oracle.seeded(s, 400 + 10 * i + j) for j, s in enumerate([(b, tq, hq, d), (b, tk, hkv, d), (b, tk, hkv, d)])]
    q, k, v = (torch.from_numpy(x).cuda().to(dtype) for x in host)
    padding = np.zeros((b, tk), dtype=bool)
    if tail:
        padding[-1, tk - tail:] = True
    mask = AttentionMask.key_padding(torch.from_numpy(padding).cuda()) if tail else AttentionMask.none()
    p, keep = A.make_params("attention", q, k, v, mask, options)
    assert _lib.lib().dash_attn_forward_workspace(ctypes.byref(p)) > 0, "the case is here because its keys are split"
    launches = _lib.probe("kernel_launches")
    o, lse = A.attention_with_lse(q, k, v, mask, options)
    assert _lib.probe("kernel_launches") - launches == 2
    kw = dict(causal=options.causal, window=(None, None) if options.window is None else (options.window.left, options.window.right))
    if tail:
        kw["key_padding"] = padding
    want_o, want_lse = oracle.forward(*(x.float().cpu().numpy() for x in (q, k, v)), **kw)
    got_o, got_lse = o.float().cpu().numpy(), lse.cpu().numpy()
    empty = np.isneginf(want_lse)
    assert np.array_equal(np.isneginf(got_lse), empty) and np.all(got_o[empty] == 0)
    scale = 1.0 if dtype == torch.bfloat16 else 0.125   # f16 keeps three more bits
    assert np.max(np.abs(got_o - want_o)) <= OUTPUT * scale * np.max(np.abs(want_o))
    seen = ~empty
    assert np.max(np.abs(got_lse[seen] - want_lse[seen])) <= SWEEP[1] * np.max(np.abs(want_lse[seen]))
    again = A.attention_with_lse(q, k, v, mask, options)
    assert torch.equal(again[0], o) and torch.equal(again[1], lse)
    # No scratch: one block a tile, the same result but for the order of the sums.
    o1, lse1 = torch.full_like(o, float("nan")), torch.full_like(lse, float("nan"))
    rc = _lib.lib().dash_attn_forward(ctypes.byref(p), A._ptr(q), A._ptr(k), A._ptr(v), A._ptr(o1), A._ptr(lse1), None, 0, A._stream(q.device))
    assert rc == _lib.OK
    assert np.max(np.abs(o1.float().cpu().numpy() - want_o)) <= OUTPUT * scale * np.max(np.abs(want_o))
    assert np.max(np.abs(lse1.cpu().numpy()[seen] - want_lse[seen])) <= SWEEP[1] * np.max(np.abs(want_lse[seen]))


@pytest.mark.parametrize("d", [64, 128, 256])
@pytest.mark.parametrize("where,bad", [("q", "nan"), ("k", "nan"), ("k", "inf"), ("v", "nan"), ("v", "inf")])
def test_a_part_hides_no_nan(d, where, bad):
    """A NaN or an infinity in a query, key or value comes out of the split forward where it comes out of the unsplit one."""
    host = [oracle.seeded(s, 70 + j) for j, s in enumerate([(1, 150, 8, d), (1, 3000, 2, d), (1, 3000, 2, d)])]
    q, k, v = (torch.from_numpy(x).cuda().to(torch.bfloat16) for x in host)
    {"q": q, "k": k, "v": v}[where][0, 100, 0, 3] = float(bad)   # every query sees key 100
    p, keep = A.make_params("attention", q, k, v, AttentionMask.none(), C)
    assert _lib.lib().dash_attn_forward_workspace(ctypes.byref(p)) > 0
    o, lse = A.attention_with_lse(q, k, v, AttentionMask.none(), C)
    o1, lse1 = torch.zeros_like(o), torch.zeros_like(lse)
    rc = _lib.lib().dash_attn_forward(ctypes.byref(p), A._ptr(q), A._ptr(k), A._ptr(v), A._ptr(o1), A._ptr(lse1), None, 0, A._stream(q.device))
    assert rc == _lib.OK
    assert not torch.isfinite(o1).all()
    assert torch.equal(torch.isfinite(o), torch.isfinite(o1)) and torch.equal(torch.isfinite(lse), torch.isfinite(lse1))
    if bad == "nan":
        assert torch.equal(torch.isnan(o), torch.isnan(o1))
    whole = torch.isfinite(o1)
    assert torch.max(torch.abs(o[whole].float() - o1[whole].float())) <= 2 * OUTPUT * torch.max(torch.abs(o1[whole].float()))
