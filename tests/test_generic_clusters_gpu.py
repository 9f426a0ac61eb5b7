"""The CUDA-core kernels whose rows a cluster of blocks shares: two and four blocks a row block, sweeps that leave blocks of the
cluster without a tile, windows and padding that do, packed sequences, every number of rows a warp, head dimensions from the smallest
that is shared, NaN in one block's run - against the f64 oracle; repeats to the bit."""
import math

import numpy as np
import pytest
import torch

from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions

from oracle import attention_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,tq,tk,hq,hkv,d,causal,window,seqs", [
    (1, 130, 130, 4, 4, 64, True, -1, 0), (1, 16, 1000, 8, 2, 64, True, -1, 0), (1, 9, 129, 2, 1, 32, False, -1, 0), (2, 33, 500, 6, 2, 96, True, 40, 0),
    (1, 590, 590, 3, 1, 96, True, -1, 2), (1, 700, 700, 4, 4, 128, True, -1, 1), (1, 384, 384, 4, 4, 64, True, -1, 2), (1, 500, 500, 8, 2, 64, True, -1, 0),
    (1, 60, 300, 2, 1, 128, True, -1, 0), (1, 40, 90, 2, 2, 36, False, -1, 0), (1, 300, 300, 8, 2, 51, True, 3, 0), (3, 70, 200, 4, 1, 128, False, -1, -1)])
def test_against_f64(b, tq, tk, hq, hkv, d, causal, window, seqs):
    q, k, v, g = (oracle.seeded(s, i) for i, s in enumerate(((b, tq, hq, d), (b, tk, hkv, d), (b, tk, hkv, d), (b, tq, hq, d))))
    options, kw, mask = AttentionOptions(causal=causal), dict(causal=causal), AttentionMask.none()
    if window >= 0:
        options, kw["window"] = options.with_window(window, 0), (window, 0)
    if seqs > 0:
        cu = np.array([tq * i // seqs for i in range(seqs + 1)], dtype=np.int64)
        mask, kw = AttentionMask.packed(*[torch.tensor(cu, device="cuda")] * 2), dict(kw, cu_q=cu, cu_k=cu)
    if seqs < 0:   # padding: one element whole, one of a single key, one with a hole
        keep = np.ones((b, tk), dtype=bool)
        keep[1, 1:], keep[2, 40:150] = False, False
        mask, kw = AttentionMask.key_padding(torch.tensor(~keep, device="cuda")), dict(kw, key_padding=~keep)
    dev = [torch.tensor(x, dtype=torch.float32, device="cuda") for x in (q, k, v, g)]
    o, lse = A.attention_with_lse(*dev[:3], mask, options)
    grads = A.attention_backward(*dev[:3], o, lse, dev[3], mask, options)
    wo, wl = oracle.forward(q, k, v, **kw)
    want = (wo, wl) + tuple(oracle.backward(q, k, v, wo, wl, g, **kw))
    for name, got, ref in zip(("o", "lse", "dq", "dk", "dv"), (o, lse) + tuple(grads), want):
        got = got.cpu().numpy()
        assert np.array_equal(np.isfinite(got), np.isfinite(ref)), name
        fine = np.isfinite(ref)
        # f32 sums of up to some thousand terms, of the largest value: the bound of the f32 kernels (tests/test_kernels_gpu.py).
        assert np.abs(got - ref)[fine].max() <= 1e-5 * max(1.0, np.abs(ref[fine]).max()), name
    again = A.attention_with_lse(*dev[:3], mask, options)
    for x, y in zip((o, lse) + tuple(grads), tuple(again) + tuple(A.attention_backward(*dev[:3], o, lse, dev[3], mask, options))):
        assert torch.equal(x, y)


@pytest.mark.parametrize("key", [0, 250, 999])
def test_a_nan_in_one_run(key):
    q, k, v = (torch.randn(s, device="cuda") for s in ((1, 16, 8, 64), (1, 1000, 2, 64), (1, 1000, 2, 64)))
    clean, _ = A.attention_with_lse(q, k, v, AttentionMask.none(), AttentionOptions())
    k[0, key, 0, 3] = math.nan
    out, lse = A.attention_with_lse(q, k, v, AttentionMask.none(), AttentionOptions())
    assert torch.isnan(out[:, :, :4]).all() and torch.equal(out[:, :, 4:], clean[:, :, 4:])
