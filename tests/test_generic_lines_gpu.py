"""The CUDA-core kernels on both sides of the lines that say how many blocks share a row block's sweep: by the number of blocks (37, 74,
148, 222, 400 and what fits at once), the steps of a sweep, rows a warp, causal and whole rows, windows that make long sweeps short,
dkdv shared with dq and alone - against the f64 oracle; repeats to the bit."""
import numpy as np
import pytest
import torch

from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions

from oracle import attention_oracle as oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,tq,tk,hq,hkv,d,causal,window,seqs", [
    (1, 96, 191, 3, 1, 64, False, -1, 0), (1, 96, 193, 3, 1, 64, False, -1, 0),     # 36 blocks: below and above three steps
    (1, 148, 256, 4, 4, 64, False, -1, 0), (1, 156, 256, 4, 4, 64, False, -1, 0),   # 76 and 80 blocks
    (1, 140, 140, 4, 2, 64, True, -1, 0), (1, 190, 190, 8, 8, 64, True, -1, 0),     # around 148 and 222 blocks
    (2, 111, 200, 8, 2, 64, False, -1, 0), (2, 113, 200, 8, 2, 64, False, -1, 0),   # 224 and 240 blocks
    (1, 294, 294, 4, 2, 64, False, -1, 0), (1, 294, 294, 4, 2, 64, True, -1, 0),    # dkdv's 74 blocks: with dq's only, alone
    (1, 161, 294, 3, 1, 64, True, -1, 0), (1, 474, 474, 3, 1, 80, True, -1, 0),
    (1, 400, 400, 4, 4, 64, True, 500, 0), (1, 400, 400, 4, 4, 64, True, 20, 0),    # a window over all, and of less than a step
    (1, 590, 590, 8, 8, 96, True, -1, 0), (1, 384, 384, 4, 4, 64, True, -1, 2), (1, 384, 384, 4, 4, 64, True, -1, 3)])
def test_against_f64(b, tq, tk, hq, hkv, d, causal, window, seqs):
    q, k, v, g = (oracle.seeded(s, i) for i, s in enumerate(((b, tq, hq, d), (b, tk, hkv, d), (b, tk, hkv, d), (b, tq, hq, d))))
    options, kw, mask = AttentionOptions(causal=causal), dict(causal=causal), AttentionMask.none()
    if window >= 0:
        options, kw["window"] = options.with_window(window, 0), (window, 0)
    if seqs > 0:
        cu = np.array([tq * i // seqs for i in range(seqs + 1)], dtype=np.int64)
        mask, kw = AttentionMask.packed(*[torch.tensor(cu, device="cuda")] * 2), dict(kw, cu_q=cu, cu_k=cu)
    dev = [torch.tensor(x, dtype=torch.float32, device="cuda") for x in (q, k, v, g)]

    def call():
        o, lse = A.attention_with_lse(*dev[:3], mask, options)
        return (o, lse) + tuple(A.attention_backward(*dev[:3], o, lse, dev[3], mask, options))
    got = call()
    wo, wl = oracle.forward(q, k, v, **kw)
    for name, x, ref in zip(("o", "lse", "dq", "dk", "dv"), got, (wo, wl) + tuple(oracle.backward(q, k, v, wo, wl, g, **kw))):
        x = x.cpu().numpy()
        assert np.array_equal(np.isfinite(x), np.isfinite(ref)), name
        fine = np.isfinite(ref)
        # f32 sums of up to some thousand terms, of the largest value: the bound of the f32 kernels (tests/test_kernels_gpu.py).
        assert np.abs(x - ref)[fine].max() <= 1e-5 * max(1.0, np.abs(ref[fine]).max()), name
    for x, y in zip(got, call()):
        assert torch.equal(x, y)
