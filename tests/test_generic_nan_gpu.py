"""NaN and infinities on the CUDA-core forward: a row is NaN exactly where the f64 oracle's is, whichever tile of 32 keys the value
sits in, with one, two and four rows a warp and where two warps share a pair of rows.  (A row that is NaN has no log-sum-exp: -inf.)"""
import numpy as np
import pytest
import torch

from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions
from oracle import attention_oracle as oracle

pytestmark = pytest.mark.gpu

# b, hq, hkv, tq, d: blocks of 8 rows shared by two warps each (the first), of 8, 16 and 32 rows.
FORMS = [(1, 2, 1, 40, 64), (1, 2, 1, 9, 100), (1, 2, 1, 40, 256), (1, 8, 8, 700, 40), (1, 16, 4, 700, 64)]


def check(form, tk, spoil, causal):
    b, hq, hkv, tq, d = form
    tq = tk if causal else tq
    q, k, v = (oracle.seeded(s, 100 + i) for i, s in enumerate([(b, tq, hq, d), (b, tk, hkv, d), (b, tk, hkv, d)]))
    spoil(q, k, v)
    with np.errstate(all="ignore"):
        want_o, want_lse = oracle.forward(q, k, v, causal=causal)
    o, lse = A.attention_with_lse(*(torch.from_numpy(x).cuda() for x in (q, k, v)), AttentionMask.none(), AttentionOptions(causal=causal))
    o, lse = o.cpu().numpy(), lse.cpu().numpy()
    assert np.array_equal(np.isnan(o), np.isnan(want_o))
    assert np.array_equal(np.isinf(o), np.isinf(want_o)) and np.array_equal(o[np.isinf(o)], want_o[np.isinf(o)])
    fine = np.isfinite(want_o)
    assert np.all(np.abs(o - want_o)[fine] <= 1e-5 * max(1.0, np.abs(want_o[fine]).max(initial=0.0)))
    seen = np.isfinite(want_lse)
    assert np.array_equal(np.isfinite(lse), seen) and np.all(np.abs(lse - want_lse)[seen] <= 1e-5 * np.maximum(1.0, np.abs(want_lse[seen])))


@pytest.mark.parametrize("form", FORMS, ids=str)
@pytest.mark.parametrize("value", [np.nan, np.inf, -np.inf], ids=str)
@pytest.mark.parametrize("key", [0, 31, 32, 33, 63, 64, 96])
def test_one_key(form, value, key):
    def a_key(q, k, v):
        k[:, key, :, 1] = value

    def a_value(q, k, v):
        v[:, key, :, 1] = value

    for tk in sorted({key + 1, 97}):
        check(form, tk, a_value, False)
        for causal in (False, True):
            check(form, tk, a_key, causal)


@pytest.mark.parametrize("form", FORMS, ids=str)
@pytest.mark.parametrize("lo,hi,tk", [(0, 32, 64), (32, 64, 64), (32, 33, 33), (0, 32, 33), (0, 64, 64), (64, 96, 160), (0, 7, 7)])
def test_a_whole_share(form, lo, hi, tk):
    """Every key of a tile or of a warp's share of the tiles."""
    def keys(q, k, v):
        k[:, lo:hi] = np.nan

    for causal in (False, True):
        check(form, tk, keys, causal)


@pytest.mark.parametrize("form", FORMS, ids=str)
def test_a_query(form):
    def query(q, k, v):
        q[:, 5, :, 0] = np.nan
        q[:, 6, :, 0] = np.inf

    check(form, 70, query, False)
