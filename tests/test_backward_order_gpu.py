"""The key and value gradients of the first keys of a long causal sequence, which every query sees with a weight that falls
with the query: sums of many small terms and a few large ones, whose small ones must not be lost to the accumulator's rounding."""
import math

import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions

pytestmark = pytest.mark.gpu

# Two roundings to f16, of P or dS and of the result, each with an error of at most 2^-11 / sqrt(3) of the value (root mean square).
BOUND = 2.0 ** -11 * math.sqrt(2 / 3)


# (Heads of 128 take the five-product form, where dq may be summed in any order, from 500 blocks of 128 keys on: two key-value heads.)
@pytest.mark.parametrize("d,deterministic,hkv", [(64, True, 1), (128, True, 1), (256, True, 1), (64, False, 1), (128, False, 2)])
def test_small_terms_count(d, deterministic, hkv):
    t, heads, first = 32768, 8, 128   # heads to a key-value head, whose first one is looked at
    g = torch.Generator(device="cuda").manual_seed(1)
    q, k, v, w = (torch.randn(1, t, h, d, generator=g, device="cuda").half() for h in (heads * hkv, hkv, hkv, heads * hkv))
    options = AttentionOptions(causal=True, deterministic=deterministic)
    o, lse = A.attention_with_lse(q, k, v, AttentionMask.none(), options)
    five = _lib.probe("atomic_runs")
    _, dk, dv = A.attention_backward(q, k, v, o, lse, w, AttentionMask.none(), options)
    assert _lib.probe("atomic_runs") == five + int(not deterministic)
    keys, values = k[0, :first, 0].double(), v[0, :first, 0].double()
    want_k, want_v = torch.zeros_like(keys), torch.zeros_like(values)
    hidden = torch.arange(first, device="cuda")[None] > torch.arange(t, device="cuda")[:, None]
    for h in range(heads):
        queries, grads = q[0, :, h].double(), w[0, :, h].double()
        p = (queries @ keys.T / math.sqrt(d) - lse[0, :, h].double()[:, None]).masked_fill(hidden, -math.inf).exp()
        delta = (grads * o[0, :, h].double()).sum(1, keepdim=True)
        want_v += p.T @ grads
        want_k += (p * (grads @ values.T - delta)).T @ queries / math.sqrt(d)
    for got, want in ((dk[0, :first, 0], want_k), (dv[0, :first, 0], want_v)):
        assert (got.double() - want).norm() <= BOUND * want.norm()
