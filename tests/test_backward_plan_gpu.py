"""The backward on both sides of the line below which no launch order is made (148 units of 128 keys and a key-value head, 37 at head
dimension 256), on packed sequences of up to 300 tokens against the same sums in f64, call after call without a synchronisation in
between: the kernels of a call start before the ones in front of them have ended."""
import math

import numpy as np
import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions

pytestmark = pytest.mark.gpu


# `five`: dq summed in any order and so by reductions, from 240 units on (never without a launch order in a packed batch).
@pytest.mark.parametrize("blocks,hkv,group,d,five", [
    (1, 1, 1, 128, None), (74, 2, 2, 128, None), (75, 2, 2, 128, None), (148, 1, 4, 64, None), (149, 1, 1, 128, None), (37, 1, 2, 256, None),
    (38, 1, 1, 256, None), (74, 2, 1, 128, False), (149, 1, 2, 64, False), (240, 1, 2, 64, True), (80, 3, 4, 64, True)])
def test_both_sides(blocks, hkv, group, d, five):
    deterministic = five is None
    rng = np.random.default_rng(blocks)
    t = 128 * blocks - int(rng.integers(0, 128))
    lens = []
    while sum(lens) < t:
        lens.append(int(min(rng.integers(1, 301), t - sum(lens))))
    g = torch.Generator(device="cuda").manual_seed(blocks)
    q, k, v, go = (torch.randn((1, t, h, d), generator=g, device="cuda").bfloat16() for h in (hkv * group, hkv, hkv, hkv * group))
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda")
    mask, options = AttentionMask.packed(cu, cu), AttentionOptions(causal=True, deterministic=deterministic)
    o, lse = A.attention_with_lse(q, k, v, mask, options)
    atomic = _lib.probe("atomic_runs")
    runs = [A.attention_backward(q, k, v, o, lse, go, mask, options) for _ in range(8)]
    assert _lib.probe("atomic_runs") == atomic + (8 if five else 0)
    for run in runs[1:]:
        for x, y, fixed in zip(run, runs[0], (not five, True, True)):
            assert not fixed or torch.equal(x, y)
    want = [torch.empty(x.shape, dtype=torch.float64, device="cuda") for x in runs[0]]
    at = 0
    for n in lens:
        qs, ks, vs, gs = (x[0, at:at + n].double() for x in (q, k, v, go))
        ks, vs = ks.repeat_interleave(group, 1), vs.repeat_interleave(group, 1)
        s = torch.einsum("ihd,jhd->hij", qs, ks) / math.sqrt(d)
        p = torch.softmax(s.masked_fill(torch.ones(n, n, device="cuda").triu(1).bool(), -math.inf), 2)
        dp = torch.einsum("ihd,jhd->hij", gs, vs)
        ds = p * (dp - (p * dp).sum(2, keepdim=True)) / math.sqrt(d)
        want[0][0, at:at + n] = torch.einsum("hij,jhd->ihd", ds, ks)
        want[1][0, at:at + n] = torch.einsum("hij,ihd->jhd", ds, qs).reshape(n, hkv, group, d).sum(2)
        want[2][0, at:at + n] = torch.einsum("hij,ihd->jhd", p, gs).reshape(n, hkv, group, d).sum(2)
        at += n
    for got, x in zip(runs[-1], want):
        # P, dS, the output that delta is taken from and the result, each rounded to 2^-9 of itself.
        assert float((got.double() - x).norm() / x.norm()) <= 4 * 2.0 ** -9
