"""The backward where two blocks share a unit's steps (few key blocks, long sweeps), and the forms of a call that leaves the order of
dq's sums free - on both sides of the lines between them, and the five-product form (the probe says that it ran) over groups, masks,
windows and dtypes - against the same sums in f64; the fixed order repeats to the bit."""
import math

import numpy as np
import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions

pytestmark = pytest.mark.gpu


def reference(q, k, v, g, seen):
    """dq, dk, dv in f64 of [T, H, D] tensors of one batch element; `seen` [Tq, Tk] or None.  And what an error in delta of all of
    sum |O| |dO| would make of them: a query that sees one key has dP = delta, gradients of zero and nothing but that error."""
    group = q.shape[1] // k.shape[1]
    q, g = q.double(), g.double()
    kk, vv = (x.double().repeat_interleave(group, 1) for x in (k, v))
    s = torch.einsum("ihd,jhd->hij", q, kk) / math.sqrt(q.shape[-1])
    if seen is not None:
        s = s.masked_fill(~seen, -math.inf)
    p = torch.softmax(s, 2).nan_to_num(0.0)
    dp = torch.einsum("ihd,jhd->hij", g, vv)
    ds = p * (dp - (p * dp).sum(2, keepdim=True)) / math.sqrt(q.shape[-1])
    fold = lambda x: x.reshape(x.shape[0], k.shape[1], group, -1).sum(2)
    slip = p * torch.einsum("ihd,ihd->hi", torch.einsum("hij,jhd->ihd", p, vv).abs(), g.abs())[..., None] / math.sqrt(q.shape[-1])
    return ((torch.einsum("hij,jhd->ihd", ds, kk), torch.einsum("hij,jhd->ihd", slip, kk.abs())),
            (fold(torch.einsum("hij,ihd->jhd", ds, q)), fold(torch.einsum("hij,ihd->jhd", slip, q.abs()))),
            (fold(torch.einsum("hij,ihd->jhd", p, g)), torch.zeros(1)))


def check(b, t, hkv, group, d, dtype, mask_kind, causal, window, deterministic, five=False, tq=None):
    """`five`: the call sums dq by reductions, five products a pair of tiles; `tq` queries (t, where not said) against t keys."""
    tq = tq or t
    gen = torch.Generator(device="cuda").manual_seed(t)
    q, k, v, g = (torch.randn((b, n, h, d), generator=gen, device="cuda").to(dtype)
                  for n, h in ((tq, hkv * group), (t, hkv), (t, hkv), (tq, hkv * group)))
    i = torch.arange(t, device="cuda")
    at = torch.arange(tq, device="cuda") + t - tq   # the queries' places among the keys
    seen = [torch.ones(tq, t, dtype=torch.bool, device="cuda") for _ in range(b)]
    if mask_kind == "packed":
        cut = [0, t // 3, t // 3 + 1, t]
        cu = torch.tensor(cut, dtype=torch.int32, device="cuda")
        mask = AttentionMask.packed(cu, cu)
        part = torch.bucketize(i, cu[1:], right=True)
        seen[0] &= part[:, None] == part[None]
    elif mask_kind == "padding":
        lens = [t, 1, t // 2, 0][:b] + [t] * max(b - 4, 0)
        pad = i[None] >= torch.tensor(lens, device="cuda")[:, None]
        mask = AttentionMask.key_padding(pad)
        seen = [s & ~p[None] for s, p in zip(seen, pad)]
    else:
        mask = AttentionMask.none()
    if causal:
        seen = [s & (at[:, None] >= i[None]) for s in seen]
    options = AttentionOptions(causal=causal, deterministic=deterministic)
    if window is not None:
        options = options.with_window(window, window)
        seen = [s & ((at[:, None] - i[None]).abs() <= window) for s in seen]
    o, lse = A.attention_with_lse(q, k, v, mask, options)
    atomic = _lib.probe("atomic_runs")
    runs = [A.attention_backward(q, k, v, o, lse, g, mask, options) for _ in range(4)]
    assert _lib.probe("atomic_runs") == atomic + (4 if five else 0)
    for run in runs[1:]:
        for x, y, fixed in zip(run, runs[0], (deterministic, True, True)):
            assert not fixed or torch.equal(x, y)
    for n in range(b):
        for name, got, (want, slip) in zip(("dq", "dk", "dv"), runs[-1], reference(q[n], k[n], v[n], g[n], seen[n])):
            # P, dS and the result, each rounded to 2^-9 (f16: 2^-12) of itself, and the output that delta is taken from.
            bound = 2.0 ** (-9 if dtype == torch.bfloat16 else -12) * (3 * float(want.norm()) + float(slip.norm()))
            assert float((got[n].double() - want).norm()) <= bound, name
    assert _lib.lib().dash_attn_device_status(0) == 0


@pytest.mark.parametrize("b,t,hkv,group,d,dtype,mask,causal,window", [
    (1, 1024, 1, 1, 128, torch.bfloat16, "none", True, None), (1, 256, 1, 4, 128, torch.bfloat16, "none", True, None),
    (1, 255, 2, 8, 64, torch.float16, "none", False, None), (1, 1029, 1, 3, 128, torch.float16, "none", True, None),
    (1, 1152, 1, 2, 128, torch.bfloat16, "none", True, None), (1, 1153, 1, 2, 128, torch.bfloat16, "none", True, None),
    (1, 1100, 2, 4, 64, torch.bfloat16, "packed", True, None), (1, 1999, 1, 8, 128, torch.bfloat16, "packed", True, 700),
    (4, 256, 2, 3, 128, torch.bfloat16, "padding", False, None), (4, 500, 1, 8, 64, torch.float16, "padding", True, None),
    (1, 4736, 1, 8, 128, torch.bfloat16, "none", True, 130), (1, 4737, 1, 8, 64, torch.bfloat16, "packed", True, None), (2, 500, 1, 5, 128, torch.bfloat16, "none", False, 60)])
def test_shared_units(b, t, hkv, group, d, dtype, mask, causal, window):
    check(b, t, hkv, group, d, dtype, mask, causal, window, True)


# Units (blocks of 128 keys by key-value heads by batch) on both sides of the lines: 90 (packed: 240) at heads of 64, 500 (packed: never) at 128.
@pytest.mark.parametrize("b,t,hkv,group,d,mask,five", [
    (30, 300, 1, 1, 64, "padding", True), (29, 300, 1, 1, 64, "padding", False), (1, 3840, 8, 1, 64, "packed", True), (1, 3700, 8, 1, 64, "packed", False),
    (125, 260, 2, 1, 128, "padding", True), (100, 200, 2, 1, 128, "padding", False), (1, 1000, 2, 4, 128, "packed", False), (2, 1000, 2, 4, 64, "none", False)])
def test_free_order_on_both_sides(b, t, hkv, group, d, mask, five):
    check(b, t, hkv, group, d, torch.bfloat16, mask, False, None, False, five)


B, H = torch.bfloat16, torch.float16


# Tiles of 128 / 2^p tokens by 2^p heads: p = 0 (groups 1, 3), 1 (2, 6), 2 (4, 12), 3 (8, 16).
@pytest.mark.parametrize("b,tq,t,hkv,group,d,dtype,mask,causal,window", [
    (12, 130, 130, 4, 2, 64, B, "none", True, None), (16, 257, 257, 2, 3, 64, H, "padding", False, None), (10, 300, 300, 3, 4, 64, B, "none", True, 60),
    (13, 300, 300, 3, 8, 64, H, "none", True, None), (50, 129, 200, 1, 16, 64, B, "none", True, None), (45, 255, 131, 1, 6, 64, B, "none", True, None),
    (24, 500, 500, 1, 12, 64, H, "padding", True, 100), (1, 3840, 3840, 8, 2, 64, B, "packed", True, None), (1, 3840, 3840, 8, 4, 64, H, "packed", True, 300),
    (1, 5250, 5250, 6, 3, 64, B, "packed", False, 90), (45, 256, 256, 1, 1, 64, B, "none", True, None),
    (50, 130, 130, 5, 2, 128, B, "none", True, None), (45, 260, 260, 4, 3, 128, H, "padding", False, None), (64, 140, 140, 4, 4, 128, H, "none", True, 40),
    (32, 256, 256, 8, 8, 128, B, "none", True, None), (84, 129, 300, 2, 6, 128, B, "none", False, 70), (125, 5, 200, 2, 16, 128, H, "none", True, None),
    (125, 257, 129, 2, 1, 128, H, "none", True, None), (64, 200, 200, 4, 12, 128, B, "padding", True, None)], ids=str)
def test_five_products(b, tq, t, hkv, group, d, dtype, mask, causal, window):
    check(b, t, hkv, group, d, dtype, mask, causal, window, False, True, tq)
