"""Key padding on the tensor-core kernels: batches whose keys that are not padding are one run - looked at once, the sweep cut to it -
and batches with holes, runs at either end and inside tiles, elements of padding alone, flags of one and four bytes and with strides, on
both sides of the longest mask that is looked at once; forward and backward against the same sums in f64."""
import math

import pytest
import torch

from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions

pytestmark = pytest.mark.gpu


def reference(q, k, v, grad, padding, causal, window):
    q, k, v = (x.double().requires_grad_() for x in (q, k, v))
    b, tq, hq, d = q.shape
    tk, group = k.shape[1], hq // k.shape[2]
    s = torch.einsum("bqhd,bkhd->bhqk", q, k.repeat_interleave(group, 2)) / math.sqrt(d)
    at = torch.arange(tq, device="cuda")[:, None] + tk - tq
    key = torch.arange(tk, device="cuda")[None, :]
    shut = padding[:, None, None, :] | ((key > at) if causal else torch.zeros_like(key > at)) | ((key < at - window) if window >= 0 else torch.zeros_like(key > at))
    s = s.masked_fill(shut, -math.inf)
    seen = ~shut.all(-1, keepdim=True)
    p = torch.where(seen, torch.softmax(s.masked_fill(~seen, 0.0), -1), 0.0).masked_fill(shut, 0.0)
    o = torch.einsum("bhqk,bkhd->bqhd", p, v.repeat_interleave(group, 2))
    lse = torch.logsumexp(s, -1).transpose(1, 2)
    return (o.detach(), lse.detach()) + torch.autograd.grad(o, (q, k, v), grad.double())


@pytest.mark.parametrize("tq,tk,d,causal,window", [
    (200, 200, 64, False, -1), (300, 333, 128, False, -1), (256, 513, 128, True, -1), (190, 700, 64, True, 100), (130, 2047, 64, False, -1),
    (150, 2048, 128, False, -1), (150, 2049, 128, False, -1)])
@pytest.mark.parametrize("bytes4", [False, True], ids=["u8", "i32"])
def test_runs_and_holes(tq, tk, d, causal, window, bytes4):
    b, hq, hkv, dtype = 7, 4, 2, torch.float16
    g = torch.Generator(device="cuda").manual_seed(tk + d)
    q, k, v, grad = (torch.randn(s, generator=g, device="cuda").to(dtype) for s in ((b, tq, hq, d), (b, tk, hkv, d), (b, tk, hkv, d), (b, tq, hq, d)))
    padding = torch.zeros(b, tk, dtype=torch.bool, device="cuda")
    padding[1, tk - 37:] = True                 # right
    padding[2, :65] = True                      # left
    padding[3, :1], padding[3, tk - 130:] = True, True
    padding[4, tk // 2] = True                  # one hole
    padding[5] = True                           # nothing but padding
    padding[6] = torch.rand(tk, generator=g, device="cuda") < 0.5
    wide = torch.zeros(b, 2 * tk, dtype=torch.int32 if bytes4 else torch.bool, device="cuda")
    wide[:, ::2] = padding.to(wide.dtype)
    mask = AttentionMask.key_padding(wide[:, ::2])
    options = AttentionOptions(causal=causal)
    if window >= 0:
        options = options.with_window(window, 0)
    o, lse = A.attention_with_lse(q, k, v, mask, options)
    grads = A.attention_backward(q, k, v, o, lse, grad, mask, options)
    want = reference(q, k, v, grad, padding, causal, window)
    assert torch.equal(torch.isfinite(lse), torch.isfinite(want[1]))
    # The sweep's bounds of the f16 kernels (tests/test_random_shapes_gpu.py), of the largest value.
    for name, got, ref, bound in zip(("o", "lse", "dq", "dk", "dv"), (o, lse) + tuple(grads), want, (5.0e-4, 4.4e-7, 7.3e-4, 6.8e-4, 5.5e-4)):
        ref, got = ref.nan_to_num(0.0, 0.0, 0.0), got.double().nan_to_num(0.0, 0.0, 0.0)
        assert (got - ref).abs().max() <= bound * ref.abs().max(), name
    for x, y in zip((o, lse) + tuple(grads), A.attention_with_lse(q, k, v, mask, options) + tuple(A.attention_backward(q, k, v, o, lse, grad, mask, options))):
        assert torch.equal(x, y)
    assert not o[5].any() and not any(x[5].any() for x in grads)
