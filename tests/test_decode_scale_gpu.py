"""The decoding step under scales of zero and below: every head dimension and dtype, calls that chunks and clusters would take, sequences
without keys, a window, and the step that rotates and appends - against the same sums in f64."""
import pytest
import torch

from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionOptions
from dashmag_b200.rope import Rope, attention_decode_append_rope

pytestmark = pytest.mark.gpu
UNIT = {torch.float32: 2.0 ** -20, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}


def reference(q, k, v, n, scale, left=None):
    first = 0 if left is None else max(0, n - 1 - left)
    kk, vv = (x[first:n].double().repeat_interleave(q.shape[0] // k.shape[1], 1) for x in (k, v))
    if n == 0:
        return torch.zeros_like(q, dtype=torch.float64)
    return torch.einsum("hs,shd->hd", torch.softmax(torch.einsum("hd,shd->hs", q.double(), kk) * scale, 1), vv)


@pytest.mark.parametrize("b,s,hq,hkv,d", [(1, 2000, 8, 2, 128), (4, 300, 16, 4, 64), (3, 1500, 8, 2, 256), (2, 700, 20, 1, 128), (3, 200, 4, 2, 40), (2, 900, 3, 3, 128)])
@pytest.mark.parametrize("dtype", list(UNIT), ids=["f32", "bf16", "f16"])
@pytest.mark.parametrize("scale", [0.0, -0.0, -0.1, -2e-3, 0.05])
def test_against_f64(b, s, hq, hkv, d, dtype, scale):
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").to(dtype) for shape in ((b, hq, d), (b, s, hkv, d), (b, s, hkv, d)))
    lengths = torch.tensor([s, 0, 17, 1][:b], dtype=torch.int32, device="cuda")
    for options, left in ((AttentionOptions(scale=scale), None), (AttentionOptions(scale=scale).with_window(50, 0), 50)):
        out = A.attention_decode(q, k, v, lengths, options)
        for i, n in enumerate(lengths.tolist()):
            want = reference(q[i], k[i], v[i], n, scale, left)
            # One rounding of the result; the sums before it are f32.
            assert ((out[i].double() - want).abs() <= UNIT[dtype] * want.abs() + 1e-5).all(), i


@pytest.mark.parametrize("s,d", [(300, 128), (1200, 128), (900, 64), (900, 256)])
@pytest.mark.parametrize("scale", [0.0, -0.1])
def test_a_step_that_rotates(s, d, scale):
    g = torch.Generator(device="cuda").manual_seed(s)
    q, kn, vn, k, v = (torch.randn(shape, generator=g, device="cuda").bfloat16() for shape in ((2, 8, d), (2, 2, d), (2, 2, d), (2, s, 2, d), (2, s, 2, d)))
    rope = Rope(d, 10000.0, s, torch.bfloat16, device="cuda")
    lengths = torch.tensor([s - 1, 20], dtype=torch.int32, device="cuda")
    rq, rk = rope.apply_at(q, lengths, other=kn)
    k2, v2 = k.clone(), v.clone()
    for i, n in enumerate(lengths.tolist()):
        k2[i, n], v2[i, n] = rk[i], vn[i]
    out = attention_decode_append_rope(rope, q, kn, vn, k, v, lengths, AttentionOptions(scale=scale))
    assert torch.equal(k, k2) and torch.equal(v, v2)
    for i, n in enumerate(lengths.tolist()):
        want = reference(rq[i], k2[i], v2[i], n + 1, scale)
        assert ((out[i].double() - want).abs() <= UNIT[torch.bfloat16] * want.abs() + 1e-5).all(), i
