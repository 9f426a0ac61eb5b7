"""The decoding step on both sides of the line between blocks of two warps and of eight (2304 and 2368 warps), with ragged
lengths, against the same sums in f64; repeats to the bit."""
import math

import pytest
import torch

from dashmag_b200 import attention as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b", [36, 37])
def test_both_sides(b):
    s, heads, d = 8192, 16, 128
    g = torch.Generator(device="cuda").manual_seed(b)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").bfloat16() for shape in ((b, heads, d), (b, s, 1, d), (b, s, 1, d)))
    lengths = torch.randint(0, s + 1, (b,), generator=g, device="cuda", dtype=torch.int32)
    lengths[0], lengths[1] = s, 0
    out = A.attention_decode(q, k, v, lengths)
    for i, n in enumerate(lengths.tolist()):
        scores = q[i].double() @ k[i, :n, 0].double().T / math.sqrt(d)
        want = torch.softmax(scores, 1) @ v[i, :n, 0].double() if n else torch.zeros(heads, d, dtype=torch.float64, device="cuda")
        # One rounding of the result; the sums before it are f32.
        assert ((out[i].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all(), i
    for _ in range(3):
        assert torch.equal(A.attention_decode(q, k, v, lengths), out)
