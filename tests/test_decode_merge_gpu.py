"""The decoding step's merge at the numbers of partials where its form changes - all of them asked for at once by 128, 256 or 512
threads, in passes beyond, head dimensions that do not divide the threads - against the same sums in f64; repeats to the bit."""
import math

import pytest
import torch

from dashmag_b200 import attention as A

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,hq,hkv,d", [
    (1, 1, 8, 2, 128), (1, 64, 8, 2, 128), (2, 65, 8, 2, 64), (1, 2048, 32, 8, 128), (1, 2049, 32, 8, 128), (1, 4096, 32, 8, 128),
    (1, 4097, 32, 8, 128), (2, 5919, 32, 8, 128), (1, 8200, 4, 1, 128), (8, 6144, 8, 2, 256), (1, 60000, 2, 1, 256), (1, 33000, 2, 1, 128),
    (3, 700, 6, 2, 36), (2, 300, 4, 2, 250), (40, 3000, 8, 8, 64), (1, 20000, 3, 3, 52)])
def test_against_f64(b, s, hq, hkv, d):
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").bfloat16() for shape in ((b, hq, d), (b, s, hkv, d), (b, s, hkv, d)))
    lengths = torch.randint(0, s + 1, (b,), generator=g, device="cuda", dtype=torch.int32)
    lengths[0] = s
    out = A.attention_decode(q, k, v, lengths)
    for i, n in enumerate(lengths.tolist()):
        kk, vv = (x[i, :n].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
        scores = torch.einsum("hd,shd->hs", q[i].double(), kk) / math.sqrt(d)
        want = torch.einsum("hs,shd->hd", torch.softmax(scores, 1), vv)
        # One rounding of the result; the sums before it are f32.
        assert ((out[i].double() - want).abs() <= 2.0 ** -8 * want.abs() + 1e-5).all(), i
    for _ in range(3):
        assert torch.equal(A.attention_decode(q, k, v, lengths), out)
