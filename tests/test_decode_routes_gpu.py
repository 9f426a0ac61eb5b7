"""Which decoding steps clusters take (one launch) and which go in chunks (two), on both sides of each line of the rule: where blocks run
at once or do not, shares up to the longest for how many blocks there are, for lengths given and whole caches, windows up to half the
cache, f16's shorter shares - each against the same sums in f64."""
import math

import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionOptions

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,hq,hkv,d,left,dtype,whole,ragged", [
    (9, 20576, 16, 4, 128, -1, "bf16", 2, 2),      # few blocks, a long share
    (18, 6156, 8, 2, 256, -1, "bf16", 2, 2),
    (3, 20000, 32, 8, 128, -1, "bf16", 2, 2),
    (4, 11776, 32, 8, 128, -1, "bf16", 1, 1),      # eight blocks a head, all of the room: 23 tiles a share, then 24
    (4, 11792, 32, 8, 128, -1, "bf16", 2, 2),
    (4, 6144, 32, 8, 128, -1, "f16", 1, 1),        # f16: 12 tiles, the most where the chunk is no longer, then 13
    (4, 6160, 32, 8, 128, -1, "f16", 2, 2),
    (1, 12288, 32, 8, 128, -1, "bf16", 1, 1),      # sixteen blocks a head: 12 tiles, then 13
    (1, 12304, 32, 8, 128, -1, "bf16", 2, 2),
    (1, 6144, 4, 2, 128, -1, "bf16", 1, 1),        # two heads: 6 tiles, then 7
    (1, 6160, 4, 2, 128, -1, "bf16", 2, 2),
    (1, 2048, 16, 8, 256, -1, "bf16", 1, 1),       # heads of 256, sixteen blocks: 4 tiles, then 5
    (1, 2064, 16, 8, 256, -1, "bf16", 2, 2),
    (16, 4096, 32, 8, 128, -1, "bf16", 2, 1),      # nearly twice the blocks that run at once: where lengths are given
    (16, 4112, 32, 8, 128, -1, "bf16", 2, 2),      # 17 tiles
    (12, 4096, 16, 8, 128, -1, "bf16", 2, 1),      # 1.41 times, then 1.29
    (11, 4096, 16, 8, 128, -1, "bf16", 2, 2),
    (40, 900, 16, 8, 256, 449, "bf16", 1, 1),      # a window of half the cache, then of a key more
    (40, 900, 16, 8, 256, 450, "bf16", 2, 2)])
def test_both_sides(b, s, hq, hkv, d, left, dtype, whole, ragged):
    dtype = {"bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").to(dtype) for shape in ((b, hq, d), (b, s, hkv, d), (b, s, hkv, d)))
    lengths = torch.randint(0, s + 1, (b,), generator=g, device="cuda", dtype=torch.int32)
    lengths[0] = s
    options = AttentionOptions().with_window(left, 0) if left >= 0 else AttentionOptions()
    for lens, launches in ((None, whole), (lengths, ragged)):
        before = _lib.probe("kernel_launches")
        out = A.attention_decode(q, k, v, lens, options)
        assert _lib.probe("kernel_launches") - before == launches
        unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        for i in range(0, b, 5):
            n = s if lens is None else int(lens[i])
            first = max(0, n - 1 - left) if left >= 0 else 0
            kk, vv = (x[i, first:n].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
            scores = torch.einsum("hd,shd->hs", q[i].double(), kk) / math.sqrt(d)
            want = torch.einsum("hs,shd->hd", torch.softmax(scores, 1), vv) if n else torch.zeros(hq, d, dtype=torch.float64, device="cuda")
            # One rounding of the result; the sums before it are f32.
            assert ((out[i].double() - want).abs() <= unit * want.abs() + 1e-5).all(), i
        assert torch.equal(A.attention_decode(q, k, v, lens, options), out)
