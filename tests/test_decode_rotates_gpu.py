"""The decoding step whose split pass rotates the queries and the new key as it reads them: the bits of the steps taken one by
one (rotation, then the appending step), in the result and in the caches - partial rotations with halves of whole and of
broken 16-byte chunks (the latter take a launch of their own), heads of 256 whose pairs sit in two warps, groups of more than
sixteen heads, the new row on both sides of a chunk's and a tile's edge, positions outside the tables - in one chunk's worth of
units and in several waves of them (both block shapes)."""
import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.rope import Rope, attention_decode_append_rope

pytestmark = pytest.mark.gpu

LENGTHS = [0, 1, 15, 16, 63, 64, 65, 127, 128, 300, 511, 512]   # 512: the cache is full, no row is written


# (d, rotated, query heads per key-value head, key-value heads, whether the pass rotates)
@pytest.mark.parametrize("d,dim,group,hkv,fused", [
    (128, 128, 2, 2, True), (128, 64, 20, 1, True), (128, 96, 4, 3, True), (128, 24, 4, 2, False), (128, 2, 4, 2, False), (64, 64, 16, 1, True),
    (64, 32, 33, 1, True), (256, 256, 4, 2, True), (256, 160, 3, 1, True), (256, 16, 8, 1, True), (128, 128, 1, 2, False), (128, 128, 4, 64, True)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
def test_the_pass_rotates_to_the_bit(d, dim, group, hkv, fused, dtype):
    b, s = len(LENGTHS), 512
    g = torch.Generator(device="cuda").manual_seed(d + dim + group)
    rnd = lambda *shape: torch.randn(shape, device="cuda", generator=g).to(dtype)
    q, kn, vn, k, v = rnd(b, group * hkv, d), rnd(b, hkv, d), rnd(b, hkv, d), rnd(b, s, hkv, d), rnd(b, s, hkv, d)
    k2, v2 = k.clone(), v.clone()
    rope = Rope(dim, 10000.0, 600, dtype, device="cuda")
    lens = torch.tensor(LENGTHS, dtype=torch.int32, device="cuda")
    bits = lambda x: x.view(torch.int16)
    for positions in (None, torch.arange(b, device="cuda") * 54):   # the last, 594, still inside the tables
        launches = _lib.probe("kernel_launches")
        got = attention_decode_append_rope(rope, q, kn, vn, k, v, lens, positions=positions)
        assert _lib.probe("kernel_launches") - launches == (2 if fused else 3)
        rq, rk = rope.apply_at(q, lens if positions is None else positions, other=kn)
        want = A.attention_decode_append(rq, rk, vn, k2, v2, lens)
        assert torch.equal(bits(got), bits(want)) and torch.equal(bits(k), bits(k2)) and torch.equal(bits(v), bits(v2))
    outside = torch.full((b,), 600, device="cuda")
    outside[3] = -1
    got = attention_decode_append_rope(rope, q, kn, vn, k, v, lens, positions=outside)
    rq, rk = rope.apply_at(q, outside, other=kn)
    want = A.attention_decode_append(rq, rk, vn, k2, v2, lens)
    assert torch.equal(bits(k), bits(k2)) and torch.equal(torch.isnan(got), torch.isnan(want))
