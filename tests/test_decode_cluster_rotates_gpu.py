"""The decoding step that rotates and appends in a cluster's launch: the bits of the rotation, then the appending step, in the result and in the
caches - heads of 64, 128 and of 256, whose partner columns sit in another warp; whole and partial rotations; the new row at the edges
of tiles and of a warp's share, in the first and in the last block; full caches; positions given and outside the tables."""
import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.rope import Rope, attention_decode_append_rope

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("b,s,group,hkv,d,dim", [
    (1, 4096, 4, 8, 128, 128), (4, 4096, 4, 8, 128, 64), (2, 1000, 8, 2, 128, 96), (3, 700, 2, 4, 64, 64), (6, 2000, 5, 4, 64, 32),
    (2, 700, 4, 2, 256, 256), (8, 600, 8, 2, 256, 160), (12, 1500, 4, 4, 256, 16), (16, 700, 3, 8, 256, 256)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
def test_to_the_bit(b, s, group, hkv, d, dim, dtype):
    g = torch.Generator(device="cuda").manual_seed(s + d)
    rnd = lambda *shape: torch.randn(shape, device="cuda", generator=g).to(dtype)
    bits = lambda x: x.view(torch.int16)
    rope = Rope(dim, 10000.0, s + 100, dtype, device="cuda")
    q, kn, vn, k0, v0 = rnd(b, group * hkv, d), rnd(b, hkv, d), rnd(b, hkv, d), rnd(b, s, hkv, d), rnd(b, s, hkv, d)
    edges = [s - 1, 0, 15, 16, s, s // 2, 1, s - 17, 63, 64, s // 3, 127, 128, 255, 256, s - 2]   # s: the cache is full, no row is written
    for turn in range(0, 16, b):
        lengths = torch.tensor((edges[turn:] + edges)[:b], dtype=torch.int32, device="cuda")
        for positions in (None, lengths + 50, torch.full_like(lengths, s + 100)):
            k, v, k2, v2 = k0.clone(), v0.clone(), k0.clone(), v0.clone()
            before = _lib.probe("kernel_launches")
            got = attention_decode_append_rope(rope, q, kn, vn, k, v, lengths, positions=positions)
            assert _lib.probe("kernel_launches") - before == 1
            rq, rk = rope.apply_at(q, lengths if positions is None else positions, other=kn)
            before = _lib.probe("kernel_launches")
            want = A.attention_decode_append(rq, rk, vn, k2, v2, lengths)
            assert _lib.probe("kernel_launches") - before == 1
            assert torch.equal(bits(k), bits(k2)) and torch.equal(bits(v), bits(v2))
            if positions is None or int(positions[0]) < s + 100:
                assert torch.equal(bits(got), bits(want))
            else:
                assert torch.equal(torch.isnan(got), torch.isnan(want))
