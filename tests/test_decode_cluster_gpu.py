"""The decoding step whose key-value heads are taken by clusters of blocks: every size of cluster, caches from the shortest it
takes, sequences shorter than the cluster has warps and tiles, windows, groups that fill the eight columns and that do not, a NaN
that only some warps meet - against the same sums in f64; repeats to the bit, one launch."""
import math

import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionOptions

pytestmark = pytest.mark.gpu


# Units (b x hkv) 1 to 330: clusters of sixteen down to one block; the last four stay chunks (512 keys, few units of long sweeps)
# or groups above eight.
@pytest.mark.parametrize("b,s,hq,hkv,d,left,launches", [
    (1, 513, 8, 2, 128, -1, 1), (1, 528, 4, 2, 64, -1, 1), (1, 4096, 32, 8, 128, -1, 1), (3, 700, 24, 4, 128, -1, 1), (4, 1025, 56, 8, 128, -1, 1),
    (16, 1000, 16, 4, 128, -1, 1), (16, 3000, 32, 8, 128, 1000, 1), (20, 2000, 12, 4, 64, -1, 1), (1, 529, 16, 2, 256, -1, 1),
    (12, 1500, 16, 4, 256, -1, 1), (40, 777, 16, 8, 256, 300, 1), (55, 515, 12, 6, 64, -1, 1), (1, 512, 8, 2, 128, -1, 2), (1, 9000, 4, 1, 256, -1, 2),
    (2, 600, 18, 2, 128, -1, 2), (2, 600, 16, 1, 64, -1, 2)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
def test_against_f64(b, s, hq, hkv, d, left, launches, dtype):
    g = torch.Generator(device="cuda").manual_seed(b + s + d)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").to(dtype) for shape in ((b, hq, d), (b, s, hkv, d), (b, s, hkv, d)))
    lengths = torch.randint(0, s + 1, (b,), generator=g, device="cuda", dtype=torch.int32)
    for i, n in enumerate([s, 0, 1, 15, 16, 17, 33, s - 1][:b]):
        lengths[i] = n
    options = AttentionOptions().with_window(left, 0) if left >= 0 else AttentionOptions()
    for lens in (lengths, None):
        before = _lib.probe("kernel_launches")
        out = A.attention_decode(q, k, v, lens, options)
        assert _lib.probe("kernel_launches") - before == launches
        unit = 2.0 ** -8 if dtype == torch.bfloat16 else 2.0 ** -11
        for i, n in enumerate([s] * b if lens is None else lens.tolist()):
            first = max(0, n - 1 - left) if left >= 0 else 0
            kk, vv = (x[i, first:n].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
            scores = torch.einsum("hd,shd->hs", q[i].double(), kk) / math.sqrt(d)
            want = torch.einsum("hs,shd->hd", torch.softmax(scores, 1), vv) if n else torch.zeros(hq, d, dtype=torch.float64, device="cuda")
            # One rounding of the result; the sums before it are f32.
            assert ((out[i].double() - want).abs() <= unit * want.abs() + 1e-5).all(), i
        for _ in range(3):
            assert torch.equal(A.attention_decode(q, k, v, lens, options), out)


@pytest.mark.parametrize("b,s,hq,hkv,d", [(1, 4096, 8, 2, 128), (3, 1000, 16, 4, 256), (16, 3000, 32, 8, 64)])
def test_a_nan_is_its_heads_nan(b, s, hq, hkv, d):
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").bfloat16() for shape in ((b, hq, d), (b, s, hkv, d), (b, s, hkv, d)))
    lengths = torch.full((b,), s - 1, dtype=torch.int32, device="cuda")
    clean = A.attention_decode(q, k, v, lengths)
    group = hq // hkv
    for key in (0, 31, s // 2, s - 2):
        k2, v2 = k.clone(), v.clone()
        k2[0, key, 1, 3] = math.nan            # every query head of key-value head 1
        v2[b - 1, key, 0, 5] = math.nan        # one feature of key-value head 0
        out = A.attention_decode(q, k2, v2, lengths)
        want = clean.clone()
        want[0, group:2 * group] = math.nan
        want[b - 1, :group, 5] = math.nan
        assert torch.equal(torch.isnan(out), torch.isnan(want)) and torch.equal(out.nan_to_num(), want.nan_to_num())
    beyond = k.clone()
    beyond[:, s - 1] = math.nan                # past the lengths
    assert torch.equal(A.attention_decode(q, beyond, v, lengths), clean)
