"""The decoding step's merge at the numbers of partials where its form changes - all of them asked for at once by 128, 256 or 512
threads, in passes beyond, head dimensions that do not divide the threads - against the same sums in f64; repeats to the bit.  (Of the first
list, groups of two to eight 16-bit heads with short shares are taken by clusters and have no merge; the second holds each line with calls
that go in chunks, and says so.)"""
import math

import pytest
import torch

from dashmag_b200 import _lib
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


# Partials of 64 keys each on both sides of 32, 64 and 128 of them (heads of 128; of 64 and 256 twice and half as many): 128 | 256 | 512 threads | passes.
@pytest.mark.parametrize("b,s,hq,hkv,d,dtype", [
    (1, s, 16, 1, 128, "bf16") for s in (2048, 2049, 4096, 4097, 8192, 8193)] + [(1, s, 4, 4, 128, "f32") for s in (2048, 2049, 4096, 4097, 8192, 8193)] + [
    (2, s, 9, 1, 64, "f16") for s in (4096, 4097, 8192, 8193)] + [(1, s, 12, 1, 256, "bf16") for s in (1024, 1025, 2048, 2049, 4096, 4097)] + [
    (1, 8193, 8, 8, 128, "f16"),
    # Columns of up to eight heads, blocks of two warps and of eight: 2304 and 2368 warps.
    (36, 512, 64, 16, 128, "bf16"), (37, 512, 64, 16, 128, "bf16"), (72, 512, 16, 8, 128, "f16"), (74, 512, 16, 8, 128, "f16")])
def test_chunks_are_merged(b, s, hq, hkv, d, dtype):
    dtype = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}[dtype]
    g = torch.Generator(device="cuda").manual_seed(s)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").to(dtype) for shape in ((b, hq, d), (b, s, hkv, d), (b, s, hkv, d)))
    lengths = torch.randint(0, s + 1, (b,), generator=g, device="cuda", dtype=torch.int32)
    lengths[0] = s
    before = _lib.probe("kernel_launches")
    out = A.attention_decode(q, k, v, lengths)
    assert _lib.probe("kernel_launches") - before == 2
    unit = {torch.float32: 2.0 ** -20, torch.bfloat16: 2.0 ** -8, torch.float16: 2.0 ** -11}[dtype]
    for i, n in enumerate(lengths.tolist()):
        kk, vv = (x[i, :n].double().repeat_interleave(hq // hkv, 1) for x in (k, v))
        want = torch.einsum("hs,shd->hd", torch.softmax(torch.einsum("hd,shd->hs", q[i].double(), kk) / math.sqrt(d), 1), vv)
        # One rounding of the result; the sums before it are f32.
        assert ((out[i].double() - want).abs() <= unit * want.abs() + 1e-5).all(), i
    assert torch.equal(A.attention_decode(q, k, v, lengths), out)
