"""What the forward's workspace query says about splitting a tile's keys, without a GPU: a pure function of the shape, nothing
for packed batches, f32 or calls that fill the GPU, and never more rows of parts than a few waves of tiles."""
import ctypes
import random

import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions

C, N = AttentionOptions.causal_(), AttentionOptions()


def splits(b, hq, hkv, tq, tk, d, options=C, dtype=torch.bfloat16, mask=AttentionMask.none()):
    q, k = torch.empty(b, tq, hq, d, dtype=dtype, device="meta"), torch.empty(b, tk, hkv, d, dtype=dtype, device="meta")
    p, _ = A.make_params("attention", q, k, k, mask, options)
    need = _lib.lib().dash_attn_forward_workspace(ctypes.byref(p))
    rows = b * tq * hq
    if need == 0:
        return 1
    n = need // (4 * rows * (d + 1))
    assert need == 4 * n * rows * d + (4 * n * rows + 255) // 256 * 256, "parts and their log-sum-exps, nothing else"
    return n


def test_who_is_split():
    assert splits(1, 32, 8, 500, 8200, 128) > 1 and splits(1, 32, 8, 130, 4000, 64) > 1 and splits(1, 8, 2, 130, 4000, 256) > 1
    assert splits(1, 32, 8, 16, 4000, 128) > 1
    assert splits(1, 32, 8, 500, 8200, 128, dtype=torch.float32) == 1 and splits(1, 32, 8, 500, 8200, 96) == 1
    cu = torch.tensor([0, 500], dtype=torch.int32)
    assert splits(1, 32, 8, 500, 500, 128, mask=AttentionMask.packed(cu, cu)) == 1
    assert splits(1, 32, 8, 16384, 16384, 128) == 1 and splits(16, 12, 12, 509, 509, 64, N) == 1
    assert splits(1, 32, 8, 500, 60, 128) == 1   # too few keys to share
    # What the CUDA-core kernels take is never split, and no scratch is asked for: few queries at D 64 and 256, a scale the
    # tensor-core kernels refuse, rows no tile load can read.
    assert splits(1, 32, 8, 16, 4000, 64) == 1 and splits(1, 32, 8, 100, 9100, 256) == 1
    assert splits(1, 32, 8, 500, 8200, 128, C.with_scale(-0.1)) == 1
    q = torch.empty(1, 500, 32, 128, dtype=torch.bfloat16, device="meta")
    for width, step in ((256, 2), (132, 1)):
        k = torch.empty(1, 8200, 8, width, dtype=torch.bfloat16, device="meta")[..., : 128 * step : step]
        p, _ = A.make_params("attention", q, k, k, AttentionMask.none(), C)
        assert _lib.lib().dash_attn_forward_workspace(ctypes.byref(p)) == 0


def test_the_parts_stay_a_few_waves():
    rng = random.Random(5)
    for _ in range(2000):
        hkv, group, d = rng.choice([1, 2, 3, 8]), rng.choice([1, 2, 3, 4, 8, 16]), rng.choice([64, 128, 256])
        b, tq, tk = rng.choice([1, 1, 2, 9]), rng.randint(1, 3000), rng.randint(1, 40000)
        options = rng.choice([C, N, C.with_window(rng.randint(0, 5000), 0), N.with_window(rng.randint(0, 900), rng.randint(0, 900))])
        n = splits(b, hkv * group, hkv, tq, tk, d, options)
        assert 1 <= n <= 32 and n * 64 <= max(tk, 64), "a part has a sub-step's keys at least"
        assert n == splits(b, hkv * group, hkv, tq, tk, d, options)


def test_sides_past_every_key_are_no_bound():
    big = [2 ** 63 - 1, 2 ** 63 - 2, 2 ** 62, 2 ** 40]
    for tq, tk, d in ((500, 8200, 128), (37, 3001, 64), (300, 3001, 256), (130, 4000, 128)):
        for options, sides in ((C, [(x, 0) for x in big]), (C, [(x, y) for x in big for y in big]), (N, [(x, y) for x in big for y in big])):
            for left, right in sides:
                assert splits(1, 32, 8, tq, tk, d, options.with_window(left, right)) == splits(1, 32, 8, tq, tk, d, options), (options, left, right)
        for x in big:
            assert splits(1, 32, 8, tq, tk, d, N.with_window(200, x)) == splits(1, 32, 8, tq, tk, d, N.with_window(200, None))
