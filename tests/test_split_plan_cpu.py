"""What the forward's workspace query says about splitting a tile's keys, without a GPU: a pure function of the shape, nothing
for packed batches, f32 or calls that fill the GPU, and never more parts than the sweep they shorten is worth."""
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


def test_the_parts_stay_bounded():
    rng = random.Random(5)
    most = 0
    for _ in range(2000):
        hkv, group, d = rng.choice([1, 2, 3, 8]), rng.choice([1, 2, 3, 4, 8, 16]), rng.choice([64, 128, 256])
        b, tq, tk = rng.choice([1, 1, 2, 9]), rng.randint(130, 3000), rng.randint(130, 40000)
        options = rng.choice([C, N, C.with_window(rng.randint(0, 5000), 0), N.with_window(rng.randint(0, 900), rng.randint(0, 900))])
        n = splits(b, hkv * group, hkv, tq, tk, d, options)
        most = max(most, n)
        if n == 1:
            continue
        pack = 1   # heads of a group in a tile
        while pack < 8 and group % (2 * pack) == 0:
            pack *= 2
        rows, step, step_bytes = (128, 128, 4.1e6) if d == 256 else (256, 64, 2.2e6)   # of a block; keys of a step; f32 parts that cost one
        blocks = -(-tq // (rows // pack)) * (hkv * group // pack) * b
        steps = -(-tk // step)
        assert n <= 32 and n <= steps // 2, "a part has two steps of keys at least"
        assert blocks < 2 * 148, "a call that fills the GPU is not split"
        waves = -(-blocks // 148)
        assert 4 * n * b * tq * hkv * group * d <= step_bytes * waves * (steps + 6), "the parts cost less than the sweep they shorten"
    assert most > 8


def test_many_rows_are_not_split():
    """Calls that measured slower in parts than whole: their f32 rows outweigh the shorter sweep."""
    assert splits(1, 12, 4, 3000, 3000, 128) == 1 and splits(1, 12, 4, 1500, 1500, 128) == 1 and splits(1, 12, 4, 2048, 4096, 128) == 1
    assert splits(1, 12, 4, 1000, 3000, 256) == 1 and splits(1, 5, 1, 3000, 3000, 256) == 1 and splits(1, 12, 4, 3000, 3000, 64) == 1
    assert splits(1, 8, 2, 2380, 6897, 256) == 1   # 150 blocks: the second wave is two short ones


def test_sides_past_every_key_are_no_bound():
    big = [2 ** 63 - 1, 2 ** 63 - 2, 2 ** 62, 2 ** 40]
    for tq, tk, d in ((500, 8200, 128), (37, 3001, 64), (300, 3001, 256), (130, 4000, 128)):
        for options, sides in ((C, [(x, 0) for x in big]), (C, [(x, y) for x in big for y in big]), (N, [(x, y) for x in big for y in big])):
            for left, right in sides:
                assert splits(1, 32, 8, tq, tk, d, options.with_window(left, right)) == splits(1, 32, 8, tq, tk, d, options), (options, left, right)
        for x in big:
            assert splits(1, 32, 8, tq, tk, d, N.with_window(200, x)) == splits(1, 32, 8, tq, tk, d, N.with_window(200, None))
