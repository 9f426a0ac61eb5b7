"""Tiles of query rows that hold several heads of a group (128 / 2^p tokens x 2^p heads): every power of two a
group can give (1, 2, 4, 8, and what is left of 3, 6, 12 and 16), with lengths on both sides of a tile's tokens,
on the kernels of the three head dimensions, against the f64 oracle; repeats to the bit.  (These calls are too small for the
five-product backward: test_backward_pairs_gpu.py has its tiles.)"""
import numpy as np
import pytest

import cases as K
import records as R
from adapter import B200Adapter
from dashmag_b200.contract import AttentionMask, AttentionOptions, DType
from test_kernels_gpu import oracle_results, run_case
from test_random_shapes_gpu import SWEEP

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def adapter():
    return B200Adapter()


def tile_cases():
    out = []
    # (group, kv heads, d): tokens to a tile 128, 128, 64, 32, 64, 16, 32, 16
    for i, (group, hkv, d) in enumerate([(1, 3, 128), (3, 2, 128), (2, 2, 128), (4, 2, 128), (6, 1, 64), (8, 1, 128), (12, 1, 128), (16, 1, 64),
                                         (8, 1, 256), (4, 1, 256), (16, 2, 128)]):
        for j, (tq, tk) in enumerate([(129, 129), (1, 70), (17, 200), (257, 300)]):
            if d != 128:
                tq, tk = max(tq, 128), max(tk, 128)
            options = AttentionOptions.causal_() if j % 2 == 0 else AttentionOptions.causal_().with_window(40, 0)
            out.append(K.seeded(f"group {group} d{d} tq{tq} tk{tk}", [2, group * hkv, hkv, tq, tk, d], AttentionMask.none(), options, 5000 + 10 * i + j))
        lens = [31, 0, 33, 1, 15, 64, 17]   # sequences that meet inside the tiles
        out.append(K.seeded(f"group {group} d{d} packed", [1, group * hkv, hkv, sum(lens), sum(lens), d],
                            AttentionMask.packed(K.offsets(lens), K.offsets(lens)), AttentionOptions.causal_(), 5005 + 10 * i))
    return out


CASES = tile_cases()
# With one query a gradient's sum has one term and nothing averages out: P (or dS) and the result are each rounded to
# bf16, up to 2^-8 of the largest value apiece - 2 x 2^-8 for dV - and dK takes a third rounding through delta, which
# is made from the output as stored.  The same holds for tiles of one head (group 1: 5.5e-3 of dK).
ONE_QUERY = SWEEP[:3] + [3 * 2.0 ** -8, 2 * 2.0 ** -8]


@pytest.mark.parametrize("case", CASES, ids=[c.name for c in CASES])
def test_heads_share_tiles(adapter, case):
    a = run_case(adapter, case, DType.BF16)
    want = oracle_results(case)
    bounds = ONE_QUERY if case.q.shape[1] == 1 else SWEEP
    R.check(case.name, [a.out, a.lse, *a.grads], want, bounds)
    b = run_case(adapter, case, DType.BF16)
    for x, y in zip([a.out, a.lse, *a.grads], [b.out, b.lse, *b.grads]):
        assert np.array_equal(x, y, equal_nan=True), "two runs of the same call differ"
    c = run_case(adapter, case, DType.BF16, deterministic=False)
    R.check(f"any order {case.name}", [c.out, c.lse, *c.grads], want, bounds)
