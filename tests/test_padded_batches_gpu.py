"""Batches padded at the right, at the left, at both ends and from end to end (sweeps end where the tokens do; key blocks
of padding alone are not swept), holes inside, lengths on both sides of a look's 256 flags and of a step's 64 / 128 keys,
on the kernels of the three head dimensions, against the f64 oracle."""
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


def padded_cases():
    out = []
    t = 700
    spans = [(0, 700), (0, 1), (0, 63), (0, 65), (0, 443), (0, 445), (0, 188), (257, 700), (255, 700), (699, 700), (300, 310), (0, 0)]
    keep = np.zeros((len(spans), t), dtype=bool)
    for i, (lo, hi) in enumerate(spans):
        keep[i, lo:hi] = True
    keep[0, 128:384] = False   # a hole of two whole key blocks
    for i, (d, group) in enumerate([(128, 2), (64, 1), (256, 1)]):
        for j, options in enumerate([AttentionOptions(), AttentionOptions.causal_()]):
            out.append(K.seeded(f"d{d} {'causal' if j else 'full'}", [len(spans), 2 * group, 2, t, t, d], AttentionMask.key_padding(~keep), options, 7000 + 10 * i + j))
    return out


CASES = padded_cases()


@pytest.mark.parametrize("case", CASES, ids=[c.name for c in CASES])
@pytest.mark.parametrize("deterministic", [True, False])
def test_padded_batch(adapter, case, deterministic):
    got = run_case(adapter, case, DType.BF16, deterministic)
    R.check(case.name, [got.out, got.lse, *got.grads], oracle_results(case), SWEEP)
