"""The sampler's list of candidates: rows whose list fits, rows whose list does not (ties by the thousand at the cut, a nucleus
of nearly everything) and goes back to the passes over the row, cuts wider than the threads that bound them, masked ids
above the cut, one block and several to a row - against the oracle, tokens and log-probabilities, and repeats to the bit."""
import numpy as np
import pytest

from dashmag_b200.sample import SampleOptions
from oracle import sample_oracle as S
from oracle.rope_oracle import round_to
from test_sample_gpu import close, logits_of, oracle_of, run

pytestmark = pytest.mark.gpu


def rows(kind, b, v, dtype):
    z = logits_of(b, v, dtype, 11 + v, scale=3.0)
    rng = np.random.default_rng(v)
    if kind == "ties at the top":          # a third of the row holds the maximum: more than a list
        z[:, rng.permutation(v)[: v // 3]] = np.float32(12.0)
    elif kind == "flat":
        z[:] = np.float32(1.0)
    elif kind == "one token":
        z[:] = np.float32(-40.0)
        z[:, v // 2] = np.float32(40.0)
    elif kind == "few values":             # whole classes of ties on both sides of the cut
        z = np.round(z)
    elif kind == "ruled out":              # most of the row at -inf: most threads have nothing
        z[:, rng.permutation(v)[: v - 40]] = -np.inf
    elif kind == "far from zero":          # one byte of a key does not tell the tokens apart
        z = z + np.float32(20.0)
    elif kind == "crowded blocks":         # few threads' maxima reach the bound, in blocks whose lists they overflow (eight blocks a row)
        z = z + np.where(np.arange(v) // (8 if dtype == "bf16" else 4) % 8192 < 3000, np.float32(30.0), np.float32(0.0))
    return round_to(z, dtype)


@pytest.mark.parametrize("dtype", ["bf16", "f32"])
@pytest.mark.parametrize("b,v", [(2, 151936), (64, 30011), (150, 9001)])   # eight, two blocks a row; one
@pytest.mark.parametrize("kind", ["plain", "ties at the top", "flat", "one token", "few values", "ruled out", "far from zero", "crowded blocks"])
def test_lists(kind, b, v, dtype):
    z = rows(kind, b, v, dtype)
    top = tuple(int(i) for i in np.argsort(-z[0], kind="stable")[:7])
    # The nucleus ends where the kept mass reaches p of all of it; the oracle's f32 sums know that to some 1e-6 of the mass.  With
    # forty tokens left, p = 0.9999 puts tokens of about that weight at the edge (a row of 9001 differed, with the passes over
    # the row as with the list), p = 0.99 none of less than 1e-4.
    nearly_all = 0.99 if kind == "ruled out" else 0.9999
    for options in (SampleOptions(top_k=50, top_p=0.9, temperature=0.7, seed=1), SampleOptions(top_k=1, seed=2), SampleOptions(top_k=20, seed=3),
                    SampleOptions(top_k=3000, top_p=0.5, seed=4), SampleOptions(top_p=0.9, temperature=0.7, seed=5), SampleOptions(top_p=nearly_all, seed=6),
                    SampleOptions(top_k=30, top_p=0.95, masked=top, seed=7), SampleOptions(top_p=0.6, masked=top, seed=8)):
        # A nucleus alone makes no list; and on a row of ties its end can fall closer to p (6.6e-8 of the mass, a bf16 row of 9001
        # far from zero, p = 0.9999) than the oracle's f32 sums tell (some 1e-6).
        if kind in ("far from zero", "crowded blocks") and options.top_k == 0:
            continue
        got, want = run(z, dtype, options), oracle_of(z, options)
        tau = float(S.inverse_temperature(options.temperature))
        for r in np.nonzero(got[0] != want[0])[0]:   # decided inside the last places of f32 (test_sample_gpu)
            g = S.gumbel_of_inputs(S.row_inputs(options.seed, options.offset, int(r), v))
            score = (z[r] - z[r].max()) * tau + g
            assert abs(score[got[0][r]] - score[want[0][r]]) <= 4e-6 * max(1.0, abs(score[want[0][r]])), (options, r)
        same = got[0] == want[0]
        for k in (1, 2, 3):
            assert close(got[k][same], want[k][same]), (options, k)
        again = run(z, dtype, options)
        assert all(np.array_equal(x, y, equal_nan=True) for x, y in zip(got, again))
