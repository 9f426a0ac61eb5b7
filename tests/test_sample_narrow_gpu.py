"""The list's threshold search where every key has a bin of its own: the largest logit from well within its 1024 keys of the bound to
well past them, zeros of either sign at the cut, few and many kept, one block a row and eight - against the oracle."""
import numpy as np
import pytest
import torch

from dashmag_b200.sample import SampleOptions, sample
from oracle import sample_oracle

pytestmark = pytest.mark.gpu


def value_of(key):
    """The bf16 whose order-preserving 16-bit key this is, as f32."""
    bits = key & 0x7FFF if key & 0x8000 else ~key & 0xFFFF
    return np.array([bits << 16], dtype=np.uint32).view(np.float32)[0]


def check(logits, options):
    got = sample(torch.from_numpy(logits).cuda().bfloat16(), options)
    want = sample_oracle.sample(logits, options.temperature, options.top_k, options.top_p, options.seed, options.offset)
    assert np.array_equal(got.tokens.cpu().numpy(), want[0])
    for x, y in zip((got.logprob, got.tempered_logprob, got.sampling_logprob), want[1:]):
        # The bound the reference holds its kernel to against its own CPU form, and f32's rounding of the larger ones.
        assert np.all(np.abs(x.cpu().numpy() - y) <= 4e-6 + 4e-7 * np.abs(y))


@pytest.mark.parametrize("b,v", [(3, 20000), (140, 9000)])
@pytest.mark.parametrize("k,p", [(1, 0.5), (20, 0.9), (50, 1.0), (500, 0.95)])
def test_the_largest_logit_near_and_far(b, v, k, p):
    rng = np.random.default_rng(v + k)
    z = torch.from_numpy(rng.standard_normal((b, v), dtype=np.float32) * 0.05).bfloat16().float().numpy()
    top = 0x8000 | (np.array([z.max()], dtype=np.float32).view(np.uint32)[0] >> 16)   # the key of the largest (positive) one
    for r in range(b):
        z[r, rng.integers(v)] = value_of(int(top) + (0, 300, 640, 700, 760, 820, 890, 900, 950, 1000, 1010, 1021, 1022, 1023, 1024)[r % 15])
    check(z, SampleOptions(temperature=0.7, top_k=k, top_p=p, seed=9, offset=2))


# (One sign a row: the kernel's keys order -0 below 0, in every form of the search, where the oracle ties them.)
@pytest.mark.parametrize("k", [3, 40, 300])
def test_zeros_at_the_cut(k):
    rng = np.random.default_rng(k)
    z = -np.abs(rng.standard_normal((6, 30000), dtype=np.float32)) - np.float32(1)
    z = torch.from_numpy(z).bfloat16().float().numpy()
    for r in range(6):
        z[r, rng.permutation(30000)[: (1, 30, 120)[r // 2]]] = np.float32(-0.0 if r % 2 else 0.0)
    check(z, SampleOptions(temperature=1.0, top_k=k, top_p=0.9, seed=3, offset=5))
