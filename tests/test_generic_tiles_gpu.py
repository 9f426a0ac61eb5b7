"""The CUDA-core training kernels where their tiles can go wrong: blocks of 8, 16 and 32 rows (calls on both sides of the lines,
by tokens and by heads), tiles of 32 with remainders, head dimensions on both sides of 64 and 128, of whole and of broken
16-byte vectors, inputs no vector can read, padding and packed batches, against the f64 oracle; repeats to the bit."""
import numpy as np
import pytest
import torch

import cases as K
import records as R
from adapter import B200Adapter
from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions, DType
from oracle import attention_oracle as oracle
from test_kernels_gpu import OWN, oracle_results, run_case

pytestmark = pytest.mark.gpu
C, N = AttentionOptions.causal_(), AttentionOptions()


@pytest.fixture(scope="module")
def adapter():
    return B200Adapter()


def generic_cases():
    out = []
    # b, hq, hkv, tq, tk, d: one query (of five keys: with one, dQ and dK are zero); a tile's edges; 370 and 371 blocks of 8 rows, 371 of 16; several tiles a side
    for i, (dims, options) in enumerate([((1, 2, 1, 1, 5, 64), N), ((2, 3, 3, 31, 33, 51), C), ((1, 4, 2, 65, 64, 96), C), ((1, 1, 1, 2960, 40, 4), N),
                                         ((1, 1, 1, 2961, 40, 4), N), ((1, 1, 1, 5925, 40, 4), N), ((1, 148, 4, 32, 96, 66), C), ((1, 2, 1, 130, 257, 256), C.with_window(50, 0)),
                                         ((3, 50, 50, 70, 70, 128), C), ((1, 4, 4, 300, 300, 200), N.with_window(20, 90)), ((1, 6, 2, 40, 5000, 72), C)]):
        out.append(K.seeded(f"{dims}", list(dims), AttentionMask.none(), options, 9000 + 10 * i))
    pad = np.zeros((3, 100), dtype=bool)
    pad[0, 33:] = True
    pad[1, :64] = True
    pad[2] = True
    out.append(K.seeded("padded", [3, 4, 2, 100, 100, 64], AttentionMask.key_padding(pad), N, 9500))
    lens = [1, 31, 0, 33, 64, 40, 7]
    out.append(K.seeded("packed", [1, 4, 2, sum(lens), sum(lens), 64], AttentionMask.packed(K.offsets(lens), K.offsets(lens)), C, 9510))
    ql, kl = [40, 0, 50], [7, 30, 90]
    out.append(K.seeded("packed, other keys", [1, 4, 4, sum(ql), sum(kl), 80], AttentionMask.packed(K.offsets(ql), K.offsets(kl)), N.with_window(60, 8), 9520))
    return out


CASES = generic_cases()


@pytest.mark.parametrize("dtype", [DType.F32, DType.F16], ids=["f32", "f16"])
@pytest.mark.parametrize("case", CASES, ids=[c.name for c in CASES])
def test_generic_tiles(adapter, case, dtype):
    # f16 here takes what f32 takes only by force; its inputs are rounded, which alone is 2^-11 of each product.
    _lib.lib().dash_attn_force_generic(1)
    try:
        a, b = run_case(adapter, case, dtype), run_case(adapter, case, dtype)
    finally:
        _lib.lib().dash_attn_force_generic(0)
    # One term a sum leaves nothing to average out: results of few terms get the roundings of inputs and result in full
    # (f16: 2^-10 through two rounded factors and 2^-11 of the result, of sums that cancel to a third at worst: 6e-3).
    bounds = OWN[DType.F32] if dtype == DType.F32 else [6e-3, 1e-3, 6e-3, 6e-3, 6e-3]
    R.check(case.name, [a.out, a.lse, *a.grads], oracle_results(case), bounds)
    for x, y in zip([a.out, a.lse, *a.grads], [b.out, b.lse, *b.grads]):
        assert np.array_equal(x, y, equal_nan=True)


def test_rows_no_vector_can_read():
    """f32 rows off the 16-byte grid, of broken strides, and of every other element: the bits of the same values laid out plainly."""
    t, h, d = 77, 3, 64
    g = torch.Generator(device="cuda").manual_seed(3)
    plain = [torch.randn(1, t, h, d, device="cuda", generator=g) for _ in range(4)]
    mask = AttentionMask.none()
    want = A.attention_with_lse(*plain[:3], mask, C)
    want_g = A.attention_backward(*plain[:3], *want, plain[3], mask, C)

    def off_grid(x):
        y = torch.empty(x.numel() + 1, device="cuda")[1:].view(x.shape)
        return y.copy_(x)

    def odd_stride(x):
        y = torch.empty(1, t, h, d + 1, device="cuda")[..., :d]
        return y.copy_(x)

    def every_other(x):
        y = torch.empty(1, t, h, 2 * d, device="cuda")[..., ::2]
        return y.copy_(x)

    def head_major(x):
        y = torch.empty(1, h, t, d, device="cuda").transpose(1, 2)
        return y.copy_(x)

    for lay in (off_grid, odd_stride, every_other, head_major):
        q, k, v, go = (lay(x) for x in plain)
        got = A.attention_with_lse(q, k, v, mask, C)
        got_g = A.attention_backward(q, k, v, *got, go, mask, C)
        assert all(torch.equal(x, y) for x, y in zip((*got, *got_g), (*want, *want_g))), lay.__name__


# Rows whose blocks have nothing to sweep (their own rows still arrive asynchronously, and the block waits for them before it
# leaves): b, hq, hkv, tq, tk, d with blocks of 8, 16 and 32 rows; all keys padded, or causal with more queries than keys.
@pytest.mark.parametrize("shape", [(2, 4, 2, 40, 40, 64), (1, 8, 8, 700, 60, 128), (2, 16, 16, 600, 600, 64), (1, 2, 1, 33, 9, 256)], ids=str)
@pytest.mark.parametrize("kind", ["all padding", "causal"])
def test_blocks_with_nothing_to_sweep(shape, kind):
    b, hq, hkv, tq, tk, d = shape
    host = [oracle.seeded(s, 9600 + j) for j, s in enumerate([(b, tq, hq, d), (b, tk, hkv, d), (b, tk, hkv, d), (b, tq, hq, d)])]
    q, k, v, g = (torch.from_numpy(x).cuda() for x in host)
    if kind == "causal":
        mask, options, blind = AttentionMask.none(), C, max(tq - tk, 0)
    else:
        mask, options, blind = AttentionMask.key_padding(torch.ones(b, tk, dtype=torch.bool, device="cuda")), N, tq
    for _ in range(20):
        o, lse = A.attention_with_lse(q, k, v, mask, options)
        dq, dk, dv = A.attention_backward(q, k, v, o, lse, g, mask, options)
        assert not o[:, :blind].any() and torch.isneginf(lse[:, :blind]).all() and not dq[:, :blind].any()
        if blind == tq:
            assert not dk.any() and not dv.any()
    if kind == "causal":
        want_o, want_lse = oracle.forward(*host[:3], causal=True)
        assert np.max(np.abs(o.cpu().numpy() - want_o)) <= OWN[DType.F32][0] * np.max(np.abs(want_o))
        assert torch.isfinite(lse[:, blind:]).all()
