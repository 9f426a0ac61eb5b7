"""The multi-GPU partition of the training passes, every rank's share run one after another on ONE
GPU: the shares of ``sharding.training_plan`` (head slices read in place through strides; bins of
sequences gathered into packed tensors of their own when the heads run out) put back together are
the whole call - to the bit where a share is a head slice of a packed batch with heads of 64 or 128
(the same tiles run), and to the rounding of the dtype where the sums run in another order: where a bin
of sequences is packed anew (its tiles cut the sequences elsewhere), where an unpacked call has few
enough tiles for their keys to be split over blocks, and where a call at head dimension 256 has few
enough units for two blocks to share one.  The units are independent: nothing but the partition is
under test."""
import ctypes

import numpy as np
import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200 import sharding
from dashmag_b200.contract import AttentionMask, AttentionOptions

pytestmark = pytest.mark.gpu
DEV = "cuda:0"


def normal(shape, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float32).to(torch.bfloat16)


def run(q, k, v, g, lengths, options):
    cu = torch.tensor(np.concatenate([[0], np.cumsum(lengths)]), dtype=torch.int32, device=DEV)
    mask = AttentionMask.packed(cu, cu)
    o, lse = A.attention_with_lse(q, k, v, mask, options)
    return (o, lse) + tuple(A.attention_backward(q, k, v, o, lse, g, mask, options))


def assert_rounding(name, got, want, what):
    got, want = got.float(), want.float()
    # o: its own rounding (neighbouring bf16 values) plus P rounded against other step boundaries (2^-9 of
    # each weight); lse: f32 rounding; the gradients: both results lie within the parity bound of the exact
    # gradient (dQ 7.7e-3, dK 4.6e-3, dV 5.0e-3 of the largest value, tests/test_full_size_gpu.py), so they
    # lie within twice that of each other
    if name == "o":
        bound = 2.0 ** -7 * want.abs() + 1e-3 * float(want.abs().max())
    elif name == "lse":
        bound = 1e-6 * want.abs().clamp_min(1.0)
    else:
        bound = torch.full_like(want, 2 * {"dq": 7.7e-3, "dk": 4.6e-3, "dv": 5.0e-3}[name] * float(want.abs().max()))
    finite = torch.isfinite(want)
    assert torch.equal(torch.isfinite(got), finite), name
    assert bool(((got - want).abs()[finite] <= bound[finite]).all()), f"{name}: {what} differs from the whole call"


@pytest.mark.parametrize("world,hkv,window", [(2, 4, None), (8, 4, 300), (4, 1, None), (8, 8, None)],
                         ids=["2 ranks x 2 heads", "8 ranks: 4 heads x 2 sequence bins, window", "4 ranks share one head", "a head a rank"])
def test_the_ranks_shares_put_together_are_the_whole_call(world, hkv, window):
    lengths = [700, 130, 1, 515, 260, 390, 128, 333]
    t, group, d = sum(lengths), 2, 128
    q, k, v, g = normal((1, t, hkv * group, d), 1), normal((1, t, hkv, d), 2), normal((1, t, hkv, d), 3), normal((1, t, hkv * group, d), 4)
    options = AttentionOptions.causal_() if window is None else AttentionOptions.causal_().with_window(window, 0)
    whole = run(q, k, v, g, lengths, options)
    parts = [torch.full_like(x, float("nan")) for x in whole]
    starts = np.concatenate([[0], np.cumsum(lengths)])
    plan = sharding.training_plan(lengths, hkv, group, world, window)
    for rank, entry in enumerate(plan):
        seqs, kv, qh = entry
        mine, qr, kr, vr, gr = sharding.training_share(entry, lengths, q, k, v, g)
        if qr.numel() == 0:
            continue
        if list(seqs) == list(range(len(lengths))):
            assert qr.data_ptr() == q[:, :, qh].data_ptr(), "a head share is a view of the caller's tensor"
        o, lse, dq, dk, dv = run(qr, kr, vr, gr, mine, options)
        at = 0
        for s_ in seqs:   # scatter the share's sequences back to their places
            a, b = int(starts[s_]), int(starts[s_ + 1])
            n = b - a
            parts[0][:, a:b, qh] = o[:, at:at + n]
            parts[1][:, a:b, qh] = lse[:, at:at + n]
            parts[2][:, a:b, qh] = dq[:, at:at + n]
            parts[3][:, a:b, kv] = dk[:, at:at + n]
            parts[4][:, a:b, kv] = dv[:, at:at + n]
            at += n
    torch.cuda.synchronize()
    bins = any(list(seqs) != list(range(len(lengths))) for seqs, _, _ in plan)
    for name, got, want in zip("o lse dq dk dv".split(), parts, whole):
        assert not torch.isnan(got.float()).any(), f"{name}: some unit was given to no rank"
        if not bins:
            assert torch.equal(got, want), f"{name}: the shares do not rebuild the whole call"
        else:
            assert_rounding(name, got, want, "a bin of sequences")


# Head slices whose sums run in another order than the whole call's: 4096 tokens of one key-value head are split over blocks, of two
# not; 1000 tokens of one head of 256 are 8 units, of ten 80.
@pytest.mark.parametrize("t,hkv,group,d,packed", [(4096, 2, 8, 128, False), (1000, 10, 2, 256, True)], ids=["unpacked", "head dimension 256"])
def test_head_slices_in_another_order(t, hkv, group, d, packed):
    q, k, v, g = normal((1, t, hkv * group, d), 1), normal((1, t, hkv, d), 2), normal((1, t, hkv, d), 3), normal((1, t, hkv * group, d), 4)
    options = AttentionOptions.causal_()
    cu = torch.tensor([0, t // 3, t], dtype=torch.int32, device=DEV)
    mask = AttentionMask.packed(cu, cu) if packed else AttentionMask.none()

    def step(q, k, v, g):
        o, lse = A.attention_with_lse(q, k, v, mask, options)
        return (o, lse) + tuple(A.attention_backward(q, k, v, o, lse, g, mask, options))

    def scratch(q, k):
        return _lib.lib().dash_attn_forward_workspace(ctypes.byref(A.make_params("attention", q, k, k, mask, options)[0]))

    whole = step(q, k, v, g)
    for h in range(hkv):
        kv, qh = slice(h, h + 1), slice(h * group, (h + 1) * group)
        if not packed:
            assert scratch(q, k) == 0 and scratch(q[:, :, qh], k[:, :, kv]) > 0, "the share is split, the whole call is not"
        share = step(q[:, :, qh], k[:, :, kv], v[:, :, kv], g[:, :, qh])
        for name, got, want, at in zip("o lse dq dk dv".split(), share, whole, (qh, qh, qh, kv, kv)):
            assert_rounding(name, got, want[:, :, at], "a head slice")


# The CUDA-core kernels take another form as the rows, heads and batch of a call grow: one, two or four rows a warp, which sum in one order,
# or (up to head dimension 128) two warps to a pair of rows, which sum in another.  dtype, batch, key-value heads, group, tokens, head dimension,
# mask, with the whole call and its slices on both sides of the lines: slices agree to rounding, and to the bit beyond 128.
@pytest.mark.parametrize("dtype,b,hkv,group,t,d,kind", [
    (torch.float32, 1, 4, 1, 1000, 64, "packed"), (torch.float32, 1, 4, 2, 1500, 64, "packed"), (torch.float32, 1, 8, 4, 300, 128, "window"),
    (torch.float32, 1, 16, 1, 700, 96, "packed"), (torch.float32, 1, 2, 8, 333, 40, "packed"), (torch.bfloat16, 2, 8, 2, 500, 80, "padding"),
    (torch.float32, 12, 2, 2, 200, 64, "causal"), (torch.float16, 24, 3, 1, 170, 96, "padding"), (torch.float32, 3, 6, 1, 260, 200, "window")], ids=str)
def test_slices_on_the_cuda_cores(dtype, b, hkv, group, t, d, kind):
    q, k, v, g = (normal((b, t, h, d), i).to(dtype) for i, h in enumerate((hkv * group, hkv, hkv, hkv * group)))
    options = AttentionOptions.causal_() if kind != "padding" else AttentionOptions()
    if kind == "window":
        options = options.with_window(t // 3, 0)
    cu = torch.tensor([0, 1, t // 3 + 7, t], dtype=torch.int32, device=DEV)
    pad = torch.arange(t, device=DEV)[None] >= t - 13 * torch.arange(b, device=DEV)[:, None] % t

    def step(n, kv):
        mask = AttentionMask.packed(cu, cu) if kind == "packed" else AttentionMask.key_padding(pad[n]) if kind == "padding" else AttentionMask.none()
        qh = slice(kv.start * group, kv.stop * group)
        qs, ks, vs, gs = q[n][:, :, qh], k[n][:, :, kv], v[n][:, :, kv], g[n][:, :, qh]
        o, lse = A.attention_with_lse(qs, ks, vs, mask, options)
        return (o, lse) + tuple(A.attention_backward(qs, ks, vs, o, lse, gs, mask, options))

    before = _lib.probe("generic_runs")
    whole = step(slice(0, b), slice(0, hkv))
    assert _lib.probe("generic_runs") == before + 2
    for n in (1, max(b // 3, 1)):
        for heads in (1, max(hkv // 2, 1)):
            at, kv = slice(b - n, b), slice(0, heads)
            qh = slice(0, heads * group)
            for name, got, want, h in zip("o lse dq dk dv".split(), step(at, kv), whole, (qh, qh, qh, kv, kv)):
                want = want[at][:, :, h]
                if d > 128:
                    assert torch.equal(got, want), f"{name}: {n} sequences, {heads} key-value heads"
                    continue
                # Both lie within the f32 kernels' bound of the exact result (tests/test_kernels_gpu.py: 1e-5 of the largest value, the
                # log-sum-exp 1e-6), so within twice that of each other; 16-bit results that straddle a rounding are neighbours.
                near = (2e-6 if name == "lse" else 2e-5) * want.float().abs()[torch.isfinite(want)].max()
                slack = 0.0 if name == "lse" else {torch.float32: 0.0, torch.bfloat16: 2.0 ** -7, torch.float16: 2.0 ** -10}[dtype]
                finite = torch.isfinite(want)
                assert torch.equal(torch.isfinite(got), finite)
                apart = (got.float() - want.float()).abs()[finite] - slack * want.float().abs()[finite]
                assert float(apart.max()) <= float(near), f"{name}: {n} sequences, {heads} key-value heads"
