"""The work this library is asked to do, as cases that can be prepared, run and compared.

Three kinds of call make up the attention path and each is here over its range, through the public
entry points: the training step of one attention layer (forward with its log-sum-exp, then the
backward), inference (a chunk of a prompt against the keys before it, the decoding step, and the
decoding step with rotation and append in front), and the two steps around them (rotation of a
layer's query and key, sampling of the next token).  Sizes are the benchmark's own configurations
or of their kind; values are N(0, 1) in the case's dtype, as there.
"""
import math

import numpy as np
import torch

from dashmag_b200.attention import attention, attention_backward, attention_decode, attention_with_lse
from dashmag_b200.contract import AttentionMask, AttentionOptions
from dashmag_b200.rope import Rope, attention_decode_append_rope
from dashmag_b200.sample import SampleOptions, sample

DTYPES = {"f32": torch.float32, "bf16": torch.bfloat16, "f16": torch.float16}
BYTES = {"f32": 4, "bf16": 2, "f16": 2}


def listed():
    return [
        # The smallest training call: two packed sequences in f32, the size of a unit test or a toy model.
        dict(name="train_small_f32", kind="packed", dtype="f32", seqs=2, lo=128, hi=256, total=384, hq=4, hkv=4, d=64,
             window=-1, deterministic=True, lens_seed=0),
        # The headline: a packed batch of eight sequences of 512 to 4096 tokens, grouped heads.
        dict(name="train_packed", kind="packed", dtype="bf16", seqs=8, lo=512, hi=4096, total=16384, hq=32, hkv=8, d=128,
             window=-1, deterministic=True, lens_seed=0),
        # Sliding-window training: sixteen packed sequences of 1024 to 8192 tokens, a window of 4096.
        dict(name="train_window", kind="packed", dtype="bf16", seqs=16, lo=1024, hi=8192, total=65536, hq=16, hkv=4, d=128,
             window=4096, deterministic=True, lens_seed=4),
        # Long context: one causal sequence of 131072 tokens, the share (one key-value head, eight query heads) that one
        # of eight GPUs holds of a 64 / 8-head layer.
        dict(name="train_long", kind="packed", dtype="bf16", seqs=1, lo=131072, hi=131072, total=131072, hq=8, hkv=1, d=128,
             window=-1, deterministic=True, lens_seed=0),
        # Head dimension 256, the reference's own benchmark shape.
        dict(name="train_d256", kind="packed", dtype="bf16", seqs=1, lo=6144, hi=6144, total=6144, hq=8, hkv=2, d=256,
             window=-1, deterministic=True, lens_seed=0),
        # An encoder's batch: right-padded sequences, every token sees every token that is not padding, heads of 64 without
        # grouping, f16, an odd length, the order of the query gradient's sums left free.
        dict(name="train_padded_f16", kind="padded", dtype="f16", b=16, t=509, lo=200, hq=12, hkv=12, d=64, causal=False,
             deterministic=False, lens_seed=1),
        # A chunk of a prompt against what is already in the cache (forward only; few queries, many keys).
        dict(name="prefill_chunk", kind="prefill", dtype="bf16", b=1, tq=500, past=7700, hq=32, hkv=8, d=128),
        # The serving step at a full batch: 64 sequences with 1024 to 32768 tokens in the cache.
        dict(name="decode_batch", kind="decode", dtype="bf16", b=64, s=32768, lo=1024, hq=32, hkv=8, d=128, window=-1, lens_seed=77),
        # The reference's own decoding case: eight whole caches of 6144 keys, heads of 256.
        dict(name="decode_short", kind="decode", dtype="bf16", b=8, s=6144, lo=0, hq=8, hkv=2, d=256, window=-1, lens_seed=0),
        # One user's next token: rotate, append to the cache, attend - where latency and launches count.
        dict(name="decode_single", kind="step", dtype="bf16", b=1, s=4096, lo=2047, hq=32, hkv=8, d=128, lens_seed=3),
        # The rotation of a layer's query and key over the headline batch.
        dict(name="rope_packed", kind="rope", dtype="bf16", seqs=8, lo=512, hi=4096, total=16384, hq=32, hkv=8, d=128, dim=128, lens_seed=0),
        # The next token of 64 sequences out of 151936.
        dict(name="sample_batch", kind="sample", dtype="bf16", b=64, v=151936, temperature=0.7, top_k=50, top_p=0.9),
    ]


# ------------------------------------------------------------------------------------------------
# More cases of the same ranges
# ------------------------------------------------------------------------------------------------
def _log(rng, lo, hi):
    """An integer of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def _sixteen(rng):
    return rng.choice(["bf16", "bf16", "f16"])


def _draw_packed(rng, dtype, total_lo, total_hi, seqs_hi, heads, dims, windows=(-1,)):
    total = _log(rng, total_lo, total_hi)
    seqs = rng.randint(1, max(1, min(seqs_hi, total // 48)))
    mean = total // seqs
    hq, hkv = rng.choice(heads)
    return dict(kind="packed", dtype=dtype, seqs=seqs, lo=max(1, mean // 4), hi=max(2, 2 * mean), total=total, hq=hq, hkv=hkv, d=rng.choice(dims),
                window=rng.choice(windows), deterministic=rng.random() < 0.85, lens_seed=rng.randrange(1000))


def draw(rng):
    family = rng.randrange(12)
    if family == 0:
        return _draw_packed(rng, "f32", 100, 1500, 4, [(4, 4), (4, 2), (8, 2), (3, 1)], [64, 64, 96, 128])
    if family in (1, 2):
        return _draw_packed(rng, _sixteen(rng), 1000, 32768, 16, [(32, 8), (16, 4), (16, 16), (8, 1), (24, 8)], [128, 128, 64])
    if family == 3:
        return _draw_packed(rng, _sixteen(rng), 8192, 65536, 16, [(16, 4), (16, 8), (8, 2)], [128], (512, 1024, 4096, 1000))
    if family == 4:
        return _draw_packed(rng, "bf16", 16384, 98304, 1, [(8, 1), (8, 2), (4, 1)], [128])
    if family == 5:
        return _draw_packed(rng, _sixteen(rng), 500, 8192, 4, [(8, 2), (16, 4), (4, 4)], [256])
    if family == 6:
        return dict(kind="padded", dtype=_sixteen(rng), b=rng.randint(1, 32), t=_log(rng, 130, 1024), lo=rng.randint(1, 129), hq=12, hkv=rng.choice([12, 4]),
                    d=rng.choice([64, 64, 128]), causal=rng.random() < 0.4, deterministic=rng.random() < 0.5, lens_seed=rng.randrange(1000))
    if family == 7:
        hq, hkv = rng.choice([(32, 8), (32, 8), (16, 16), (8, 1)])
        return dict(kind="prefill", dtype=_sixteen(rng), b=rng.choice([1, 1, 2]), tq=_log(rng, 16, 2048), past=_log(rng, 100, 30000), hq=hq, hkv=hkv,
                    d=rng.choice([128, 128, 64, 256]))
    if family == 8:
        hq, hkv = rng.choice([(32, 8), (32, 8), (16, 8), (16, 1)])
        return dict(kind="decode", dtype=_sixteen(rng), b=rng.randint(9, 64), s=_log(rng, 4096, 32768), lo=rng.randint(1, 1024), hq=hq, hkv=hkv, d=128,
                    window=rng.choice([-1, -1, 4096]), lens_seed=rng.randrange(1000))
    if family == 9:
        hq, hkv = rng.choice([(8, 2), (16, 4), (8, 8), (32, 8)])
        return dict(kind="decode", dtype=rng.choice(["bf16", "bf16", "f16", "f32"]), b=rng.randint(1, 16), s=_log(rng, 100, 8192), lo=rng.choice([0, 50]), hq=hq, hkv=hkv,
                    d=rng.choice([64, 128, 256]), window=rng.choice([-1, -1, 1024]), lens_seed=rng.randrange(1000))
    if family == 10:
        hq, hkv = rng.choice([(32, 8), (16, 4), (8, 8)])
        s = _log(rng, 256, 16384)
        return dict(kind="step", dtype=_sixteen(rng), b=rng.choice([1, 1, 2, 4, 16]), s=s, lo=rng.randint(1, s - 1), hq=hq, hkv=hkv, d=rng.choice([128, 128, 64]),
                    lens_seed=rng.randrange(1000))
    if rng.random() < 0.4:
        c = _draw_packed(rng, rng.choice(["bf16", "bf16", "f16", "f32"]), 7, 32768, 8, [(32, 8), (16, 4), (8, 8)], [64, 128, 256])
        return {k: c[k] for k in ("dtype", "seqs", "lo", "hi", "total", "hq", "hkv", "d", "lens_seed")} | dict(kind="rope", dim=rng.choice([c["d"], c["d"] // 2]))
    return dict(kind="sample", dtype=rng.choice(["bf16", "bf16", "f32"]), b=_log(rng, 1, 128), v=_log(rng, 5000, 200000), temperature=rng.choice([0.0, 0.7, 1.0]),
                top_k=rng.choice([0, 0, 20, 50]), top_p=rng.choice([1.0, 0.9, 0.95]))


# ------------------------------------------------------------------------------------------------
# Sizes
# ------------------------------------------------------------------------------------------------
def _lengths(c):
    """The packed sequences' lengths: integers uniform in [lo, hi], rescaled to sum to the total."""
    if c["seqs"] == 1:
        return [c["total"]]
    raw = np.random.default_rng(c["lens_seed"]).integers(c["lo"], c["hi"] + 1, size=c["seqs"]).astype(np.float64)
    lens = np.floor(raw * c["total"] / raw.sum()).astype(np.int64)
    lens[: c["total"] - lens.sum()] += 1
    return [int(x) for x in lens]


def _ragged(c, top):
    """One length per sequence of a batch, uniform in [lo, top]; lo 0: every sequence at the top."""
    if c["lo"] == 0:
        return [top] * c["b"]
    return [int(x) for x in np.random.default_rng(c["lens_seed"]).integers(min(c["lo"], top), top + 1, size=c["b"])]


def _pairs(c):
    """The (query, key) pairs of one head that the mask lets through."""
    if c["kind"] == "padded":
        t, lens = c["t"], _ragged(c, c["t"])
        return sum(n * (n + 1) // 2 + (t - n) * n if c["causal"] else t * n for n in lens)
    if c["kind"] == "prefill":
        return c["b"] * (c["tq"] * c["past"] + c["tq"] * (c["tq"] + 1) // 2)
    total, w = 0, c["window"]
    for n in _lengths(c):
        total += n * (n + 1) // 2 if w < 0 or n <= w + 1 else (w + 1) * (w + 2) // 2 + (n - w - 1) * (w + 1)
    return total


def work(case):
    c, e = case, BYTES[case["dtype"]]
    kind = c["kind"]
    if kind in ("packed", "padded"):
        tokens = c["total"] if kind == "packed" else c["b"] * c["t"]
        q, kv, stat = tokens * c["hq"] * c["d"] * e, tokens * c["hkv"] * c["d"] * e, tokens * c["hq"] * 4
        # In: q, k, v, dO.  Out: o, lse, dq, dk, dv.  Two products forward, five backward.
        return {"bytes": 4 * q + 4 * kv + stat, "flops": 14 * c["d"] * c["hq"] * _pairs(c)}
    if kind == "prefill":
        tk = c["past"] + c["tq"]
        return {"bytes": c["b"] * c["d"] * e * 2 * (c["tq"] * c["hq"] + tk * c["hkv"]), "flops": 4 * c["d"] * c["hq"] * _pairs(c)}
    if kind in ("decode", "step"):
        lens = _ragged(c, c["s"] if kind == "decode" else c["s"] - 1)
        keys = sum(min(n, c["window"] + 1) if c.get("window", -1) >= 0 else n for n in lens)
        rows = c["b"] * c["d"] * e * (2 * c["hq"] + (4 * c["hkv"] if kind == "step" else 0))
        return {"bytes": keys * c["hkv"] * c["d"] * e * 2 + rows, "flops": 4 * c["d"] * c["hq"] * keys}
    if kind == "rope":
        return {"bytes": 2 * c["total"] * (c["hq"] + c["hkv"]) * c["d"] * e, "flops": 3 * c["total"] * (c["hq"] + c["hkv"]) * c["dim"]}
    return {"bytes": c["b"] * c["v"] * e, "flops": 4 * c["b"] * c["v"]}


# ------------------------------------------------------------------------------------------------
# What a program has in hand, and the pass
# ------------------------------------------------------------------------------------------------
def prepare(case, seed):
    c = case
    g = torch.Generator(device="cuda")
    g.manual_seed(seed)

    def randn(*shape, dtype=None):
        return torch.randn(shape, generator=g, device="cuda", dtype=dtype or DTYPES[c["dtype"]])

    kind = c["kind"]
    state = {"kind": kind}
    if kind == "packed":
        t = c["total"]
        cu = torch.tensor(np.concatenate([[0], np.cumsum(_lengths(c))]), dtype=torch.int32, device="cuda")
        options = AttentionOptions(causal=True, deterministic=c["deterministic"])
        if c["window"] >= 0:
            options = options.with_window(c["window"], 0)
        state.update(q=randn(1, t, c["hq"], c["d"]), k=randn(1, t, c["hkv"], c["d"]), v=randn(1, t, c["hkv"], c["d"]),
                     grad=randn(1, t, c["hq"], c["d"]), mask=AttentionMask.packed(cu, cu), options=options)
    elif kind == "padded":
        b, t = c["b"], c["t"]
        lens = torch.tensor(_ragged(c, t), device="cuda")
        padding = torch.arange(t, device="cuda")[None, :] >= lens[:, None]
        state.update(q=randn(b, t, c["hq"], c["d"]), k=randn(b, t, c["hkv"], c["d"]), v=randn(b, t, c["hkv"], c["d"]),
                     grad=randn(b, t, c["hq"], c["d"]), mask=AttentionMask.key_padding(padding),
                     options=AttentionOptions(causal=c["causal"], deterministic=c["deterministic"]))
    elif kind == "prefill":
        b, tk = c["b"], c["past"] + c["tq"]
        state.update(q=randn(b, c["tq"], c["hq"], c["d"]), k=randn(b, tk, c["hkv"], c["d"]), v=randn(b, tk, c["hkv"], c["d"]),
                     mask=AttentionMask.none(), options=AttentionOptions.causal_())
    elif kind == "decode":
        b, s = c["b"], c["s"]
        lens = None if c["lo"] == 0 else torch.tensor(_ragged(c, s), dtype=torch.int32, device="cuda")
        options = AttentionOptions().with_window(c["window"], 0) if c["window"] >= 0 else AttentionOptions()
        state.update(q=randn(b, c["hq"], c["d"]), k=randn(b, s, c["hkv"], c["d"]), v=randn(b, s, c["hkv"], c["d"]), lens=lens, options=options)
    elif kind == "step":
        b, s = c["b"], c["s"]
        state.update(q=randn(b, c["hq"], c["d"]), k_new=randn(b, c["hkv"], c["d"]), v_new=randn(b, c["hkv"], c["d"]), k=randn(b, s, c["hkv"], c["d"]),
                     v=randn(b, s, c["hkv"], c["d"]), lens=torch.tensor(_ragged(c, s - 1), dtype=torch.int32, device="cuda"),
                     rope=Rope(c["d"], 10000.0, s, DTYPES[c["dtype"]], device="cuda"))
    elif kind == "rope":
        lens = _lengths(c)
        state.update(q=randn(c["total"], c["hq"], c["d"]), k=randn(c["total"], c["hkv"], c["d"]),
                     cu=torch.tensor(np.concatenate([[0], np.cumsum(lens)]), dtype=torch.int32, device="cuda"),
                     rope=Rope(c["dim"], 10000.0, max(lens), DTYPES[c["dtype"]], device="cuda"))
    else:
        # Logits spread like a model's: a few tokens carry most of the mass.
        state.update(logits=(randn(c["b"], c["v"], dtype=torch.float32) * 3).to(DTYPES[c["dtype"]]),
                     options=SampleOptions(temperature=c["temperature"], top_k=c["top_k"], top_p=c["top_p"], seed=seed, offset=1))
    return state


def run(state):
    s = state
    kind = s["kind"]
    if kind in ("packed", "padded"):
        o, lse = attention_with_lse(s["q"], s["k"], s["v"], s["mask"], s["options"])
        dq, dk, dv = attention_backward(s["q"], s["k"], s["v"], o, lse, s["grad"], s["mask"], s["options"])
        return {"o": o, "lse": lse, "dq": dq, "dk": dk, "dv": dv}
    if kind == "prefill":
        return attention(s["q"], s["k"], s["v"], s["mask"], s["options"])
    if kind == "decode":
        return attention_decode(s["q"], s["k"], s["v"], s["lens"], s["options"])
    if kind == "step":
        # The new row goes to the caches at the lengths the state holds: a repeated pass writes the same row again.
        out = attention_decode_append_rope(s["rope"], s["q"], s["k_new"], s["v_new"], s["k"], s["v"], s["lens"])
        return {"out": out, "k": s["k"], "v": s["v"]}
    if kind == "rope":
        return s["rope"].apply_packed(s["q"], s["cu"], other=s["k"])
    r = sample(s["logits"], s["options"])
    return {"tokens": r.tokens, "logprob": r.logprob, "tempered": r.tempered_logprob, "sampling": r.sampling_logprob}


def tolerance(case):
    kind, dtype = case["kind"], case["dtype"]
    if kind == "rope":
        return "exact"   # each product and the sum rounded once to the dtype: one right answer
    if kind == "sample":
        # f32 sums in another order move a log-probability by a few 1e-7 of it; a draw between two scores that close may differ.
        return {"rel": 1e-5, "max": 1e-4, "differ": 0.01}
    # Four times what the path shows against the same sums in f64: f32 0.7e-6 (largest 1.0e-5); 16-bit inputs, whose P, dS and
    # results are rounded to 8 (bf16) or 11 (f16) significant bits, 2.5e-3 (largest 0.12) and 3.1e-4 (largest 0.009).
    if dtype == "f32":
        return {"rel": 3e-6, "max": 5e-5}
    return {"rel": 1e-2, "max": 0.4} if dtype == "bf16" else {"rel": 1.25e-3, "max": 0.04}
