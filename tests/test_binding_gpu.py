"""The native host side makes the very call the Python side makes: the same bits out, the same refusals, and what it leaves to
the Python side (other devices' streams, transforms, layouts to copy) still runs."""
import ctypes
import pathlib
import subprocess
import threading
import time

import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions
from dashmag_b200.rope import Rope, attention_decode_append_rope
from dashmag_b200.sample import SampleOptions, sample

pytestmark = pytest.mark.gpu


class Nothing:
    """Stands in for the binding and does nothing."""

    def __getattr__(self, name):
        return lambda *args: None


def randn(*shape, dtype=torch.bfloat16, seed=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(seed + sum(shape))
    return torch.randn(shape, generator=g, device="cuda", dtype=dtype)


def train(mask, options, dtype=torch.bfloat16, d=64, swap=False):
    q, k, v, g = (randn(1 if mask.kind == "packed" else 2, 150, h, d, dtype=dtype, seed=i) for i, h in enumerate((4, 2, 2, 4)))
    if swap:
        q, g = (x.transpose(1, 2).contiguous().transpose(1, 2) for x in (q, g))
    o, lse = A.attention_with_lse(q, k, v, mask, options)
    return (o, lse, *A.attention_backward(q, k, v, o, lse, g, mask, options))


def calls():
    cu = torch.tensor([0, 70, 150], dtype=torch.int32, device="cuda")
    pad = torch.arange(150, device="cuda")[None] >= torch.tensor([[150], [90]], device="cuda")
    causal = AttentionOptions(causal=True)
    yield "none", lambda: train(AttentionMask.none(), AttentionOptions())
    yield "packed", lambda: train(AttentionMask.packed(cu, cu), causal.with_window(40, 0))
    yield "packed i64", lambda: train(AttentionMask.packed(cu.long(), cu.long()), causal.with_scale(0.2))
    yield "padding", lambda: train(AttentionMask.key_padding(pad), AttentionOptions(), torch.float16, 128)
    yield "padding i32, strided", lambda: train(AttentionMask.key_padding(pad.int()), causal.with_deterministic(True), torch.float32, 64, True)
    q, k, v = randn(3, 8, 128), randn(3, 300, 2, 128), randn(3, 300, 2, 128, seed=1)
    nk, nv = randn(3, 2, 128), randn(3, 2, 128, seed=1)
    lens = torch.tensor([299, 0, 41], dtype=torch.int32, device="cuda")
    rope = Rope(64, 10000.0, 300, torch.bfloat16)
    yield "decode", lambda: (A.attention_decode(q, k, v, lens, AttentionOptions().with_window(100, None)),)
    yield "decode all", lambda: (A.attention_decode(q, k[:, :200], v[:, :200], None, AttentionOptions(scale=0.1)),)

    def append(f):
        kk, vv = k.clone(), v.clone()
        return f(kk, vv), kk, vv

    yield "append", lambda: append(lambda kk, vv: A.attention_decode_append(q, nk, nv, kk, vv, lens.long()))
    yield "append rope", lambda: append(lambda kk, vv: attention_decode_append_rope(rope, q, nk, nv, kk, vv, lens))
    yield "append rope at", lambda: append(lambda kk, vv: attention_decode_append_rope(rope, q, nk, nv, kk, vv, lens, positions=lens // 2))
    z = randn(5, 3001, dtype=torch.float32)
    for o in (SampleOptions.greedy(), SampleOptions(temperature=0.7, top_k=20, top_p=0.9, seed=2**64 - 1, offset=3), SampleOptions(masked=(1, 7))):
        yield f"sample {o}", lambda o=o: (lambda r: (r.tokens, r.logprob, r.tempered_logprob, r.sampling_logprob))(sample(z, o))
    yield "sample of columns", lambda: (sample(z.t().contiguous().t(), SampleOptions(seed=4)).tokens,)


class Noted:
    """The binding, and whether it made each call it was asked for."""

    def __init__(self, binding):
        self.binding, self.made = binding, []

    def __getattr__(self, name):
        def call(*args):
            done = getattr(self.binding, name)(*args)
            self.made.append(done is not None)
            return done
        return call


#: Calls the Python side makes; it is not even asked for the first.
LEFT = {"append rope at": [], "sample of columns": [False]}


def test_same_results_as_the_python_side(monkeypatch):
    noted = Noted(_lib.binding())
    monkeypatch.setattr(_lib, "_binding", noted)
    made = []
    for name, call in calls():
        noted.made.clear()
        made.append((name, [x.clone() for x in call()]))
        masked = name.startswith("sample") and "masked=(1, 7)" in name
        assert noted.made == LEFT.get(name, [False] if masked else [True] * max(len(noted.made), 1)), name
    torch.cuda.synchronize()
    monkeypatch.setattr(_lib, "_binding", Nothing())
    for (name, got), (_, call) in zip(made, calls()):
        want = call()
        assert len(got) == len(want)
        for x, y in zip(got, want):
            assert x.dtype == y.dtype and x.shape == y.shape and x.stride() == y.stride() and torch.equal(x, y), name


def test_runs_on_the_current_stream_and_in_a_graph():
    q, k, v = randn(2, 8, 128), randn(2, 500, 2, 128), randn(2, 500, 2, 128, seed=1)
    want = A.attention_decode(q, k, v)
    torch.cuda.synchronize()
    side = torch.cuda.Stream()
    with torch.cuda.stream(side):
        A.attention_decode(q, k, v)
        graph = torch.cuda.CUDAGraph()
        with torch.cuda.graph(graph, stream=side):
            out = A.attention_decode(q, k, v)
        out.zero_()
        graph.replay()
    torch.cuda.synchronize()
    assert torch.equal(out, want)


def test_refusals_of_the_library_are_raised():
    q, k = randn(1, 4, 3, 64), randn(1, 4, 2, 64)
    with pytest.raises(A.AttentionError, match="multiple of the key-value heads"):
        A.attention(q, k, k)
    with pytest.raises(A.AttentionError, match="multiple of the key-value heads"):
        A.attention_decode(q[0], randn(4, 5, 2, 64), randn(4, 5, 2, 64))


def test_a_mode_that_watches_sees_the_allocations():
    from torch.overrides import TorchFunctionMode
    from torch.utils._python_dispatch import TorchDispatchMode

    seen = []

    class Watch(TorchDispatchMode):
        def __torch_dispatch__(self, func, types, args=(), kwargs=None):
            seen.append(str(func))
            return func(*args, **(kwargs or {}))

    class WatchFunctions(TorchFunctionMode):
        def __torch_function__(self, func, types, args=(), kwargs=None):
            seen.append(func.__name__)
            return func(*args, **(kwargs or {}))

    q, k = randn(1, 4, 2, 64), randn(1, 4, 2, 64)
    for mode in (Watch, WatchFunctions):
        seen.clear()
        with mode():
            A.attention(q, k, k)
        assert any("empty" in s for s in seen), mode


def test_a_default_device_does_not_watch(monkeypatch):
    q, k = randn(1, 4, 2, 64), randn(1, 4, 2, 64)
    want = A.attention(q, k, k)
    noted = Noted(_lib.binding())
    monkeypatch.setattr(_lib, "_binding", noted)
    with torch.device("cpu"):
        got = A.attention(q, k, k)
    assert noted.made == [True] and torch.equal(got, want)


def test_what_only_an_attribute_holds_outlives_the_call():
    """A mask whose tensor is made anew each time it is asked for: the call alone holds it, and must until its kernels are launched -
    while the outputs are allocated, that is, the tensor's memory is not free."""
    pad = torch.arange(60, device="cuda")[None] >= torch.tensor([[60], [31]], device="cuda")
    size = []

    class Fresh:
        kind = "key_padding"

        @property
        def key_padding_mask(self):
            large = pad.repeat(1, 1 << 16)
            size.append(large.untyped_storage().nbytes())
            return large[:, :60]

    q, k, v = randn(2, 60, 1, 64), randn(2, 60, 1, 64, seed=1), randn(2, 60, 1, 64, seed=2)
    want = A.attention_with_lse(q, k, v, AttentionMask.key_padding(pad), AttentionOptions())
    torch.cuda.synchronize()
    torch.cuda.reset_peak_memory_stats()
    before = torch.cuda.memory_allocated()
    got = A.attention_with_lse(q, k, v, Fresh(), AttentionOptions())
    assert torch.cuda.max_memory_allocated() - before >= size[0] + sum(x.untyped_storage().nbytes() for x in got)
    assert len(size) == 1 and all(torch.equal(x, y) for x, y in zip(got, want))


WAITING_ALLOCATOR = r"""
#include <cuda_runtime_api.h>
#include <sys/types.h>
#include <unistd.h>
extern "C" {
volatile int waiting = 0, go = 0, late = 0;
void *take(ssize_t size, int, cudaStream_t) {
    waiting = 1;
    for (int i = 0; i < 3000 && !go; ++i) usleep(1000);
    if (!go) late = 1;
    void *p = nullptr;
    return cudaMalloc(&p, size) == cudaSuccess ? p : nullptr;
}
void give(void *p, ssize_t, int, cudaStream_t) { cudaFree(p); }
}
"""


def test_other_threads_run_while_the_outputs_are_allocated(tmp_path):
    """An allocator that waits (three seconds at most) for another Python thread to let it go on."""
    source, path = tmp_path / "waiting.cpp", tmp_path / "waiting.so"
    source.write_text(WAITING_ALLOCATOR)
    cuda = pathlib.Path("/usr/local/cuda")
    subprocess.run(["g++", "-shared", "-fPIC", f"-I{cuda}/include", str(source), "-o", str(path), f"-L{cuda}/lib64", "-lcudart"], check=True)
    flags = ctypes.CDLL(str(path))
    waiting, go, late = (ctypes.c_int.in_dll(flags, n) for n in ("waiting", "go", "late"))
    q, k = randn(2, 8, 128), randn(2, 500, 2, 128)
    want = A.attention_decode(q, k, k)

    def let_go():
        for _ in range(5000):
            if waiting.value:
                break
            time.sleep(0.001)
        go.value = 1

    pool = torch.cuda.MemPool(torch.cuda.memory.CUDAPluggableAllocator(str(path), "take", "give").allocator())
    other = threading.Thread(target=let_go)
    other.start()
    with torch.cuda.use_mem_pool(pool):
        got = A.attention_decode(q, k, k)
    other.join()
    assert waiting.value and not late.value
    assert torch.equal(got, want)
    torch.cuda.synchronize()


def test_an_allocation_that_fails_is_raised():
    q = torch.empty(1, 1, 1, 64, dtype=torch.bfloat16, device="cuda").expand(1, 1 << 20, 2048, 64)   # 256 GB of output
    with pytest.raises(torch.OutOfMemoryError):
        A.attention(q, q, q)
    small = randn(1, 4, 2, 64)
    assert torch.isfinite(A.attention(small, small, small)).all()


def test_two_threads_on_two_streams():
    """Each thread's calls are its own: parameters, outputs and scratch, on its own stream."""
    def work(seed, out):
        with torch.cuda.stream(torch.cuda.Stream()):
            q, k = randn(3, 8, 128, seed=seed), randn(3, 900, 2, 128, seed=seed)
            tq, tk = randn(1, 200, 4, 64, seed=seed), randn(1, 200, 2, 64, seed=seed)
            cu = torch.tensor([0, 90 + seed, 200], dtype=torch.int32, device="cuda")
            mask, options = AttentionMask.packed(cu, cu), AttentionOptions(causal=True)
            for _ in range(60):
                o, lse = A.attention_with_lse(tq, tk, tk, mask, options)
                out.append((A.attention_decode(q, k, k), o, lse, *A.attention_backward(tq, tk, tk, o, lse, tq, mask, options)))
            torch.cuda.current_stream().synchronize()

    alone = [[], []]
    for seed in (0, 1):
        work(seed, alone[seed])
    both = [[], []]
    threads = [threading.Thread(target=work, args=(seed, both[seed])) for seed in (0, 1)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    for seed in (0, 1):
        assert len(both[seed]) == 60
        for made in both[seed]:
            assert all(torch.equal(x, y) for x, y in zip(made, alone[seed][0]))
