"""The backward's kernels run side by side (dq beside dkdv's last waves, delta beside the plan): what follows in the
stream sees every gradient whole, eagerly and from a captured graph, with few and with many more blocks than
multiprocessors in either kernel."""
import numpy as np
import pytest
import torch

from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionMask, AttentionOptions

pytestmark = pytest.mark.gpu


# kv heads, group, tokens, d: dkdv short of the GPU (8 units of long sweeps), of its size, several waves; one key block (no plan)
@pytest.mark.parametrize("hkv,group,t,d", [(1, 8, 1000, 128), (4, 2, 4700, 128), (2, 4, 3000, 64), (2, 4, 2000, 256), (2, 2, 100, 128)])
def test_the_gradients_are_whole_when_the_call_is_over(hkv, group, t, d):
    g = torch.Generator(device="cuda").manual_seed(t)
    q, go = (torch.randn(1, t, hkv * group, d, device="cuda", generator=g).bfloat16() for _ in range(2))
    k, v = (torch.randn(1, t, hkv, d, device="cuda", generator=g).bfloat16() for _ in range(2))
    mask, options = AttentionMask.none(), AttentionOptions.causal_()
    o, lse = A.attention_with_lse(q, k, v, mask, options)
    want = A.attention_backward(q, k, v, o, lse, go, mask, options)
    torch.cuda.synchronize()
    for _ in range(5):   # read by the next kernel in the stream, without a synchronisation
        got = [x.clone() for x in A.attention_backward(q, k, v, o, lse, go, mask, options)]
        assert all(torch.equal(a, b) for a, b in zip(got, want))
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph):
        grads = A.attention_backward(q, k, v, o, lse, go, mask, options)
        copies = [x.clone() for x in grads]
    for _ in range(3):
        for x in (*grads, *copies):
            x.fill_(float("nan"))
        graph.replay()
        torch.cuda.synchronize()
        assert all(torch.equal(a, b) for a, b in zip(copies, want))
        assert all(torch.equal(a, b) for a, b in zip(grads, want))
