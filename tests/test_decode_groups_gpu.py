"""The decoding step in chunks: a head's bits are its own, whether one to seven others share its key-value head (heads as the products'
columns) or eight and more (heads as rows) - every head dimension, both 16-bit dtypes, ragged lengths, windows, one chunk and many,
tiles cut short, both block shapes; and so are those of a step that rotates and appends."""
import pytest
import torch

from dashmag_b200 import _lib
from dashmag_b200 import attention as A
from dashmag_b200.contract import AttentionOptions
from dashmag_b200.rope import Rope, attention_decode_append_rope

pytestmark = pytest.mark.gpu


# Caches of at most 512 keys or so few units of long sweeps that no cluster takes them: two launches.
@pytest.mark.parametrize("b,s,hkv,d,left", [
    (1, 1, 1, 128, -1), (2, 17, 2, 64, -1), (3, 300, 2, 128, -1), (5, 511, 1, 256, 100), (16, 512, 4, 64, -1), (8, 6144, 2, 256, -1), (2, 8192, 1, 128, -1),
    (1, 9000, 2, 256, 5000), (1, 20000, 1, 64, -1), (40, 512, 24, 128, -1)])
@pytest.mark.parametrize("dtype", [torch.bfloat16, torch.float16], ids=["bf16", "f16"])
def test_a_heads_bits_are_its_own(b, s, hkv, d, left, dtype):
    g = torch.Generator(device="cuda").manual_seed(b + s + d)
    q, k, v = (torch.randn(shape, generator=g, device="cuda").to(dtype) for shape in ((b, hkv, 16, d), (b, s, hkv, d), (b, s, hkv, d)))
    lengths = torch.randint(0, s + 1, (b,), generator=g, device="cuda", dtype=torch.int32)
    lengths[0] = s
    options = AttentionOptions().with_window(left, 0) if left >= 0 else AttentionOptions()
    for lens in (lengths, None):
        def heads(n):
            before = _lib.probe("kernel_launches")
            out = A.attention_decode(q[:, :, :n].reshape(b, hkv * n, d).contiguous(), k, v, lens, options)
            return out.view(torch.int16).reshape(b, hkv, n, d) if _lib.probe("kernel_launches") - before == 2 else None
        whole = heads(16)
        for n in (2, 3, 4, 7, 8, 9):
            assert torch.equal(heads(n), whole[:, :, :n]), n


@pytest.mark.parametrize("d,dim,b,s", [(64, 32, 6, 400), (128, 128, 2, 512), (256, 256, 3, 512)])
def test_a_step_that_rotates(d, dim, b, s):
    g = torch.Generator(device="cuda").manual_seed(d)
    q, kn, vn, k, v = (torch.randn(shape, generator=g, device="cuda").bfloat16() for shape in ((b, 2, 12, d), (b, 2, d), (b, 2, d), (b, s, 2, d), (b, s, 2, d)))
    rope = Rope(dim, 10000.0, s, torch.bfloat16, device="cuda")
    lengths = torch.tensor([s - 1, 16, 0, 15, 100, 63][:b], dtype=torch.int32, device="cuda")
    def heads(n):
        return attention_decode_append_rope(rope, q[:, :, :n].reshape(b, 2 * n, d).contiguous(), kn, vn, k, v, lengths).view(torch.int16).reshape(b, 2, n, d)
    whole = heads(12)
    for n in (2, 5, 8):
        assert torch.equal(heads(n), whole[:, :, :n]), n
