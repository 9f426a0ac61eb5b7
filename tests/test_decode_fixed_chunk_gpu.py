"""DASH_ATTN_DECODE_CHUNK: a number fixes the chunk, and the call goes in chunks; 0 leaves the call to the planner, as if it were not set."""
import os
import subprocess
import sys

import pytest

pytestmark = pytest.mark.gpu

CALL = """
import torch
from dashmag_b200 import _lib, attention as A
q, k = torch.randn(1, 8, 128, device="cuda").bfloat16(), torch.randn(1, 2000, 2, 128, device="cuda").bfloat16()
before = _lib.probe("kernel_launches")
A.attention_decode(q, k, k)
print("launches", _lib.probe("kernel_launches") - before)
"""


@pytest.mark.parametrize("value,launches", [(None, 1), ("0", 1), ("256", 2)])
def test_launches(value, launches):
    env = {k: v for k, v in os.environ.items() if k != "DASH_ATTN_DECODE_CHUNK"} | ({} if value is None else {"DASH_ATTN_DECODE_CHUNK": value})
    run = subprocess.run([sys.executable, "-c", CALL], env=env, cwd=os.path.dirname(os.path.dirname(os.path.abspath(__file__))), capture_output=True, text=True, timeout=300)
    assert run.returncode == 0, run.stderr
    assert f"launches {launches}\n" in run.stdout
