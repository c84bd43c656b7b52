"""Which kernel the per-head products of a few tokens go to (CPU): the lines that were measured."""
import os
import subprocess
import sys

import pytest

from llmi_b200.ops import kernels


@pytest.mark.parametrize("batch,N,K,alone,with_rotation", [(16, 512, 128, 3, 7), (16, 128, 512, 8, 8), (32, 512, 128, 2, 5), (128, 512, 128, 2, 3),
                                                           (128, 128, 512, 2, 3), (8, 256, 64, 3, 8), (3, 64, 64, 3, 8), (32, 128, 1024, 6, 8)])
def test_lines(batch, N, K, alone, with_rotation):
    """The most tokens that go to the kernel that is the latency of its loads; one more goes to the tensor cores, as do nine of anything."""
    for most, saved in ((alone, 0.0), (with_rotation, kernels.HEADS_LAUNCH_US)):
        takes = [kernels.heads_token_faster(n, batch, N, K, saved) for n in range(1, 12)]
        assert takes == [n <= most for n in range(1, 12)]


@pytest.mark.parametrize("value,most", [(None, 8), ("1", 0), ("5", 0)])
def test_variable_sends_them_to_the_tensor_cores(value, most):
    """LLMI_HEADS_MMA_MIN names the tokens from which on the tensor cores run: no third kernel then."""
    env = {k: v for k, v in os.environ.items() if k != "LLMI_HEADS_MMA_MIN"}
    if value is not None:
        env["LLMI_HEADS_MMA_MIN"] = value
    code = ("from llmi_b200.ops import kernels as k\n"
            "print(k.HEADS_MMA_MIN_TOKENS, sum(k.heads_token_faster(n, 16, 128, 512) for n in range(1, 12)))")
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    out = subprocess.run([sys.executable, "-c", code], env=env, cwd=root, capture_output=True, text=True, check=True).stdout.split()
    assert out == [value or "1", str(most)]
