"""Lengths beyond the keys mean that all keys are valid, up to the largest 32-bit number."""
import re
import shutil
import subprocess
from pathlib import Path

import pytest
import torch

from spiraltorch_b200.ops import attention as A
from spiraltorch_b200.ops import native

SOURCE = Path(__file__).resolve().parents[1] / "csrc" / "attention" / "attn_bwd.cu"
LENGTHS = (-2 ** 31, -1, 0, 1, 127, 128, 129, 300, 301, 1024, 2 ** 31 - 128, 2 ** 31 - 127, 2 ** 31 - 1)


@pytest.mark.skipif(shutil.which("g++") is None, reason="needs g++")
def test_sums_per_query(tmp_path):
    """How many sums of dQ a query belongs to, by the kernel's own function compiled for the host, where an overflow ends it."""
    function = re.search(r"__device__ __forceinline__ int dq_buffers\(.*?\n}\n", SOURCE.read_text(), re.S).group(0)
    program = tmp_path / "sums.cpp"
    program.write_text("#include <algorithm>\n#include <cstdio>\n#include <cstdlib>\nusing std::min; using std::max;\n"
                       "#define __device__\n#define __forceinline__ inline\nconstexpr int BLK = 128;\n" + function +
                       "int main(int, char** v) {\n  const int length = (int)strtol(v[1], nullptr, 10);\n"
                       "  for (int n = 1; n <= 8; ++n) for (int c = 0; c < 2; ++c) for (int s = 0; s < 1100; s += 50)\n"
                       "    printf(\"%d \", dq_buffers(s, n, c, &length, 0));\n}\n")
    subprocess.run(["g++", "-O1", "-fsanitize=signed-integer-overflow", "-fno-sanitize-recover=all", str(program), "-o", str(tmp_path / "sums")], check=True)
    for length in LENGTHS:
        run = subprocess.run([str(tmp_path / "sums"), str(length)], capture_output=True, text=True)
        assert run.returncode == 0, run.stderr
        want = []
        for n in range(1, 9):
            for causal in (False, True):
                for s in range(0, 1100, 50):
                    live = min(n, -(-max(0, length) // 128))
                    tiles = 0 if s // 128 >= live else min(live, s // 128 + 1) if causal else live
                    want.append((tiles + 1) // 2)
        assert [int(x) for x in run.stdout.split()] == want


@pytest.mark.gpu
@pytest.mark.parametrize("seq,dim", [(300, 64), (1100, 64), (300, 128)])
def test_no_limit_is_all_keys(seq, dim):
    torch.manual_seed(0)
    q, k, v, g = (torch.randn(2, seq, 2, dim, device="cuda").bfloat16() for _ in range(4))

    def run(length):
        lengths = torch.full((2,), length, dtype=torch.int32, device="cuda")
        o, lse = A.attention_forward(q, k, v, False, lengths=lengths)
        return (o, lse, *A.attention_backward(q, k, v, o, lse, g, False, lengths=lengths))

    want = run(seq)
    assert want[2].float().norm() > 0
    for length in (seq + 1, 2 ** 31 - 127, 2 ** 31 - 1):
        for x, y in zip(run(length), want):
            assert torch.equal(x, y)
    native.raise_on_device_error()
