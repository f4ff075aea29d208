"""The correctly rounded quotients and roots of nmhd_b200/csrc/rounded.cuh on
the GPU, on every case in which they could differ from the IEEE operations.

Tolerance: none may differ."""
import os
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.mark.gpu
def test_quotients_and_roots_are_correctly_rounded(tmp_path):
    exe = tmp_path / "rounded_check"
    subprocess.run(["/usr/local/cuda/bin/nvcc", "-gencode", "arch=compute_100a,code=sm_100a", "-std=c++17", "-O3",
                    "-fmad=false", "-o", str(exe), os.path.join(HERE, "native", "rounded_check.cu")], check=True)
    out = subprocess.run([str(exe)], capture_output=True, text=True, check=True).stdout
    counts = [[int(v) for v in line.split()] for line in out.splitlines()]
    assert [c for c, _ in counts[:2]] == [3 << 24, 3 << 23] and counts[2][0] > 1e8, out
    assert [bad for _, bad in counts] == [0, 0, 0], out
