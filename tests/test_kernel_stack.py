"""Kernels of the coarse correction run over every sheet of a batch in every step, also where they return at
once: none may keep a copy of its launch parameters on its threads' stacks."""
import os
import re
import shutil
import subprocess

import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_coarse_kernels_need_no_stack_for_their_parameters(tmp_path):
    nvcc = shutil.which("nvcc")
    if nvcc is None:
        pytest.skip("no nvcc")
    log = subprocess.run([nvcc, "-std=c++17", "-O3", "-gencode", "arch=compute_100a,code=sm_100a", "-Xptxas", "-v", "-I", os.path.join(ROOT, "include"), "-c",
                          os.path.join(ROOT, "clothsimulator_b200", "csrc", "coarse.cu"), "-o", str(tmp_path / "coarse.o")],
                         check=True, capture_output=True, text=True)
    text = log.stdout + log.stderr
    frames = re.findall(r"Function properties for (\w+)\s+(\d+) bytes stack frame", text)
    assert len(frames) >= 6
    assert all(int(size) <= 64 for _, size in frames), frames
