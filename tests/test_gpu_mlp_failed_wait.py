"""A training step whose tensor-core wait gave up (reported by hand,
tests/cuda/mlp_failed_wait.cu) leaves the model as it was."""
import os
import subprocess

import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


def test_a_failed_step_leaves_the_model_unchanged(tmp_path):
    exe = str(tmp_path / "mlp_failed_wait")
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17", "-I",
                    os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cuda", "mlp_failed_wait.cu"), "-o", exe], check=True)
    out = subprocess.run([exe], check=True, capture_output=True, text=True).stdout
    lines = out.splitlines()
    assert lines[0] == "timeout 1 kept 1 same 1 moved 1"
    assert lines[1].startswith("wait gave up 1 within 3 s 1")
