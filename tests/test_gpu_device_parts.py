"""Device functions of the lattice and cell-update kernels by themselves
(tests/cuda/device_parts.cu), at the ends of the ranges that whole runs do not
reach."""
import ctypes as C
import os
import subprocess

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.fixture(scope="module")
def parts(tmp_path_factory):
    so = str(tmp_path_factory.mktemp("parts") / "device_parts.so")
    subprocess.run(["nvcc", "-gencode", "arch=compute_103a,code=sm_103a", "-O3", "-std=c++17",
                    "-shared", "-Xcompiler", "-fPIC", "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cuda", "device_parts.cu"), "-o", so], check=True)
    return C.CDLL(so)


def _p(a):
    return a.ctypes.data_as(C.c_void_p)


@pytest.mark.parametrize("rows", [1, 14, 31, 32, 33, 64, 441, 5100])
def test_output_sums_are_32_strided_sums_joined_by_a_tree(parts, rows):
    """The statistics of an output record: row r joins partial sum r % 32, and
    the 32 partial sums are added pairwise (16 apart, then 8, 4, 2, 1), which
    keeps the error at the size of one rounding whatever the cell's size."""
    rng = np.random.default_rng(rows)
    n, first = parts.part_row_length(), parts.part_first_statistic()
    a = np.exp(rng.uniform(-3, 3, (rows, n)))
    a[:, -1] = 0.0
    a[rows // 2, -1] = 1.0 if rows % 2 else 0.0
    got = np.zeros(n - first)
    assert parts.part_output_sums(_p(a), rows, _p(got)) == n - first
    s = np.zeros((32, n - first))
    for r in range(rows):
        s[r % 32] += a[r, first:]
    for off in (16, 8, 4, 2, 1):
        s[:off] = s[:off] + s[off:2 * off]
    np.testing.assert_array_equal(got[:-1], s[0, :-1])
    assert got[-1] == float(rows % 2)
