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


@pytest.mark.parametrize("dt", [0.025, 0.1, 2.0])
def test_estimated_draws_are_the_fp64_ones_or_none(parts, dt):
    """Wherever the FP32 estimates decide a CRU's RyR transitions, the counts
    and the draws taken are those of the FP64 comparisons: over rates from
    nothing to the cap, and inputs that are zero, tiny, huge, infinite or NaN,
    alone and together (0/0 among the rates included)."""
    rng = np.random.default_rng(int(1000 * dt))
    n = 400_000
    scale = [np.exp(rng.uniform(np.log(a), np.log(b), n)) for a, b in
             [(1e-2, 300.0), (20.0, 1500.0), (1e-3, 1.0), (1e-1, 100.0), (1e-3, 10.0), (1e-3, 10.0)]]
    odd = np.array([0.0, 5e-324, 1e-310, 1e-60, 1e-39, 1e39, 1e300, np.inf, np.nan, -1.0, -0.0])
    v = np.stack(scale)
    hit = rng.random(v.shape) < 0.15
    hit[:, : n // 2] = False  # half of the CRUs are ordinary
    v[hit] = rng.choice(odd, hit.sum())
    both = slice(n - n // 8, n)  # closed RyRs on an empty dyad: ku / cp is 0/0
    v[0, both], v[3, both] = 0.0, 0.0
    counts = rng.multinomial(100, [0.02, 0.5, 0.03, 0.45], n).astype(np.int32)
    few = slice(n // 4, n)
    counts[few] = rng.integers(0, 2, (n - n // 4, 4))
    est = np.zeros(n, np.uint32)
    e, x = np.zeros((n, 2), np.uint32), np.zeros((n, 2), np.uint32)
    v, counts = np.ascontiguousarray(v), np.ascontiguousarray(counts)
    assert parts.part_draws(n, _p(v), C.c_double(dt), _p(counts), _p(est), _p(e), _p(x)) == 0
    assert np.count_nonzero(est == 0xffffffff) == 0
    bad = (est != 0) & (e != x).any(axis=1)
    assert not bad.any(), (int(bad.sum()), v[:, bad][:, :5], counts[bad][:5])
    if dt == 0.025:  # the model's step, no Gaussian draws: the estimates do decide
        assert np.count_nonzero(est[: n // 2]) > 0.9 * (n // 2)


@pytest.mark.parametrize("lo,hi", [(1e-300, 1e-100), (1e-3, 1e3), (1e290, 1.7e308)])
def test_stencil_sums_equal_the_fp64_differences(parts, lo, hi):
    """The integer sums against the same sums of FP64 differences: within the
    rounding of both (8 differences of at most the largest value, a half unit
    in the last place each), and overflowing where those overflow."""
    rng = np.random.default_rng(2)
    n, kt, kl = 100_000, 0.125, 0.03125
    # neighbours within three decades of each other, at levels from lo to hi
    level = np.exp(rng.uniform(np.log(lo), np.log(hi), (n, 1)))
    v = np.minimum(level * np.exp(rng.uniform(-7, 0, (n, 12))), 1.79e308)
    v[::7] = np.where(rng.random((len(v[::7]), 12)) < 0.5, v[::7], level[::7])
    v = np.ascontiguousarray(v)
    got = np.zeros((n, 2))
    assert parts.part_stencil(n, _p(v), C.c_double(kt), C.c_double(kl), _p(got)) == 0
    with np.errstate(over="ignore", invalid="ignore"):
        for h in (0, 1):
            c, z, far = v[:, h], v[:, 1 - h], v[:, 2 + h]
            t = (((z - c) + (far - c)) + (v[:, 4 + h] - c)) + (v[:, 6 + h] - c)
            want = t * kt + ((v[:, 8 + h] - c) + (v[:, 10 + h] - c)) * kl
            inf = ~np.isfinite(want)
            np.testing.assert_array_equal(got[inf, h], want[inf])
            big = v.max(axis=1)
            assert np.all(np.abs(got[~inf, h] - want[~inf]) <= 8 * 2.0**-53 * big[~inf])
