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


@pytest.mark.parametrize("lo,hi", [(1e-3, 3e3), (1e-30, 1e30), (1e30, 1e160), (1e-320, 1e308)])
def test_uptake_and_leak_equal_their_quotients(parts, lo, hi):
    """SERCA uptake and leak, which share one reciprocal, against a division
    each: within their roundings (at most six a side, a half unit in the last
    place each), and infinite or NaN where those are."""
    rng = np.random.default_rng(4)
    m, sviup = 200_000, 0.91
    v = np.exp(rng.uniform(np.log(lo), np.log(hi), (m, 4)))
    if hi > 1e300:
        odd = np.array([0.0, np.inf, np.nan, 5e-324, 1.79e308])
        hit = rng.random((m, 2)) < 0.1
        v[:, :2][hit] = rng.choice(odd, hit.sum())
    with np.errstate(all="ignore"):
        v[:, 2], v[:, 3] = (v[:, 0] / 0.123) ** 1.787, (v[:, 1] / 1700.0) ** 1.787
        c, n, pa, pb = v.T
        up = sviup * ((0.3 * (pa - pb)) / (1.0 + pa + pb))
        lk = ((0.00001035 * (n - c)) * (n * n)) / (n * n + 500.0 * 500.0)
    got = np.zeros((m, 2))
    v = np.ascontiguousarray(v)
    assert parts.part_serca_leak(m, _p(v), C.c_double(sviup), _p(got)) == 0
    for g, want in ((got[:, 0], up), (got[:, 1], lk)):
        np.testing.assert_array_equal(np.isnan(g), np.isnan(want))
        ok = np.isfinite(want)
        np.testing.assert_array_equal(g[np.isinf(want)], want[np.isinf(want)])
        # below 1e-290 products of the numerators lose bits to underflow
        tol = np.where(np.abs(want[ok]) > 1e-290, 12 * 2.0**-53 * np.abs(want[ok]), 1e-300)
        assert np.all(np.abs(g[ok] - want[ok]) <= tol)


@pytest.mark.parametrize("kind", ["model", "normal", "small_numerator", "any_bits", "special"])
def test_refined_division_equals_the_rounded_quotient(parts, kind):
    """div_refined against the correctly rounded quotient, bit for bit: the
    model's magnitudes, all normal numbers, numerators whose residual is
    subnormal, arbitrary bit patterns, and every pair of special values."""
    rng = np.random.default_rng(6)
    n = 4_000_000
    special = np.array([0.0, 5e-324, 2.2e-308, 2.3e-308, 1e-290, 1e-20, 1.0, 3.0, 1e20, 1e290,
                        1.7e308, np.inf, np.nan])
    if kind == "special":
        special = np.concatenate([special, -special])
        a, b = (x.ravel() for x in np.meshgrid(special, special))
    elif kind == "any_bits":
        a, b = (rng.integers(0, 1 << 64, n, dtype=np.uint64).view(np.float64) for _ in range(2))
    else:
        def draw(lo, hi):
            return np.ldexp(1.0 + rng.random(n), rng.integers(lo, hi, n)) * rng.choice([-1.0, 1.0], n)
        e = {"model": (-40, 40), "normal": (-1022, 1024), "small_numerator": (-1022, -900)}[kind]
        a, b = draw(*e), draw(*((-60, 60) if kind == "small_numerator" else e))
    a, b, q = (np.ascontiguousarray(x, np.float64) for x in (a, b, np.zeros(len(a))))
    assert parts.part_divide(len(a), _p(a), _p(b), _p(q)) == 0
    with np.errstate(all="ignore"):
        want = a / b
    bad = (q.view(np.uint64) != want.view(np.uint64)) & ~(np.isnan(q) & np.isnan(want))
    assert not bad.any(), (int(bad.sum()), a[bad][:5], b[bad][:5], q[bad][:5], want[bad][:5])


def test_a_wait_that_nothing_ends_gives_up_within_seconds(parts):
    import time
    parts.part_output_sums(_p(np.zeros((1, parts.part_row_length()))), 1, _p(np.zeros(64)))
    t = time.perf_counter()
    assert parts.part_wait_runs_out() == 1
    assert time.perf_counter() - t < 3.0
