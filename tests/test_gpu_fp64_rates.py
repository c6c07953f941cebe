"""The FP64 lattice's SERCA and leak rates against numpy over the whole input
range: table intervals and their edges, powers of two, and the values that
leave the table (zero, below 2^-32, above 2^32)."""
import numpy as np
import pytest

from ryr_hyperactivity_gb300.abi import cell_params
from ryr_hyperactivity_gb300.sim import Simulator

pytestmark = pytest.mark.gpu

VUP, KI, KNSR, HH = 0.3, 0.123, 1700.0, 1.787  # subroutine_cuda.c:128-146
GLEAK, KJSR = 0.00001035, 500.0


def _inputs(kind, n, rng):
    if kind == "physiological":
        return np.exp(rng.uniform(np.log(1e-3), np.log(1e3), n)), rng.uniform(1.0, 2500.0, n)
    if kind == "interval_edges":  # m at k/128 and one step below, exponents over the table
        m = 1.0 + rng.integers(0, 128, n) / 128.0
        x = np.ldexp(m, rng.integers(-12, 12, n))
        return np.where(np.arange(n) % 2, np.nextafter(x, 0), x), np.ldexp(m, rng.integers(0, 11, n))
    x = np.ldexp(1.0, rng.integers(-60, 60, n))  # across both ends of the table
    return np.where(np.arange(n) % 5 == 0, 0.0, x), np.ldexp(1.0 + rng.random(n), rng.integers(-40, 40, n))


@pytest.mark.parametrize("kind", ["physiological", "interval_edges", "outside_the_table"])
def test_fp64_serca_and_leak_match_numpy(kind):
    p = cell_params(nx=11, ny=7, nz=5, iso2=1, lqt=0)
    with Simulator(p, precision="fp64") as sim:
        st = sim.get_state(0)
        rng = np.random.default_rng(3)
        ci, cn = _inputs(kind, 8 * st.n, rng)
        st["ci"][...] = ci
        st["cnsr"][...] = cn
        sim.set_state(0, st)
        sim.lattice_step()
        got = sim.get_state(0)
    scale = 1.75 * 1.75 * VUP
    pa, pb = (ci / KI) ** HH, (cn / KNSR) ** HH
    up = scale * (pa - pb) / (1 + pa + pb)
    # a few units in the last place of each power, of their difference's terms
    # (not of the difference, which cancels) and of the quotient
    assert np.all(np.abs(got["xiup"] - up) <= 1e-14 * scale * (pa + pb) / (1 + pa + pb))
    lk = GLEAK * (cn - ci) * cn * cn / (cn * cn + KJSR * KJSR)
    assert np.all(np.abs(got["xileak"] - lk) <= 1e-14 * np.abs(lk))


@pytest.mark.parametrize("seed,v,params", [
    (0, -80.0, dict()), (1, 0.5, dict(ku2=3.0)), (2, 30.0, dict(kb=0.0)), (3, -40.0, dict(ku=0.5, ku2=3.0)),
])
def test_fp64_channel_draws_are_those_of_the_fp64_comparisons(seed, v, params):
    """The FP64 lattice decides most draws from FP32 estimates and repeats the
    close ones in FP64: over half a million draws at rates from zero to the
    Gaussian branch, every count equals the oracle's."""
    from oracle import oracle as O
    from tests.gpu_helpers import count_mismatch

    p = cell_params(nx=100, ny=30, nz=20, lqt=0, seed=seed, **params)
    o = O.Oracle(p)
    st, m = o.get_state(), o.get_membrane()
    rng = np.random.default_rng(seed)
    st["cp"][...] = np.exp(rng.uniform(np.log(1e-2), np.log(300.0), st.n))
    st["cp"][::97] = 0.0
    st["cjsr"][...] = rng.uniform(20.0, 1500.0, st.n)
    occ = rng.multinomial(100, [0.02, 0.5, 0.03, 0.45], st.n)
    for i, f in enumerate(["nou", "ncu", "nob", "ncb"]):
        st[f][...] = occ[:, i]
    st["lcc"].reshape(8, -1)[:4] = rng.integers(0, 16, (4, st.n))
    m.v = v
    o.set_state(st)
    o.set_membrane(m)
    o.lattice_step()
    with Simulator(p, precision="fp64") as sim:
        sim.set_state(0, st)
        sim.set_membrane(0, m)
        sim.lattice_step()
        got = sim.get_state(0)
    bad = count_mismatch(got, o.get_state())
    assert not bad.any(), np.flatnonzero(bad)[:10]


@pytest.mark.parametrize("kind", ["smooth", "wide", "with_zeros"])
def test_fp64_stencil_sums_match_oracle(kind):
    """One lattice step from sub-voxel fields that are nearly constant (the
    sums cancel), spread over five decades (mantissas shifted out) or zero in
    places (the FP64 form): ci and cnsr within a few units in the last place of
    the largest value around."""
    from oracle import oracle as O

    p = cell_params(nx=11, ny=9, nz=6, lqt=0, tapsi=1)  # no SERCA
    o = O.Oracle(p)
    st, m = o.get_state(), o.get_membrane()
    rng = np.random.default_rng(8)
    for f, level in (("ci", 0.1), ("cnsr", 500.0)):
        n = st[f].size
        if kind == "smooth":
            st[f][...] = level * (1 + 1e-6 * rng.standard_normal(n))
        else:
            st[f][...] = level * np.exp(rng.uniform(-6, 6, n))
        if kind == "with_zeros":
            st[f][rng.random(n) < 0.2] = 0.0
    o.set_state(st)
    o.set_membrane(m)
    o.lattice_step()
    ref = o.get_state()
    with Simulator(p, precision="fp64") as sim:
        sim.set_state(0, st)
        sim.set_membrane(0, m)
        sim.lattice_step()
        got = sim.get_state(0)
    for f in ("ci", "cnsr"):
        assert np.max(np.abs(got[f] - ref[f])) <= 1e-14 * max(st[f].max(), ref[f].max()), f
