"""A cell updated by four warps (a small simulation) and by one (the same
cell in a batch that fills the GPU) gives the same bits: state, records and
beat statistics, for every protocol and build option."""
import numpy as np
import pytest

from ryr_hyperactivity_gb300.abi import cell_params
from ryr_hyperactivity_gb300.sim import Simulator

pytestmark = pytest.mark.gpu

OPTIONS = [dict(), dict(lqt=1), dict(iso2=0), dict(protocol="vclamp", clamp_mv=-20.0),
           dict(protocol="brownvclamp"), dict(protocol="linearapclamp"), dict(perm=1),
           dict(iso=1, pcl_ms=40.0), dict(slowncx=1), dict(ncx_form="oldncx"),
           dict(ncx_form="ncx_noallo"), dict(randomlcc=1)]


def _run(cells, precision, keep):
    # one cell group: every cell runs the lattice kernel's option variant in
    # both batches (its FP64 rounding may differ from the plain variant's)
    with Simulator(cells, precision=precision, record_cadist=1, cell_groups=1) as sim:
        for c in range(keep):  # through a stimulus: threshold branches of the gates
            m = sim.get_membrane(c)
            m.v = -45.0 + 7.0 * c
            sim.set_membrane(c, m)
        sim.run_steps(230)
        return [(sim.get_state(c).snapshot(), sim.get_membrane(c).as_dict(), sim.drain_wholecell(c),
                 sim.drain_cadist(c), sim.drain_stats(c), sim.status(c)) for c in range(keep)]


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
def test_four_warp_cell_update_equals_one_warp(precision):
    small = [cell_params(**dict(dict(nx=12 + i, ny=7, nz=5, lqt=0, seed=5, cell_id=i, pcl_ms=300.0), **o))
             for i, o in enumerate(OPTIONS)]
    big = cell_params(nx=100, ny=40, nz=18, seed=5, cell_id=99)  # 1,862 warps
    a = _run(small, precision, len(small))
    b = _run(small + [big], precision, len(small))
    for (sa, ma, wa, ca, ta, ua), (sb, mb, wb, cb, tb, ub) in zip(a, b):
        # (a NaN is the model's own: the IKr rate is 0/0 at V = -10 mV)
        np.testing.assert_equal(ma, mb)
        assert ta == tb and ua == ub
        np.testing.assert_array_equal(wa, wb)
        np.testing.assert_array_equal(ca, cb)
        for f in sa:
            np.testing.assert_array_equal(sa[f], sb[f], err_msg=f)


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("tile", [0, 128])
def test_a_cell_does_not_depend_on_its_group(precision, tile):
    """A plain cell beside a permeabilised one runs the lattice kernel's plain
    variant in a group of its own and the option variant in a shared one."""
    p = cell_params(nx=35, ny=17, nz=9, lqt=0, seed=5, ku2=3.0)
    q = cell_params(nx=15, ny=7, nz=5, seed=5, cell_id=4, perm=1)
    out = []
    for groups in (1, 2):
        with Simulator([p, q], precision=precision, cell_groups=groups, block_size=tile) as sim:
            sim.run_steps(430)
            out.append((sim.drain_wholecell(0), sim.get_state(0).snapshot()))
    np.testing.assert_array_equal(out[0][0], out[1][0])
    for f in out[0][1]:
        np.testing.assert_array_equal(out[0][1][f], out[1][1][f], err_msg=f)
