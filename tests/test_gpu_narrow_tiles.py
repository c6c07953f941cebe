"""The narrow tiles the library uses for small lattices by itself (32 CRUs by
five warps or one), and the staging it chooses for large ones, give the state
and records of the default launch shape, in both precisions and with the build
options' kernel variant."""
import numpy as np
import pytest

from ryr_hyperactivity_gb300.abi import cell_params
from ryr_hyperactivity_gb300.sim import Simulator

pytestmark = pytest.mark.gpu


def _run(cells, precision, **opts):
    with Simulator(cells, precision=precision, **opts) as sim:
        sim.run_steps(230)  # two whole windows and a partial one
        return ([sim.get_state(c).snapshot() for c in range(len(cells))],
                [sim.drain_wholecell(c) for c in range(len(cells))],
                [sim.drain_linescan(c) for c in range(len(cells))])


@pytest.mark.parametrize("precision", ["fp64", "mixed"])
@pytest.mark.parametrize("extents,options", [
    ([(3, 3, 3)], [{}]),                          # one CRU
    ([(10, 6, 3)], [{}]),                         # exactly one tile
    ([(35, 9, 4)], [{}]),                         # a row longer than a tile, one CRU over
    ([(60, 24, 17)], [{}]),                       # too many tiles for five warps each
    ([(100, 60, 30), (99, 61, 30)], [{}, {}]),    # three waves of default tiles: tensor copies
    ([(12, 7, 5), (41, 8, 6), (5, 4, 13)], [{}, dict(perm=1), dict(slowncx=1, ncx_form="oldncx")]),
])
def test_narrow_tiles_equal_default_tiles(precision, extents, options):
    cells = [cell_params(nx=x, ny=y, nz=z, lqt=0, seed=9, cell_id=i, ku2=2.0, **o)
             for i, ((x, y, z), o) in enumerate(zip(extents, options))]
    a = _run(cells, precision)                    # the library's choice
    b = _run(cells, precision, block_size=128)
    for sa, sb in zip(a[0], b[0]):
        for f in sa:
            np.testing.assert_array_equal(sa[f], sb[f], err_msg=f)
    for ra, rb in zip(a[1], b[1]):
        # FP64 statistics are summed warp by warp over the same 32-CRU ranges
        np.testing.assert_array_equal(ra, rb)
    for ra, rb in zip(a[2], b[2]):
        np.testing.assert_array_equal(ra, rb)
