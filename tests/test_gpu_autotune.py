"""The launch-shape autotuners on small simulations: what a trial times is what
a window then takes, and the library's own choice of tiles is among the
candidates, can be kept and can be asked for."""
import time

import pytest

from ryr_hyperactivity_gb300.abi import cell_params
from ryr_hyperactivity_gb300.sim import Simulator

pytestmark = pytest.mark.gpu


def _population(n):
    return [cell_params(nx=20, ny=10, nz=5, lqt=0, seed=3, cell_id=i, ku2=2.0) for i in range(n)]


def _window_ms(sim):
    sim.run_steps(200)
    best = 1e9
    for _ in range(4):
        t = time.perf_counter()
        sim.run_steps(400)
        sim.get_membrane(0)  # waits
        best = min(best, time.perf_counter() - t)
    return best / 4 * 1e3


def test_trials_take_what_windows_take():
    """50 small cells in 8 groups: 16 launches a step, which the host issues
    more slowly one by one than a window's graph runs them."""
    with Simulator(_population(50), precision="mixed", record_linescan=0) as sim:
        sim.run_steps(100)
        _, tried = sim.autotune_shapes(50)
        shape, per = next((t, ms) for t, ms in tried
                          if (t["persistent"], t["tile_crus"], t["cell_groups"],
                              t["bulk_staging"]) == (0, 128, 8, 0))
        sim.set_launch_shape(0, 128, 0, 8, 0)
        window = _window_ms(sim)
        assert 100 * per < 1.4 * window, (100 * per, window)


def _state(sim):
    return sim.get_membrane(0).as_dict(), sim.drain_wholecell(0)


def test_the_library_s_own_choice_is_a_candidate_and_a_shape():
    """One 432-unit FP64 cell runs 32-CRU tiles by itself, at half the time of
    any launch shape: tuning keeps that, also from the cache, and a shape that
    was read can be set again."""
    p = cell_params(nx=20, ny=10, nz=5, lqt=0, seed=4)
    with Simulator(p, precision="fp64", record_linescan=0) as a, \
            Simulator(p, precision="fp64", record_linescan=0) as b, \
            Simulator(p, precision="fp64", record_linescan=0, block_size=128) as c:
        assert a.tile_size() == 32 and c.tile_size() == 128
        own = a.launch_shape()
        assert own["tile_crus"] == 0 and own["bulk_staging"] == 0
        a.set_launch_shape(**own)
        assert a.tile_size() == 32
        a.run_steps(120)
        best, tried = a.autotune_shapes(40)
        assert sum(t["tile_crus"] == 0 for t, _ in tried) == 1
        assert best["tile_crus"] == 0 and a.tile_size() == 32 and a.launch_shape() == own
        best2, tried2 = b.autotune_shapes(40)
        assert tried2 == [] and best2 == best and b.tile_size() == 32
        b.run_steps(120)
        # a shape asked for is run, and the choice can be given back
        b.set_launch_shape(0, 64)
        assert b.tile_size() == 64 and b.launch_shape()["tile_crus"] == 64
        b.run_steps(60)
        b.set_launch_shape(**own)
        assert b.tile_size() == 32
        tile, ms = c.autotune(40)
        assert tile in (64, 128, 256) and all(m > 0 for m in ms) and c.tile_size() == 32
        a.run_steps(180)
        b.run_steps(120)
        c.run_steps(300)
        ref = _state(a)
        for sim in (b, c):
            m, w = _state(sim)
            assert m == ref[0]
            assert (w == ref[1]).all()


@pytest.mark.parametrize("shape", [(1, 0, 0, 0, 0), (0, 0, 0, 0, 1), (0, 0, 0, 0, 2), (0, 32, 0, 0, 0)])
def test_shapes_that_are_none_are_refused(shape):
    from ryr_hyperactivity_gb300.native import NativeError
    with Simulator(_population(2), precision="mixed") as sim:
        was = sim.launch_shape()
        with pytest.raises(NativeError):
            sim.set_launch_shape(*shape)
        assert sim.launch_shape() == was
