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
