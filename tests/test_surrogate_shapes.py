"""Arrays that hold fewer values than a call of the surrogate reads are refused
before the call (no GPU needed: the check comes first)."""
import numpy as np
import pytest

from ryr_hyperactivity_gb300.surrogate import Surrogate


def _unconnected():
    m = Surrogate.__new__(Surrogate)  # no handle, no library
    m.batch_max = 4096
    return m


@pytest.mark.parametrize("x", [np.zeros((8, 3)), np.zeros(8), np.zeros((8, 0))])
def test_short_inputs_are_refused(x):
    t = np.zeros((8, 3))
    for call in (lambda m: m.predict(x), lambda m: m.gradients(x, t),
                 lambda m: m.fit(x, t, epochs=1, batch=4)):
        with pytest.raises(ValueError, match="samples take"):
            call(_unconnected())


@pytest.mark.parametrize("t", [np.zeros((8, 2)), np.zeros(8), np.zeros((7, 3)), np.zeros(24)])
def test_short_targets_are_refused(t):
    x = np.zeros((8, 4))
    if t.shape != (24,):  # 24 values are enough for one pass, as a flat list
        with pytest.raises(ValueError, match="samples take"):
            _unconnected().gradients(x, t)
    with pytest.raises((ValueError, IndexError)):
        _unconnected().fit(x, t, epochs=1, batch=8)
