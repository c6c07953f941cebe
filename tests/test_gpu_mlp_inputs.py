"""The network's host calls take arrays at any address: numpy makes arrays off
a 4-byte boundary from the middle of a buffer, and passes them on unchanged."""
import ctypes as C

import numpy as np
import pytest

from ryr_hyperactivity_gb300.surrogate import Surrogate, _fptr, init_params

pytestmark = pytest.mark.gpu


def _off(a, by):
    """A copy of `a` that starts `by` bytes past a 16-byte boundary."""
    buf = np.zeros(a.nbytes + 32, np.uint8)
    start = (-buf.ctypes.data) % 16 + by
    out = np.frombuffer(buf.data, np.float32, a.size, start).reshape(a.shape)
    out.setflags(write=True)
    out[...] = a
    assert out.ctypes.data % 16 == by
    return out


def _batch(n):
    rng = np.random.default_rng(n)
    return (rng.random((n, 4)).astype(np.float32),
            np.stack([rng.random(n), rng.random(n) * 0.5, rng.random(n) * 0.2], 1).astype(np.float32))


@pytest.mark.parametrize("by", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 300, 40001])
def test_predict_takes_arrays_at_any_address(n, by):
    x, _ = _batch(n)
    m = Surrogate(batch_max=256, seed=1)
    want = m.predict(x)
    xo, y = _off(x, by), _off(np.zeros((n, 3), np.float32), by)
    np.testing.assert_array_equal(m.predict(xo), want)
    m._ck(m.L.rh_mlp_forward(m.h, _fptr(xo), n, _fptr(y)))
    np.testing.assert_array_equal(y, want)


@pytest.mark.parametrize("by", [1, 2, 3, 4])
@pytest.mark.parametrize("n", [1, 300, 4096])
def test_gradients_and_steps_take_arrays_at_any_address(n, by):
    x, t = _batch(n)
    a, b = Surrogate(batch_max=n, seed=2), Surrogate(batch_max=n, seed=2)
    loss, g = a.gradients(x, t)
    for xo, to in ((_off(x, by), _off(t, by)), (x, _off(t, by)), (_off(x, by), t)):
        loss_o, g_o = b.gradients(xo, to)
        assert loss_o == loss
        np.testing.assert_array_equal(g_o, g)
    for m, xs, ts in ((a, x, t), (b, _off(x, by), _off(t, by))):
        l = C.c_float()
        m._ck(m.L.rh_mlp_train_step(m.h, _fptr(xs), _fptr(ts), n, 1e-3, C.byref(l)))
        m.set_params(_off(m.get_params(), by))
    np.testing.assert_array_equal(a.get_params(), b.get_params())
    assert not np.array_equal(a.get_params(), init_params(2))


@pytest.mark.parametrize("batch_max", [(1 << 26) + 1, (1 << 31) - 1])
def test_a_batch_no_memory_holds_is_refused(batch_max):
    from ryr_hyperactivity_gb300.surrogate import _lib
    h = C.c_void_p()
    assert _lib().rh_mlp_create(batch_max, 0, C.byref(h)) == -3  # RH_ERR_NOMEM
    assert not h.value
