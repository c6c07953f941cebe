"""The network's one-kernel passes at the sizes where their tiling changes
(tiles of 128 samples, one CTA up to 256, one tile per CTA above, launches of
16,384 samples) and with inputs off a 16-byte boundary, against the CPU
oracle with the tolerances of the other network tests."""
import ctypes as C

import numpy as np
import pytest

from oracle import mlp_oracle as MO
from ryr_hyperactivity_gb300 import native
from ryr_hyperactivity_gb300.surrogate import Surrogate, init_params

pytestmark = pytest.mark.gpu


def _case(n, seed):
    rng = np.random.default_rng(seed)
    p = (init_params(seed) * rng.uniform(0.8, 1.2, 36232)).astype(np.float32)
    o = 0
    for r, k in MO.SHAPES:
        o += r * k
        p[o:o + r] = rng.uniform(-0.2, 0.2, r)
        o += r
    buf = rng.random(4 * n + 1).astype(np.float32)
    x = buf[n % 2:4 * n + n % 2].reshape(n, 4)  # odd n: 4 bytes past a 16-byte boundary
    t = np.stack([rng.random(n), rng.random(n) * 0.5, rng.random(n) * 0.2], 1).astype(np.float32)
    return p, x, t


@pytest.mark.parametrize("n", [1, 2, 127, 128, 129, 256, 257, 2049])
def test_predict_matches_oracle(n):
    p, x, _ = _case(n, n)
    m = Surrogate(batch_max=100)
    m.set_params(p)
    np.testing.assert_allclose(m.predict(x), MO.forward(p, x)[0], rtol=2e-3, atol=2e-3)
    np.testing.assert_array_equal(m.get_params()[:2048].reshape(128, 16)[:, 4:], 0)


@pytest.mark.parametrize("n", [257, 16384, 16385, 40001])
def test_a_sample_s_prediction_does_not_depend_on_its_batch(n):
    """Many tiles, several launches: bit for bit what one tile at a time gives
    (which the test above compares with the oracle; over tens of thousands of
    samples some activation lies on a BF16 rounding boundary, where the
    oracle's FP64 sums and the FP32 ones round differently)."""
    p, x, _ = _case(n, n)
    m = Surrogate(batch_max=100)
    m.set_params(p)
    one = np.concatenate([m.predict(x[i:i + 128]) for i in range(0, n, 128)])
    np.testing.assert_array_equal(m.predict(x), one)


@pytest.mark.parametrize("n", [1, 127, 128, 129, 256, 257, 511, 4096, 20000])
def test_gradients_match_oracle(n):
    p, x, t = _case(n, n)
    m = Surrogate(batch_max=n)
    m.set_params(p)
    loss, g = m.gradients(x, t)
    loss_ref, g_ref = MO.loss_and_grads(p, x, t)
    assert loss == pytest.approx(loss_ref, rel=2e-3)
    o = 0
    for r, k in MO.SHAPES:
        for size in (r * k, r):
            a, b = g[o:o + size], g_ref[o:o + size]
            assert np.max(np.abs(a - b)) <= 2e-2 * (np.max(np.abs(b)) + 1e-12), (r, k, size)
            assert np.linalg.norm(a - b) <= 1e-2 * (np.linalg.norm(b) + 1e-12)
            o += size
    # the same pass again: the sums' order is fixed
    loss2, g2 = m.gradients(x, t)
    assert loss2 == loss
    np.testing.assert_array_equal(g2, g)


@pytest.mark.parametrize("n,shift", [(1, 0), (129, 1), (4096, 0)])
def test_noalloc_equals_handle_forward(n, shift):
    torch = pytest.importorskip("torch")
    p, x, _ = _case(n, n + 7)
    m = Surrogate()
    m.set_params(p)
    f = native.load().rh_mlp_forward_noalloc
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_char_p, C.c_size_t]
    dp = torch.zeros(p.size + 4, device="cuda")[shift:shift + p.size]
    dp.copy_(torch.from_numpy(p))
    dx = torch.zeros(x.size + 4, device="cuda")[shift:shift + x.size]
    dx.copy_(torch.from_numpy(x.copy()).reshape(-1))
    dy = torch.full((n, 3), float("nan"), device="cuda")
    torch.cuda.synchronize()
    assert f(dp.data_ptr(), dx.data_ptr(), n, dy.data_ptr(), None, None, 0) == 0
    torch.cuda.synchronize()
    np.testing.assert_array_equal(dy.cpu().numpy(), m.predict(x))
