"""rh_mlp_forward_noalloc with outputs that lie in the inputs' or the
parameters' memory gives what it gives with memory of their own."""
import ctypes as C

import numpy as np
import pytest

from ryr_hyperactivity_gb300 import native
from ryr_hyperactivity_gb300.surrogate import init_params

pytestmark = pytest.mark.gpu

NPAR = 36232


def _call(p, x, n, y, stream=None):
    f = native.load().rh_mlp_forward_noalloc
    f.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_char_p, C.c_size_t]
    err = C.create_string_buffer(256)
    assert f(p, x, n, y, stream, err, 256) == 0, err.value.decode()


@pytest.mark.parametrize("n", [1, 128, 129, 256, 300, 1000, 1025, 4095, 4096])
@pytest.mark.parametrize("where", ["in_place", "later", "earlier", "last_input", "params"])
def test_outputs_may_overlap_what_is_read(n, where):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(n)
    p = torch.from_numpy(init_params(n)).cuda()
    x = torch.from_numpy(rng.random(4 * n).astype(np.float32)).cuda()
    want = torch.full((3 * n,), float("nan"), device="cuda")
    _call(p.data_ptr(), x.data_ptr(), n, want.data_ptr())
    # one buffer: 3n floats, the parameters or the inputs, 3n floats
    held = p if where == "params" else x
    m = held.numel()
    buf = torch.zeros(6 * n + m, device="cuda")
    at = {"in_place": 3 * n, "later": 3 * n + n // 2, "earlier": 2 * n, "last_input": 3 * n + m - 1,
          "params": 3 * n + min(m - 1, 77)}[where]
    for _ in range(3):
        buf.zero_()
        buf[3 * n:3 * n + m] = held
        src = buf.data_ptr() + 4 * 3 * n
        _call(src if where == "params" else p.data_ptr(),
              x.data_ptr() if where == "params" else src, n, buf.data_ptr() + 4 * at)
        torch.cuda.synchronize()
        np.testing.assert_array_equal(buf[at:at + 3 * n].cpu().numpy(), want.cpu().numpy())
        rest = buf.clone()
        rest[at:at + 3 * n] = 0  # nothing else is written
        was = torch.zeros_like(buf)
        was[3 * n:3 * n + m] = held
        was[at:at + 3 * n] = 0
        assert torch.equal(rest, was)


def test_overlapping_call_can_be_captured():
    torch = pytest.importorskip("torch")
    n = 1000
    rng = np.random.default_rng(1)
    p = torch.from_numpy(init_params(3)).cuda()
    x0 = torch.from_numpy(rng.random(4 * n).astype(np.float32)).cuda()
    want = torch.zeros(3 * n, device="cuda")
    _call(p.data_ptr(), x0.data_ptr(), n, want.data_ptr())
    x = x0.clone()
    torch.cuda.synchronize()
    g = torch.cuda.CUDAGraph()
    with torch.cuda.graph(g):
        x.copy_(x0)
        _call(p.data_ptr(), x.data_ptr(), n, x.data_ptr(), torch.cuda.current_stream().cuda_stream)
    for _ in range(2):
        g.replay()
    torch.cuda.synchronize()
    assert torch.equal(x[:3 * n], want) and torch.equal(x[3 * n:], x0[3 * n:])
