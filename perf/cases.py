"""The work users have this framework do, as measurable cases.

A simulation case advances a batch of cells by one output window (100 time
steps, 2.5 ms) and drains what the window recorded: the call pattern of the
drop-in program, the ensemble drivers and the surrogate's data generator.  A
network case is one call of the surrogate: predictions of a sweep, gradients
of a batch, an epoch of training, or the forward pass on the caller's own
device memory.

A case is a dict of plain values.  Lattice sizes come from the case alone
(`layout` seeds the uneven ones); the seed given to prepare() sets the random
streams, the cells' physiological parameters, the network's weights and its
inputs.
"""
from __future__ import annotations

import ctypes as C

import numpy as np
import torch

from ryr_hyperactivity_gb300 import native
from ryr_hyperactivity_gb300.abi import cell_params
from ryr_hyperactivity_gb300.sim import Simulator
from ryr_hyperactivity_gb300.surrogate import Surrogate, init_params
from ryr_hyperactivity_gb300.workloads import HYPER, STAB

STEPS = 100  # one output window
H, KIN, NOUT = 128, 16, 8
SHAPES = [(H, KIN), (H, H), (H, H), (NOUT, H)]
#: options one batch of protocol cells goes through (the program's build switches)
PROTOCOLS = [dict(), dict(protocol="vclamp", clamp_mv=-20.0), dict(perm=1), dict(iso=1),
             dict(slowncx=1), dict(ncx_form="oldncx"), dict(ncx_form="ncx_noallo"),
             dict(protocol="linearapclamp"), dict(randomlcc=1), dict(protocol="nopacing")]


def _sim(precision, cells, lo, hi, base, warm, **more):
    """A simulation case: `cells` lattices with extents uniform in lo..hi
    (ghost shell included), `warm` steps taken before the measured windows."""
    return dict(kind="sim", precision=precision, cells=cells, nx_lo=lo[0], nx_hi=hi[0], ny_lo=lo[1],
                ny_hi=hi[1], nz_lo=lo[2], nz_hi=hi[2], base=base, warm=warm, **more)


# the ensemble's lattice range
LO, HI = (60, 12, 6), (100, 20, 10)


def listed():
    return [
        # the smallest cell (432 units), double precision, as a quick look at a
        # parameter is run: launches and the whole-cell update's latency count
        dict(_sim("fp64", 1, (20, 10, 5), (20, 10, 5), "stab", 4000), name="cell_fp64_20x10x5"),
        # one full-size cell, double precision: what the drop-in program runs
        dict(_sim("fp64", 1, (100, 20, 10), (100, 20, 10), "stab", 4000),
             name="cell_fp64_100x20x10"),
        # an uneven ensemble in double precision (the reference arm of a
        # mixed-precision report)
        dict(_sim("fp64", 64, LO, HI, "hyper", 400, layout=12345), name="ensemble_fp64_64"),
        # cells of every protocol and build switch in one batch, odd lattice
        # (3,705 units each), double precision
        dict(_sim("fp64", 10, (41, 21, 7), (41, 21, 7), "stab", 1000, protocols=True),
             name="protocols_fp64_10"),
        # one full-size cell, mixed precision
        dict(_sim("mixed", 1, (100, 20, 10), (100, 20, 10), "stab", 4000),
             name="cell_mixed_100x20x10"),
        # a population of small cells: seeds per parameter point
        dict(_sim("mixed", 200, (20, 10, 5), (20, 10, 5), "hyper", 4000), name="population_mixed_200"),
        # the 512-cell uneven ensemble: the batched study, the largest work here
        dict(_sim("mixed", 512, LO, HI, "hyper", 400, layout=12345), name="ensemble_mixed_512"),
        # the same kind of ensemble kept in host memory between windows
        dict(_sim("mixed", 128, LO, HI, "hyper", 400, layout=777, host=True),
             name="ensemble_mixed_host_128"),
        # the surrogate over a parameter sweep
        dict(kind="predict", n=65536, name="surrogate_predict_65536"),
        # one epoch of the surrogate's training at its default batch
        dict(kind="fit", n=3276, batch=256, name="surrogate_fit_3276"),
        # gradients of the largest batch a default handle takes
        dict(kind="gradients", n=4096, name="surrogate_gradients_4096"),
        # the forward pass on the caller's device memory, ragged batch
        dict(kind="noalloc", n=1000, name="surrogate_noalloc_1000"),
    ]


def _log(rng, lo, hi):
    return int(round(lo * (hi / lo) ** rng.random()))


def draw(rng):
    kind = rng.choice(["cell", "cell", "cells", "ensemble", "ensemble", "population", "protocols",
                       "host", "predict", "gradients", "fit", "noalloc"])
    if kind == "cell":
        s = (_log(rng, 12, 110), rng.randint(6, 28), rng.randint(5, 12))
        p = rng.choice(["fp64", "fp64", "mixed"])
        return _sim(p, 1, s, s, rng.choice(["stab", "hyper"]), rng.choice([1000, 4000]))
    if kind == "cells":  # a few uneven cells, double precision
        return _sim("fp64", _log(rng, 2, 48), (14, 8, 5), HI, "hyper", 400,
                    layout=rng.randint(1, 1 << 20))
    if kind == "ensemble":
        return _sim("mixed", _log(rng, 8, 500), LO, HI, "hyper", 400, layout=rng.randint(1, 1 << 20))
    if kind == "population":
        s = (rng.randint(14, 62), rng.randint(8, 16), rng.randint(5, 8))
        return _sim("mixed", _log(rng, 16, 256), s, s, "hyper", 1000)
    if kind == "protocols":
        s = (rng.randint(12, 48), rng.randint(7, 22), rng.randint(5, 8))
        return _sim(rng.choice(["fp64", "mixed"]), rng.randint(4, 20), s, s, "stab", 1000,
                    protocols=True)
    if kind == "host":
        return _sim("mixed", _log(rng, 4, 128), LO, HI, "hyper", 400,
                    layout=rng.randint(1, 1 << 20), host=True)
    if kind == "predict":
        return dict(kind=kind, n=_log(rng, 1, 65536))
    if kind == "fit":
        return dict(kind=kind, n=_log(rng, 300, 4096), batch=rng.choice([64, 100, 128, 256]))
    return dict(kind=kind, n=_log(rng, 1, 4096))


# ------------------------------------------------------------ simulations

def _lattices(case):
    rng = np.random.default_rng(case.get("layout", 0))
    n = case["cells"]
    return np.stack([rng.integers(case[d + "_lo"], case[d + "_hi"] + 1, n)
                     for d in ("nx", "ny", "nz")], 1)


def _interior(case):
    return int(np.prod(_lattices(case) - 2, axis=1).sum())


def _cells(case, seed):
    rng = np.random.default_rng(seed)
    cells = []
    for c, (nx, ny, nz) in enumerate(_lattices(case)):
        d = dict(HYPER if case["base"] == "hyper" else STAB)
        d.update(nx=int(nx), ny=int(ny), nz=int(nz), nbeats=1000, lqt=0, iso2=1, cell_id=c,
                 seed=int(seed) & 0xFFFFFFFF, ku2=float(rng.uniform(1.0, 3.0)),
                 ikr_scale=float(rng.uniform(0.0, 1.0)), pcl_ms=float(rng.uniform(500.0, 3000.0)))
        if case.get("protocols"):
            d.update(PROTOCOLS[c % len(PROTOCOLS)])
        cells.append(cell_params(**d))
    return cells


def _records(sim):
    """What the window recorded (V, concentrations, currents, channel counts
    of every cell); of a single cell also its linescan and membrane state."""
    out = {"wholecell": np.concatenate(sim.drain_wholecell_all())}
    if sim.ncells == 1:
        out["linescan"] = sim.drain_linescan(0, 4)
        out["membrane"] = np.array(list(sim.get_membrane(0).as_dict().values()), np.float64)
    return out


# --------------------------------------------------------------- network

def _params(seed):
    p = init_params(seed)
    rng = np.random.default_rng(seed + 1)
    o = 0
    for n, k in SHAPES:  # a trained network's biases are not zero
        o += n * k
        p[o:o + n] = rng.uniform(-0.1, 0.1, n)
        o += n
    return p


def _batch(case, seed):
    """Points of the unit parameter box and targets of the kind a simulated
    ensemble gives: EAD probability, scaled APD90 mean and variance."""
    rng = np.random.default_rng(seed + 2)
    x = rng.random((case["n"], 4)).astype(np.float32)
    ead = 1 / (1 + np.exp(-(8 * x[:, 0] - 6 * x[:, 1] + 2 * x[:, 2] - 3)))
    t = np.stack([np.round(ead * 4) / 4, 0.2 + 0.3 * x[:, 2] - 0.1 * x[:, 1], 0.05 * ead], 1)
    return x, t.astype(np.float32)


def prepare(case, seed):
    if case["kind"] == "sim":
        sim = Simulator(_cells(case, seed), precision=case["precision"])
        sim.run_steps(case["warm"])
        for _ in range(2):
            sim.drain_wholecell_all()
        if sim.ncells == 1:
            sim.drain_linescan(0)
        st = {"kind": "host" if case.get("host") else "sim", "sim": sim}
        if case.get("host"):
            nb = sim.state_bytes()
            st["image"] = torch.empty(nb, dtype=torch.uint8, pin_memory=True)
            sim.export_state(st["image"].data_ptr(), nb)
        return st
    x, t = _batch(case, seed)
    if case["kind"] == "noalloc":
        f = native.load().rh_mlp_forward_noalloc
        f.argtypes = [C.c_void_p, C.c_void_p, C.c_int32, C.c_void_p, C.c_void_p, C.c_char_p,
                      C.c_size_t]
        return {"kind": "noalloc", "call": f, "p": torch.from_numpy(_params(seed)).cuda(),
                "x": torch.from_numpy(x).cuda(), "y": torch.zeros((case["n"], 3), device="cuda"),
                "err": C.create_string_buffer(256)}
    m = Surrogate()
    m.set_params(_params(seed))
    return {"kind": case["kind"], "model": m, "x": x, "t": t, "batch": case.get("batch")}


def run(state):
    kind = state["kind"]
    if kind == "sim":
        state["sim"].run_steps(STEPS)
        return _records(state["sim"])
    if kind == "host":  # the batch's state goes to the GPU and back
        sim, im = state["sim"], state["image"]
        sim.run_steps_host(STEPS, im.data_ptr(), im.data_ptr(), im.numel())
        return _records(sim)
    if kind == "noalloc":
        rc = state["call"](state["p"].data_ptr(), state["x"].data_ptr(), state["x"].shape[0],
                           state["y"].data_ptr(), torch.cuda.current_stream().cuda_stream,
                           state["err"], 256)
        if rc != 0:
            raise RuntimeError(state["err"].value.decode())
        return state["y"]
    m, x, t = state["model"], state["x"], state["t"]
    if kind == "predict":
        return m.predict(x)
    if kind == "gradients":
        loss, g = m.gradients(x, t)
        return {"loss": loss, "gradients": g}
    losses = m.fit(x, t, epochs=1, batch=state["batch"])
    return {"losses": losses, "params": m.get_params()}


def work(case):
    """Simulation: every field of every unit read and written once a step (73
    reals and 16 bytes of counts) and about 1,400 arithmetic operations.
    Network: parameters, inputs and outputs once, two operations per weight
    and sample (six with gradients)."""
    if case["kind"] == "sim":
        n = _interior(case)
        real = 8 if case["precision"] == "fp64" else 4
        b = 2.0 * n * (73 * real + 16) * STEPS
        if case.get("host"):
            b += 2.0 * n * (90 * real + 16)
        return {"bytes": b, "flops": 1400.0 * n * STEPS}
    n, p = case["n"], sum(a * b + a for a, b in SHAPES)
    per = 2.0 * (4 * H + 2 * H * H + 3 * H)
    if case["kind"] in ("predict", "noalloc"):
        return {"bytes": 4.0 * (7 * n + p), "flops": per * n}
    if case["kind"] == "gradients":
        return {"bytes": 4.0 * (7 * n + 2 * p), "flops": 3 * per * n}
    steps = n // min(case["batch"], n)
    return {"bytes": 4.0 * (7 * n + 6 * p * steps), "flops": 3 * per * n}


# ------------------------------------------------- the same in 64 bits

def _network(p, x):
    p = p.astype(np.float64)
    ws, bs, o = [], [], 0
    for n, k in SHAPES:
        ws.append(p[o:o + n * k].reshape(n, k).copy())
        o += n * k
        bs.append(p[o:o + n])
        o += n
    ws[0][:, 4:] = 0  # padding
    ws[3][3:, :] = 0
    a = [np.zeros((x.shape[0], KIN))]
    a[0][:, :4] = x
    for l in range(3):
        a.append(np.maximum(a[-1] @ ws[l].T + bs[l], 0))
    z = a[3] @ ws[3].T + bs[3]
    y = np.stack([1 / (1 + np.exp(-z[:, 0])), z[:, 1], np.log1p(np.exp(z[:, 2]))], 1)
    return ws, a, z, y


def exact(case, seed):
    """The network in 64 bits.  The simulations have no closed value: a
    stochastic model's window in plain numpy would take minutes, and an epoch
    of training is a sequence of sign-like Adam steps."""
    if case["kind"] in ("sim", "fit"):
        return None
    x, t = _batch(case, seed)
    ws, a, z, y = _network(_params(seed), x.astype(np.float64))
    if case["kind"] in ("predict", "noalloc"):
        return torch.from_numpy(y) if case["kind"] == "noalloc" else y
    n, t = case["n"], t.astype(np.float64)
    loss = np.mean(-(t[:, 0] * np.log(y[:, 0]) + (1 - t[:, 0]) * np.log(1 - y[:, 0]))
                   + (y[:, 1] - t[:, 1]) ** 2 + (y[:, 2] - t[:, 2]) ** 2)
    d = np.zeros((n, NOUT))
    d[:, 0] = (y[:, 0] - t[:, 0]) / n
    d[:, 1] = 2 * (y[:, 1] - t[:, 1]) / n
    d[:, 2] = 2 * (y[:, 2] - t[:, 2]) / (1 + np.exp(-z[:, 2])) / n
    parts = []
    for l in (3, 2, 1, 0):
        parts = [(d.T @ a[l]).ravel(), d.sum(0)] + parts
        if l:
            d = (d @ ws[l]) * (a[l] > 0)
    return {"loss": float(loss), "gradients": np.concatenate(parts)}
