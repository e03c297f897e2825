"""The Euler and shallow-water steps at the edges of their tiles and of the
interface solves (claw2_dense.cuh), against the oracle bit for bit.

Quotients and square roots without branches, the bound that stands in for the
star states' speeds, the splits that leave clipped terms out and the lines
passed over because they carry no waves must all give the bits of the plain
solver: velocities through the sound speed in both directions, momenta that
are zero, subnormal or far smaller than the density, states outside 2^-100 ..
2^100, regions of one state next to a jump, limiters that differ by wave.  The
tolerance is therefore none (a zero's sign aside, which == does not see).
"""
import ctypes

import numpy as np
import pytest

import gpu_helpers as H
from pyclaw_b200 import _lib

pytestmark = pytest.mark.gpu

NAMES = ["euler4", "euler5", "shallow"]
SHAPES = [(4, 4), (27, 5), (28, 3), (29, 28), (56, 29), (57, 61), (85, 4), (4, 40)]
KINDS = ["transonic", "still", "small", "subnormal", "tails", "jump", "column", "high", "low"]


def data(kind, p, seed):
    rng = np.random.default_rng(seed)
    mx, my = p.mx, p.my
    X, Y = np.meshgrid((np.arange(mx) + 0.5) / mx, (np.arange(my) + 0.5) / my, indexing="ij")
    q = np.empty((p.num_eqn, mx, my), order="F")
    rho, pr = 1.0 + 0.2 * rng.random((mx, my)), 1.0 + 0.2 * rng.random((mx, my))
    u, v = 0.3 * np.sin(7 * Y), 0.2 * np.cos(5 * X)
    if kind == "transonic":
        u, v = 2.5 * np.sin(6 * X + 3 * Y), 2.5 * np.cos(4 * X - 7 * Y)
    elif kind == "still":
        u, v = np.zeros((mx, my)), np.zeros((mx, my))
    elif kind == "small":
        u, v = u * 2.0 ** -500, v * 2.0 ** rng.integers(-900, -400, (mx, my)).astype(float)
    elif kind == "tails":                  # through every binade down to zero, in still gas
        u, v = 10.0 ** (-330.0 * X) * rng.choice([-1.0, 1.0], (mx, my)), 10.0 ** (-330.0 * Y)
        rho[:], pr[:] = 1.0, 1.0
    elif kind == "subnormal":
        u, v = rng.integers(-9, 10, (2, mx, my)) * 5e-324
    elif kind in ("jump", "column"):
        rho[:], pr[:], u, v = 1.0, 1.0, np.full((mx, my), 0.1), np.full((mx, my), -0.2)
        at = (X - 0.4) ** 2 + (Y - 0.6) ** 2 < 0.04 if kind == "jump" else X > 0.55
        rho[at], pr[at] = 1.7, 2.0
    scale = {"high": 2.0 ** 150, "low": 2.0 ** -150}.get(kind, 1.0)
    q[0] = rho * scale
    q[1], q[2] = q[0] * u, q[0] * v
    if p.num_eqn >= 4:
        q[3] = scale * pr / 0.4 + 0.5 * q[0] * (u * u + v * v)
    elif scale != 1.0:                     # gravity is 1: speeds grow with the depth's root
        q[1], q[2] = q[1] * np.sqrt(scale), q[2] * np.sqrt(scale)
    if p.num_eqn == 5:
        q[4] = rho * (X > 0.5)
    return q


def check(orc, p, q, cfl, steps=3):
    qbc = orc.new_qbc(p, q)
    orc.fill_ghosts(p, qbc)
    dt = 1e-3 / max(p.mx, p.my)
    dt *= cfl / orc.step_hyperbolic(p, qbc.copy(order="F"), None, dt)
    for _ in range(steps):
        got, c = H.dev_step(p, qbc, None, dt)
        ref = orc.step_hyperbolic(p, qbc, None, dt)
        orc.fill_ghosts(p, qbc)
        assert np.isfinite(qbc).all()
        assert np.array_equal(got, qbc), np.nanmax(np.abs(got - qbc))
        assert c == ref


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("mode", [2, -1])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bcs", [((1, 3), (3, 1)), ((2, 2), (2, 2))])
def test_tile_edges(orc, name, mode, shape, bcs):
    p = H.problem(name, shape[0], shape[1], mode, bcl=bcs[0], bcu=bcs[1])
    check(orc, p, data("smooth", p, sum(shape)), 0.4)


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("mode,order", [(2, 2), (1, 2), (0, 2), (2, 1), (-1, 2), (-1, 1)])
@pytest.mark.parametrize("kind", KINDS)
def test_states(orc, name, mode, order, kind):
    p = H.problem(name, 60, 43, mode, order=order)
    check(orc, p, data(kind, p, 3), 0.3)


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("mode", [2, -1])
@pytest.mark.parametrize("lim", [(0,), (1,), (2,), (3,), (5,), (4, 2, 4, 4, 4), (4, 4, 4, 4, 2), (0, 4, 0, 1, 3)])
def test_limiters(orc, name, mode, lim):
    p = H.problem(name, 45, 33, mode, mthlim=lim[:H.SOLVERS[name]["num_waves"]])
    check(orc, p, data("transonic", p, 8), 0.3)


# 28-cell tiles: one CTA per SM (147 and 128 tiles), two per SM (303 and 602)
@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("mode", [2, -1])
@pytest.mark.parametrize("shape", [(29, 2030), (1790, 56), (57, 2802), (8401, 29)])
def test_large_tile_edges(orc, name, mode, shape):
    p = H.problem(name, shape[0], shape[1], mode, bcl=(2, 1), bcu=(2, 3))
    check(orc, p, data("transonic", p, 1), 0.3, steps=2)


@pytest.mark.parametrize("name", NAMES)
def test_split_step_of_buffers_off_16_bytes(orc, name):
    """The halo copies need 16-byte boundaries; split, other buffers are stepped
    by the general body."""
    t, lib = H.torch(), _lib.load()
    p = H.problem(name, 61, 40, -1)
    qbc = orc.new_qbc(p, data("transonic", p, 4))
    orc.fill_ghosts(p, qbc)
    L = _lib.layout(p)
    src = H.to_dev(p, qbc, L)
    qin, qout = t.empty(src.numel() + 1, dtype=t.float64, device="cuda")[1:], t.empty_like(src)
    qin.copy_(src)
    scratch = t.zeros(lib.claw2_scratch_bytes(ctypes.byref(p)), dtype=t.uint8, device="cuda")
    cfl = t.zeros(1, dtype=t.float64, device="cuda")
    dt = 1e-3
    rc = lib.claw2_step(ctypes.byref(p), ctypes.c_void_p(qin.data_ptr()), ctypes.c_void_p(qout.data_ptr()), None, dt,
                        ctypes.c_void_p(scratch.data_ptr()), ctypes.c_void_p(cfl.data_ptr()), H.stream())
    assert rc == 0
    got = H.from_dev(p, qout, p.num_eqn, L)
    ref = orc.step_hyperbolic(p, qbc, None, dt)
    orc.fill_ghosts(p, qbc)
    assert np.array_equal(got, qbc)
    assert float(cfl.item()) == ref


# more than 16 tiles of 28 cells per SM: one-state tiles are stepped by a pass of their own
@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("mode", [2, -1])
@pytest.mark.parametrize("kind", ["jump", "rest", "transonic"])
@pytest.mark.parametrize("shape,bcs", [((66401, 5), ((1, 3), (3, 1))), ((30, 33199), ((2, 2), (2, 2)))])
def test_listed_tiles(orc, name, mode, kind, shape, bcs):
    p = H.problem(name, shape[0], shape[1], mode, bcl=bcs[0], bcu=bcs[1])
    q = data("column" if kind == "rest" else kind, p, 2)
    if kind == "rest":                     # every tile holds the one state
        q[:] = q[:, :1, :1]
    check(orc, p, q, 0.3, steps=1)


@pytest.mark.parametrize("name,mode", [("euler5", 2), ("shallow", 2), ("euler4", -1)])
def test_listed_steps_in_one_call_equal_single_calls(name, mode):
    from pyclaw_b200 import _abi
    from pyclaw_b200.device import DeviceState
    t, lib = H.torch(), _lib.load()
    p = H.problem(name, 1400, 1400, mode, bcl=(1, 3), bcu=(3, 1))
    q = data("jump", p, 6)
    results = []
    for calls in (1, 8):
        dev = DeviceState(p)
        dev.upload_q(q)
        c = _abi.Control.from_address(dev.ctrl_host.data_ptr())
        _lib.check(lib.claw2_control_init(ctypes.byref(c), 0.0, 0.2 / 1400, 1e9, 1.0, 0.9, 1e99, 1, 0, 1 << 40, 0.9),
                   "claw2_control_init")
        dev.ctrl.copy_(dev.ctrl_host)
        for _ in range(calls):
            _lib.check(lib.claw2_advance(ctypes.byref(p), dev.ptr(dev.q[0]), dev.ptr(dev.q[1]), dev.ptr(dev.aux),
                                         dev.ptr(dev.ctrl), dev.ptr(dev.scratch), 8 // calls, dev.stream), "claw2_advance")
        dev.ctrl_host.copy_(dev.ctrl)
        t.cuda.synchronize()
        c = _abi.Control.from_address(dev.ctrl_host.data_ptr())
        assert c.numsteps == 8 and c.error == 0
        assert not dev.scratch[:64].any()
        dev.cur = c.cur
        results.append((dev.download_q(), c.t, c.dt))
    assert results[0][1:] == results[1][1:]
    assert np.array_equal(results[0][0], results[1][0])
