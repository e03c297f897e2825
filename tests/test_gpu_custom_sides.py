"""Steps beside custom sides: the ghost cells of custom sides stay as the caller
left them, the step writes the others' and, in the corners, their images of the
custom sides' ghost cells, in the order of the boundary fill (x sides over all
rows, then y sides over all columns).  Against the oracle's step and fill, bit
for bit.
"""
import ctypes

import numpy as np
import pytest

import gpu_helpers as H
from pyclaw_b200 import _lib

pytestmark = pytest.mark.gpu

# (lower x, lower y), (upper x, upper y): 0 custom, 1 extrapolation, 2 periodic, 3 wall
SIDES = [((0, 3), (1, 1)), ((1, 0), (3, 1)), ((0, 2), (0, 2)), ((2, 0), (2, 1)), ((3, 1), (0, 3)), ((0, 0), (1, 3)),
         ((0, 0), (0, 0))]


def run(orc, p, seed):
    rng = np.random.default_rng(seed)
    t, lib, L = H.torch(), _lib.load(), _lib.layout(p)
    q, aux = H.init_fields(p, seed)
    qbc = orc.new_qbc(p, q)
    # ghost cells of custom sides: smooth values of the caller's
    for axis in (1, 2):
        n = qbc.shape[axis] - 4
        for g, src in ((0, 2), (1, 2), (n + 2, n + 1), (n + 3, n + 1)):
            sl, so = [slice(None)] * 3, [slice(None)] * 3
            sl[axis], so[axis] = g, src
            qbc[tuple(sl)] = qbc[tuple(so)]
    orc.fill_ghosts(p, qbc)
    auxbc = None
    if aux is not None:
        auxbc = orc.new_qbc(p, aux, p.num_aux)
        orc.fill_aux_ghosts(p, auxbc)
    out0 = np.asfortranarray(qbc + 0.01 * rng.random(qbc.shape))     # what q_out holds before the step
    dt = 0.1 / max(p.mx, p.my)
    ref = qbc.copy(order="F")
    cfl_ref = orc.step_hyperbolic(p, ref, auxbc, dt)
    want = out0.copy(order="F")
    want[:, 2:-2, 2:-2] = ref[:, 2:-2, 2:-2]
    orc.fill_ghosts(p, want)
    qin, qout = H.to_dev(p, qbc, L), H.to_dev(p, out0, L)
    daux = H.to_dev(p, auxbc, L) if auxbc is not None else t.zeros(1, dtype=t.float64, device="cuda")
    scratch = t.zeros(lib.claw2_scratch_bytes(ctypes.byref(p)), dtype=t.uint8, device="cuda")
    cfl = t.zeros(1, dtype=t.float64, device="cuda")
    _lib.check(lib.claw2_step(ctypes.byref(p), ctypes.c_void_p(qin.data_ptr()), ctypes.c_void_p(qout.data_ptr()),
                              ctypes.c_void_p(daux.data_ptr()), dt, ctypes.c_void_p(scratch.data_ptr()),
                              ctypes.c_void_p(cfl.data_ptr()), H.stream()), "claw2_step")
    got = H.from_dev(p, qout, p.num_eqn, L)
    assert np.isfinite(want).all()
    assert np.array_equal(got, want), np.argwhere(got != want)[:5]
    assert float(cfl.item()) == cfl_ref


@pytest.mark.parametrize("name", ["euler5", "shallow", "vc_acoustics", "acoustics"])
@pytest.mark.parametrize("mode", [2, -1])
@pytest.mark.parametrize("shape", [(40, 31), (4, 25), (3, 9), (29, 2030)])
@pytest.mark.parametrize("sides", SIDES)
def test_custom_sides(orc, name, mode, shape, sides):
    run(orc, H.problem(name, shape[0], shape[1], mode, bcl=sides[0], bcu=sides[1]), 5)


# a capacity function: the general body; more than 16 tiles per SM: one-state tiles in a pass of their own
@pytest.mark.parametrize("sides", SIDES)
def test_custom_sides_of_the_general_body(orc, sides):
    p = H.problem("vc_acoustics", 33, 40, 2, bcl=sides[0], bcu=sides[1])
    p.index_capa = 1
    run(orc, p, 6)


@pytest.mark.parametrize("sides", SIDES)
def test_custom_sides_of_listed_tiles(orc, sides):
    run(orc, H.problem("shallow", 66401, 5, 2, bcl=sides[0], bcu=sides[1]), 7)


@pytest.mark.parametrize("lower,upper", [((0, 3), (1, 1)), ((1, 0), (3, 1)), ((0, 0), (1, 3)), ((0, 0), (0, 0)), ((0, 2), (1, 2))])
@pytest.mark.parametrize("solver", ["euler", "acoustics"])
def test_fixed_sides_set_on_the_device_equal_the_host_fill(solver, lower, upper):
    import pyclaw_b200 as pc

    class OnHost(pc.hooks.FixedStateBC):
        """a subclass: the host fills the sides"""

    res = []
    for cls in (pc.hooks.FixedStateBC, OnHost):
        domain = pc.Domain([pc.Dimension("x", 0.0, 1.0, 41), pc.Dimension("y", 0.0, 1.0, 30)])
        st = pc.State(domain, 4 if solver == "euler" else 3)
        rng = np.random.default_rng(3)
        if solver == "euler":
            st.problem_data["gamma"], st.problem_data["gamma1"] = 1.4, 0.4
            st.q[...] = 0.1 * rng.random(st.q.shape)
            st.q[0] += 1.0
            st.q[3] += 2.5
            sol = pc.ClawSolver2D(pc.riemann.rp2_euler_4wave)
            lo, up = [1.2, 0.3, 0.1, 3.0], [0.9, -0.1, 0.2, 2.2]
        else:
            for k, v in dict(rho=1.0, bulk=4.0, cc=2.0, zz=2.0).items():
                st.problem_data[k] = v
            st.q[...] = rng.random(st.q.shape)
            sol = pc.ClawSolver2D(pc.riemann.rp2_acoustics)
            lo, up = [0.3, 0.1, -0.2], [0.0, 0.2, 0.1]
        sol.limiters = 4
        sol.dimensional_split = False
        sol.dt_initial = 1e-3
        sol.bc_lower, sol.bc_upper = list(lower), list(upper)
        sol.user_bc_lower, sol.user_bc_upper = cls(lo, side="lower"), cls(up, side="upper")
        solution = pc.Solution(st, domain)
        sol.setup(solution)
        for t in (0.02, 0.03):
            sol.evolve_to_time(solution, t)
        res.append((solution.state.get_q_host().copy(), solution.t, sol.dt))
    assert res[0][1:] == res[1][1:]
    assert np.array_equal(res[0][0], res[1][0])
