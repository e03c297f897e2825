"""The unsplit p-system step (claw2_psystem.cuh) at the edges of its tiles and of
its quotients' ranges, against the oracle: linear materials bit for bit (a zero's
sign aside, which == does not see); exponential ones, whose exponential the
device and the host may round differently by an ulp each, within 2e-12: stresses
up to e^5 = 150 carry 2 x 1.1e-16 x 150 = 3e-14, a cell takes it from 12 interfaces
(its own and the transverse ones), twice through the limiter's slopes (at most 2)
and over two steps with dt/dx below 1.
"""
import numpy as np
import pytest

import gpu_helpers as H
from pyclaw_b200 import _abi

pytestmark = pytest.mark.gpu

# 12-cell tiles, then 28-cell ones: one CTA per SM and two
SHAPES = [(4, 4), (13, 5), (12, 3), (25, 24), (4, 40), (61, 47), (29, 2030), (57, 2802)]


def problem(mx, my, mode, order=2, lim=(2,), bcl=(3, 3), bcu=(1, 1)):
    return _abi.make_problem(rp=_abi.RP_PSYSTEM, num_eqn=3, num_waves=2, num_aux=4, mx=mx, my=my, dx=1.0 / mx,
                             dy=1.0 / my, order=order, transverse=mode, mthlim=list(lim), use_fwave=True,
                             bc_lower=bcl, bc_upper=bcu, aux_bc_lower=bcl, aux_bc_upper=bcu)


def fields(p, kind, law, seed):
    rng = np.random.default_rng(seed)
    mx, my = p.mx, p.my
    q = np.zeros((3, mx, my), order="F")
    q[0] = 0.3 * rng.uniform(-3, 3, (mx, my))
    q[1:] = 0.1 * rng.standard_normal((2, mx, my))
    aux = np.ones((4, mx, my), order="F")
    aux[0], aux[1] = rng.choice([1.0, 4.0, 1.7], (2, mx, my))
    aux[2] = law if law else rng.choice([1.0, 2.0], (mx, my))
    if kind == "pulse":                 # still outside
        X, Y = np.meshgrid(np.arange(mx) / mx, np.arange(my) / my, indexing="ij")
        q *= (X - 0.4) ** 2 + (Y - 0.3) ** 2 < 0.05
    elif kind == "tiny":
        q *= 2.0 ** -480
    elif kind == "subnormal":
        q[:] = rng.integers(-9, 10, q.shape) * 5e-324
    elif kind == "stiff":               # impedance sums on both sides of the reciprocals' range
        aux[1] *= 2.0 ** rng.choice([-140, 0, 130], (mx, my))
        q *= 2.0 ** -140
    aux[3] = q[0] if kind != "old" else q[0] + 0.1 * rng.standard_normal((mx, my))
    return q, aux


def state(orc, p, q, aux):
    qbc, auxbc = orc.new_qbc(p, q), orc.new_qbc(p, aux, p.num_aux)
    orc.fill_ghosts(p, qbc)
    orc.fill_aux_ghosts(p, auxbc)
    return qbc, auxbc


def against_oracle(orc, p, q, aux, steps=2):
    qbc, auxbc = state(orc, p, q, aux)
    dt = 1e-3
    dt *= 0.4 / orc.step_hyperbolic(p, qbc.copy(order="F"), auxbc, dt)
    for _ in range(steps):
        got, cfl = H.dev_step(p, qbc, auxbc, dt)
        ref = orc.step_hyperbolic(p, qbc, auxbc, dt)
        orc.fill_ghosts(p, qbc)
        assert np.isfinite(qbc).all()
        assert np.array_equal(got, qbc), np.nanmax(np.abs(got - qbc))
        assert cfl == ref


@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bcs", [((3, 3), (1, 1)), ((2, 2), (2, 2))])
def test_tile_edges(orc, shape, bcs):
    p = problem(*shape, 1, bcl=bcs[0], bcu=bcs[1])
    against_oracle(orc, p, *fields(p, "noise", 1.0, sum(shape)))


@pytest.mark.parametrize("kind", ["noise", "old", "pulse", "tiny", "subnormal", "stiff"])
@pytest.mark.parametrize("mode,order", [(2, 2), (1, 2), (0, 2), (2, 1)])
@pytest.mark.parametrize("lim", [(4,), (0,), (1,), (2,), (3,), (5,), (4, 2), (0, 1)])
def test_states_and_limiters(orc, kind, mode, order, lim):
    p = problem(43, 30, mode, order=order, lim=lim)
    against_oracle(orc, p, *fields(p, kind, 1.0, 7))


@pytest.mark.parametrize("kind", ["noise", "old", "pulse", "tiny"])
@pytest.mark.parametrize("mode", [0, 1, 2])
@pytest.mark.parametrize("shape", [(61, 47), (203, 200), (57, 2802)])
def test_exponential_materials(orc, kind, mode, shape):
    p = problem(*shape, mode)
    q, aux = fields(p, kind, None, 3)
    assert np.max(np.abs(q[0] * aux[1])) < 5.0 and np.max(np.abs(aux[3] * aux[1])) < 5.5
    qbc, auxbc = state(orc, p, q, aux)
    dt = 0.1 / max(shape)
    for _ in range(2):
        got, cfl = H.dev_step(p, qbc, auxbc, dt)
        ref = orc.step_hyperbolic(p, qbc, auxbc, dt)
        orc.fill_ghosts(p, qbc)
        assert np.isfinite(qbc).all()
        assert np.max(np.abs(got - qbc)) <= 2e-12
        assert abs(cfl - ref) <= 1e-14 * ref
        qbc = got
