"""The unsplit acoustics step (claw2_march.cuh) at the edges of its strips and
row runs and of its quotients' ranges, against the oracle bit for bit.

The marching body divides through claw2_exact.cuh, whose quotients must be the
bits of an IEEE division for every operand, in or out of the range of the
branch-free path: zero and subnormal waves, tails of a pulse down to the
smallest numbers, large amplitudes, impedances outside 2^-60 .. 2^60, zero and
negative sound speeds.  The tolerance is therefore none: values and the CFL
number must be equal (a zero's sign aside, which == does not see).
"""
import numpy as np
import pytest

import gpu_helpers as H
from pyclaw_b200 import _abi

pytestmark = pytest.mark.gpu

SHAPES = [(4, 4), (27, 5), (28, 3), (29, 28), (56, 29), (57, 61), (85, 2), (3, 40)]


def _data(kind, p, seed):
    rng = np.random.default_rng(seed)
    mx, my = p.mx, p.my
    X, Y = np.meshgrid((np.arange(mx) + 0.5) / mx, (np.arange(my) + 0.5) / my, indexing="ij")
    r2 = (X - 0.3) ** 2 + (Y - 0.4) ** 2
    q = np.zeros((3, mx, my), order="F")
    if kind == "tails":                 # down to subnormal pressures and below
        q[0] = np.exp(-r2 * 900.0)
        q[1] = np.exp(-r2 * 1500.0)
    elif kind == "compact":             # zeros next to a pulse
        q[0] = np.where(r2 < 0.04, 1.0 + np.cos(np.pi * np.sqrt(r2) / 0.2), 0.0)
    elif kind == "tiny":
        q[:] = rng.standard_normal(q.shape) * 2.0 ** -470
    elif kind == "subnormal":
        q[:] = rng.integers(-40, 41, q.shape) * 5e-324
    elif kind == "huge":
        q[:] = rng.standard_normal(q.shape) * 2.0 ** 300
    else:
        q[:] = rng.standard_normal(q.shape)
    aux = None
    if p.num_aux:
        aux = np.empty((2, mx, my), order="F")
        aux[0], aux[1] = 1.0 + 3.0 * rng.random((mx, my)), 1.0 + rng.random((mx, my))
        if kind == "impedance":         # face sums on both sides of the reciprocals' range
            aux[0] *= 2.0 ** rng.choice([-70, 0, 65], (mx, my))
        elif kind == "negative":
            aux[1] *= rng.choice([-1.0, 1.0, 1.0], (mx, my))
        elif kind == "still":           # zero sound speeds, no two side by side
            inner = aux[1][1:-1:2, 1:-1:2]
            inner[rng.random(inner.shape) < 0.5] = 0.0
    return q, aux


def _check(orc, p, q, aux, dt, steps=3):
    qbc = orc.new_qbc(p, q)
    orc.fill_ghosts(p, qbc)
    auxbc = None
    if aux is not None:
        auxbc = orc.new_qbc(p, aux, ncomp=p.num_aux)
        orc.fill_aux_ghosts(p, auxbc)
    for _ in range(steps):
        got, cfl = H.dev_step(p, qbc, auxbc, dt)
        cfl_ref = orc.step_hyperbolic(p, qbc, auxbc, dt)
        orc.fill_ghosts(p, qbc)
        assert np.isfinite(qbc).all()
        assert np.array_equal(got, qbc), np.nanmax(np.abs(got - qbc))
        assert cfl == cfl_ref


@pytest.mark.parametrize("name", ["acoustics", "vc_acoustics"])
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bcs", [((1, 3), (3, 1)), ((2, 2), (2, 2))])
def test_strip_and_run_edges(orc, name, shape, bcs):
    p = H.problem(name, shape[0], shape[1], 2, bcl=bcs[0], bcu=bcs[1], abcl=bcs[0], abcu=bcs[1])
    q, aux = _data("noise", p, sum(shape))
    _check(orc, p, q, aux, 0.2 / max(shape))


@pytest.mark.parametrize("name", ["acoustics", "vc_acoustics"])
@pytest.mark.parametrize("kind", ["tails", "compact", "tiny", "subnormal", "huge"])
@pytest.mark.parametrize("lim", [(4,), (1,), (2,), (3,), (5,), (0,), (4, 2), (0, 1)])
def test_amplitudes_and_limiters(orc, name, kind, lim):
    p = H.problem(name, 60, 43, 2, mthlim=lim)
    q, aux = _data(kind, p, 5)
    _check(orc, p, q, aux, 0.2 / 60)


@pytest.mark.parametrize("kind", ["impedance", "negative", "still"])
@pytest.mark.parametrize("transverse,order", [(2, 2), (1, 2), (0, 2), (2, 1)])
def test_materials(orc, kind, transverse, order):
    p = H.problem("vc_acoustics", 60, 43, transverse, order=order)
    q, aux = _data(kind, p, 9)
    _check(orc, p, q, aux, 0.1 / 60)


@pytest.mark.parametrize("params", [(1.0, 4.0, -2.0, -2.0), (1e25, 1e25, 1.0, 1e25), (1e-30, 1.0, 1e15, 1e-15 * 2.0 ** -60),
                                    (3.0, 7.0, np.sqrt(7.0 / 3.0), np.sqrt(21.0))])
def test_constant_coefficients_of_any_size(orc, params):
    p = H.problem("acoustics", 60, 43, 2)
    for k, v in enumerate(params):
        p.params[k] = v
    q, _ = _data("noise", p, 3)
    _check(orc, p, q, None, 0.1 / 60 / abs(params[2]))


@pytest.mark.parametrize("name", ["acoustics", "vc_acoustics"])
def test_march_variants_of_the_batch(orc, name):
    """Batch variants 14-16 (28, 14 and 7 rows a tile) on instances with
    partial tiles equal the variants of the tile body."""
    from pyclaw_b200.batch import BatchSolver
    p = H.problem(name, 32, 32, 2)
    insts = []
    for k, (mx, my) in enumerate([(5, 90), (28, 28), (57, 33), (100, 7)]):
        pk = H.problem(name, mx, my, 2)
        q, aux = _data("noise", pk, k)
        insts.append(dict(q=q, aux=aux, dx=1.0 / mx, dy=1.0 / my, dt=0.1 / max(mx, my)))
    want = None
    for v in (0, 11, 14, 15, 16):
        bs = BatchSolver(p, insts)
        bs.variant = v
        bs.advance(4)
        got = [bs.solution(k) for k in range(len(insts))]
        ctl = [(c.t, c.dt, c.cfl, c.numsteps) for c in bs.controls()]
        if want is None:
            want = (got, ctl)
        assert all(np.array_equal(a, b) for a, b in zip(got, want[0])), v
        assert ctl == want[1], v
