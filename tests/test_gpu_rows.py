"""The split acoustics step (claw2_rows.cuh) at the edges of its tiles and of its
quotients' ranges, against the oracle bit for bit (a zero's sign aside): the
states, materials and tolerance of the unsplit step's tests.
"""
import pytest

import gpu_helpers as H
from test_gpu_march import _check, _data

pytestmark = pytest.mark.gpu

NAMES = ["acoustics", "vc_acoustics"]
# 12-cell tiles, then 28-cell ones: one CTA per SM and more
SHAPES = [(4, 4), (13, 5), (12, 3), (25, 24), (61, 47), (29, 2030), (57, 4202), (8401, 29)]


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("shape", SHAPES)
@pytest.mark.parametrize("bcs", [((1, 3), (3, 1)), ((2, 2), (2, 2))])
def test_tile_edges(orc, name, shape, bcs):
    p = H.problem(name, shape[0], shape[1], -1, bcl=bcs[0], bcu=bcs[1], abcl=bcs[0], abcu=bcs[1])
    q, aux = _data("noise", p, sum(shape))
    _check(orc, p, q, aux, 0.2 / max(shape), steps=2)


@pytest.mark.parametrize("name", NAMES)
@pytest.mark.parametrize("kind", ["tails", "compact", "tiny", "subnormal", "huge"])
@pytest.mark.parametrize("lim", [(4,), (1,), (2,), (3,), (5,), (0,), (4, 2), (0, 1)])
def test_amplitudes_and_limiters(orc, name, kind, lim):
    p = H.problem(name, 60, 43, -1, mthlim=lim)
    q, aux = _data(kind, p, 5)
    _check(orc, p, q, aux, 0.2 / 60)


@pytest.mark.parametrize("kind", ["impedance", "negative", "still"])
@pytest.mark.parametrize("order", [1, 2])
def test_materials(orc, kind, order):
    p = H.problem("vc_acoustics", 57, 45, -1, order=order)
    q, aux = _data(kind, p, 9)
    _check(orc, p, q, aux, 0.05 / 57)


@pytest.mark.parametrize("params", [(1.0, 4.0, -2.0, -2.0), (1e25, 1e25, 1.0, 1e25), (1e-30, 1.0, 1e15, 1e-15 * 2.0 ** -60)])
def test_constant_coefficients_of_any_size(orc, params):
    p = H.problem("acoustics", 60, 43, -1)
    for k, v in enumerate(params):
        p.params[k] = v
    q, _ = _data("noise", p, 3)
    _check(orc, p, q, None, 0.1 / 60 / abs(params[2]))
