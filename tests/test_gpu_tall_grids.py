"""A grid of more rows than a launch's second dimension holds tiles of 28
(65535 x 28), for each body that steps it unsplit, against the oracle bit for bit."""
import numpy as np
import pytest

import gpu_helpers as H
from pyclaw_b200 import _abi

pytestmark = pytest.mark.gpu

MX, MY = 4, 65535 * 28 + 31


@pytest.mark.parametrize("name", ["psystem", "shallow", "acoustics"])
def test_tall_grid(orc, name):
    kw = dict(mx=MX, my=MY, dx=1.0, dy=1.0, order=2, transverse=2, bc_lower=(3, 2), bc_upper=(1, 2))
    rng = np.random.default_rng(4)
    if name == "psystem":
        p = _abi.make_problem(rp=_abi.RP_PSYSTEM, num_eqn=3, num_waves=2, num_aux=4, mthlim=[2], use_fwave=True,
                              aux_bc_lower=(3, 2), aux_bc_upper=(1, 2), **kw)
    else:
        p = _abi.make_problem(mthlim=[4], **H.SOLVERS[name], **kw)
    q = np.asfortranarray(0.1 * rng.standard_normal((p.num_eqn, MX, MY)))
    q[0] += 1.0 if name == "shallow" else 0.0
    qbc, auxbc = orc.new_qbc(p, q), None
    orc.fill_ghosts(p, qbc)
    if name == "psystem":
        aux = np.ones((4, MX, MY), order="F")
        aux[0], aux[1] = rng.choice([1.0, 4.0], (2, MX, MY))
        aux[3] = q[0]
        auxbc = orc.new_qbc(p, aux, 4)
        orc.fill_aux_ghosts(p, auxbc)
    got, cfl = H.dev_step(p, qbc, auxbc, 0.1)
    want = orc.step_hyperbolic(p, qbc, auxbc, 0.1)
    orc.fill_ghosts(p, qbc)
    assert np.isfinite(qbc).all() and 0.05 < want < 1.0
    assert np.array_equal(got, qbc)
    assert cfl == want
