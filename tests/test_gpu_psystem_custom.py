"""p-system steps beside custom sides: the step leaves their ghost cells alone and writes
the others' and the corners (see test_gpu_custom_sides), on both tile sizes and on grids
whose ghost cells are filled by a kernel of their own, bit for bit (linear materials)."""
import pytest

import gpu_helpers as H
from test_gpu_custom_sides import SIDES, run
from test_gpu_psystem import fields, problem

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", [(40, 31), (4, 25), (3, 9), (29, 2030), (57, 2802)])
@pytest.mark.parametrize("sides", SIDES)
def test_custom_sides(orc, monkeypatch, shape, sides):
    monkeypatch.setattr(H, "init_fields", lambda p, seed: fields(p, "noise", 1.0, seed))
    p = problem(*shape, 1, bcl=sides[0], bcu=sides[1])
    for d in range(2):
        p.aux_bc_lower[d], p.aux_bc_upper[d] = 3, 1
    run(orc, p, 5)
