"""The CFL numbers of the multi-shot step (claw2_shots_step): every shot's is the one
of the same step taken alone, in every step, and counters and CFL cells are ready
for the next one.  All shots share aux and dt, so their numbers are equal; the
array is overwritten before each step, so a shot that reported nothing shows."""
import ctypes

import numpy as np
import pytest

import gpu_helpers as H
from pyclaw_b200 import _lib

pytestmark = pytest.mark.gpu


def runner(mx, my, shots, steps):
    from pyclaw_b200.adjoint import AcousticShots
    rng = np.random.default_rng(shots)
    src = rng.integers(0, mx * my, shots)
    return AcousticShots(mx, my, 1.0 / mx, 1.0 / my, shots, src, [0], rng.standard_normal((steps, shots)), 0.1 / max(mx, my))


@pytest.mark.parametrize("shape,shots", [((61, 47), 4), ((61, 47), 5), ((256, 256), 12), ((90, 203), 61), ((61, 47), 64),
                                         ((30, 9), 130)])
def test_every_shot_reports_its_own_cfl(orc, shape, shots):
    t, lib = H.torch(), _lib.load()
    steps = 6
    r = runner(*shape, shots, steps)
    rng = np.random.default_rng(1)
    aux = np.asfortranarray(1.0 + rng.random((2,) + shape))
    r.set_aux(t.from_numpy(aux))
    q, out = r.new_states(1)[0], r.new_states(1)[0]
    r.set_state(q, t.from_numpy(rng.standard_normal((shots, 3) + shape)))
    qbc, auxbc = orc.new_qbc(r.p, np.asfortranarray(np.zeros((3,) + shape))), orc.new_qbc(r.p, aux, 2)
    orc.fill_aux_ghosts(r.p, auxbc)
    bad = shots // 2
    for n in range(steps):
        if n == steps - 1:                       # a state that is not finite, in one shot
            r._interior(q, 3)[bad, 0, 3, 4] = float("nan")
        r.dt = 0.1 / max(shape) * (1.0 + 0.3 * n)
        r.cfl.fill_(-7.0)
        r.step(q, out, n)
        want = t.full((shots,), orc.step_hyperbolic(r.p, qbc.copy(order="F"), auxbc, r.dt), dtype=t.float64)
        if n == steps - 1:
            want[bad] = float("nan")
        assert np.array_equal(r.cfl.cpu().numpy(), want.numpy(), equal_nan=True), n
        assert not bool(r.scratch.any()), n
        q, out = out, q


def test_one_shot_equals_the_plain_step():
    t, lib = H.torch(), _lib.load()
    r = runner(83, 40, 1, 1)
    rng = np.random.default_rng(2)
    r.set_aux(t.from_numpy(1.0 + rng.random((2, 83, 40))))
    q, out = r.new_states(1)[0], r.new_states(1)[0]
    r.set_state(q, t.from_numpy(rng.standard_normal((1, 3, 83, 40))))
    r.step(q, out, 0)
    scratch = t.zeros(lib.claw2_scratch_bytes(ctypes.byref(r.p)), dtype=t.uint8, device="cuda")
    cfl = t.zeros(1, dtype=t.float64, device="cuda")
    _lib.check(lib.claw2_step(ctypes.byref(r.p), ctypes.c_void_p(q.data_ptr()), ctypes.c_void_p(out.data_ptr()),
                              ctypes.c_void_p(r.aux.data_ptr()), r.dt, ctypes.c_void_p(scratch.data_ptr()),
                              ctypes.c_void_p(cfl.data_ptr()), H.stream()), "claw2_step")
    assert float(cfl.item()) == float(r.cfl.item())
