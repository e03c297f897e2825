"""Performance cases of pyclaw_b200: the calls that its users make, over the
range of sizes, solvers, modes and options that they make them with.

A pass of a case goes through the package's public entry points only
(DeviceState.evolve, ClawSolver2D.evolve_to_time, BatchSolver, shots_traces and
the host-buffer session of include/claw2.h).  ``exact`` computes the same
outputs with plain torch in 64 bits, without the package.

Case kinds
  loop   a grid stepped `steps` times by the device-controlled loop
         (evolve_to_time's own path once the state is on the GPU)
  app    the reference's shock-bubble application through ClawSolver2D: host
         arrays in and out, inflow boundary and radial source as device hooks
  batch  many uneven variable-coefficient acoustics instances, one controlled
         step of each per launch, replayed from CUDA graphs
  shots  a seismic inversion step: receiver traces of several shots and the
         gradient with respect to the material
  host   one step through the host-buffer session, the f2py contract of the
         reference's step2 (host arrays in, host arrays out)
"""
import ctypes
import math

import numpy as np
import torch

from pyclaw_b200 import _abi, _lib

G = 2                                     # ghost cells on each side
GAMMA = 1.4
F64 = torch.float64
BCS = {"extrap": ((1, 1), (1, 1)), "periodic": ((2, 2), (2, 2)), "wall": ((3, 3), (3, 3)),
       "mixed": ((3, 3), (1, 1)), "tube": ((1, 3), (1, 3))}      # (lower x, y), (upper x, y)
SOLVERS = {
    "acoustics": dict(rp=_abi.RP_ACOUSTICS, num_eqn=3, num_waves=2, num_aux=0, params=(1.0, 4.0, 2.0, 2.0)),
    "vc": dict(rp=_abi.RP_VC_ACOUSTICS, num_eqn=3, num_waves=2, num_aux=2, params=()),
    "euler4": dict(rp=_abi.RP_EULER_4WAVE, num_eqn=4, num_waves=4, num_aux=0, params=(GAMMA, GAMMA - 1.0)),
    "euler5": dict(rp=_abi.RP_EULER_5WAVE, num_eqn=5, num_waves=5, num_aux=0, params=(GAMMA, GAMMA - 1.0)),
    "shallow": dict(rp=_abi.RP_SHALLOW_ROE, num_eqn=3, num_waves=3, num_aux=0, params=(1.0,)),
    "psystem": dict(rp=_abi.RP_PSYSTEM, num_eqn=3, num_waves=2, num_aux=4, params=()),
}
# floating-point operations of one cell in one unsplit step (normal solves of
# both directions, limiter, corrections, transverse splits, update), counted
# from the formulas; dimensional splitting has no transverse splits
FLOPS = {"acoustics": 170, "vc": 210, "euler4": 900, "euler5": 1000, "shallow": 480, "psystem": 300}


def listed():
    return [
        # the smallest call: a coarse acoustics grid (a first look, a convergence study's first level);
        # launches and latency are all there is
        dict(name="acoustics_64x48", kind="loop", solver="acoustics", mx=64, my=48, mode=2, order=2, lim=4,
             bc="wall", data="pulse", steps=24),
        # the 256 x 256 acoustics run of the benchmark, part of its 171 steps
        dict(name="acoustics_256", kind="loop", solver="acoustics", mx=256, my=256, mode=2, order=2, lim=4,
             bc="wall", data="pulse", steps=60),
        # heterogeneous acoustics on an odd grid, the variable-coefficient application's options (transverse 1)
        dict(name="vc_803x541", kind="loop", solver="vc", mx=803, my=541, mode=1, order=2, lim=4,
             bc="mixed", data="pulse", steps=20),
        # the benchmark's headline: the Euler shock bubble, shocked, smooth and still cells side by side
        dict(name="euler_1280x320", kind="loop", solver="euler4", mx=1280, my=320, mode=2, order=2, lim=4,
             bc="tube", data="shock", steps=20),
        # the reference's default mode (dimensional splitting) with the tracer, an odd grid
        dict(name="euler5_split_641x163", kind="loop", solver="euler5", mx=641, my=163, mode=-1, order=2, lim=4,
             bc="tube", data="shock", steps=40),
        # shallow water with waves everywhere (no still water), periodic, minmod
        dict(name="shallow_500x333", kind="loop", solver="shallow", mx=500, my=333, mode=1, order=2, lim=1,
             bc="periodic", data="waves", steps=30),
        # the largest grid of the benchmark: the 4096^2 dam break, most of it still
        dict(name="shallow_dam_4096", kind="loop", solver="shallow", mx=4096, my=4096, mode=2, order=2, lim=2,
             bc="extrap", data="dam", steps=6),
        # the f-wave application (nonlinear elasticity in a checkerboard), at its own 200 x 200 cells
        dict(name="psystem_200", kind="loop", solver="psystem", mx=200, my=200, mode=1, order=2, lim=2,
             bc="mixed", data="pulse", steps=40),
        # the batched form: uneven instances of 64..384 cells a side
        dict(name="batch_192", kind="batch", n=192, nmin=64, nmax=384, lim=4, steps=10),
        # one gradient of a small inversion: forward, recomputation and adjoint
        dict(name="shots_256x12", kind="shots", mx=256, my=256, shots=12, steps=20, nrec=48, lim=4, every=8),
        # the shock-bubble application as its script runs it: host arrays, callbacks as device hooks
        dict(name="app_shockbubble_320x80", kind="app", mx=320, my=80, tend=0.06),
        # one step through the host-buffer session, as the reference's solver loop would call it
        dict(name="host_step2_320x160", kind="host", solver="euler4", mx=320, my=160, mode=-1, order=2, lim=4,
             bc="tube", data="shock"),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["loop"] * 7 + ["batch", "shots", "app", "host"])
    if kind == "batch":
        return dict(kind="batch", n=_log(rng, 8, 192), nmin=rng.randint(16, 96), nmax=rng.randint(128, 384),
                    lim=rng.choice([1, 2, 3, 4]), steps=rng.randint(6, 12))
    if kind == "shots":
        return dict(kind="shots", mx=_log(rng, 64, 300), my=_log(rng, 64, 300), shots=_log(rng, 1, 12),
                    steps=rng.randint(10, 20), nrec=rng.randint(8, 64), lim=rng.choice([1, 2, 3, 4]),
                    every=rng.randint(4, 10))
    if kind == "app":
        mx = 4 * rng.randint(20, 110)
        return dict(kind="app", mx=mx, my=max(10, mx // 4 + rng.randint(-3, 3)), tend=rng.uniform(0.02, 0.06))
    solver = rng.choice(["acoustics", "vc", "euler4", "euler5", "shallow"] + (["psystem"] if kind == "loop" else []))
    data = {"euler4": "shock", "euler5": "shock", "shallow": rng.choice(["dam", "waves"])}.get(solver, "pulse")
    # the shock's flow has no wall on its left side, which it would leave behind as a vacuum
    bcs = {"psystem": ["extrap", "wall", "mixed"], "euler4": ["extrap", "periodic", "tube"],
           "euler5": ["extrap", "periodic", "tube"]}
    bc = rng.choice(bcs.get(solver, sorted(BCS)))
    mode = rng.choice([0, 1, 2]) if solver == "psystem" else rng.choice([-1, -1, 0, 1, 2, 2])
    order = rng.choice([1, 2, 2, 2, 2])
    lim = rng.choice([1, 2, 3, 4, 4])
    cells = math.exp(rng.uniform(math.log(2000), math.log(200000 if kind == "host" else 1200000)))
    aspect = math.exp(rng.uniform(math.log(0.25), math.log(4.0)))
    mx = max(11, int(math.sqrt(cells * aspect)))
    my = max(11, int(cells / mx))
    case = dict(kind=kind, solver=solver, mx=mx, my=my, mode=mode, order=order, lim=lim, bc=bc, data=data)
    if kind == "loop":
        case["steps"] = max(6, min(60, int(2.0e7 / (mx * my))))
    return case


# ---------------------------------------------------------------------------
# initial data (plain torch on the GPU; [m, j, i], interior cells)
# ---------------------------------------------------------------------------
def _lengths(mx, my):
    return (1.0, my / mx) if mx >= my else (mx / my, 1.0)


def _grid(mx, my):
    lx, ly = _lengths(mx, my)
    dx, dy = lx / mx, ly / my
    x = (torch.arange(mx, dtype=F64, device="cuda") + 0.5) * dx
    y = (torch.arange(my, dtype=F64, device="cuda") + 0.5) * dy
    return x[None, :].expand(my, mx), y[:, None].expand(my, mx), dx, dy, lx, ly


def _modes(rng, X, Y, n, amp):
    """A smooth random field: a few sine waves."""
    f = torch.zeros_like(X)
    for _ in range(n):
        kx, ky = rng.uniform(-40, 40, 2)
        f += amp / n * torch.sin(kx * X + ky * Y + rng.uniform(0, 2 * np.pi))
    return f


def _initial(solver, data, mx, my, seed):
    """(q [m, j, i], aux or None, dx, dy, largest wave speed)."""
    rng = np.random.default_rng([seed, mx, my])
    X, Y, dx, dy, lx, ly = _grid(mx, my)
    q = torch.zeros((SOLVERS[solver]["num_eqn"], my, mx), dtype=F64, device="cuda")
    if solver in ("euler4", "euler5"):
        # a planar shock running into still air and a light bubble, the flow behind the shock already stirred
        pinf = rng.uniform(3.0, 6.0)
        r2 = (GAMMA - 1 + pinf * (GAMMA + 1)) / ((GAMMA + 1) + (GAMMA - 1) * pinf)
        u2 = (pinf - 1) / math.sqrt(0.5 * ((GAMMA + 1) * pinf + GAMMA - 1))
        behind = X < rng.uniform(0.35, 0.55) * lx
        bubble = (X - rng.uniform(0.6, 0.7) * lx) ** 2 + (Y - rng.uniform(0.3, 0.7) * ly) ** 2 < (0.12 * min(lx, 2 * ly)) ** 2
        stir = behind.to(F64)
        rho = torch.where(behind, torch.full_like(X, r2), torch.where(bubble, 0.1, 1.0)) * (1 + stir * _modes(rng, X, Y, 8, 0.8))
        u = stir * (u2 + _modes(rng, X, Y, 6, 0.8))
        v = stir * _modes(rng, X, Y, 6, 0.8)
        p = torch.where(behind, torch.full_like(X, pinf), torch.ones_like(X)) * (1 + stir * _modes(rng, X, Y, 6, 0.3))
        q[0], q[1], q[2] = rho, rho * u, rho * v
        q[3] = p / (GAMMA - 1) + 0.5 * rho * (u * u + v * v)
        if solver == "euler5":
            q[4] = bubble.to(F64)
        return q, None, dx, dy, 2.0 * (u2 + math.sqrt(GAMMA * 2.0 * pinf / r2))
    if solver == "shallow":
        cx, cy = rng.uniform(0.4, 0.6, 2)
        r = torch.sqrt((X - cx * lx) ** 2 + (Y - cy * ly) ** 2)
        q[0] = torch.where(r < 0.1 * min(lx, ly), 2.0, 1.0)
        if data == "waves":
            q[0] += _modes(rng, X, Y, 8, 0.5)
            q[1] = q[0] * _modes(rng, X, Y, 8, 0.4)
            q[2] = q[0] * _modes(rng, X, Y, 8, 0.4)
        return q, None, dx, dy, 3.0
    width = 0.05 * min(lx, ly)
    for _ in range(3):
        cx, cy = rng.uniform(0.2, 0.8, 2)
        q[0] += rng.uniform(0.5, 1.0) * torch.exp(-((X - cx * lx) ** 2 + (Y - cy * ly) ** 2) / width ** 2)
    if solver == "acoustics":
        return q, None, dx, dy, 2.0
    if solver == "vc":
        n = int(rng.integers(2, 7))
        cuts = np.sort(rng.uniform(0, lx, n - 1))
        layer = torch.bucketize(X.contiguous(), torch.tensor(cuts, dtype=F64, device="cuda"))
        rho = torch.tensor(rng.uniform(1, 4, n), dtype=F64, device="cuda")[layer]
        K = torch.tensor(rng.uniform(1, 4, n), dtype=F64, device="cuda")[layer]
        return q, torch.stack([rho, torch.sqrt(K / rho)]), dx, dy, 2.0
    # psystem: a checkerboard of two materials, stress sigma = exp(K eps) - 1
    odd = (torch.floor(X / lx * 20) + torch.floor(Y / ly * 20)) % 2
    K = 1.0 + 3.0 * odd
    q[0] = torch.log(1 + 4 * q[0]) / K
    return q, torch.stack([K, K, torch.full_like(K, 2.0), q[0]]), dx, dy, 2.5


def _fill(a, lo, hi, negate):
    """Ghost cells of [m, j, i] (already padded): x sides, then y sides."""
    for axis, dim in ((0, 2), (1, 1)):
        n = a.shape[dim] - 2 * G
        for g in range(G):
            for upper, bc in ((False, lo[axis]), (True, hi[axis])):
                if bc == 0:
                    continue
                dst = n + G + g if upper else G - 1 - g
                if bc == 1:
                    src = n + G - 1 if upper else G
                elif bc == 2:
                    src = G + g if upper else n + G - 1 - g
                else:
                    src = n + G - 1 - g if upper else G + g
                v = a.select(dim, src).clone()
                if bc == 3 and negate:
                    v[axis + 1] = -v[axis + 1]
                a.select(dim, dst).copy_(v)
    return a


def _ghosted(q, lo, hi, negate):
    a = torch.zeros((q.shape[0], q.shape[1] + 2 * G, q.shape[2] + 2 * G), dtype=F64, device=q.device)
    a[:, G:-G, G:-G] = q
    return _fill(a, lo, hi, negate)


def _cfl(case):
    return (0.5, 0.45) if case["mode"] == 0 else (1.0, 0.9)


def _problem(case, dx, dy):
    lo, hi = BCS[case["bc"]]
    return _abi.make_problem(mx=case["mx"], my=case["my"], dx=dx, dy=dy, order=case["order"], transverse=case["mode"],
                             mthlim=(case["lim"],), bc_lower=lo, bc_upper=hi, aux_bc_lower=lo, aux_bc_upper=hi,
                             use_fwave=case["solver"] == "psystem", **SOLVERS[case["solver"]])


# ---------------------------------------------------------------------------
# prepare / run
# ---------------------------------------------------------------------------
def prepare(case, seed):
    return globals()["_prepare_" + case["kind"]](case, seed)


def run(state):
    return state["run"](state)


def _prepare_loop(case, seed):
    from pyclaw_b200.device import DeviceState
    q, aux, dx, dy, smax = _initial(case["solver"], case["data"], case["mx"], case["my"], seed)
    dev = DeviceState(_problem(case, dx, dy))
    lo, hi = BCS[case["bc"]]
    q0 = torch.zeros_like(dev.qview(0))
    q0[:, :, :case["mx"] + 2 * G] = _ghosted(q, lo, hi, True)
    if aux is not None:
        dev.aux.view(aux.shape[0], dev.L.rows, dev.L.ld)[:, :, :case["mx"] + 2 * G] = _ghosted(aux, lo, hi, False)
    hooks = None
    if case["solver"] == "psystem":            # the application copies the strain into aux before each step
        hooks = _abi.Hooks()
        hooks.aux_from_q, hooks.aux_q = 4, 1
    return dict(run=_run_loop, dev=dev, q0=q0, hooks=hooks, dt=0.5 * _cfl(case)[0] * min(dx, dy) / smax, case=case)


def _run_loop(s):
    dev, case = s["dev"], s["case"]
    dev.qview(0).copy_(s["q0"])
    dev.cur = 0
    cfl_max, cfl_desired = _cfl(case)
    c = _abi.Control()
    _lib.check(dev.lib.claw2_control_init(ctypes.byref(c), 0.0, s["dt"], 1e9, cfl_max, cfl_desired, 1e99, 1, 0,
                                          case["steps"], cfl_desired), "claw2_control_init")
    out = dev.evolve(c, hooks=s["hooks"])
    return {"q": dev.interior(dev.cur), "t": out.t, "dt": out.dt, "cfl": out.cfl, "numsteps": int(out.numsteps)}


def _prepare_batch(case, seed):
    from pyclaw_b200.batch import BatchSolver
    insts = [dict(q=q, aux=aux, dx=dx, dy=dy, dt=dt) for q, aux, dx, dy, dt in _instances(case, seed)]
    prob = _abi.make_problem(mx=64, my=64, dx=1.0, dy=1.0, order=2, transverse=2, mthlim=(case["lim"],),
                             bc_lower=(3, 3), bc_upper=(1, 1), aux_bc_lower=(3, 3), aux_bc_upper=(1, 1),
                             **SOLVERS["vc"])
    bs = BatchSolver(prob, insts)
    bs.autotune(steps=2, repeats=1)
    return dict(run=_run_batch, bs=bs, q0=bs.qarena.clone(), dts=[i["dt"] for i in insts], case=case)


def _instances(case, seed):
    sizes = np.random.default_rng([case["n"], case["nmin"], case["nmax"]])      # the same grids for every seed
    rng = np.random.default_rng([seed, case["n"]])
    for _ in range(case["n"]):
        nx, ny = (int(v) for v in sizes.integers(case["nmin"], case["nmax"] + 1, 2))
        n = int(rng.integers(2, 7))
        cuts = np.sort(rng.uniform(0, 1, n - 1))
        rho, K = rng.uniform(1, 4, n), rng.uniform(1, 4, n)
        x, y = (np.arange(nx) + 0.5) / nx, (np.arange(ny) + 0.5) / ny
        layer = np.searchsorted(cuts, x)
        aux = np.empty((2, nx, ny), order="F")
        aux[0], aux[1] = rho[layer][:, None], np.sqrt(K / rho)[layer][:, None]
        x0, y0 = rng.uniform(0.1, 0.9, 2)
        q = np.zeros((3, nx, ny), order="F")
        q[0] = np.exp(-((x - x0) / 0.05) ** 2)[:, None] * np.exp(-((y - y0) / 0.05) ** 2)[None, :]
        yield q, aux, 1.0 / nx, 1.0 / ny, 0.9 * min(1.0 / nx, 1.0 / ny) / float(np.sqrt(K / rho).max())


def _run_batch(s):
    bs, case = s["bs"], s["case"]
    bs.qarena.copy_(s["q0"])
    bs.init_controls(s["dts"], max_steps=case["steps"])
    bs.advance_graph(case["steps"], chunk=case["steps"])
    ctl = bs.controls()
    k = max(range(bs.n), key=lambda i: bs.problems[i].mx * bs.problems[i].my)
    return {"largest": bs._qview(k, ctl[k].cur)[:, G:G + bs.problems[k].my, G:G + bs.problems[k].mx],
            "states": bs.qarena, "t": np.array([c.t for c in ctl]), "dt": np.array([c.dt for c in ctl]),
            "numsteps": np.array([c.numsteps for c in ctl])}


def _shots_setup(case, seed):
    rng = np.random.default_rng([seed, case["mx"], case["shots"]])
    mx, my, n = case["mx"], case["my"], case["steps"]
    dx, dy = 2.0 / mx, 2.0 / my
    x, y = -1 + (np.arange(mx) + 0.5) * dx, -1 + (np.arange(my) + 0.5) * dy
    X, Y = np.meshgrid(x, y, indexing="ij")
    rho, K = np.ones((mx, my)), np.full((mx, my), 4.0)
    for _ in range(3):
        cx, cy = rng.uniform(-0.6, 0.6), rng.uniform(-0.7, 0.3)
        inside = (X - cx) ** 2 + (Y - cy) ** 2 < 0.3 ** 2
        rho[inside], K[inside] = rng.uniform(1.5, 3.0), rng.uniform(2.0, 8.0)
    dt = 0.8 * min(dx, dy) / math.sqrt(8.0 / 1.0)
    q0 = np.zeros((case["shots"], 3, mx, my))
    for s in range(case["shots"]):              # the wavefield some way into the run, its pulse under way
        cx, cy = rng.uniform(-0.7, 0.7, 2)
        q0[s, 0] = np.exp(-((X - cx) ** 2 + (Y - cy) ** 2) / 0.15 ** 2)
    a = (np.pi * 15.0 * (dt * (np.arange(n) + 1) - 0.02)) ** 2
    wav = (1 - 2 * a) * np.exp(-a) * 0.3
    src = [int(i) + mx * (my - 1) for i in rng.integers(0, mx, case["shots"])]
    rec = [int(i) + mx * (my - 1) for i in np.linspace(0, mx - 1, case["nrec"]).round()]
    target = rng.normal(0, 0.1, (n, case["shots"], case["nrec"]))
    return rho, K, q0, wav, src, rec, target, dx, dy, dt


def _prepare_shots(case, seed):
    from pyclaw_b200.adjoint import AcousticShots
    rho, K, q0, wav, src, rec, target, dx, dy, dt = _shots_setup(case, seed)
    runner = AcousticShots(case["mx"], case["my"], dx, dy, case["shots"], src, rec, wav, dt, bc_lower=(1, 1),
                           bc_upper=(1, 3), order=2, transverse=2, limiters=(case["lim"],) * 2,
                           checkpoint=("uniform", case["every"]))
    cu = lambda v: torch.tensor(v, dtype=F64, device="cuda")                                  # noqa: E731
    return dict(run=_run_shots, runner=runner, q0=cu(q0).requires_grad_(), rho=cu(rho).requires_grad_(),
                K=cu(K).requires_grad_(), target=cu(target))


def _run_shots(s):
    from pyclaw_b200.adjoint import material_aux, shots_traces
    traces = shots_traces(s["q0"], material_aux(s["rho"], s["K"]), s["runner"])
    loss = 0.5 * ((traces - s["target"]) ** 2).sum()
    gq, gr, gk = torch.autograd.grad(loss, [s["q0"], s["rho"], s["K"]])
    return {"traces": traces.detach(), "g_q0": gq, "g_rho": gr, "g_K": gk}


def _app_data(case, seed):
    """apps/euler_2d/shockbubble.py's set-up (classic solver), the bubble's place and the shock's strength varied."""
    rng = np.random.default_rng([seed, case["mx"]])
    mx, my = case["mx"], case["my"]
    pinf = rng.uniform(4.0, 6.0)
    rinf = (GAMMA - 1 + pinf * (GAMMA + 1)) / ((GAMMA + 1) + (GAMMA - 1) * pinf)
    vinf = (pinf - 1) / math.sqrt(GAMMA) / math.sqrt(0.5 * ((GAMMA + 1) / GAMMA) * pinf + 0.5 * (GAMMA - 1) / GAMMA)
    einf = 0.5 * rinf * vinf ** 2 + pinf / (GAMMA - 1)
    x, y = (np.arange(mx) + 0.5) * (2.0 / mx), (np.arange(my) + 0.5) * (0.5 / my)
    X, Y = np.meshgrid(x, y, indexing="ij")
    inside = (X - rng.uniform(0.45, 0.6)) ** 2 + Y ** 2 < 0.2 ** 2
    shock = X < 0.2
    q = np.zeros((5, mx, my), order="F")
    q[0] = np.where(shock, rinf, np.where(inside, 0.1, 1.0))
    q[1] = np.where(shock, rinf * vinf, 0.0)
    q[3] = np.where(shock, einf, 1.0 / (GAMMA - 1))
    q[4] = inside
    aux = np.empty((1, mx, my), order="F")
    aux[0] = Y
    return q, aux, [rinf, rinf * vinf, 0.0, einf, 0.0]


APP_DT, APP_CFL = 0.002, (0.5, 0.45)


def _prepare_app(case, seed):
    import pyclaw_b200 as pc
    from pyclaw_b200 import hooks
    q, aux, inflow = _app_data(case, seed)
    x, y = pc.Dimension("x", 0.0, 2.0, case["mx"]), pc.Dimension("y", 0.0, 0.5, case["my"])
    domain = pc.Domain([x, y])
    st = pc.State(domain, 5, 1)
    st.problem_data["gamma"], st.problem_data["gamma1"] = GAMMA, GAMMA - 1.0
    st.q[...] = q
    st.aux[...] = aux
    sol = pc.ClawSolver2D(pc.riemann.rp2_euler_5wave)
    sol.limiters = [4, 4, 4, 4, 2]
    sol.cfl_max, sol.cfl_desired = APP_CFL
    sol.dt_initial = APP_DT
    sol.bc_lower, sol.bc_upper = [pc.BC.custom, pc.BC.wall], [pc.BC.extrap, pc.BC.extrap]
    sol.aux_bc_lower, sol.aux_bc_upper = [pc.BC.extrap] * 2, [pc.BC.extrap] * 2
    sol.user_bc_lower = hooks.FixedStateBC(inflow)
    sol.step_source = hooks.EulerRadialSource(0)
    solution = pc.Solution(st, domain)
    sol.setup(solution)
    return dict(run=_run_app, solver=sol, solution=solution, q=q, case=case)


def _run_app(s):
    sol, solution = s["solver"], s["solution"]
    solution.state.q = s["q"]
    solution.t = 0.0
    sol.dt = APP_DT
    sol.evolve_to_time(solution, s["case"]["tend"])
    return {"q": solution.state.get_q_host(), "t": float(solution.t), "dt": float(sol.dt),
            "numsteps": int(sol.status["numsteps"])}


class _Session(object):
    """The host-buffer session, closed with its owner."""

    def __init__(self, prob):
        self.lib, self.h = _lib.load(), ctypes.c_void_p()
        _lib.check(self.lib.claw2_session_create(ctypes.byref(prob), ctypes.byref(self.h)), "claw2_session_create")

    def __del__(self):
        self.lib.claw2_session_destroy(self.h)


def _host_arrays(case, seed):
    """qbc and auxbc with ghost cells in the reference's layout (m fastest), on the host, and dx, dy, dt."""
    q, aux, dx, dy, smax = _initial(case["solver"], case["data"], case["mx"], case["my"], seed)
    lo, hi = BCS[case["bc"]]
    ref = lambda a, neg: _ghosted(a, lo, hi, neg).permute(1, 2, 0).contiguous().cpu().pin_memory()   # noqa: E731
    return ref(q, True), None if aux is None else ref(aux, False), dx, dy, 0.9 * _cfl(case)[0] * min(dx, dy) / smax


def _prepare_host(case, seed):
    qold, aux, dx, dy, dt = _host_arrays(case, seed)
    return dict(run=_run_host, session=_Session(_problem(case, dx, dy)), qold=qold, qnew=torch.empty_like(qold).pin_memory(),
                aux=aux, dt=dt)


def _run_host(s):
    cfl = ctypes.c_double()
    _lib.check(s["session"].lib.claw2_session_step2(
        s["session"].h, s["qold"].data_ptr(), s["qnew"].data_ptr(), None if s["aux"] is None else s["aux"].data_ptr(),
        s["dt"], ctypes.byref(cfl)), "claw2_session_step2")
    return {"q": s["qnew"], "cfl": cfl.value}


# ---------------------------------------------------------------------------
# work: a step reads the state (and aux) and writes the new state once; the
# steps of a pass depend on one another through the global CFL number
# ---------------------------------------------------------------------------
def work(case):
    kind = case["kind"]
    if kind in ("loop", "host"):
        s = SOLVERS[case["solver"]]
        cells, steps = case["mx"] * case["my"], case.get("steps", 1)
        return {"bytes": 8.0 * (2 * s["num_eqn"] + s["num_aux"]) * cells * steps,
                "flops": FLOPS[case["solver"]] * (0.55 if case["mode"] <= 0 else 1.0) * cells * steps}
    if kind == "app":
        cells = case["mx"] * case["my"]
        steps = 1 + case["tend"] / (0.45 * (2.0 / case["mx"]) / 4.5)
        return {"bytes": 8.0 * 11 * cells * steps, "flops": 600.0 * cells * steps}
    if kind == "batch":
        cells = case["n"] * ((case["nmin"] + case["nmax"]) / 2.0) ** 2
        return {"bytes": 8.0 * 8 * cells * case["steps"], "flops": FLOPS["vc"] * cells * case["steps"]}
    # a forward step, its recomputation and an adjoint step (about three times the forward's operations) per step
    cells = case["mx"] * case["my"] * case["shots"] * case["steps"]
    return {"bytes": 8.0 * (6 + 6 + 13) * cells, "flops": 5.0 * FLOPS["vc"] * cells}


# ---------------------------------------------------------------------------
# exact: the same step in plain torch, 64 bits
# ---------------------------------------------------------------------------
def _limiter(r, lim):
    """TVD limiter of r; ties take the branch that the comparisons below take."""
    one = torch.ones_like(r)
    if lim == 3:
        return (r + r.abs()) / (1 + r.abs())
    if lim == 2:
        t, w = torch.where(1 < 2 * r, one, 2 * r), torch.where(2 < r, 2 * one, r)
        t = torch.where(t > w, t, w)
    elif lim == 4:
        t = torch.where((1 + r) / 2 < 2, (1 + r) / 2, 2 * one)
        t = torch.where(t < 2 * r, t, 2 * r)
    else:
        t = torch.where(1 < r, one, r)
    return torch.where(0 > t, torch.zeros_like(t), t)


def _rpn_linear(qL, qR, aL, aR, prm):
    """Acoustics: constant (aL is None) or variable coefficients."""
    if aL is None:
        cL = cR = torch.full_like(qL[0], prm[2])
        zL = zR = torch.full_like(qL[0], prm[3])
    else:
        cL, cR, zL, zR = aL[1], aR[1], aL[0] * aL[1], aR[0] * aR[1]
    d1, d2 = qR[0] - qL[0], qR[1] - qL[1]
    b1, b2 = (-d1 + zR * d2) / (zL + zR), (d1 + zL * d2) / (zL + zR)
    o = torch.zeros_like(b1)
    W, s = [torch.stack([-b1 * zL, b1, o]), torch.stack([b2 * zR, b2, o])], [-cL, cR]
    return W, s, s[0] * W[0], s[1] * W[1], None


def _rpt_linear(a, asdq, ctx, a1, a2, a3, prm):
    if a1 is None:
        cm = cp = torch.full_like(asdq[0], prm[2])
        zm = zz = zp = torch.full_like(asdq[0], prm[3])
    else:
        cm, cp, zm, zz, zp = a1[1], a3[1], a1[0] * a1[1], a2[0] * a2[1], a3[0] * a3[1]
    b1, b2 = (-asdq[0] + zz * asdq[2]) / (zm + zz), (asdq[0] + zz * asdq[2]) / (zz + zp)
    o = torch.zeros_like(b1)
    return torch.stack([cm * b1 * zm, o, -cm * b1]), torch.stack([cp * b2 * zp, o, cp * b2])


def _psys(aux, eps):
    e = torch.exp(aux[1] * eps)
    c = torch.sqrt(aux[1] * e / aux[0])
    return e - 1, c, aux[0] * c


def _rpn_psystem(qL, qR, aL, aR, prm):
    sL, cL, zL = _psys(aL, qL[0])
    sR, cR, zR = _psys(aR, qR[0])
    f1, f2 = -(qR[1] / aR[0]) + qL[1] / aL[0], sL - sR
    b1, b2 = (zR * f1 + f2) / (zL + zR), (zL * f1 - f2) / (zL + zR)
    o = torch.zeros_like(b1)
    W = [torch.stack([b1, b1 * zL, o]), torch.stack([b2, -b2 * zR, o])]
    return W, [-cL, cR], W[0], W[1], None


def _rpt_psystem(a, asdq, ctx, a1, a2, a3, prm):
    _, cb, zb = _psys(a1, a1[3])
    _, ca, za = _psys(a3, a3[3])
    gb, ga = (za * asdq[0] + asdq[2]) / (zb + za), (zb * asdq[0] - asdq[2]) / (zb + za)
    o = torch.zeros_like(gb)
    return torch.stack([-cb * gb, o, -cb * gb * zb]), torch.stack([ca * ga, o, -ca * ga * za])


def _transonic(s0, s1, sr):
    """Harten-Hyman: the part of a genuinely nonlinear wave that goes left."""
    return torch.where((s0 < 0) & (s1 > 0), s0 * (s1 - sr) / (s1 - s0), torch.where(sr < 0, sr, torch.zeros_like(sr)))


def _rpn_euler(qL, qR, aL, aR, prm):
    g, g1 = prm
    tracer = qL.shape[0] == 5

    def press(q):
        return g1 * (q[3] - 0.5 * (q[1] ** 2 + q[2] ** 2) / q[0])
    pL, pR, rl, rr = press(qL), press(qR), torch.sqrt(qL[0]), torch.sqrt(qR[0])
    u, v = (qL[1] / rl + qR[1] / rr) / (rl + rr), (qL[2] / rl + qR[2] / rr) / (rl + rr)
    H = ((qL[3] + pL) / rl + (qR[3] + pR) / rr) / (rl + rr)
    a2 = g1 * (H - 0.5 * (u * u + v * v))
    a = torch.sqrt(a2)
    d = qR - qL
    b3 = g1 / a2 * ((H - u * u - v * v) * d[0] + u * d[1] + v * d[2] - d[3])
    b2 = d[2] - v * d[0]
    b4 = (d[1] + (a - u) * d[0] - a * b3) / (2 * a)
    b1 = d[0] - b3 - b4
    o = torch.zeros_like(u)
    pad = [o] if tracer else []
    W = [torch.stack([b1, b1 * (u - a), b1 * v, b1 * (H - u * a)] + pad), torch.stack([o, o, b2, b2 * v] + pad),
         torch.stack([b3, b3 * u, b3 * v, b3 * 0.5 * (u * u + v * v)] + pad),
         torch.stack([b4, b4 * (u + a), b4 * v, b4 * (H + u * a)] + pad)]
    s = [u - a, u, u, u + a]
    if tracer:
        W.append(torch.stack([o, o, o, o, d[4]]))
        s.append(u)
    s0 = qL[1] / qL[0] - torch.sqrt(g * pL / qL[0])
    m = qL + W[0]
    s1 = m[1] / m[0] - torch.sqrt(g * press(m) / m[0])
    n = qR - W[3]
    s2 = n[1] / n[0] + torch.sqrt(g * press(n) / n[0])
    s3 = qR[1] / qR[0] + torch.sqrt(g * pR / qR[0])
    am = _transonic(s0, s1, s[0]) * W[0]
    mid = u * (W[1] + W[2]) + (u * W[4] if tracer else 0)
    am = torch.where(u < 0, am + mid + _transonic(s2, s3, s[3]) * W[3], am)
    am = torch.where((s0 >= 0) & (s[0] > 0), torch.zeros_like(am), am)
    return W, s, am, sum(sp * w for sp, w in zip(s, W)) - am, (u, v, a, H, g1 / a2)


def _rpt_euler(a_, x, ctx, a1, a2, a3, prm):
    u, v, a, H, g1a2 = ctx
    b3 = g1a2 * ((H - u * u - v * v) * x[0] + u * x[1] + v * x[2] - x[3])
    b2 = x[1] - u * x[0]
    b4 = (x[2] + (a - v) * x[0] - a * b3) / (2 * a)
    b1 = x[0] - b3 - b4
    W = [torch.stack([b1, b1 * u, b1 * (v - a), b1 * (H - v * a)]),
         torch.stack([b3, b3 * u + b2, b3 * v, b3 * 0.5 * (u * u + v * v) + b2 * u]),
         torch.stack([b4, b4 * u, b4 * (v + a), b4 * (H + v * a)])]
    s = [v - a, v, v + a]
    bm, bp = sum(sp.clamp(max=0) * w for sp, w in zip(s, W)), sum(sp.clamp(min=0) * w for sp, w in zip(s, W))
    if x.shape[0] == 5:
        bm, bp = torch.cat([bm, (v.clamp(max=0) * x[4])[None]]), torch.cat([bp, (v.clamp(min=0) * x[4])[None]])
    return bm, bp


def _rpn_shallow(qL, qR, aL, aR, prm):
    g = prm[0]
    hl, hr = torch.sqrt(qL[0]), torch.sqrt(qR[0])
    u, v = (qL[1] / hl + qR[1] / hr) / (hl + hr), (qL[2] / hl + qR[2] / hr) / (hl + hr)
    c = torch.sqrt(g * 0.5 * (qL[0] + qR[0]))
    d = qR - qL
    b1, b2, b3 = ((u + c) * d[0] - d[1]) / (2 * c), d[2] - v * d[0], (d[1] - (u - c) * d[0]) / (2 * c)
    o = torch.zeros_like(u)
    W = [torch.stack([b1, b1 * (u - c), b1 * v]), torch.stack([o, o, b2]), torch.stack([b3, b3 * (u + c), b3 * v])]
    s = [u - c, u, u + c]
    s0, s3 = qL[1] / qL[0] - torch.sqrt(g * qL[0]), qR[1] / qR[0] + torch.sqrt(g * qR[0])
    m, n = qL + W[0], qR - W[2]
    s1, s2 = m[1] / m[0] - torch.sqrt(g * m[0]), n[1] / n[0] + torch.sqrt(g * n[0])
    am = _transonic(s0, s1, s[0]) * W[0]
    am = torch.where(u < 0, am + u * W[1] + _transonic(s2, s3, s[2]) * W[2], am)
    am = torch.where((s0 >= 0) & (s[0] > 0), torch.zeros_like(am), am)
    return W, s, am, sum(sp * w for sp, w in zip(s, W)) - am, (u, v, c)


def _rpt_shallow(a_, x, ctx, a1, a2, a3, prm):
    u, v, c = ctx
    b1, b2, b3 = ((v + c) * x[0] - x[2]) / (2 * c), x[1] - u * x[0], (x[2] - (v - c) * x[0]) / (2 * c)
    o = torch.zeros_like(u)
    W = [torch.stack([b1, b1 * u, b1 * (v - c)]), torch.stack([o, b2, o]), torch.stack([b3, b3 * u, b3 * (v + c)])]
    s = [v - c, v, v + c]
    return sum(sp.clamp(max=0) * w for sp, w in zip(s, W)), sum(sp.clamp(min=0) * w for sp, w in zip(s, W))


RPN = {"acoustics": _rpn_linear, "vc": _rpn_linear, "euler4": _rpn_euler, "euler5": _rpn_euler,
       "shallow": _rpn_shallow, "psystem": _rpn_psystem}
RPT = {"acoustics": _rpt_linear, "vc": _rpt_linear, "euler4": _rpt_euler, "euler5": _rpt_euler,
       "shallow": _rpt_shallow, "psystem": _rpt_psystem}


def _slices(o, q, aux, dtd):
    """The 1D slices q[m, line, cell] (ghost cells along the slice) of one
    direction, momentum along the slice second: per interior cell the
    fluctuation and correction updates and, with transverse waves, the two
    transverse fluxes; and the CFL number.  aux has one line more on each side."""
    rpn, rpt, prm = RPN[o["solver"]], RPT[o["solver"]], SOLVERS[o["solver"]]["params"]
    a2 = None if aux is None else aux[:, 1:-1]
    aL, aR = (None, None) if aux is None else (a2[..., :-1], a2[..., 1:])
    W, s, am, ap, ctx = rpn(q[..., :-1], q[..., 1:], aL, aR, prm)
    used = slice(1, -1)                                   # interfaces of interior cells
    cfl = max(float((dtd * sp[..., used]).abs().max()) for sp in s)
    cq = torch.zeros_like(am)
    if o["order"] == 2:
        for w, sp, lim in zip(W, s, o["lims"]):
            lw = w
            if lim:
                wn, dot = (w * w).sum(0), torch.zeros_like(sp)
                dr = (w[..., :-1] * w[..., 1:]).sum(0)
                dot[..., used] = torch.where(sp[..., used] > 0, dr[..., :-1], dr[..., 1:])
                # a wave too small to square changes nothing that can be seen
                ok = wn > 1e-290
                phi = _limiter(dot / torch.where(ok, wn, torch.ones_like(wn)), lim)
                lw = torch.where(ok, phi, torch.ones_like(phi)) * w
            f = torch.sign(sp) * (1 - sp.abs() * dtd) if o["solver"] == "psystem" else sp.abs() * (1 - sp.abs() * dtd)
            cq = cq + f * lw
    n = q.shape[-1] - 2 * G
    L, R = slice(1, n + 1), slice(2, n + 2)               # the left and right interfaces of the interior cells
    qadd = -dtd * (ap[..., L] + am[..., R])
    dF = 0.5 * (cq[..., R] - cq[..., L])
    if o["mode"] <= 0:
        return qadd, dF, None, None, cfl
    k = 1.0 if o["mode"] == 2 else 0.0
    lines = (None,) * 3 if aux is None else (aux[:, :-2], aux[:, 1:-1], aux[:, 2:])
    left = [None if b is None else b[..., :-1] for b in lines]
    right = [None if b is None else b[..., 1:] for b in lines]
    bmL, bpL = rpt(1, am + k * cq, ctx, *left, prm)
    bmR, bpR = rpt(2, ap - k * cq, ctx, *right, prm)
    return qadd, dF, -0.5 * dtd * (bmL[..., R] + bmR[..., L]), -0.5 * dtd * (bpL[..., R] + bpR[..., L]), cfl


def _turn(a, q):
    """[m, j, i] <-> [m, i, j], with the momentum along the slice second (q only)."""
    if a is None:
        return None
    a = a.transpose(1, 2)
    return a if not q else torch.cat([a[:1], a[2:3], a[1:2], a[3:]])


def _exact_step(o, q, aux, dt):
    """One step of the ghosted q[m, j, i]; returns (interior, CFL number)."""
    dtx, dty = dt / o["dx"], dt / o["dy"]
    if o["mode"] < 0:
        pad = None if aux is None else torch.cat([aux[:, :1], aux, aux[:, -1:]], 1)
        qa, dF, _, _, cx = _slices(o, q, pad, dtx)
        mid = q.clone()
        mid[..., G:-G] = q[..., G:-G] + qa - dtx * dF
        t, ta = _turn(mid, True), _turn(aux, False)
        pad = None if ta is None else torch.cat([ta[:, :1], ta, ta[:, -1:]], 1)
        qa, dF, _, _, cy = _slices(o, t, pad, dty)
        return _turn(t[..., G:-G] + qa - dty * dF, True)[:, :, G:-G], max(cx, cy)
    qa, dF, g1, g2, cx = _slices(o, q[:, 1:-1], aux, dtx)
    v = q[:, G:-G, G:-G] + qa[:, 1:-1] - dtx * dF[:, 1:-1]
    if o["mode"] > 0:
        v = v + dty * (g2[:, :-2] - (g2 - g1)[:, 1:-1] - g1[:, 2:])
    qa, dF, g1, g2, cy = _slices(o, _turn(q, True)[:, 1:-1], _turn(aux, False), dty)
    w = qa[:, 1:-1] - dty * dF[:, 1:-1]
    if o["mode"] > 0:
        w = w + dtx * (g2[:, :-2] - (g2 - g1)[:, 1:-1] - g1[:, 2:])
    return v + _turn(w, True), max(cx, cy)


def _evolve(o, q, aux, dt, cfl_max, cfl_desired, steps=None, tend=None, fill=None, before=None, source=None):
    """Solver.evolve_to_time: (ghosted q, t, dt, CFL number, accepted steps)."""
    t, done, cfl, it = 0.0, 0, cfl_desired, 0
    while steps is None or it < steps:
        if tend is not None:
            if t + dt > tend or tend - t - dt < 1e-14 * t:
                dt = tend - t
        if before is not None:
            before(q, aux)
        v, cfl = _exact_step(o, q, aux, dt)
        it += 1
        if cfl <= cfl_max:
            q = q.clone()
            q[:, G:-G, G:-G] = v if source is None else source(v, dt)
            fill(q)
            t += dt
            done += 1
        dt = dt * cfl_desired / cfl
        if tend is not None and t >= tend:
            break
    return q, t, dt, cfl, done


def exact(case, seed):
    return globals()["_exact_" + case["kind"]](case, seed)


def _options(case, dx, dy):
    return dict(solver=case["solver"], mode=case["mode"], order=case["order"],
                lims=[case["lim"]] * SOLVERS[case["solver"]]["num_waves"], dx=dx, dy=dy)


def _exact_loop(case, seed):
    q, aux, dx, dy, smax = _initial(case["solver"], case["data"], case["mx"], case["my"], seed)
    lo, hi = BCS[case["bc"]]
    cfl_max, cfl_desired = _cfl(case)

    def before(q, aux):
        aux[3] = q[0]
    q, t, dt, cfl, n = _evolve(_options(case, dx, dy), _ghosted(q, lo, hi, True),
                               None if aux is None else _ghosted(aux, lo, hi, False),
                               0.5 * cfl_max * min(dx, dy) / smax, cfl_max, cfl_desired, steps=case["steps"],
                               fill=lambda v: _fill(v, lo, hi, True),
                               before=before if case["solver"] == "psystem" else None)
    return {"q": q[:, G:-G, G:-G], "t": t, "dt": dt, "cfl": cfl, "numsteps": n}


def _exact_host(case, seed):
    qold, aux, dx, dy, dt = _host_arrays(case, seed)
    lo, hi = BCS[case["bc"]]
    dev = lambda a: None if a is None else a.cuda().permute(2, 0, 1).contiguous()              # noqa: E731
    v, cfl = _exact_step(_options(case, dx, dy), dev(qold), dev(aux), dt)
    return {"q": _ghosted(v, lo, hi, True).permute(1, 2, 0).contiguous(), "cfl": cfl}


def _exact_batch(case, seed):
    o = dict(solver="vc", mode=2, order=2, lims=[case["lim"]] * 2)
    insts = list(_instances(case, seed))
    k = max(range(len(insts)), key=lambda i: insts[i][0].shape[1] * insts[i][0].shape[2])
    q, aux, dx, dy, dt = insts[k]
    cu = lambda a: torch.tensor(np.ascontiguousarray(a.transpose(0, 2, 1)), device="cuda")     # noqa: E731
    lo, hi = (3, 3), (1, 1)
    out = _evolve(dict(o, dx=dx, dy=dy), _ghosted(cu(q), lo, hi, True), _ghosted(cu(aux), lo, hi, False), dt, 1.0, 0.9,
                  steps=case["steps"], fill=lambda v: _fill(v, lo, hi, True))
    return {"largest": out[0][:, G:-G, G:-G], "states": None, "t": None, "dt": None, "numsteps": None}


def _exact_app(case, seed):
    q, aux, inflow = _app_data(case, seed)
    cu = lambda a: torch.tensor(np.ascontiguousarray(a.transpose(0, 2, 1)), device="cuda")     # noqa: E731
    o = dict(solver="euler5", mode=-1, order=2, lims=[4, 4, 4, 4, 2], dx=2.0 / case["mx"], dy=0.5 / case["my"])
    rad = cu(aux)[0]

    def fill(a):
        a[:, :, :G] = torch.tensor(inflow, dtype=F64, device="cuda")[:, None, None]
        return _fill(a, (0, 3), (1, 1), True)

    def source(v, dt):
        def rhs(w):
            u, s = w[1] / w[0], w[2] / w[0]
            p = (GAMMA - 1) * (w[3] - 0.5 * w[0] * (u * u + s * s))
            return torch.stack([w[2], w[0] * u * s, w[0] * s * s, s * (w[3] + p), torch.zeros_like(u)]) / rad
        return v - dt * rhs(v - 0.5 * dt * rhs(v))
    q0 = torch.zeros((5, case["my"] + 2 * G, case["mx"] + 2 * G), dtype=F64, device="cuda")
    q0[:, G:-G, G:-G] = cu(q)
    out, t, dt, _, n = _evolve(o, fill(q0), None, APP_DT, APP_CFL[0], APP_CFL[1], tend=case["tend"], fill=fill,
                               source=source)
    return {"q": out[:, G:-G, G:-G].permute(0, 2, 1).contiguous(), "t": t, "dt": dt, "numsteps": n}


def _exact_shots(case, seed):
    rho, K, q0, wav, src, rec, target, dx, dy, dt = _shots_setup(case, seed)
    o = dict(solver="vc", mode=2, order=2, lims=[case["lim"]] * 2, dx=dx, dy=dy)
    cu = lambda a: torch.tensor(a, dtype=F64, device="cuda")                                   # noqa: E731
    rho, K = cu(rho).requires_grad_(), cu(K).requires_grad_()
    q0, wav, target = cu(q0).requires_grad_(), cu(wav), cu(target)
    mx, my = case["mx"], case["my"]
    lo, hi = (1, 1), (1, 3)

    def ghosts(a, negate):               # out of place, for autograd
        a = torch.cat([a[..., :1], a[..., :1], a, a[..., -1:], a[..., -1:]], -1)
        m = torch.stack([a[:, -1], a[:, -2]], 1)
        if negate:
            m = m * cu([1.0, 1.0, -1.0])[:, None, None]
        return torch.cat([a[:, :1], a[:, :1], a, m], 1)
    ri = torch.tensor([r % mx for r in rec], device="cuda")
    rj = torch.tensor([r // mx for r in rec], device="cuda")
    traces, grads = [], None
    for s in range(case["shots"]):
        aux = ghosts(torch.stack([rho, torch.sqrt(K / rho)]).transpose(1, 2), False)
        q, row = q0[s].transpose(1, 2), []
        spike = torch.zeros_like(q)
        spike[0, src[s] // mx, src[s] % mx] = 1.0
        for n in range(case["steps"]):
            q = _exact_step(o, ghosts(q, True), aux, dt)[0] + wav[n] * spike
            row.append(q[0][rj, ri])
        tr = torch.stack(row)
        g = torch.autograd.grad(0.5 * ((tr - target[:, s]) ** 2).sum(), [q0, rho, K])
        grads = g if grads is None else [a + b for a, b in zip(grads, g)]
        traces.append(tr.detach())
    return {"traces": torch.stack(traces, 1), "g_q0": grads[0], "g_rho": grads[1], "g_K": grads[2]}
