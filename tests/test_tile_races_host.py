"""The tile bodies' use of shared memory under a thread sanitizer: whole steps of small
grids, a host thread per CUDA thread of a CTA, barriers and shuffles as the device code
has them.  No access to shared or global memory may be unordered with a write, and the
result is the oracle's, bit for bit (a zero's sign aside)."""
import os
import subprocess

import numpy as np
import pytest

import gpu_helpers as H
from host_device import compile_host
from pyclaw_b200 import _abi

SOURCE = r"""
#include <cuda_runtime.h>
#include "../../include/claw2.h"
#include "claw2_lean.cuh"
#include "claw2_psystem.cuh"
#include "claw2_rows.cuh"

using namespace claw2;

static const int THREADS = 256;
static std::vector<double> smem(1 << 15);

template <class RP, int T, bool SPLIT> static void lean(StepArgs a, const TileId& t)
{
    using SM = LeanSmem<RP, T, THREADS, SPLIT>;
    constexpr int TR = SM::TR, MEQN = RP::MEQN;
    double *H = smem.data(), *Qx = H + SM::HS, *CX = Qx + SM::QX, *red = CX + SM::CX;
    const int i0 = t.bx * T, j0 = t.by * T;
    for (int m = 0; m < MEQN; m++)
        for (int r = 0; r < TR; r++)
            for (int c = 0; c < TR; c++)
                H[lean_hidx<MEQN, TR>(m, r, c)] =
                    i0 + c < a.mx + 4 && j0 + r < a.my + 4 ? a.qin[m * a.plane + (j0 + r) * a.ld + i0 + c] : 0.0;
    emu::run_cta(THREADS, [&] {
        DevCtx ctx{H};
        const double c = lean_tile_sweeps<RP, T, THREADS, SPLIT>(a, ctx, H, Qx, CX, i0, j0, a.dt / a.dx, a.dt / a.dy);
        ctx.sync();
        const bool bad = store_tile<MEQN, T, T, THREADS, SM::QP>(a, ctx, Qx, T * SM::QP, a.qout, i0, j0, a.dt);
        report_cell<THREADS>(a, ctx, t.ntiles, red, c, bad, false);
    });
}

int main(int argc, char** argv)
{
    // body meqn naux mx my mode dt mthlim prm0..prm3 file: the two arrays, then the result is written over them
    const std::string body = argv[1];
    const int meqn = atoi(argv[2]), naux = atoi(argv[3]);
    StepArgs a;
    std::memset(&a, 0, sizeof a);
    a.mx = atoi(argv[4]); a.my = atoi(argv[5]);
    a.ld = (a.mx + 4 + 15) / 16 * 16;
    a.plane = a.ld * (a.my + 4);
    a.dx = 1.0 / a.mx; a.dy = 1.0 / a.my; a.dt = atof(argv[7]);
    a.order = 2; a.trans = atoi(argv[6]); a.capa = -1; a.fwave = body == "psystem";
    a.limit_any = 1;
    for (int& m : a.mthlim) m = atoi(argv[8]);
    a.limit_first = a.mthlim[0];
    for (int k = 0; k < 4; k++) a.prm[k] = atof(argv[9 + k]);
    a.ghost_fused = 1;
    for (int d = 0; d < 2; d++) { a.bcl[d] = CLAW2_BC_WALL; a.bcu[d] = CLAW2_BC_EXTRAP; }
    std::vector<double> q(meqn * a.plane), out(q.size()), aux(naux * a.plane + 1);
    FILE* f = fopen(argv[13], "rb");
    if (fread(q.data(), 8, q.size(), f) != q.size() || fread(aux.data(), 8, naux * a.plane, f) != naux * (size_t)a.plane) return 3;
    fclose(f);
    unsigned header[16] = {0};
    double cfl = 0.0;
    a.qin = q.data(); a.qout = out.data(); a.aux = aux.data(); a.cfl_out = &cfl;
    a.ticket = header;
    a.partials = reinterpret_cast<double*>(header) + 1;
    const int t = body == "march" || body == "march_vc" ? 28 : body.find("28") != std::string::npos ? 28 : 12, rows = body[0] == 'm' ? 5 : t;
    const int nbx = (a.mx + t - 1) / t, nby = (a.my + rows - 1) / rows;
    for (int by = 0; by < nby; by++)
        for (int bx = 0; bx < nbx; bx++) {
            const TileId T{bx, by, nbx, nby, by * nbx + bx, nbx * nby};
            auto cta = [&](int n, auto run) { emu::run_cta(n, [&] { DevCtx ctx{smem.data()}; run(ctx); }); };
            if (body == "rows") cta(THREADS, [&](DevCtx& c) { rows_tile<false, 12, THREADS>(a, c, T); });
            else if (body == "rows_vc") cta(THREADS, [&](DevCtx& c) { rows_tile<true, 12, THREADS>(a, c, T); });
            else if (body == "rows28") cta(THREADS, [&](DevCtx& c) { rows_tile<false, 28, THREADS>(a, c, T); });
            else if (body == "psystem") cta(THREADS, [&](DevCtx& c) { psys_tile<12, THREADS>(a, c, T); });
            else if (body == "march") cta(MARCH_NT, [&](DevCtx&) { march_tile<RpAcoustics, true>(a, T, rows); });
            else if (body == "march_vc") cta(MARCH_NT, [&](DevCtx&) { march_tile<RpVcAcoustics, true>(a, T, rows); });
            else if (body == "euler_split") lean<RpEuler<false>, 12, true>(a, T);
            else if (body == "shallow_split") lean<RpShallow, 12, true>(a, T);
            else if (body == "shallow_split28") lean<RpShallow, 28, true>(a, T);
            else if (body == "shallow") lean<RpShallow, 12, false>(a, T);
            else return 4;
        }
    f = fopen(argv[13], "wb");
    fwrite(out.data(), 8, out.size(), f);
    fwrite(&cfl, 8, 1, f);
    fclose(f);
    return 0;
}
"""

# body -> solver, mode; the grids leave warps without a line in the last pass over the lines
BODIES = {"rows": ("acoustics", -1), "rows28": ("acoustics", -1), "rows_vc": ("vc_acoustics", -1),
          "euler_split": ("euler4", -1), "shallow_split": ("shallow", -1), "shallow_split28": ("shallow", -1),
          "shallow": ("shallow", 2), "psystem": ("psystem", 2), "march": ("acoustics", 2), "march_vc": ("vc_acoustics", 1)}


@pytest.fixture(scope="module")
def program(tmp_path_factory):
    d = tmp_path_factory.mktemp("tiles")
    probe = d / "probe.cpp"
    probe.write_text("int main() { return 0; }")
    ok = subprocess.run(["g++", "-fsanitize=thread", "-o", str(d / "probe"), str(probe)], capture_output=True).returncode == 0
    if not ok or subprocess.run([str(d / "probe")], capture_output=True).returncode:
        pytest.skip("no thread sanitizer on this machine")
    return compile_host(SOURCE, d / "src", shared=False, flags=["-fsanitize=thread"])


@pytest.mark.parametrize("shape", [(5, 7), (14, 6)])
@pytest.mark.parametrize("body", sorted(BODIES))
def test_no_unordered_access(orc, program, tmp_path, body, shape):
    solver, mode = BODIES[body]
    bcs = dict(bcl=(3, 3), bcu=(1, 1), abcl=(3, 3), abcu=(1, 1))
    if solver == "psystem":
        p = _abi.make_problem(rp=_abi.RP_PSYSTEM, num_eqn=3, num_waves=2, num_aux=4, mx=shape[0], my=shape[1],
                              dx=1.0 / shape[0], dy=1.0 / shape[1], order=2, transverse=mode, mthlim=[4], use_fwave=True,
                              bc_lower=(3, 3), bc_upper=(1, 1), aux_bc_lower=(3, 3), aux_bc_upper=(1, 1))
        rng = np.random.default_rng(1)
        q, aux = np.asfortranarray(0.1 * rng.standard_normal((3,) + shape)), np.ones((4,) + shape, order="F")
        aux[3] = q[0]
    else:
        p = H.problem(solver, shape[0], shape[1], mode, **bcs)
        q, aux = H.init_fields(p, 1)
    qbc = orc.new_qbc(p, q)
    orc.fill_ghosts(p, qbc)
    auxbc = None
    if aux is not None:
        auxbc = orc.new_qbc(p, aux, p.num_aux)
        orc.fill_aux_ghosts(p, auxbc)
    ld = (shape[0] + 4 + 15) // 16 * 16

    def planes(a):
        d = np.full((a.shape[0], shape[1] + 4, ld), np.nan)
        d[:, :, :shape[0] + 4] = a.transpose(0, 2, 1)
        return d.tobytes()

    path = tmp_path / "state.bin"
    path.write_bytes(planes(qbc) + (planes(auxbc) if auxbc is not None else b""))
    dt, prm = 0.02 / max(shape), (list(H.SOLVERS.get(solver, {}).get("params", ())) + [0.0] * 4)[:4]
    r = subprocess.run([program, body, str(p.num_eqn), str(p.num_aux), str(shape[0]), str(shape[1]), str(mode), repr(dt), "4"] +
                       [repr(v) for v in prm] + [str(path)], capture_output=True, text=True, timeout=300,
                       env=dict(os.environ, TSAN_OPTIONS="exitcode=66"))
    assert r.returncode == 0, r.stderr[:3000]
    res = np.frombuffer(path.read_bytes())
    got = res[:-1].reshape(p.num_eqn, shape[1] + 4, ld)[:, :, :shape[0] + 4].transpose(0, 2, 1)
    cfl = orc.step_hyperbolic(p, qbc, auxbc, dt)
    orc.fill_ghosts(p, qbc)
    assert np.array_equal(got, qbc)
    assert res[-1] == cfl
