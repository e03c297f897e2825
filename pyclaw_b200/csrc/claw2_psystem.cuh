// claw2_psystem.cuh -- the unsplit step of the p-system with f-waves
// (apps/psystem_2d/psystem.py), on square tiles of T = 28 or 12 cells.
//
// Same step as step_tile_at (step2.f90:92-248, flux2.f90:104-206) with the same
// operations in the same order per cell, so the results are the same bits (only
// the sign of an exact zero can differ).  The tile's lines are swept as in
// claw2_lean.cuh (T + 4 lanes a line, neighbours by shuffle, the two cross-line
// terms through a double-buffered shared array, one block barrier per chunk of
// lines).  What differs:
//  - stress, sound speed and impedance are functions of one cell (an
//    exponential, a division and a square root): they are computed once per cell
//    of the tile's halo and staged in shared memory, instead of two times per
//    interface for the normal solve and four for the transverse ones;
//  - the f-waves are (b1, b1 Z_left) and (b2, -b2 Z_right) in the strain and one
//    momentum, the transverse splits have the strain and the other momentum: the
//    components that are zero are left out;
//  - quotients by one impedance sum share its reciprocal (claw2_exact.cuh);
//    operands outside its range are divided out of line;
//  - lines without waves are passed over.
//
// Bound by the latency of the FP64 chains (two chunks of lines a step on grids of
// one wave).  us a step on a B200, the general body and this one, with the copy of the
// strain before it: 64 x 48 64 and 10, 200 x 200 68 and 12, 641 x 163 77 and 18,
// 800 x 400 137 and 38, 1500^2 681 and 184.
#pragma once

#include "claw2_exact.cuh"
#include "claw2_kernels.cuh"
#include "claw2_march.cuh"
#include "claw2_riemann.cuh"

namespace claw2 {

// Shared memory (doubles): per cell of the halo q[1]/rho, q[2]/rho, the stress, speed
// and impedance of the cell's strain and the speed and impedance of the strain
// before the step; the tile's new state; the exchange (2 buffers x 2 terms x 2
// components x cells of a chunk); the reduction scratch.
template <int T, int NT> struct PsysSmem {
    static constexpr int MEQN = 3, TR = T + 4, HP = TR + 1;      // odd pitches: columns without bank conflicts
    static constexpr int QP = T | 1, LPC = NT / TR, NX = LPC * T;
    enum { U, V, SG, C, Z, CT, ZT, FIELDS };
    static constexpr int HS = FIELDS * TR * HP, QX = MEQN * T * QP, CX = 2 * 2 * 2 * NX;
    static constexpr int total = HS + QX + CX + NT / 32, bytes = total * 8;
    static_assert(TR == 16 || TR == 32, "lines of 16 or 32 lanes");
};

template <int T, int NT>
__device__ __forceinline__ void psys_stage(const StepArgs& a, const double* __restrict__ qin, double* H, int i0, int j0)
{
    using SM = PsysSmem<T, NT>;
    const double* __restrict__ aux = a.aux;
    for (int e = threadIdx.x; e < SM::TR * SM::TR; e += NT) {
        const int r = e / SM::TR, c = e % SM::TR;
        double f[SM::FIELDS] = {0.0, 0.0, 0.0, 0.0, 1.0, 0.0, 1.0};
        if (i0 - 2 + c <= a.mx + 1 && j0 - 2 + r <= a.my + 1) {
            const long long o = (long long)(j0 + r) * a.ld + (i0 + c);             // ghosted row j0 is row j0-2
            const double ax[4] = {aux[o], aux[o + a.plane], aux[o + 2 * a.plane], aux[o + 3 * a.plane]};
            const double eps = qin[o], m1 = qin[o + a.plane], m2 = qin[o + 2 * a.plane];
            f[SM::U] = m1 / ax[0];
            f[SM::V] = m2 / ax[0];
            RpPsystem::cell(ax, eps, f[SM::SG], f[SM::C], f[SM::Z]);
            f[SM::CT] = f[SM::C];
            f[SM::ZT] = f[SM::Z];
            double st;
            if (ax[3] != eps) RpPsystem::cell(ax, ax[3], st, f[SM::CT], f[SM::ZT]);
        }
#pragma unroll
        for (int k = 0; k < SM::FIELDS; k++) H[k * SM::TR * SM::HP + r * SM::HP + c] = f[k];
    }
}

// x1 / y and x2 / y; r: 1 / y where y is in range
__device__ __forceinline__ double2 psys_quots(double x1, double x2, double y, double r, bool used)
{
    double2 q = make_double2(quot_rn(x1, y, r), quot_rn(x2, y, r));
    const bool safe = max(word_above<960>(x1), word_above<960>(x2)) < WordSpan<960, 900>::value && quot_den_ok(y);
    if (used && !safe && !(quot_den_ok(y) && quot_num_ok(x1) && quot_num_ok(x2))) q = slow_quots(x1, x2, y);
    return q;
}

// One chunk of one sweep direction; CX is the half of the exchange array that it uses.
template <int IXY, int T, int NT>
__device__ __forceinline__ void psys_chunk(const StepArgs& a, const double* __restrict__ qin, const double* H, double* Qx,
                                           double* CX, int i0, int j0, int line, int cfirst, int clast, bool lineok,
                                           double dtn, double dtt, double& cflm)
{
    using SM = PsysSmem<T, NT>;
    constexpr int TR = SM::TR, NX = SM::NX, NSLOT = T + 3;
    constexpr int MU = Dir<IXY>::MU, MV = Dir<IXY>::MV;
    const int tid = threadIdx.x, slot = tid & (TR - 1);
    const int len = IXY == 1 ? a.mx : a.my;
    const int k = (IXY == 1 ? i0 : j0) - 1 + slot;
    const bool ifok = lineok && slot < NSLOT && k <= len + 1;
    const bool lim = ifok && slot >= 1 && slot <= NSLOT - 2 && k >= 0 && k <= len;
    const int kr = slot < NSLOT ? k : k - 1;
    auto h = [&](int f, int kk, int ll) -> double {
        const int r = IXY == 1 ? ll - j0 + 2 : kk - j0 + 2, c = IXY == 1 ? kk - i0 + 2 : ll - i0 + 2;
        return H[f * TR * SM::HP + r * SM::HP + c];
    };

    // ---------------- normal solve ----------------
    const double cl = h(SM::C, k - 1, line), zl = h(SM::Z, k - 1, line), cr = h(SM::C, kr, line), zr = h(SM::Z, kr, line);
    double b1, b2;
    {
        const double ul = h(IXY == 1 ? SM::U : SM::V, k - 1, line), ur = h(IXY == 1 ? SM::U : SM::V, kr, line);
        const double df1 = (-ur) - (-ul), df2 = (-h(SM::SG, kr, line)) - (-h(SM::SG, k - 1, line));
        const double den = zl + zr;
        const double2 b = psys_quots(zr * df1 + df2, zl * df1 - df2, den, recip_rn(den), ifok);
        b1 = b.x; b2 = b.y;
    }
    const double b1z = b1 * zl, b2z = -b2 * zr;
    if (lim) {
        const double cm = fabs(dtn) * (cl > cr ? cl : cr);
        cflm = cflm > cm ? cflm : cm;
    }
    const bool flat = __all_sync(0xffffffffu, (b1 == 0.0 && b2 == 0.0) || !ifok);

    // ---------------- limiter, corrections ----------------
    double cq0 = 0.0, cqm = 0.0;
    if (!flat && a.order == 2) {
        double w10 = b1, w1m = b1z, w20 = b2, w2m = b2z;
        if (a.limit_any) {
            const double dr1 = b1 * from_right(b1) + b1z * from_right(b1z), dr2 = b2 * from_right(b2) + b2z * from_right(b2z);
            const double dl2 = from_left(dr2);
            const int m0 = a.mthlim[0], m1 = a.mthlim[1];
            // the left-going wave's upwind side is the right, the other's the left
            const double2 ph = march_limit(dr1, cr > 0.0 ? dl2 : dr2, b1 * b1 + b1z * b1z, b2 * b2 + b2z * b2z, m0, m1,
                                           m0 == m1 ? m0 : -1, lim);
            w10 = ph.x * b1; w1m = ph.x * b1z;
            w20 = ph.y * b2; w2m = ph.y * b2z;
        }
        const double f1 = -(1.0 - cl * dtn), f2 = 1.0 - cr * dtn;
        cq0 = f1 * w10 + f2 * w20;
        cqm = f1 * w1m + f2 * w2m;
    }

    // ---------------- transverse splits ----------------
    // left-going part in cell k-1, right-going in cell k: down (strain, momentum) and up
    double dL0 = 0.0, dLv = 0.0, uL0 = 0.0, uLv = 0.0, dR0 = 0.0, dRv = 0.0, uR0 = 0.0, uRv = 0.0;
    if (!flat && a.trans > 0) {
        const bool cor = a.order == 2 && a.trans == 2;
        const double A = cor ? b1 + cq0 : b1, P = cor ? b2 - cq0 : b2;
        const int ld = line - 1, lu = line + 1;
        const double zb = h(SM::ZT, kr, ld), za = h(SM::ZT, kr, lu), cb = h(SM::CT, kr, ld), ca = h(SM::CT, kr, lu);
        const double zbl = h(SM::ZT, k - 1, ld), zal = h(SM::ZT, k - 1, lu), cbl = h(SM::CT, k - 1, ld),
                     cal = h(SM::CT, k - 1, lu);
        const double den = zb + za, denl = zbl + zal, r = recip_rn(den);
        // the lane on the left has the reciprocal of cell k-1's sum (lane 0 uses none)
        const double2 gl = psys_quots(zal * A, zbl * A, denl, from_left(r), lim);
        const double2 gr = psys_quots(za * P, zb * P, den, r, lim);
        dL0 = -cbl * gl.x; dLv = dL0 * zbl;
        uL0 = cal * gl.y; uLv = -uL0 * zal;
        dR0 = -cb * gr.x; dRv = dR0 * zb;
        uR0 = ca * gr.y; uRv = -uR0 * za;
    }

    // ---------------- the slice's contributions to cell k ----------------
    const double hh = 0.5 * dtn;
    const double y00 = from_right(dtn * b1), y0m = from_right(dtn * b1z);
    const double y10 = from_right(0.5 * cq0), y1m = from_right(0.5 * cqm);
    const double y20 = from_right(hh * dL0), y2v = from_right(hh * dLv), y30 = from_right(hh * uL0), y3v = from_right(hh * uLv);
    const bool cellok = lim && slot <= T && k < len;
    const bool trans = a.trans > 0;
    const double C10 = -(dtn * b2) - y00, C1m = -(dtn * b2z) - y0m;
    const double C20 = dtn * (y10 - 0.5 * cq0), C2m = dtn * (y1m - 0.5 * cqm);
    const double g10 = -y20 - hh * dR0, g1v = -y2v - hh * dRv, g20 = -y30 - hh * uR0, g2v = -y3v - hh * uRv;
    const double C00 = dtt * g20, C0v = dtt * g2v, C30 = dtt * (g20 - g10), C3v = dtt * (g2v - g1v), C40 = dtt * g10,
                 C4v = dtt * g1v;
    const int mine = tid / TR * T + slot - 1;
    if (cellok) {
        CX[mine] = C00; CX[NX + mine] = C0v;
        CX[2 * NX + mine] = C40; CX[3 * NX + mine] = C4v;
    }
    __syncthreads();

    // ---------------- combine slices line-1, line, line+1 per cell ----------------
    if (!cellok) return;
    auto qx = [&](int m, int ll) -> double& {
        const int ci = IXY == 1 ? k : ll, cj = IXY == 1 ? ll : k;
        return Qx[(m * T + (cj - j0)) * SM::QP + (ci - i0)];
    };
    auto old = [&](int m, int ll) -> double {
        if (IXY == 2) return qx(m, ll);
        return qin[(long long)m * a.plane + (long long)(ll + CLAW2_NUM_GHOST) * a.ld + (k + CLAW2_NUM_GHOST)];
    };
    auto in_tile_line = [&](int ll) {
        return IXY == 1 ? (ll >= j0 && ll < j0 + T && ll < a.my) : (ll >= i0 && ll < i0 + T && ll < a.mx);
    };
    if (in_tile_line(line)) {
        double v0, vm, vv;
        if (line == cfirst) {                      // has up(line-1) already
            v0 = qx(0, line); vm = qx(MU, line); vv = qx(MV, line);
        } else {
            v0 = old(0, line); vm = old(MU, line); vv = old(MV, line);
            if (trans) { v0 = v0 + CX[mine - T]; vv = vv + CX[NX + mine - T]; }
        }
        if (IXY == 1) {
            v0 = v0 + C10 - C20;
            if (trans) v0 = v0 - C30;
            vm = vm + C1m - C2m;
        } else {
            v0 = v0 + (trans ? (C10 - C20 - C30) : (C10 - C20));
            vm = vm + (C1m - C2m);
        }
        if (trans) vv = vv - C3v;
        if (trans && line != clast) { v0 = v0 - CX[2 * NX + mine + T]; vv = vv - CX[3 * NX + mine + T]; }
        qx(0, line) = v0; qx(MU, line) = vm; qx(MV, line) = vv;
    }
    if (line == clast && in_tile_line(line + 1)) {
        double v0 = old(0, line + 1), vv = old(MV, line + 1);
        if (trans) { v0 = v0 + C00; vv = vv + C0v; }
        qx(0, line + 1) = v0; qx(MU, line + 1) = old(MU, line + 1); qx(MV, line + 1) = vv;
    }
    if (trans && line == cfirst && in_tile_line(line - 1)) {
        qx(0, line - 1) = qx(0, line - 1) - C40;
        qx(MV, line - 1) = qx(MV, line - 1) - C4v;
    }
}

template <int T, int NT>
__device__ __forceinline__ void psys_tile(const StepArgs& a, DevCtx& ctx, const TileId& tile)
{
    using SM = PsysSmem<T, NT>;
    double* H = ctx.smem();
    double* Qx = H + SM::HS;
    double* CX = Qx + SM::QX;
    double* red = CX + SM::CX;
    const int i0 = tile.bx * T, j0 = tile.by * T;
    const double* qin = a.qin;
    double* qout = a.qout;
    double dt = a.dt;
    if (a.ctrl) {
        const int done = a.ctrl->done, cur = a.ctrl->cur;           // loaded together
        dt = a.ctrl->dt;
        if (done) return;                          // uniform across the grid
        qin = cur ? a.q1 : a.q0;
        qout = cur ? a.q0 : a.q1;
    }
    const double dtdx = dt / a.dx, dtdy = dt / a.dy;
    psys_stage<T, NT>(a, qin, H, i0, j0);
    __syncthreads();
    const int mine = threadIdx.x / SM::TR;
    double cflm = 0.0;
    int chunk = 0;
    {
        const int first = j0 - 1, last = j0 + T < a.my ? j0 + T : a.my;
        for (int c0 = first; c0 <= last; c0 += SM::LPC, chunk++) {
            const int line = c0 + mine, clast = c0 + SM::LPC - 1 < last ? c0 + SM::LPC - 1 : last;
            psys_chunk<1, T, NT>(a, qin, H, Qx, CX + (chunk & 1) * 4 * SM::NX, i0, j0, line < last ? line : last, c0, clast,
                                 line <= last, dtdx, dtdy, cflm);
        }
    }
    {
        const int first = i0 - 1, last = i0 + T < a.mx ? i0 + T : a.mx;
        for (int c0 = first; c0 <= last; c0 += SM::LPC, chunk++) {
            const int line = c0 + mine, clast = c0 + SM::LPC - 1 < last ? c0 + SM::LPC - 1 : last;
            psys_chunk<2, T, NT>(a, qin, H, Qx, CX + (chunk & 1) * 4 * SM::NX, i0, j0, line < last ? line : last, c0, clast,
                                 line <= last, dtdy, dtdx, cflm);
        }
    }
    __syncthreads();
    const bool bad = store_tile<3, T, T, NT, SM::QP>(a, ctx, Qx, T * SM::QP, qout, i0, j0, dt);
    report_cell<NT>(a, ctx, tile.ntiles, red, cflm, bad, false);
}

}  // namespace claw2
