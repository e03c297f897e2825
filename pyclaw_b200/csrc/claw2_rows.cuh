// claw2_rows.cuh -- the split step of the acoustics solvers, on square tiles of
// T = 28 or 12 cells.
//
// Same step as step_tile_at (step2ds.f90:96-252, flux2.f90:104-180 without
// transverse terms) with the same operations in the same order per cell, so the
// results are the same bits (only the sign of an exact zero can differ).  A split
// line depends on no other, so nothing is exchanged between lines:
//  - the tile's halo (T + 4 rows and columns; with variable coefficients also
//    impedance and speed) is staged in shared memory, pitched so that rows and
//    columns are read without bank conflicts;
//  - T + 4 lanes hold a line, one cell each; neighbours' waves come by shuffle;
//  - the x sweep rewrites the halo's rows in place, one block barrier later the y
//    sweep its columns;
//  - the waves and corrections are those of claw2_march.cuh (no divergent
//    divisions, lines without waves passed over).
//
// Bound by the latency of the FP64 chains; 64 registers a thread keep 32 warps on
// an SM (80 and 24 warps: 73.8 us instead of 68.9 on acoustics 1500^2).  us a step
// on a B200, the general body and this one, a pulse over the whole grid: acoustics
// 64 x 48 19.4 and 6.2, 256^2 22.7 and 8.5, 1280 x 320 37 and 24, 1500^2 169 and 67;
// variable coefficients 20.8 and 7.2, 25.6 and 9.5, 43 and 27, 205 and 80.  At rest
// (lines without waves) 1280 x 320 takes 11 and 12, 1500^2 36 and 45.
#pragma once

#include "claw2_march.cuh"

namespace claw2 {

template <bool VC, int T, int NT> struct RowsSmem {
    static constexpr int TR = T + 4, HP = TR + 1, FS = TR * HP, LPC = NT / TR;
    enum { Z = 3, C = 4 };
    static constexpr int total = (VC ? 5 : 3) * FS + NT / 32, bytes = total * 8;
    static_assert(TR == 16 || TR == 32, "lines of 16 or 32 lanes");
};

// One line of one sweep.  `own`: its cells are swept (ghost columns only count in
// the CFL number).  Returns the largest |c| of the lane's interface.
template <bool VC, int IXY, int T, int NT>
__device__ __forceinline__ double rows_line(const StepArgs& a, const MarchJob& J, double* H, int i0, int j0, int line,
                                            bool lineok, bool own, double dtn)
{
    using SM = RowsSmem<VC, T, NT>;
    constexpr int TR = SM::TR, NSLOT = T + 3, MU = Dir<IXY>::MU;
    const int slot = threadIdx.x & (TR - 1);
    const int len = IXY == 1 ? a.mx : a.my;
    const int k = (IXY == 1 ? i0 : j0) - 1 + slot;
    const bool ifok = lineok && slot < NSLOT && k <= len + 1;
    const bool lim = ifok && slot >= 1 && slot <= NSLOT - 2 && k >= 0 && k <= len;
    constexpr int step = IXY == 1 ? 1 : SM::HP;
    const int across = IXY == 1 ? (line - j0 + 2) * SM::HP : line - i0 + 2;
    double* L = H + across + slot * step;          // cell k-1; the last lane has no cell k and repeats it
    double* R = L + (slot < NSLOT ? step : 0);
    const double pl = L[0], p1 = R[0], ul = L[MU * SM::FS], u1 = R[MU * SM::FS];
    double zl = J.czz, cl = J.ccc, z1 = J.czz, c1 = J.ccc, dx = J.cden, rx = J.crec;
    bool odd = J.cbad;
    if (VC) {
        zl = L[SM::Z * SM::FS]; cl = L[SM::C * SM::FS]; z1 = R[SM::Z * SM::FS]; c1 = R[SM::C * SM::FS];
        dx = zl + z1;
        rx = recip_rn(dx);
        odd = __any_sync(0xffffffffu, ifok && !quot_den_ok(dx));
    }
    const double top = lim ? (fabs(cl) > fabs(c1) ? fabs(cl) : fabs(c1)) : 0.0;
    const double d1 = p1 - pl, d2 = u1 - ul;
    if (__all_sync(0xffffffffu, (d1 == 0.0 && d2 == 0.0) || !ifok) && !odd) return top;
    double a1, a2;
    march_strengths(a1, a2, -d1 + z1 * d2, d1 + zl * d2, dx, rx, odd, ifok);
    const double w1p = -a1 * zl, w2p = a2 * z1;
    double cq_p = 0.0, cq_n = 0.0;
    if (J.second) {
        const double dr1 = w1p * from_right(w1p) + a1 * from_right(a1), dr2 = w2p * from_right(w2p) + a2 * from_right(a2);
        const double dl1 = from_left(dr1), dl2 = from_left(dr2);
        march_correct(J, w1p, a1, w2p, a2, -cl > 0.0 ? dl1 : dr1, c1 > 0.0 ? dl2 : dr2, cl, c1, dtn, lim, cq_p, cq_n);
    }
    const double ap_p = c1 * w2p, ap_n = c1 * a2, am_p = -cl * w1p, am_n = -cl * a1;
    const double yp = from_right(dtn * am_p), yn = from_right(dtn * am_n);
    const double fp = from_right(0.5 * cq_p), fn = from_right(0.5 * cq_n);
    __syncwarp();                                  // the line has been read
    if (own && lim && slot <= T && k < len) {
        R[0] = p1 + (-(dtn * ap_p) - yp) - dtn * (fp - 0.5 * cq_p);
        R[MU * SM::FS] = u1 + (-(dtn * ap_n) - yn) - dtn * (fn - 0.5 * cq_n);
    }
    return top;
}

template <bool VC, int T, int NT>
__device__ __forceinline__ void rows_tile(const StepArgs& a, DevCtx& ctx, const TileId& tile)
{
    using SM = RowsSmem<VC, T, NT>;
    double* H = ctx.smem();
    double* red = H + (VC ? 5 : 3) * SM::FS;
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
    MarchJob J;
    J.second = a.order == 2;
    J.m0 = a.limit_any ? a.mthlim[0] : 0; J.m1 = a.limit_any ? a.mthlim[1] : 0;
    J.mm = J.m0 == J.m1 ? J.m0 : -1;
    J.czz = VC ? 0.0 : a.prm[3]; J.ccc = VC ? 0.0 : a.prm[2];
    J.cden = J.czz + J.czz; J.crec = VC ? 0.0 : recip_rn(J.cden);
    J.cbad = !VC && !quot_den_ok(J.cden);
    const double dtdx = dt / a.dx, dtdy = dt / a.dy;
#pragma unroll
    for (int it = 0; it < SM::TR * SM::TR / NT; it++) {
        const int e = threadIdx.x + it * NT, r = e / SM::TR, c = e % SM::TR, s = r * SM::HP + c;
        const bool in = i0 - 2 + c <= a.mx + 1 && j0 - 2 + r <= a.my + 1;
        const long long o = in ? (long long)(j0 + r) * a.ld + (i0 + c) : 0;        // ghosted row j0 is row j0-2
#pragma unroll
        for (int m = 0; m < 3; m++) H[m * SM::FS + s] = qin[o + m * a.plane];
        if (VC) {
            const double rho = a.aux[o], cs = a.aux[o + a.plane];
            H[SM::Z * SM::FS + s] = rho * cs;
            H[SM::C * SM::FS + s] = cs;
        }
    }
    __syncthreads();
    // A warp past the last line leaves its loop (`lead`: its first line of a pass): the
    // lines are rewritten in place, and it would read one that another warp writes.
    const int mine = threadIdx.x / SM::TR, lead = threadIdx.x / 32 * (32 / SM::TR);
    double cx = 0.0, cy = 0.0;
    {
        // rows of the halo
        const int first = j0 - 2, last = j0 + T + 1 < a.my + 1 ? j0 + T + 1 : a.my + 1;
        for (int c0 = first; c0 + lead <= last; c0 += SM::LPC) {
            const int line = c0 + mine;
            const double t = rows_line<VC, 1, T, NT>(a, J, H, i0, j0, line < last ? line : last, line <= last, true, dtdx);
            cx = cx > t ? cx : t;
        }
    }
    __syncthreads();
    {
        // the tile's columns of the swept rows, and the ghost columns beside it
        const int own = i0 + T < a.mx ? i0 + T : a.mx;
        const int first = i0 == 0 ? -2 : i0, last = own == a.mx ? a.mx + 1 : own - 1;
        for (int c0 = first; c0 + lead <= last; c0 += SM::LPC) {
            const int line = c0 + mine;
            const double t = rows_line<VC, 2, T, NT>(a, J, H, i0, j0, line < last ? line : last, line <= last,
                                                     line >= 0 && line < own, dtdy);
            cy = cy > t ? cy : t;
        }
    }
    const double vx = fabs(dtdx) * cx, vy = fabs(dtdy) * cy;
    __syncthreads();
    const bool bad = store_tile<3, T, T, NT, SM::HP>(a, ctx, H + 2 * SM::HP + 2, SM::FS, qout, i0, j0, dt);
    report_cell<NT>(a, ctx, tile.ntiles, red, vx > vy ? vx : vy, bad, false);
}

}  // namespace claw2
