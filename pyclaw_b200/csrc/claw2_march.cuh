// claw2_march.cuh -- the unsplit step of the two-wave acoustics solvers: a pair of
// warps marching over rows.
//
// A CTA of two warps owns a strip of 28 columns (the 32 lanes hold columns
// i0-2 .. i0+29) and marches up a run of rows, one row per iteration:
//  - the x warp takes the x slices.  The lane of cell i owns the interface on
//    its left and exchanges with its neighbours by shuffle; what slice j adds
//    to rows j-1 and j+1 stays in the lane, carried to the next iteration.  It
//    hands the row that its slices have finished to the y warp;
//  - the y warp takes the y slices, a column per lane, meeting one interface
//    of each per iteration: limiter neighbours and what the cell below still
//    needs are carried in registers, the contributions to the neighbouring
//    columns are shuffles.  It writes the new row and its ghost images, and
//    prepares the rows' impedances (variable coefficients).
// The two run in lockstep, one barrier per iteration, with a ring of rows in
// shared memory between them.  Every state value is read from global memory by
// the warps that need it, coalesced and one row ahead.
//
// Same operations on the same operands in the same order per cell as
// step2.f90:92-248 / flux2.f90:104-206 (see step_tile_at), so the results are
// the same bits (only the sign of an exact zero can differ).  Divisions go
// through claw2_exact.cuh: a face between two cells has one impedance sum,
// which is the denominator of its normal solve and of the four transverse
// splits on its two sides, so a cell takes two reciprocals and three
// operations per quotient instead of sixteen divisions.
//
// A slice row without any difference between neighbouring cells carries zero
// waves and is passed over.
#pragma once

#include "claw2_exact.cuh"
#include "claw2_kernels.cuh"
#include "claw2_limit.cuh"

namespace claw2 {

constexpr int MARCH_TX = 28;                 // columns a warp owns
constexpr int MARCH_NT = 64;                 // the x warp and the y warp

// MINB: CTAs per SM that the register budget is sized for
struct MarchVc { static constexpr bool VC = true; static constexpr int MINB = 8; };
struct MarchConst { static constexpr bool VC = false; static constexpr int MINB = 10; };
template <class RP> struct MarchOf;
template <> struct MarchOf<RpAcoustics> { using type = MarchConst; };
template <> struct MarchOf<RpVcAcoustics> { using type = MarchVc; };

__device__ __forceinline__ double from_left(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double from_right(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }

// Ghost images of one cell (write_ghosts), out of line: only cells within two
// of a side have any.  bcs: the four boundary codes, two bits each.
template <int MEQN>
__device__ __noinline__ void march_ghosts(double* qo, long long ld, long long plane, int mx, int my, int bcs, int i, int j,
                                          double v0, double v1, double v2, double v3, double v4)
{
    StepArgs a;
    a.ld = ld; a.plane = plane; a.mx = mx; a.my = my;
    a.bcl[0] = bcs & 3; a.bcl[1] = (bcs >> 2) & 3; a.bcu[0] = (bcs >> 4) & 3; a.bcu[1] = (bcs >> 6) & 3;
    const double w[5] = {v0, v1, v2, v3, v4};
    double v[MEQN];
#pragma unroll
    for (int m = 0; m < MEQN; m++) v[m] = w[m];
    write_ghosts<MEQN>(a, qo, i, j, v);
}

// The ring between the two warps: field f of row j at [f][j & 7][lane].  V: the
// finished row (three fields); impedance, speed, reciprocals of the impedance
// sums with the left neighbour (RX) and with the row above (RY).  In iteration
// it (x slice l = j0-1+it, y interface below row r = l) the x warp writes V(l-1) and
// RX(l) and reads Z, C of rows l and l+1 and RY(l); the y warp reads V, RX, Z, C
// of row r-2, Z, C of row r and RY(r-1), and writes Z, C of row r+2 and RY(r+1):
// no row is written while it is read.
struct MarchRing {
    static constexpr int V = 0, Z = 3, C = 4, RX = 5, RY = 6;
    double* s;
    __device__ __forceinline__ double& at(int f, int j, int lane) const { return s[(f * 8 + (j & 7)) * 32 + lane]; }
};
template <bool VC> struct MarchRingSize { static constexpr int value = (VC ? 7 : 3) * 8 * 32; };

// Quotients n1 / d and n2 / d by a face sum with reciprocal r; odd: d has none.
__device__ __forceinline__ void march_strengths(double& a1, double& a2, double n1, double n2, double d, double r, bool odd,
                                                bool used)
{
    a1 = quot_rn(n1, d, r);
    a2 = quot_rn(n2, d, r);
    const bool safe = max(word_above<960>(n1), word_above<960>(n2)) < WordSpan<960, 900>::value;
    if (odd || (used && !safe)) {
        if (odd || !quot_num_ok(n1) || !quot_num_ok(n2)) {
            const double2 s = slow_quots(n1, n2, d);
            a1 = s.x; a2 = s.y;
        }
    }
}

// the other limiters, and mixed ones
static __device__ __noinline__ double2 march_limit_other(double r0, double r1, int m0, int m1)
{
    return make_double2(m0 != 0 ? philim_r(r0, m0) : 1.0, m1 != 0 ? philim_r(r1, m1) : 1.0);
}

// A zero, or far from a pulse, where the squared waves are tiny: both terms
// of the ratio scaled up by 2^600 (exactly), else the plain division.
static __device__ __noinline__ double2 march_limit_cold(double dot0, double dot1, double wn0, double wn1, int m0, int m1)
{
    const double dot[2] = {dot0, dot1}, wn[2] = {wn0, wn1};
    double ph[2];
#pragma unroll
    for (int k = 0; k < 2; k++) {
        const bool tiny = abs_word(wn[k]) < ExpWord<-800>::value;
        const double sc = __hiloint2double(tiny ? (int)ExpWord<600>::value : (int)ExpWord<0>::value, 0);
        const double x = dot[k] * sc, y = wn[k] * sc;
        ph[k] = quot_rn(x, y, recip_rn(y));
        if (!is_zero(y) && !ratio_ok(x, y)) ph[k] = slow_quot(dot[k], wn[k]);
        const int m = k ? m1 : m0;
        ph[k] = m != 0 && wn[k] != 0.0 ? philim_r(ph[k], m) : 1.0;
    }
    return make_double2(ph[0], ph[1]);
}

// The limiter's value for two waves: philim of dot / wn, 1 where the wave is
// too small to square.  mm: the two waves' limiter, -1 if they differ.
__device__ __forceinline__ double2 march_limit(double dot0, double dot1, double wn0, double wn1, int m0, int m1, int mm,
                                              bool used)
{
    const double r0 = quot_rn(dot0, wn0, recip_rn(wn0)), r1 = quot_rn(dot1, wn1, recip_rn(wn1));
    const bool safe = max(max(word_above<900>(wn0), word_above<900>(wn1)),
                          max(word_above<900>(dot0), word_above<900>(dot1))) < WordSpan<900, 100>::value;
    if (used && !safe) return march_limit_cold(dot0, dot1, wn0, wn1, m0, m1);
    if (mm == 4) return make_double2(philim_mc(r0), philim_mc(r1));
    if (mm == 1) return make_double2(philim_minmod(r0), philim_minmod(r1));
    if (mm == 2) return make_double2(philim_superbee(r0), philim_superbee(r1));
    return march_limit_other(r0, r1, m0, m1);
}

// Transverse splits of a cell's left-going part A and right-going part P
// (pressure components) into the lines below and above: contributions
// dtt g1, dtt g2 (pressure, transverse velocity) and dtt (g2 - g1).  zm, cm,
// zp, cp: impedance and speed of the cells below / above; dm, dp, rm, rp: the
// impedance sums with them and their reciprocals; h = dtn / 2.
struct MarchTrans { double c0p, c0t, c3p, c3t, c4p, c4t; };
__device__ __forceinline__ MarchTrans march_trans(double A, double P, double zm, double cm, double zp, double cp, double dm,
                                                  double dp, double rm, double rp, double h, double dtt, bool odd, bool used)
{
    double am = quot_rn(A, dm, rm), ap = quot_rn(A, dp, rp);
    double pm = quot_rn(P, dm, rm), pp = quot_rn(P, dp, rp);
    const bool safe = max(word_above<960>(A), word_above<960>(P)) < WordSpan<960, 900>::value;
    if (odd || (used && !safe)) {
        if (odd || !quot_num_ok(A) || !quot_num_ok(P)) {
            const double2 sm = slow_quots(A, P, dm), sp = slow_quots(A, P, dp);
            am = sm.x; pm = sm.y; ap = sp.x; pp = sp.y;
        }
    }
    // bmasdq = (cm b1 zm, -cm b1) with b1 = -A/dm; bpasdq = (cp b2 zp, cp b2), b2 = A/dp
    const double a1 = cm * am, a2 = cp * ap, b1 = cm * pm, b2 = cp * pp;
    const double g1p = h * (a1 * zm) + h * (b1 * zm), g1t = -(h * a1) - h * b1;
    const double g2p = -(h * (a2 * zp)) - h * (b2 * zp), g2t = -(h * a2) - h * b2;
    return MarchTrans{dtt * g2p, dtt * g2t, dtt * (g2p - g1p), dtt * (g2t - g1t), dtt * g1p, dtt * g1t};
}

// What the warps share: the problem's options and the strip.
struct MarchJob {
    int i0, j0, n, lane, i, ic;
    long long P;
    double dtdx, dtdy, czz, ccc, cden, crec;
    bool second, trans, cor, cbad;
    int m0, m1, mm;
};

// One interface's limited correction: waves (w1p, a1), (w2p, a2) of speeds -cl
// and cr; dot1 / dot2: products with the waves upwind.
__device__ __forceinline__ void march_correct(const MarchJob& J, double w1p, double a1, double w2p, double a2, double dot1,
                                              double dot2, double cl, double cr, double dtn, bool used, double& cq_p,
                                              double& cq_n)
{
    double l1p = w1p, l1n = a1, l2p = w2p, l2n = a2;
    if (J.m0 != 0 || J.m1 != 0) {
        const double2 ph = march_limit(dot1, dot2, w1p * w1p + a1 * a1, w2p * w2p + a2 * a2, J.m0, J.m1, J.mm, used);
        l1p = ph.x * w1p; l1n = ph.x * a1;
        l2p = ph.y * w2p; l2n = ph.y * a2;
    }
    const double sl = fabs(cl), sr = fabs(cr);
    const double f1 = sl * (1.0 - sl * dtn), f2 = sr * (1.0 - sr * dtn);
    cq_p = f1 * l1p + f2 * l2p;
    cq_n = f1 * l1n + f2 * l2n;
}

// x warp.  Slices l = j0-1 .. j0+n, one per iteration; finished rows go to the
// ring.  Returns the lane's largest |c| over the cells whose interfaces count
// in the CFL number (columns i0-1 .. i0+28, rows j0-1 .. j0+n).
template <class L>
__device__ __forceinline__ double march_x(const StepArgs& a, const MarchJob& J, const MarchRing& ring,
                                          const double* __restrict__ qin)
{
    constexpr bool VC = L::VC;
    const int lane = J.lane, lanel = lane > 0 ? lane - 1 : 0;
    const long long P = J.P, ld = a.ld;
    const double dtn = J.dtdx, dtt = J.dtdy, h = 0.5 * dtn;
    const bool cfl_col = lane >= 1 && lane <= 2 + MARCH_TX && J.i <= a.mx;
    // lanes whose normal solve / limited waves some result depends on
    const bool usedn = lane >= 1 && J.i <= a.mx + 1, usedl = lane >= 2 && lane <= 2 + MARCH_TX && J.i <= a.mx;
    const double* q = qin + (long long)(J.j0 + 1) * ld + (J.ic + CLAW2_NUM_GHOST);               // row j0-1
    double pn = q[0], un = q[P], vn = q[2 * P];
    double z1 = J.czz, c1 = J.ccc, z0 = J.czz, c0 = J.ccc;
    double rya = J.crec;                            // face between rows l and l+1
    __syncthreads();
    if (VC) {
        z1 = ring.at(ring.Z, J.j0 - 2, lane); c1 = ring.at(ring.C, J.j0 - 2, lane);
        z0 = ring.at(ring.Z, J.j0 - 1, lane); c0 = ring.at(ring.C, J.j0 - 1, lane);
        rya = ring.at(ring.RY, J.j0 - 2, lane);     // face above row j0-2
    }
    double cmax = 0.0;
    double Vp = 0.0, Vu = 0.0, Vv = 0.0, up_p = 0.0, up_t = 0.0;
    for (int it = 0; it <= J.n + 2; it++, __syncthreads()) {
        if (it > J.n + 1) continue;
        const int l = J.j0 - 1 + it;
        // rows l-1 (z2), l (p, u, v, z1) and l+1 (z0)
        const double z2 = z1, c2 = c1, ry = rya;
        z1 = z0; c1 = c0;
        const double p1 = pn, u1 = un, v1 = vn;
        if (it <= J.n) {
            q += ld;
            pn = q[0]; un = q[P]; vn = q[2 * P];
        }
        const double pl = from_left(p1), ul = from_left(u1);
        double zl = J.czz, cl = J.ccc, dx = J.cden, rx = J.crec;
        bool odd = J.cbad;
        if (VC) {
            z0 = ring.at(ring.Z, l + 1, lane); c0 = ring.at(ring.C, l + 1, lane);
            zl = ring.at(ring.Z, l, lanel); cl = ring.at(ring.C, l, lanel);
            rya = ring.at(ring.RY, l, lane);
            dx = zl + z1;
            rx = recip_rn(dx);
            ring.at(ring.RX, l, lane) = rx;
            odd = __any_sync(0xffffffffu, !quot_den_ok(dx) || c1 < 0.0);
            if (cfl_col) {
                const double ca = fabs(c1);
                cmax = cmax > ca ? cmax : ca;
            }
        }
        const double d1 = p1 - pl, d2 = u1 - ul;
        double vp = Vp, vv = Vv;                    // row l-1
        const double vu = Vu;
        Vp = p1; Vu = u1; Vv = v1;                  // row l
        if (J.trans) { Vp = Vp + up_p; Vv = Vv + up_t; }
        if (__all_sync(0xffffffffu, d1 == 0.0 && d2 == 0.0) && !odd) {
            up_p = 0.0; up_t = 0.0;
        } else {
            double a1, a2;
            march_strengths(a1, a2, -d1 + z1 * d2, d1 + zl * d2, dx, rx, odd, usedn);
            // wave 1 of the right neighbour interface starts in this cell, wave
            // 2 of the left one ends in the left cell
            const double a1r = from_right(a1), a2l = from_left(a2);
            const double w1p = -a1 * zl, w2p = a2 * z1, w1pr = -a1r * z1;
            double cq_p = 0.0, cq_n = 0.0;
            if (J.second) {
                // s1 = -c <= 0 meets the right neighbour's wave, s2 = c > 0 the left
                // one's (c = 0: the wave's correction is zero anyway)
                double dot1 = w1p * w1pr + a1 * a1r, dot2 = w2p * (a2l * zl) + a2 * a2l;
                if (odd) {                          // negative sound speeds turn the sides around
                    const double a1l = from_left(a1), a2r = from_right(a2), zll = from_left(zl), zr = from_right(z1);
                    if (-cl > 0.0) dot1 = w1p * (-a1l * zll) + a1 * a1l;
                    if (!(c1 > 0.0)) dot2 = w2p * (a2r * zr) + a2 * a2r;
                }
                march_correct(J, w1p, a1, w2p, a2, dot1, dot2, cl, c1, dtn, usedl, cq_p, cq_n);
            }
            // cell (i, l): fluctuations and corrections of its two interfaces
            const double ap_p = c1 * w2p, ap_n = c1 * a2;
            const double am_p = -c1 * w1pr, am_n = -c1 * a1r;
            const double cr_p = from_right(cq_p), cr_n = from_right(cq_n);
            Vp = Vp + (-(dtn * ap_p) - dtn * am_p) - dtn * (0.5 * cr_p - 0.5 * cq_p);
            Vu = Vu + (-(dtn * ap_n) - dtn * am_n) - dtn * (0.5 * cr_n - 0.5 * cq_n);
            if (J.trans) {
                const double dm = VC ? z2 + z1 : J.cden, dp = VC ? z1 + z0 : J.cden;
                const bool oddt = VC ? !quot_den_ok(dm) || !quot_den_ok(dp) : J.cbad;
                const double A = J.cor ? am_p + cr_p : am_p, Q = J.cor ? ap_p - cq_p : ap_p;
                const MarchTrans T = march_trans(A, Q, z2, c2, z0, c0, dm, dp, ry, rya, h, dtt, oddt, usedl);
                Vp = Vp - T.c3p; Vv = Vv - T.c3t;
                vp = vp - T.c4p; vv = vv - T.c4t;
                up_p = T.c0p; up_t = T.c0t;
            }
        }
        ring.at(ring.V, l - 1, lane) = vp; ring.at(ring.V + 1, l - 1, lane) = vu; ring.at(ring.V + 2, l - 1, lane) = vv;
    }
    return VC ? cmax : fabs(J.ccc);
}

// y warp.  Iteration it meets the interface between rows r-1 and r = j0-1+it of
// its columns, limits the one below it and finishes row r-2.  Returns whether a
// new value is not finite.
template <class L>
__device__ __forceinline__ bool march_y(const StepArgs& a, const MarchJob& J, const MarchRing& ring,
                                        const double* __restrict__ qin, double* __restrict__ qout)
{
    constexpr bool VC = L::VC;
    const int lane = J.lane, lanel = lane > 0 ? lane - 1 : 0, laner = lane < 31 ? lane + 1 : 31;
    const long long P = J.P, ld = a.ld;
    const double dtn = J.dtdy, dtt = J.dtdx, h = 0.5 * dtn;
    const bool own = lane >= 2 && lane < 2 + MARCH_TX && J.i < a.mx;
    const bool used = lane >= 1 && lane <= 2 + MARCH_TX && J.i <= a.mx;      // columns some result depends on
    const bool edge_cols = J.i0 <= 1 || J.i0 + MARCH_TX >= a.mx - 2;
    const double* q = qin + (long long)J.j0 * ld + (J.ic + CLAW2_NUM_GHOST);                     // row j0-2
    double* d = qout + (long long)(J.j0 - 1) * ld + (J.i + CLAW2_NUM_GHOST);                     // row j0-3
    const double* x = VC ? a.aux + (long long)J.j0 * ld + (J.ic + CLAW2_NUM_GHOST) : nullptr;    // row j0-2
    double p0 = q[0], v0 = q[2 * P];
    q += ld;
    double pn = q[0], vn = q[2 * P];
    // interface m (below the new one): strengths; the one below it: second
    // strength, right-going fluctuation and correction
    double y1 = 0.0, y2 = 0.0, y2b = 0.0, apb_p = 0.0, apb_n = 0.0, cqb_p = 0.0, cqb_n = 0.0;
    double zt = 0.0, rn = 0.0, cn = 0.0;            // impedance of row r+1, aux of row r+2
    if (VC) {
        const double ca = x[P], za = x[0] * ca;     // row j0-2
        x += ld;
        const double cb = x[P], zb = x[0] * cb;     // row j0-1
        x += ld;
        const double ct = x[P];                     // row j0
        zt = x[0] * ct;
        ring.at(ring.Z, J.j0 - 2, lane) = za; ring.at(ring.C, J.j0 - 2, lane) = ca;
        ring.at(ring.Z, J.j0 - 1, lane) = zb; ring.at(ring.C, J.j0 - 1, lane) = cb;
        ring.at(ring.Z, J.j0, lane) = zt; ring.at(ring.C, J.j0, lane) = ct;
        ring.at(ring.RY, J.j0 - 2, lane) = recip_rn(za + zb);
        ring.at(ring.RY, J.j0 - 1, lane) = recip_rn(zb + zt);
        x += ld;
        rn = x[0]; cn = x[P];                       // row j0+1
    }
    bool quietm = true, quietb = true, oddm = J.cbad;
    unsigned top = 0;                               // largest exponent word of the new values
    __syncthreads();
    for (int it = 0; it <= J.n + 2; it++, __syncthreads()) {
        const int r = J.j0 - 1 + it, j = r - 2;
        const double p1 = p0, v1 = v0;
        p0 = pn; v0 = vn;
        if (it <= J.n + 1) {
            q += ld;
            pn = q[0]; vn = q[2 * P];
        }
        double dy = J.cden, ry = J.crec, z0 = J.czz, z1 = J.czz, c1 = J.ccc;
        bool odd0 = J.cbad;
        if (VC) {
            z0 = ring.at(ring.Z, r, lane); z1 = ring.at(ring.Z, r - 1, lane); c1 = ring.at(ring.C, r - 1, lane);
            ry = ring.at(ring.RY, r - 1, lane);
            dy = z1 + z0;
            odd0 = __any_sync(0xffffffffu, !quot_den_ok(dy) || c1 < 0.0);
            if (it <= J.n) {
                const double z = rn * cn;           // row r+2
                ring.at(ring.Z, r + 2, lane) = z; ring.at(ring.C, r + 2, lane) = cn;
                ring.at(ring.RY, r + 1, lane) = recip_rn(zt + z);
                zt = z;
                if (it < J.n) { x += ld; rn = x[0]; cn = x[P]; }
            }
        }
        const double d1 = p0 - p1, d2 = v0 - v1;
        const bool quiet0 = __all_sync(0xffffffffu, d1 == 0.0 && d2 == 0.0) && !odd0;
        double vp = 0.0, vu = 0.0, vv = 0.0;
        if (it >= 3) { vp = ring.at(ring.V, j, lane); vu = ring.at(ring.V + 1, j, lane); vv = ring.at(ring.V + 2, j, lane); }
        double a1 = 0.0, a2 = 0.0;
        if (!quiet0) march_strengths(a1, a2, -d1 + z0 * d2, d1 + z1 * d2, dy, ry, odd0, used);
        if (quietm && quietb) {
            apb_p = 0.0; apb_n = 0.0; cqb_p = 0.0; cqb_n = 0.0;
        } else {
            double z2 = J.czz, c2 = J.ccc;
            if (VC) { z2 = ring.at(ring.Z, j, lane); c2 = ring.at(ring.C, j, lane); }
            const double w1p = -y1 * z2, w2p = y2 * z1;
            double cq_p = 0.0, cq_n = 0.0;
            if (J.second) {
                double dot1 = w1p * (-a1 * z1) + y1 * a1, dot2 = w2p * (y2b * z2) + y2 * y2b;
                if (odd0 || oddm) {
                    if (-c2 > 0.0 && it >= 2) {
                        // first strength of the interface between rows r-3 and r-2
                        const double* b = qin + (long long)(r - 1) * ld + (J.ic + CLAW2_NUM_GHOST);
                        const double* e = b + ld;
                        double zb = J.czz;
                        if (VC) {
                            const double* ab = a.aux + (b - qin);
                            zb = ab[0] * ab[P];
                        }
                        const double ba1 = slow_quot(-(e[0] - b[0]) + z2 * (e[2 * P] - b[2 * P]), zb + z2);
                        dot1 = w1p * (-ba1 * zb) + y1 * ba1;
                    }
                    if (!(c1 > 0.0)) dot2 = w2p * (a2 * z0) + y2 * a2;
                }
                march_correct(J, w1p, y1, w2p, y2, dot1, dot2, c2, c1, dtn, used, cq_p, cq_n);
            }
            // cell (i, j): its lower interface (carried) and interface m
            const double am_p = -c2 * w1p, am_n = -c2 * y1;
            const double c1p = -(dtn * apb_p) - dtn * am_p, c1n = -(dtn * apb_n) - dtn * am_n;
            const double c2p = dtn * (0.5 * cq_p - 0.5 * cqb_p), c2n = dtn * (0.5 * cq_n - 0.5 * cqb_n);
            if (J.trans) {
                double zl = J.czz, cl = J.ccc, zr = J.czz, cr = J.ccc, dl = J.cden, dr = J.cden, rl = J.crec, rr = J.crec;
                bool oddt = J.cbad;
                if (VC) {
                    zl = ring.at(ring.Z, j, lanel); cl = ring.at(ring.C, j, lanel);
                    zr = ring.at(ring.Z, j, laner); cr = ring.at(ring.C, j, laner);
                    rl = ring.at(ring.RX, j, lane); rr = ring.at(ring.RX, j, laner);
                    dl = zl + z2; dr = z2 + zr;
                    oddt = !quot_den_ok(dl) || !quot_den_ok(dr);
                }
                const double A = J.cor ? am_p + cq_p : am_p, Q = J.cor ? apb_p - cqb_p : apb_p;
                const MarchTrans T = march_trans(A, Q, zl, cl, zr, cr, dl, dr, rl, rr, h, dtt, oddt, used);
                vp = vp + from_left(T.c0p); vu = vu + from_left(T.c0t);
                vp = vp + (c1p - c2p - T.c3p); vv = vv + (c1n - c2n); vu = vu - T.c3t;
                vp = vp - from_right(T.c4p); vu = vu - from_right(T.c4t);
            } else {
                vp = vp + (c1p - c2p); vv = vv + (c1n - c2n);
            }
            apb_p = c1 * w2p; apb_n = c1 * y2; cqb_p = cq_p; cqb_n = cq_n;
        }
        y2b = y2; y1 = a1; y2 = a2;
        quietb = quietm; quietm = quiet0; oddm = odd0;
        if (it >= 3 && own) {
            d[0] = vp; d[P] = vu; d[2 * P] = vv;
            top = max(top, max(abs_word(vp), max(abs_word(vu), abs_word(vv))));
            if (a.ghost_fused && (edge_cols || j <= 1 || j >= a.my - 2)) {
                if (J.i <= 1 || J.i >= a.mx - 2 || j <= 1 || j >= a.my - 2) {
                    const int bcs = a.bcl[0] | a.bcl[1] << 2 | a.bcu[0] << 4 | a.bcu[1] << 6;
                    march_ghosts<3>(qout, ld, P, a.mx, a.my, bcs, J.i, j, vp, vu, vv, 0.0, 0.0);
                }
            }
        }
        d += ld;
    }
    return top >= 0x7ff00000u;
}

// One CTA's tile: MARCH_TX columns by up to `rows` rows.  CELL: the CFL maximum
// is collected by collect_cfl, else by report_cfl through one partial per tile.
template <class RP, bool CELL>
__device__ __forceinline__ void march_tile(const StepArgs& a, const TileId& tile, int rows)
{
    using L = typename MarchOf<RP>::type;
    constexpr bool VC = L::VC;
    __shared__ double red[MARCH_NT / 32 + 1];
    __shared__ double ring_mem[MarchRingSize<VC>::value];
    DevCtx ctx{red};
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
    J.i0 = tile.bx * MARCH_TX; J.j0 = tile.by * rows;
    J.n = a.my - J.j0 < rows ? a.my - J.j0 : rows;
    J.lane = threadIdx.x & 31;
    J.i = J.i0 - 2 + J.lane;
    J.ic = J.i < a.mx + 1 ? J.i : a.mx + 1;        // lanes beyond the ghosted array repeat its last column
    J.P = a.plane;
    J.dtdx = dt / a.dx; J.dtdy = dt / a.dy;
    J.second = a.order == 2; J.trans = a.trans > 0; J.cor = J.second && a.trans == 2;
    J.m0 = a.limit_any ? a.mthlim[0] : 0; J.m1 = a.limit_any ? a.mthlim[1] : 0;
    J.mm = J.m0 == J.m1 ? J.m0 : -1;
    // constant coefficients: every impedance is zz, every face sum 2 zz
    J.czz = VC ? 0.0 : a.prm[3]; J.ccc = VC ? 0.0 : a.prm[2];
    J.cden = J.czz + J.czz; J.crec = VC ? 0.0 : recip_rn(J.cden);
    J.cbad = !VC && (!quot_den_ok(J.cden) || J.ccc < 0.0);
    const MarchRing ring{ring_mem};
    double cflm = 0.0;
    bool bad = false;
    if (threadIdx.x < 32) {
        const double cmax = march_x<L>(a, J, ring, qin);
        const double tx = fabs(J.dtdx), ty = fabs(J.dtdy);
        cflm = (tx > ty ? tx : ty) * cmax;         // the largest of all dtdx |s| and dtdy |s|
    } else {
        bad = march_y<L>(a, J, ring, qin, qout);
    }
    if constexpr (CELL) {
        const bool nf = __syncthreads_or(bad || cflm != cflm);
        const double mw = ctx.warp_max(cflm);      // the x warp's, in thread 0
        if (threadIdx.x == 0) collect_cfl(a, ctx, tile.ntiles, mw, nf, false);
    }
    else report_cfl<MARCH_NT>(a, ctx, tile, red, cflm, bad);
}

}  // namespace claw2
