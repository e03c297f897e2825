// claw2_dense.cuh -- the interface solves of the solvers with dense waves (Euler
// 4- and 5-wave Roe, shallow-water Roe) as the tile bodies use them.
//
// Same operations on the same operands in the same order as the solvers of
// claw2_riemann.cuh and flux2.f90:104-206, so the results are the same bits
// (only the sign of an exact zero can differ).  What is saved is work that
// cannot change them:
//  - quotients by one denominator share its reciprocal, and none has a branch
//    (claw2_exact.cuh).  Numerators below its range (the momenta ahead of a shock
//    decay through every binade to zero) are divided out of line (low_quot);
//    denominators outside it send the interface through the plain solver.  The
//    plain solver for the former too made the tiles ahead of the shock take 59 us
//    instead of 21, and the step of the developed 1280 x 320 shock bubble 121 instead
//    of 77 (97 with the solves of claw2_riemann.cuh);
//  - the entropy fix needs the star states' speeds s1 and s2 only where they
//    change sign against the cells': a bound on rhou^2 - gamma p rho without
//    divisions rules that out nearly everywhere (star_subsonic);
//  - transverse splits where every lane's velocity is subsonic drop the two
//    terms whose speeds are clipped to zero.
// An unsplit Euler 4-wave step of 1280 x 320 cells, the shock bubble shortly after its
// start, executes 28.2 M warp instructions with them (11.2 M in FP64; 26.9 M and
// 10.8 M before low_quot), 31.0 M (12.0 M) with the plain solves.  The developed flow at
// t = 0.32 takes 37.6 M (15.9 M).
#pragma once

#include "claw2_exact.cuh"
#include "claw2_kernels.cuh"
#include "claw2_limit.cuh"

namespace claw2 {

// max(s, 0) and min(s, 0) as the solvers' fmax / fmin give them (a NaN gives 0)
__device__ __forceinline__ double clip_low(double s) { return s > 0.0 ? s : 0.0; }
__device__ __forceinline__ double clip_high(double s) { return s < 0.0 ? s : 0.0; }

// true unless some |x| is below 2^kNumLow without being zero
template <int K>
__device__ __forceinline__ bool nums_ok(const double (&x)[K])
{
    unsigned low = abs_word(x[0]);
#pragma unroll
    for (int k = 1; k < K; k++) low = min(low, abs_word(x[k]));
    if (low >= ExpWord<kNumLow>::value) return true;
    bool ok = true;
#pragma unroll
    for (int k = 0; k < K; k++) ok = ok && (abs_word(x[k]) >= ExpWord<kNumLow>::value || is_zero(x[k]));
    return ok;
}

// ---------------------------------------------------------------------------
// Euler
// ---------------------------------------------------------------------------
template <bool TRACER> struct DenseEuler {
    using RP = RpEuler<TRACER>;
    static constexpr int N = RP::MEQN, MW = RP::MW;
    static constexpr int NCD = 6;                      // cell: sq, U, V (normal, transverse), H, s0, s3
    static constexpr int S0 = 4, S3 = 5;
    static constexpr int NR = 8;                       // RP's Roe averages and 1 / (2 a)
    // whether component m of wave p is not a structural zero
    template <int IXY> static constexpr __host__ __device__ bool wave_has(int p, int m)
    {
        return p == 4 ? m == 4 : m != 4 && (p != 1 || m == Dir<IXY>::MV || m == 3);
    }

    // The quantities of one cell (RpEuler::Cell; s0 and s3 are its normal
    // velocity minus and plus its sound speed).  False if an operand leaves
    // the quotients' range.
    template <int IXY>
    static __device__ __forceinline__ bool cell(const double (&q)[N], const double* prm, double (&c)[NCD])
    {
        constexpr int mu = Dir<IXY>::MU, mv = Dir<IXY>::MV;
        const double gamma = prm[0], gamma1 = prm[1];
        const double r0 = recip_rn(q[0]), sq = sqrt_rn(q[0]), rs = recip_rn(sq);
        const double kin = 0.5 * (q[1] * q[1] + q[2] * q[2]);
        const double p = gamma1 * (q[3] - quot_rn(kin, q[0], r0));
        const double ep = q[3] + p, gp = gamma * p;
        const double c2 = quot_rn(gp, q[0], r0), cs = sqrt_rn(c2), un = quot_rn(q[mu], q[0], r0);
        c[0] = sq;
        c[1] = quot_rn(q[mu], sq, rs);
        c[2] = quot_rn(q[mv], sq, rs);
        c[3] = quot_rn(ep, sq, rs);
        c[S0] = un - cs; c[S3] = un + cs;
        // A kinetic energy or velocity too small for its quotient to be exact is
        // nothing beside the energy or the sound speed.
        const bool ok = max(pos_word(q[0]), max(pos_word(gp), pos_word(c2))) < WordSpan<100, 100>::value &&
                        min(abs_word(q[3]), abs_word(ep)) >= ExpWord<-600>::value;
        const double x[2] = {q[1], q[2]};
        if (!nums_ok(x)) { c[1] = low_quot(q[mu], sq, rs); c[2] = low_quot(q[mv], sq, rs); }
        return ok;
    }
    template <int IXY>
    static __device__ __noinline__ void cell_plain(const double* q, double prm0, double prm1, double* c)
    {
        const double prm[2] = {prm0, prm1};
        double a[N];
#pragma unroll
        for (int m = 0; m < N; m++) a[m] = q[m];
        const typename RP::Cell x = RP::template cell<IXY>(a, prm);
        c[0] = x.sq; c[1] = x.U; c[2] = x.V; c[3] = x.H;
        c[S0] = x.un - x.c; c[S3] = x.un + x.c;
    }

    // True where the state's normal velocity is certainly not above its sound
    // speed: rho > 0 and rhou <= 0 or rhou^2 < gamma p rho by a margin far above
    // the rounding errors of both sides.
    static __device__ __forceinline__ bool star_subsonic(double rho, double ru, double rv, double en, double gg1)
    {
        const double u2 = ru * ru, e = en * rho;
        const double k = 0.5 * __fma_rn(rv, rv, u2);
        const double cc = gg1 * (e - k);                       // gamma p rho
        const double scale = __fma_rn(gg1, fabs(e) + k, u2);
        return rho > 0.0 && (ru <= 0.0 || cc - u2 > 0x1p-40 * scale);
    }
    // s1 (sign -1) or s2 (+1): the star state's velocity -+ sound speed
    static __device__ __noinline__ double star_speed(double rho, double ru, double rv, double en, double gamma,
                                                     double gamma1, double sign)
    {
        const double kin = 0.5 * (ru * ru + rv * rv);
        {
            const double r = recip_rn(rho), gp = gamma * (gamma1 * (en - quot_rn(kin, rho, r)));
            const double c2 = quot_rn(gp, rho, r), c = sqrt_rn(c2), u = quot_rn(ru, rho, r);
            const double x[2] = {kin, ru};
            if (max(pos_word(rho), max(pos_word(gp), pos_word(c2))) < WordSpan<100, 100>::value && nums_ok(x))
                return sign < 0.0 ? u - c : u + c;
        }
        const double p = gamma1 * (en - kin / rho);
        const double c = sqrt(gamma * p / rho);
        return sign < 0.0 ? ru / rho - c : ru / rho + c;
    }

    // Normal solve between cells L and R (RpEuler::rpn2a).  False if an operand
    // leaves the quotients' range.
    template <int IXY>
    static __device__ __forceinline__ bool normal(const double (&qL)[N], const double (&qR)[N], const double (&L)[NCD],
                                                  const double (&R)[NCD], const double* prm, double (&al)[MW],
                                                  double (&am)[N], double (&ap)[N], double (&roe)[NR])
    {
        constexpr int mu = Dir<IXY>::MU, mv = Dir<IXY>::MV;
        const double gamma1 = prm[1];
        const double s0 = L[S0], s3 = R[S3];
        const double rhsq2 = L[0] + R[0], rr = recip_rn(rhsq2);
        const double nu = L[1] + R[1], nv = L[2] + R[2], nh = L[3] + R[3];
        double u = quot_rn(nu, rhsq2, rr), v = quot_rn(nv, rhsq2, rr);
        const double enth = quot_rn(nh, rhsq2, rr), num[2] = {nu, nv};
        if (!nums_ok(num)) { u = low_quot(nu, rhsq2, rr); v = low_quot(nv, rhsq2, rr); }
        const double u2v2 = u * u + v * v;
        const double asq = gamma1 * (enth - .5 * u2v2);
        const double a = sqrt_rn(asq), g1a2 = quot_rn(gamma1, asq, recip_rn(asq));
        const double euv = enth - u2v2, a2x = 2.0 * a, r2a = recip_rn(a2x);
        roe[0] = u; roe[1] = v; roe[2] = a; roe[3] = enth; roe[4] = u2v2; roe[5] = g1a2; roe[6] = euv; roe[7] = r2a;
        const double d0 = qR[0] - qL[0], d1 = qR[mu] - qL[mu], d2 = qR[mv] - qL[mv], d3 = qR[3] - qL[3];
        const double a3 = g1a2 * (euv * d0 + u * d1 + v * d2 - d3);
        const double a2 = d2 - v * d0;
        const double n4 = d1 + (a - u) * d0 - a * a3;
        double a4 = quot_rn(n4, a2x, r2a);
        if (abs_word(n4) < ExpWord<kNumLow>::value && !is_zero(n4)) a4 = low_quot(n4, a2x, r2a);
        const double a1 = d0 - a3 - a4;
        al[0] = a1; al[1] = a2; al[2] = a3; al[3] = a4;
        if constexpr (TRACER) al[4] = qR[4] - qL[4];
        const bool ok = max(pos_word(rhsq2), max(pos_word(asq), pos_word(a2x))) < WordSpan<100, 100>::value &&
                        abs_word(nh) >= ExpWord<kNumLow>::value;

        double w0[N], w1[N], w2[N], w3[N];
        RP::template wave_of<IXY, 0>(a1, rn(roe), w0);
        RP::template wave_of<IXY, 1>(a2, rn(roe), w1);
        RP::template wave_of<IXY, 2>(a3, rn(roe), w2);
        RP::template wave_of<IXY, 3>(a4, rn(roe), w3);
        const double sm = u - a, sp = u + a, gg1 = prm[0] * gamma1;
        // entropy fix.  With s0 >= 0 the wave has a positive speed or none at all
        // goes left; s1 matters only against s0 < 0.
        double s1 = s0;
        {
            const double r = qL[0] + w0[0], ru = qL[mu] + w0[mu], rv = qL[mv] + w0[mv], en = qL[3] + w0[3];
            if (s0 < 0.0 && !star_subsonic(r, ru, rv, en, gg1)) s1 = star_speed(r, ru, rv, en, prm[0], gamma1, -1.0);
        }
        const double f0 = s0 < 0.0 && s1 > 0.0 ? s0 * (s1 - sm) / (s1 - s0) : clip_high(sm);
#pragma unroll
        for (int m = 0; m < N; m++) am[m] = 0.0;
        am[0] = f0 * w0[0]; am[mu] = f0 * w0[mu]; am[mv] = f0 * w0[mv]; am[3] = f0 * w0[3];
        if (u < 0.0) {
            am[0] = am[0] + u * w2[0];
            am[mu] = am[mu] + u * w2[mu];
            am[mv] = am[mv] + u * w1[mv];
            am[mv] = am[mv] + u * w2[mv];
            am[3] = am[3] + u * w1[3];
            am[3] = am[3] + u * w2[3];
            if constexpr (TRACER) am[4] = am[4] + u * al[4];
            // right-going wave: s2 matters only against s3 > 0; mirrored, -s2 is
            // the speed of a left-going wave
            double s2 = s3;
            const double r = qR[0] - w3[0], ru = qR[mu] - w3[mu], rv = qR[mv] - w3[mv], en = qR[3] - w3[3];
            if (s3 > 0.0 && !star_subsonic(r, -ru, rv, en, gg1)) s2 = star_speed(r, ru, rv, en, prm[0], gamma1, 1.0);
            const double f3 = s2 < 0.0 && s3 > 0.0 ? s2 * (s3 - sp) / (s3 - s2) : clip_high(sp);
#pragma unroll
            for (int m = 0; m < 4; m++) am[m] = am[m] + f3 * w3[m];
        }
        double df0 = sm * w0[0];
        df0 = df0 + u * w2[0];
        df0 = df0 + sp * w3[0];
        double dfu = sm * w0[mu];
        dfu = dfu + u * w2[mu];
        dfu = dfu + sp * w3[mu];
        double dfv = sm * w0[mv];
        dfv = dfv + u * w1[mv];
        dfv = dfv + u * w2[mv];
        dfv = dfv + sp * w3[mv];
        double dfe = sm * w0[3];
        dfe = dfe + u * w1[3];
        dfe = dfe + u * w2[3];
        dfe = dfe + sp * w3[3];
        ap[0] = df0 - am[0]; ap[mu] = dfu - am[mu]; ap[mv] = dfv - am[mv]; ap[3] = dfe - am[3];
        if constexpr (TRACER) ap[4] = u * al[4] - am[4];
        return ok;
    }
    // the first NROE of roe, as RP's functions take them
    static __device__ __forceinline__ const double (&rn(const double (&roe)[NR]))[RP::NROE]
    {
        return reinterpret_cast<const double (&)[RP::NROE]>(roe);
    }
    static __device__ __forceinline__ double top_speed(const double (&roe)[NR]) { return fabs(roe[0]) + roe[2]; }
    template <int P> static __device__ __forceinline__ double speed(const double (&roe)[NR]) { return RP::template speed<P>(rn(roe)); }

    // Transverse split (RpEuler::rpt2).  sub: every lane that counts has
    // |v| < a, so v - a and v + a keep their signs.
    static __device__ __forceinline__ bool subsonic(const double (&roe)[NR]) { return fabs(roe[1]) < roe[2]; }
    template <int IXY>
    static __device__ __forceinline__ void split(const double (&x)[N], const double (&roe)[NR], bool sub, double (&bm)[N],
                                                 double (&bp)[N])
    {
        constexpr int mu = Dir<IXY>::MU, mv = Dir<IXY>::MV;
        const double u = roe[0], v = roe[1], a = roe[2], enth = roe[3], u2v2 = roe[4], g1a2 = roe[5], euv = roe[6];
        const double a3 = g1a2 * (euv * x[0] + u * x[mu] + v * x[mv] - x[3]);
        const double a2 = x[mu] - u * x[0];
        const double n4 = x[mv] + (a - v) * x[0] - a * a3;
        double a4 = quot_rn(n4, 2.0 * a, roe[7]);
        if (abs_word(n4) < ExpWord<kNumLow>::value && !is_zero(n4)) a4 = low_quot(n4, 2.0 * a, roe[7]);
        const double a1 = x[0] - a3 - a4;
        const double sb0 = v - a, sb2 = v + a;
        double wb[3][4];
        wb[0][0] = a1; wb[0][mu] = a1 * u; wb[0][mv] = a1 * sb0; wb[0][3] = a1 * (enth - v * a);
        wb[1][0] = a3; wb[1][mu] = a3 * u + a2; wb[1][mv] = a3 * v; wb[1][3] = a3 * 0.5 * u2v2 + a2 * u;
        wb[2][0] = a4; wb[2][mu] = a4 * u; wb[2][mv] = a4 * sb2; wb[2][3] = a4 * (enth + v * a);
        const double mn1 = clip_high(v), mx1 = clip_low(v);
        if (sub) {
#pragma unroll
            for (int m = 0; m < 4; m++) {
                bm[m] = sb0 * wb[0][m] + mn1 * wb[1][m];
                bp[m] = mx1 * wb[1][m] + sb2 * wb[2][m];
            }
        } else {
            const double mn0 = clip_high(sb0), mn2 = clip_high(sb2), mx0 = clip_low(sb0), mx2 = clip_low(sb2);
#pragma unroll
            for (int m = 0; m < 4; m++) {
                double b = mn0 * wb[0][m];
                b = b + mn1 * wb[1][m];
                bm[m] = b + mn2 * wb[2][m];
                double c = mx0 * wb[0][m];
                c = c + mx1 * wb[1][m];
                bp[m] = c + mx2 * wb[2][m];
            }
        }
        if constexpr (TRACER) { bm[4] = mn1 * x[4]; bp[4] = mx1 * x[4]; }
    }
};

// ---------------------------------------------------------------------------
// shallow water
// ---------------------------------------------------------------------------
struct DenseShallow {
    using RP = RpShallow;
    static constexpr int N = 3, MW = 3;
    static constexpr int NCD = 5;                      // cell: sq, U, V (normal, transverse), s0, s3
    static constexpr int S0 = 3, S3 = 4;
    static constexpr int NR = 4;                       // ubar, vbar, cbar, 1 / (2 cbar)
    template <int IXY> static constexpr __host__ __device__ bool wave_has(int p, int m) { return p != 1 || m == Dir<IXY>::MV; }

    template <int IXY>
    static __device__ __forceinline__ bool cell(const double (&q)[N], const double* prm, double (&c)[NCD])
    {
        constexpr int mu = Dir<IXY>::MU, mv = Dir<IXY>::MV;
        const double gh = prm[0] * q[0];
        const double r0 = recip_rn(q[0]), sq = sqrt_rn(q[0]), rs = recip_rn(sq), cs = sqrt_rn(gh);
        const double un = quot_rn(q[mu], q[0], r0);
        c[0] = sq;
        c[1] = quot_rn(q[mu], sq, rs);
        c[2] = quot_rn(q[mv], sq, rs);
        c[S0] = un - cs; c[S3] = un + cs;          // a velocity too small to be exact is nothing beside cs
        const bool ok = max(pos_word(q[0]), pos_word(gh)) < WordSpan<100, 100>::value;
        const double x[2] = {q[1], q[2]};
        if (!nums_ok(x)) { c[1] = low_quot(q[mu], sq, rs); c[2] = low_quot(q[mv], sq, rs); }
        return ok;
    }
    template <int IXY>
    static __device__ __noinline__ void cell_plain(const double* q, double prm0, double, double* c)
    {
        const double prm[1] = {prm0};
        const double a[N] = {q[0], q[1], q[2]};
        const RP::Cell x = RP::cell<IXY>(a, prm);
        c[0] = x.sq; c[1] = x.U; c[2] = x.V;
        c[S0] = x.un - x.c; c[S3] = x.un + x.c;
    }
    // hu <= 0, or hu^2 < g h^3 by a margin far above the rounding errors
    static __device__ __forceinline__ bool star_subsonic(double h, double hu, double grav)
    {
        const double u2 = hu * hu, cc = grav * h * (h * h);
        return h > 0.0 && (hu <= 0.0 || cc - u2 > 0x1p-40 * (cc + u2));
    }
    static __device__ __noinline__ double star_speed(double h, double hu, double grav, double sign)
    {
        const double gh = grav * h, c = sqrt(gh);
        const double u = abs_word(hu) >= ExpWord<kNumLow>::value && pos_word(h) < WordSpan<100, 100>::value
                             ? quot_rn(hu, h, recip_rn(h)) : hu / h;
        return sign < 0.0 ? u - c : u + c;
    }
    template <int IXY>
    static __device__ __forceinline__ bool normal(const double (&qL)[N], const double (&qR)[N], const double (&L)[NCD],
                                                  const double (&R)[NCD], const double* prm, double (&al)[MW],
                                                  double (&am)[N], double (&ap)[N], double (&roe)[NR])
    {
        constexpr int mu = Dir<IXY>::MU, mv = Dir<IXY>::MV;
        const double grav = prm[0];
        const double s0 = L[S0], s3 = R[S3];
        const double hsq2 = L[0] + R[0], rr = recip_rn(hsq2);
        const double nu = L[1] + R[1], nv = L[2] + R[2];
        double ubar = quot_rn(nu, hsq2, rr), vbar = quot_rn(nv, hsq2, rr);
        const double num[2] = {nu, nv};
        if (!nums_ok(num)) { ubar = low_quot(nu, hsq2, rr); vbar = low_quot(nv, hsq2, rr); }
        const double hbar = 0.5 * (qL[0] + qR[0]);
        const double ghb = grav * hbar, cbar = sqrt_rn(ghb), c2x = 2.0 * cbar, r2c = recip_rn(c2x);
        const double d1 = qR[0] - qL[0], d2 = qR[mu] - qL[mu], d3 = qR[mv] - qL[mv];
        roe[0] = ubar; roe[1] = vbar; roe[2] = cbar; roe[3] = r2c;
        const double sm = ubar - cbar, sp = ubar + cbar;
        const double n1 = sp * d1 - d2, n3 = d2 - sm * d1;
        double a1 = quot_rn(n1, c2x, r2c), a3 = quot_rn(n3, c2x, r2c);
        const double a2 = d3 - vbar * d1, x[2] = {n1, n3};
        if (!nums_ok(x)) { a1 = low_quot(n1, c2x, r2c); a3 = low_quot(n3, c2x, r2c); }
        al[0] = a1; al[1] = a2; al[2] = a3;
        const bool ok = max(pos_word(hsq2), max(pos_word(ghb), pos_word(c2x))) < WordSpan<100, 100>::value;
        const double w0u = a1 * sm, w0v = a1 * vbar, w2u = a3 * sp, w2v = a3 * vbar;
        double s1 = s0;
        {
            const double h1 = qL[0] + a1, hu1 = qL[mu] + w0u;
            if (s0 < 0.0 && !star_subsonic(h1, hu1, grav)) s1 = star_speed(h1, hu1, grav, -1.0);
        }
        const double f0 = s0 < 0.0 && s1 > 0.0 ? s0 * (s1 - sm) / (s1 - s0) : clip_high(sm);
        am[0] = f0 * a1; am[mu] = f0 * w0u; am[mv] = f0 * w0v;
        if (ubar < 0.0) {
            am[mv] = am[mv] + ubar * a2;
            double s2 = s3;
            const double h2 = qR[0] - a3, hu2 = qR[mu] - w2u;
            if (s3 > 0.0 && !star_subsonic(h2, -hu2, grav)) s2 = star_speed(h2, hu2, grav, 1.0);
            const double f2 = s2 < 0.0 && s3 > 0.0 ? s2 * (s3 - sp) / (s3 - s2) : clip_high(sp);
            am[0] = am[0] + f2 * a3;
            am[mu] = am[mu] + f2 * w2u;
            am[mv] = am[mv] + f2 * w2v;
        }
        const double df0 = sm * a1 + sp * a3, dfu = sm * w0u + sp * w2u;
        double dfv = sm * w0v;
        dfv = dfv + ubar * a2;
        dfv = dfv + sp * w2v;
        ap[0] = df0 - am[0]; ap[mu] = dfu - am[mu]; ap[mv] = dfv - am[mv];
        return ok;
    }
    static __device__ __forceinline__ const double (&rn(const double (&roe)[NR]))[RP::NROE]
    {
        return reinterpret_cast<const double (&)[RP::NROE]>(roe);
    }
    static __device__ __forceinline__ double top_speed(const double (&roe)[NR]) { return fabs(roe[0]) + roe[2]; }
    template <int P> static __device__ __forceinline__ double speed(const double (&roe)[NR]) { return RP::speed<P>(rn(roe)); }
    static __device__ __forceinline__ bool subsonic(const double (&roe)[NR]) { return fabs(roe[1]) < roe[2]; }
    template <int IXY>
    static __device__ __forceinline__ void split(const double (&x)[N], const double (&roe)[NR], bool sub, double (&bm)[N],
                                                 double (&bp)[N])
    {
        constexpr int mu = Dir<IXY>::MU, mv = Dir<IXY>::MV;
        const double u = roe[0], v = roe[1], c = roe[2], c2x = 2.0 * c;
        const double sb0 = v - c, sb2 = v + c;
        const double n1 = sb2 * x[0] - x[mv], n3 = x[mv] - sb0 * x[0];
        double a1 = quot_rn(n1, c2x, roe[3]), a3 = quot_rn(n3, c2x, roe[3]);
        const double a2 = x[mu] - u * x[0], y[2] = {n1, n3};
        if (!nums_ok(y)) { a1 = low_quot(n1, c2x, roe[3]); a3 = low_quot(n3, c2x, roe[3]); }
        const double w0u = a1 * u, w0v = a1 * sb0, w2u = a3 * u, w2v = a3 * sb2;
        const double mn1 = clip_high(v), mx1 = clip_low(v);
        if (sub) {
            bm[0] = sb0 * a1; bp[0] = sb2 * a3;
            bm[mu] = sb0 * w0u + mn1 * a2; bp[mu] = mx1 * a2 + sb2 * w2u;
            bm[mv] = sb0 * w0v; bp[mv] = sb2 * w2v;
        } else {
            const double mn0 = clip_high(sb0), mn2 = clip_high(sb2), mx0 = clip_low(sb0), mx2 = clip_low(sb2);
            bm[0] = mn0 * a1 + mn2 * a3;
            bp[0] = mx0 * a1 + mx2 * a3;
            double b = mn0 * w0u;
            b = b + mn1 * a2;
            bm[mu] = b + mn2 * w2u;
            double e = mx0 * w0u;
            e = e + mx1 * a2;
            bp[mu] = e + mx2 * w2u;
            bm[mv] = mn0 * w0v + mn2 * w2v;
            bp[mv] = mx0 * w0v + mx2 * w2v;
        }
    }
};

template <class RP> struct DenseOf;
template <bool T> struct DenseOf<RpEuler<T>> { using type = DenseEuler<T>; };
template <> struct DenseOf<RpShallow> { using type = DenseShallow; };

// The plain solver for an interface whose operands leave the quotients' range:
// in[0 .. 2N) the two states, out: al, am, ap, roe.
template <class D, int IXY>
static __device__ __noinline__ void dense_normal_plain(const double* in, double prm0, double prm1, double* out)
{
    const double prm[2] = {prm0, prm1};
    using RP = typename D::RP;
    constexpr int N = D::N, MW = D::MW, NR = D::NR;
    double qL[N], qR[N], al[MW], am[N], ap[N], roe[RP::NROE];
#pragma unroll
    for (int m = 0; m < N; m++) { qL[m] = in[m]; qR[m] = in[N + m]; }
    RP::template rpn2a<IXY>(qL, qR, RP::template cell<IXY>(qL, prm), RP::template cell<IXY>(qR, prm), prm, al, am, ap, roe);
#pragma unroll
    for (int p = 0; p < MW; p++) out[p] = al[p];
#pragma unroll
    for (int m = 0; m < N; m++) { out[MW + m] = am[m]; out[MW + N + m] = ap[m]; }
#pragma unroll
    for (int r = 0; r < RP::NROE; r++) out[MW + 2 * N + r] = roe[r];
    out[MW + 2 * N + NR - 1] = 1.0 / (2.0 * roe[2]);
}
// Limiter values of an interface's waves: philim of dot / wn, 1 for a wave too
// small to square.  ma: the limiter of waves 0 .. MA-1 if they share it (else
// -1), mt that of the tracer's wave.
static __device__ __noinline__ double philim_other(double r, int m) { return m != 0 ? philim_r(r, m) : 1.0; }
// dot / wn out of ratio_ok's range.  Far from a wave's front the squares are tiny:
// both scaled up (exactly), or dot alone, else the division itself.
static __device__ __noinline__ double ratio_cold(double dot, double wn)
{
    const double sc = abs_word(wn) < ExpWord<-800>::value ? 0x1p600 : 1.0;
    const double x = dot * sc, y = wn * sc;
    if (word_in<900, 100>(y)) {
        const double r = recip_rn(y);
        if (ratio_ok(x, y)) return quot_rn(x, y, r);
        if (abs_word(x) < ExpWord<-900>::value) {
            const double s = quot_rn(x * 0x1p300, y, r);
            if (abs_word(s) >= ExpWord<-721>::value) return s * 0x1p-300;
        }
    }
    return dot / wn;
}
template <class D>
__device__ __forceinline__ void dense_limit(double (&ph)[D::MW], const double (&dot)[D::MW], const double (&wn)[D::MW],
                                            const StepArgs& a, bool used)
{
    constexpr int MW = D::MW, MA = MW == 5 ? 4 : MW;
    const int ma = a.limit_first, mt = a.mthlim[MW - 1];
    unsigned top = 0;
#pragma unroll
    for (int p = 0; p < MW; p++) {
        ph[p] = quot_rn(dot[p], wn[p], recip_rn(wn[p]));
        top = max(top, max(word_above<900>(wn[p]), word_above<900>(dot[p])));
    }
    const bool odd = used && top >= WordSpan<900, 100>::value;      // zeros among them, or out of range
    if (odd) {
#pragma unroll
        for (int p = 0; p < MW; p++)
            if (!is_zero(wn[p]) && !ratio_ok(dot[p], wn[p])) ph[p] = ratio_cold(dot[p], wn[p]);
    }
    if (ma == 4) {
#pragma unroll
        for (int p = 0; p < MA; p++) ph[p] = philim_mc(ph[p]);
    } else if (ma == 1) {
#pragma unroll
        for (int p = 0; p < MA; p++) ph[p] = philim_minmod(ph[p]);
    } else if (ma == 2) {
#pragma unroll
        for (int p = 0; p < MA; p++) ph[p] = philim_superbee(ph[p]);
    } else {
#pragma unroll
        for (int p = 0; p < MA; p++) ph[p] = philim_other(ph[p], a.mthlim[p]);
    }
    if constexpr (MW > MA) {
        if (mt == 4) ph[MA] = philim_mc(ph[MA]);
        else if (mt == 2) ph[MA] = philim_superbee(ph[MA]);
        else ph[MA] = philim_other(ph[MA], mt);
    }
    if (odd) {
#pragma unroll
        for (int p = 0; p < MW; p++) ph[p] = is_zero(wn[p]) ? 1.0 : ph[p];
    }
}

// A cell's quantities, with the plain solver's where an operand leaves the range.
template <class D, int IXY>
__device__ __forceinline__ void dense_cell(const StepArgs& a, const double (&q)[D::N], bool used, double (&c)[D::NCD])
{
    if (!D::template cell<IXY>(q, a.prm, c) && used) {
        double t[D::N], o[D::NCD];
#pragma unroll
        for (int m = 0; m < D::N; m++) t[m] = q[m];
        D::template cell_plain<IXY>(t, a.prm[0], a.prm[1], o);
#pragma unroll
        for (int k = 0; k < D::NCD; k++) c[k] = o[k];
    }
}

template <class D, int IXY>
__device__ __forceinline__ void dense_normal(const StepArgs& a, const double (&qL)[D::N], const double (&qR)[D::N],
                                             const double (&L)[D::NCD], const double (&R)[D::NCD], bool used,
                                             double (&al)[D::MW], double (&am)[D::N], double (&ap)[D::N],
                                             double (&roe)[D::NR])
{
    constexpr int N = D::N, MW = D::MW, NR = D::NR;
    if (!D::template normal<IXY>(qL, qR, L, R, a.prm, al, am, ap, roe) && used) {
        double in[2 * N], out[MW + 2 * N + NR];
#pragma unroll
        for (int m = 0; m < N; m++) { in[m] = qL[m]; in[N + m] = qR[m]; }
        dense_normal_plain<D, IXY>(in, a.prm[0], a.prm[1], out);
#pragma unroll
        for (int p = 0; p < MW; p++) al[p] = out[p];
#pragma unroll
        for (int m = 0; m < N; m++) { am[m] = out[MW + m]; ap[m] = out[MW + N + m]; }
#pragma unroll
        for (int r = 0; r < NR; r++) roe[r] = out[MW + 2 * N + r];
    }
}

// sum over the components of wave p of two interfaces, in component order
template <class D, int IXY, int P>
__device__ __forceinline__ double wave_dot(const double (&w)[D::N], const double (&v)[D::N])
{
    double s = 0.0;
    bool any = false;
#pragma unroll
    for (int m = 0; m < D::N; m++)
        if (D::template wave_has<IXY>(P, m)) {
            const double t = w[m] * v[m];
            s = any ? s + t : t;
            any = true;
        }
    return s;
}

// Correction of one interface from its waves (strengths al) and dot products
// with the waves on its right (dr) and left (dl).
template <class D, int IXY>
__device__ __forceinline__ void dense_correct(const StepArgs& a, const double (&al)[D::MW], const double (&roe)[D::NR], const double (&dr)[D::MW],
                                              const double (&dl)[D::MW], double dtn, bool used, double (&cq)[D::N])
{
    using RP = typename D::RP;
    constexpr int N = D::N, MW = D::MW;
    double ph[MW];
    if (a.limit_any) {
        double wn[MW], dot[MW];
        static_for<MW>([&](auto P) {
            constexpr int p = decltype(P)::value;
            double w[N];
            RP::template wave_of<IXY, p>(al[p], D::rn(roe), w);
            wn[p] = wave_dot<D, IXY, p>(w, w);
            dot[p] = D::template speed<p>(roe) > 0.0 ? dl[p] : dr[p];
        });
        dense_limit<D>(ph, dot, wn, a, used);
    } else {
#pragma unroll
        for (int p = 0; p < MW; p++) ph[p] = 1.0;
    }
    bool any[N];
#pragma unroll
    for (int m = 0; m < N; m++) { cq[m] = 0.0; any[m] = false; }
    static_for<MW>([&](auto P) {
        constexpr int p = decltype(P)::value;
        double w[N];
        RP::template wave_of<IXY, p>(al[p], D::rn(roe), w);
        const double as = fabs(D::template speed<p>(roe));
        const double f = as * (1.0 - as * dtn);
#pragma unroll
        for (int m = 0; m < N; m++)
            if (D::template wave_has<IXY>(p, m)) {
                const double t = f * (ph[p] * w[m]);
                cq[m] = any[m] ? cq[m] + t : t;
                any[m] = true;
            }
    });
}

// products of the waves of two neighbouring interfaces, summed in component order
template <class D, int IXY>
__device__ __forceinline__ void dense_dots(const double (&al)[D::MW], const double (&roe)[D::NR], const double (&bl)[D::MW],
                                           const double (&roeb)[D::NR], double (&dr)[D::MW])
{
    using RP = typename D::RP;
    constexpr int N = D::N;
    static_for<D::MW>([&](auto P) {
        constexpr int p = decltype(P)::value;
        double w[N], v[N];
        RP::template wave_of<IXY, p>(al[p], D::rn(roe), w);
        RP::template wave_of<IXY, p>(bl[p], D::rn(roeb), v);
        dr[p] = wave_dot<D, IXY, p>(w, v);
    });
}

}  // namespace claw2
