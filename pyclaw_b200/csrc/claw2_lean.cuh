// claw2_lean.cuh -- the step of the solvers with dense waves and no aux arrays
// (Euler 4- and 5-wave Roe, shallow-water Roe), unsplit or split, on square
// tiles of T = 28 or 12 cells.
//
// Same step as step_tile_at (step2.f90:92-248, step2ds.f90:96-252, flux2.f90:
// 104-206) with the same operations in the same order, so the results are the
// same values; only the data movement differs:
//  - a line of the tile (a row in the x sweep, a column in the y sweep) is held
//    by T + 4 lanes, one cell each, cells i0-2 .. i0+T+1: a warp holds one line
//    of a 28-tile or two of a 12-tile;
//  - each lane computes the quantities of its cell that the normal solve needs
//    (dense_cell: square roots, pressures, Roe-average numerators) and takes
//    those of the cell right of its interface from the next lane, so each
//    cell's are computed once per line instead of once per interface;
//  - the solves are those of claw2_dense.cuh: the same bits from fewer
//    instructions and no divergent divisions;
//  - the normal solve stays in registers; for the limiter each lane takes its
//    right neighbour's wave strengths and Roe averages by warp shuffle and forms
//    dotr = wave(k).wave(k+1); dotl of lane k is dotr of lane k-1 (one more
//    shuffle), the same products summed in the same component order (a*b ==
//    b*a exactly);
//  - a line whose cells hold one state carries no waves: its corrections and
//    splits are passed over;
//  - what the cell left of an interface needs from it (dtdx*amdq, fadd and
//    the two transverse splits) moves one lane by shuffle;
//  - unsplit, a cell's own-line contributions stay in registers; only the two
//    cross-line terms (to the line above and below) go through a
//    double-buffered shared array: one block barrier per chunk of lines;
//  - split, a line depends on no other: the x sweep rewrites the rows of the
//    staged halo in place, and one block barrier later the y sweep reads its
//    columns;
//  - the tile's whole input halo (rows j0-2..j0+T+1, columns i0-2..i0+T+1)
//    is staged in shared memory once by the tensor memory accelerator (boxes
//    of 16 columns x T+4 rows x MEQN fields, 128-byte swizzle; see
//    claw2_tma.cuh) while the threads wait on an mbarrier; x lines read rows
//    of it and y lines read down its columns;
//  - a tile whose halo holds one state skips both sweeps: every interface
//    would join two equal states, so its cells keep their values and its CFL
//    number comes from one Riemann solve (uniform_cfl).  On large grids a pass
//    of its own looks for such tiles (lean_scan_tile).
//
// Bound by the latency of the FP64 chains and by issue: 128 registers a thread
// leave 4 warps per SM quarter, which issue 51% of the cycles (the developed Euler
// 1280 x 320; FP64 pipe 41% busy; stalled on dependences 1.9 and barriers 0.7 of the
// 7.7 warp-cycles per instruction).  80 registers and 6 warps spill and lose (Euler 1500^2 391 us
// against 280, split 197 against 175).  us a step on a B200, before (the solves
// of claw2_riemann.cuh; split, the general body; 28-tiles only) and now:
//                     64 x 48      256^2        641 x 163    1500^2
//   Euler 4 unsplit   36.5  14.0   36.7  25.2   36.8  26.6   331  261
//   Euler 4 split     44.5  11.0   47.9  20.6   49.9  21.7   394  189
//   Euler 5 unsplit   40.0  15.2   40.0  29.3   40.0  30.7   532  313
//   Euler 5 split     47.8  12.3   48.9  22.5   49.2  23.7   697  224
//   shallow unsplit   25.8  10.3   26.4  18.4   26.6  19.5   367  284
//   shallow split     29.5   8.7   31.5  14.6   32.7  16.1   275  183
// (1500^2 without still tiles: the pass that looks for them costs the split forms
// up to 4% there, see launch_lean_rp.)
#pragma once

#include "claw2_dense.cuh"
#include "claw2_kernels.cuh"
#include "claw2_tma.cuh"

namespace claw2 {

// Shared memory of the lean body (doubles): the staged input halo (T+4 rows and
// columns, in boxes of 16 columns, at a 1024-byte boundary for the swizzle), the
// tile's new state, unsplit the cross-line exchange (2 buffers x 2 terms x MEQN x
// cells of a chunk), and the reduction scratch; `bytes` includes up to 1 KB of alignment
// padding in front of the halo.
template <class RP, int T, int NT, bool SPLIT> struct LeanSmem {
    static constexpr int MEQN = RP::MEQN;
    static constexpr int QP = T | 1;             // row pitch of the tile state: odd, so that
                                                 // y lines walking down a column avoid bank conflicts
    static constexpr int QX = MEQN * T * QP;
    static constexpr int LPC = NT / (T + 4);      // lines of a chunk
    static constexpr int NX = LPC * T;           // their cells
    static constexpr int CX = SPLIT ? 0 : 2 * 2 * MEQN * NX;
    static constexpr int TR = T + 4;             // rows j0-2 .. j0+T+1; also the lanes of a line
    static constexpr int NBOX = TR / 16;
    static constexpr int BOX = MEQN * TR * 16;   // one box: columns 16b .. 16b+15 of the halo
    static constexpr int HS = NBOX * BOX;
    static constexpr int total = HS + QX + CX + NT / 32;
    static constexpr int bytes = total * 8 + 1024;
    static_assert(TR == 16 || TR == 32, "lines of 16 or 32 lanes, boxes of 16 columns");
    static_assert((BOX * 8) % 1024 == 0, "each box starts on a 1024-byte boundary");
};

// The staged input of halo row r, column c, field m: H holds q(m, i0-2+c, j0-2+r).
template <int MEQN, int TR>
__device__ __forceinline__ int lean_hidx(int m, int r, int c)
{
    return (c >> 4) * (MEQN * TR * 16) + m * (TR * 16) + swz128(r, c & 15);
}

// The part of a line that both forms of the step share.  `line` is a line of the
// halo, the lane's interface is k, its left cell k-1.
template <class RP, int IXY, int T> struct LeanLine {
    using D = typename DenseOf<RP>::type;
    static constexpr int MEQN = RP::MEQN, MW = RP::MW, TR = T + 4, NSLOT = T + 3;
    int slot, k, len;
    bool ifok, lim;              // a limiter neighbour; an interface whose flux counts
    bool flat;                   // the warp's lines carry no waves
    double q[MEQN];              // cell k
    double amdq[MEQN], apdq[MEQN], roe[D::NR], cqxx[MEQN];

    // the staged input of cell (kk along the line, ll across it)
    static __device__ __forceinline__ int at(int m, int kk, int ll, int i0, int j0)
    {
        return IXY == 1 ? lean_hidx<MEQN, TR>(m, ll - j0 + 2, kk - i0 + 2) : lean_hidx<MEQN, TR>(m, kk - j0 + 2, ll - i0 + 2);
    }
    // normal solve, CFL number, second-order correction
    template <class Ctx>
    __device__ __forceinline__ void solve(const StepArgs& a, Ctx& ctx, const double* H, int i0, int j0, int line, bool lineok,
                                          double dtn, double& cflm)
    {
        constexpr int NR = D::NR, NCD = D::NCD;
        slot = ctx.tid() & (TR - 1);
        len = IXY == 1 ? a.mx : a.my;
        k = (IXY == 1 ? i0 : j0) - 1 + slot;
        ifok = lineok && slot < NSLOT && k <= len + 1;
        lim = ifok && slot >= 1 && slot <= NSLOT - 2 && k >= 0 && k <= len;
        double al[MW];
        {
            // this lane's cell k-1, and cell k from the next lane
            double qL[MEQN], L[NCD], R[NCD];
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                qL[m] = H[at(m, k - 1, line, i0, j0)];
                q[m] = H[at(m, slot < NSLOT ? k : k - 1, line, i0, j0)];
            }
            dense_cell<D, IXY>(a, qL, lineok && k - 1 <= len + 1, L);
#pragma unroll
            for (int f = 0; f < NCD; f++) R[f] = f != D::S0 ? ctx.shfl_down(L[f]) : 0.0;
            bool eq = true;
#pragma unroll
            for (int m = 0; m < MEQN; m++) eq = eq && qL[m] == q[m];
            flat = __all_sync(0xffffffffu, eq || !ifok);
            dense_normal<D, IXY>(a, qL, q, L, R, ifok, al, amdq, apdq, roe);
        }
        if (lim) {
            const double c = fabs(dtn) * D::top_speed(roe);     // the largest of dtn s and -dtn s over the waves
            cflm = cflm > c ? cflm : c;
        }
#pragma unroll
        for (int m = 0; m < MEQN; m++) cqxx[m] = 0.0;
        if (flat || a.order != 2) return;
        double dr[MW], dl[MW];
        if (a.limit_any) {
            double alr[MW], roer[NR];
#pragma unroll
            for (int p = 0; p < MW; p++) alr[p] = ctx.shfl_down(al[p]);
#pragma unroll
            for (int r = 0; r < NR; r++) roer[r] = r < RP::NROE_WAVE ? ctx.shfl_down(roe[r]) : 0.0;
            dense_dots<D, IXY>(al, roe, alr, roer, dr);
#pragma unroll
            for (int p = 0; p < MW; p++) dl[p] = ctx.shfl_up(dr[p]);
        }
        dense_correct<D, IXY>(a, al, roe, dr, dl, dtn, lim, cqxx);
    }
};

// One line of the split step (step2ds.f90:96-252): the x sweep rewrites its row of
// H, the y sweep writes its column of the new state; `own`: the line's cells are
// swept (ghost columns only count in the CFL number).
template <class RP, int IXY, int T, int NT, class Ctx>
__device__ __forceinline__ void lean_split_line(const StepArgs& a, Ctx& ctx, double* H, double* Qx, int i0, int j0, int line,
                                                bool lineok, bool own, double dtn, double& cflm)
{
    using LL = LeanLine<RP, IXY, T>;
    using SM = LeanSmem<RP, T, NT, true>;
    constexpr int MEQN = RP::MEQN;
    LL S;
    S.solve(a, ctx, H, i0, j0, line, lineok, dtn, cflm);
    double v[MEQN];
#pragma unroll
    for (int m = 0; m < MEQN; m++) {
        const double y0 = ctx.shfl_down(dtn * S.amdq[m]), y1 = ctx.shfl_down(0.5 * S.cqxx[m]);
        v[m] = S.q[m] + (-(dtn * S.apdq[m]) - y0) - dtn * (y1 - 0.5 * S.cqxx[m]);
    }
    __syncwarp();                                  // the row has been read
    if (own && S.lim && S.slot <= T && S.k < S.len) {
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            if (IXY == 1) H[LL::at(m, S.k, line, i0, j0)] = v[m];
            else Qx[(m * T + (S.k - j0)) * SM::QP + (line - i0)] = v[m];
        }
    }
}

// One chunk of one sweep direction (arguments as in sweep_chunk); CXb is the
// half of the exchange array this chunk uses.
template <class RP, int IXY, int T, int NT, class Ctx>
__device__ __forceinline__ void lean_chunk(const StepArgs& a, Ctx& ctx, const double* H, double* Qx, double* CXb, int i0, int j0,
                         int line, int cfirst, int clast, bool lineok, double dtn, double dtt, double& cflm)
{
    constexpr int MEQN = RP::MEQN;
    using SM = LeanSmem<RP, T, NT, false>;
    using LL = LeanLine<RP, IXY, T>;
    using D = typename LL::D;
    constexpr int NCELL = T, LANES = SM::TR;
    LL S;
    S.solve(a, ctx, H, i0, j0, line, lineok, dtn, cflm);
    const int tid = ctx.tid(), slot = S.slot, k = S.k, len = S.len;
    const bool lim = S.lim;
    const double (&amdq)[MEQN] = S.amdq, (&apdq)[MEQN] = S.apdq, (&cqxx)[MEQN] = S.cqxx;
    auto hq = [&](int m, int kk, int ll) -> double { return H[LL::at(m, kk, ll, i0, j0)]; };

    double fadd[MEQN], bmL[MEQN], bpL[MEQN], bmR[MEQN], bpR[MEQN];
#pragma unroll
    for (int m = 0; m < MEQN; m++) { bmL[m] = 0.0; bpL[m] = 0.0; bmR[m] = 0.0; bpR[m] = 0.0; }
    // ---------------- transverse splits (a line of one state carries no waves) ----------------
    if (!S.flat && a.trans > 0) {
        const bool cor = a.order == 2 && a.trans == 2;
        double A[MEQN], Pf[MEQN];
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            A[m] = cor ? amdq[m] + cqxx[m] : amdq[m];
            Pf[m] = cor ? apdq[m] - cqxx[m] : apdq[m];
        }
        const bool sub = __all_sync(0xffffffffu, D::subsonic(S.roe) || !lim);
        D::template split<IXY>(A, S.roe, sub, bmL, bpL);
        D::template split<IXY>(Pf, S.roe, sub, bmR, bpR);
    }
#pragma unroll
    for (int m = 0; m < MEQN; m++) fadd[m] = 0.5 * cqxx[m];

    // ---------------- the slice's contributions to cell k ----------------
    // what interface k+1 hands to its left cell (this lane's cell k)
    const double hl = 0.5 * dtn;
    double y0[MEQN], y1[MEQN], y2[MEQN], y3[MEQN];
#pragma unroll
    for (int m = 0; m < MEQN; m++) {
        // a cell-owning lane (cellok) takes these from lane k+1, which is
        // always a limited interface (lim), so no lane needs them zeroed
        y0[m] = ctx.shfl_down(dtn * amdq[m]);
        y1[m] = ctx.shfl_down(fadd[m]);
        y2[m] = ctx.shfl_down(hl * bmL[m]);
        y3[m] = ctx.shfl_down(hl * bpL[m]);
    }
    const bool cellok = lim && slot <= NCELL && k < len;
    const bool trans = a.trans > 0;
    double C0[MEQN], C1[MEQN], C2[MEQN], C3[MEQN], C4[MEQN];
#pragma unroll
    for (int m = 0; m < MEQN; m++) {
        C0[m] = 0.0; C1[m] = 0.0; C2[m] = 0.0; C3[m] = 0.0; C4[m] = 0.0;
    }
    if (cellok) {
        const double hr = 0.5 * dtn;
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            const double qadd = -(dtn * apdq[m]) - y0[m];
            const double dF = y1[m] - fadd[m];
            const double g1 = -y2[m] - hr * bmR[m];
            const double g2 = -y3[m] - hr * bpR[m];
            C0[m] = dtt * g2;
            C1[m] = qadd;
            C2[m] = dtn * dF;
            C3[m] = dtt * (g2 - g1);
            C4[m] = dtt * g1;
        }
    }
    constexpr int NX = SM::NX;
    const int mine = tid / LANES * T + slot - 1;
    if (cellok) {
#pragma unroll
        for (int m = 0; m < MEQN; m++) {
            CXb[m * NX + mine] = C0[m];
            CXb[(MEQN + m) * NX + mine] = C4[m];
        }
    }
    ctx.sync();

    // ---------------- combine slices line-1, line, line+1 per cell ----------------
    if (cellok) {
        auto qx = [&](int m, int kk, int ll) -> double& {
            const int ci = IXY == 1 ? kk : ll, cj = IXY == 1 ? ll : kk;
            return Qx[(m * T + (cj - j0)) * SM::QP + (ci - i0)];
        };
        auto qi = [&](int m, int kk, int ll) -> double { return IXY == 1 ? hq(m, kk, ll) : qx(m, kk, ll); };
        auto in_tile_line = [&](int ll) {
            return IXY == 1 ? (ll >= j0 && ll < j0 + T && ll < a.my) : (ll >= i0 && ll < i0 + T && ll < a.mx);
        };
        const int up = mine - T, dn = mine + T;         // the lanes of lines line-1 and line+1
        if (in_tile_line(line)) {
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                double v;
                if (line == cfirst) v = qx(m, k, line);                 // has up(line-1) already
                else {
                    v = qi(m, k, line);
                    if (trans) v = v + CXb[m * NX + up];
                }
                if (IXY == 1) {
                    v = v + C1[m] - C2[m];
                    if (trans) v = v - C3[m];
                } else {
                    v = v + (trans ? (C1[m] - C2[m] - C3[m]) : (C1[m] - C2[m]));
                }
                if (trans && line != clast) v = v - CXb[(MEQN + m) * NX + dn];
                qx(m, k, line) = v;
            }
        }
        if (line == clast && in_tile_line(line + 1)) {
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                double v = qi(m, k, line + 1);
                if (trans) v = v + C0[m];
                qx(m, k, line + 1) = v;
            }
        }
        if (trans && line == cfirst && in_tile_line(line - 1)) {
#pragma unroll
            for (int m = 0; m < MEQN; m++) qx(m, k, line - 1) = qx(m, k, line - 1) - C4[m];
        }
    }
}

// True in every thread when the tile's input halo (rows j0-2..j0+T+1,
// columns i0-2..i0+T+1, clipped to the ghosted array: every cell either sweep
// reads) holds one state.  A NaN never compares equal, so a non-finite halo
// is never uniform.
template <class RP, int TR>
__device__ __forceinline__ bool lean_uniform_halo(const StepArgs& a, const double* H, int i0, int j0, int tid, int nt)
{
    constexpr int MEQN = RP::MEQN;
    const int rmax = a.my + 3 - j0, cmax = a.mx + 3 - i0;   // last halo row / column inside the array
    double q0[MEQN];
#pragma unroll
    for (int m = 0; m < MEQN; m++) q0[m] = H[lean_hidx<MEQN, TR>(m, 0, 0)];
    bool same = true;
    // columns c, c+1 (c even) sit side by side in the swizzled box: one
    // 16-byte load per pair
    for (int e = tid; e < TR * (TR / 2); e += nt) {
        const int r = e / (TR / 2), c = (e % (TR / 2)) * 2;
        if (r <= rmax && c <= cmax) {
#pragma unroll
            for (int m = 0; m < MEQN; m++) {
                const double2 v = *reinterpret_cast<const double2*>(H + lean_hidx<MEQN, TR>(m, r, c));
                same = same && v.x == q0[m] && (c + 1 > cmax || v.y == q0[m]);
            }
        }
    }
    return __syncthreads_and(same);
}

// The two sweeps of the full tile step over the staged halo H; returns this
// thread's running CFL maximum.
template <class RP, int T, int NT, bool SPLIT, class Ctx>
__device__ __forceinline__ double lean_tile_sweeps(const StepArgs& a, Ctx& ctx, double* H, double* Qx, double* CX, int i0,
                                                   int j0, double dtdx, double dtdy)
{
    constexpr int MEQN = RP::MEQN;
    using SM = LeanSmem<RP, T, NT, SPLIT>;
    constexpr int LPC = SM::LPC;
    const int mine = ctx.tid() / (T + 4);
    double cflm = 0.0;
    if constexpr (SPLIT) {
        // rows of the halo, each by itself; then the tile's columns of the swept
        // rows, and the ghost columns beside it
        // A warp past the last line leaves (`lead`: its first line of a pass): the lines
        // are rewritten in place, and it would read one that another warp writes.
        const int lead = ctx.tid() / 32 * (32 / (T + 4));
        const int first = j0 - 2, last = j0 + T + 1 < a.my + 1 ? j0 + T + 1 : a.my + 1;
        for (int c0 = first; c0 + lead <= last; c0 += LPC) {
            const int line = c0 + mine;
            lean_split_line<RP, 1, T, NT>(a, ctx, H, Qx, i0, j0, line < last ? line : last, line <= last, true, dtdx, cflm);
        }
        ctx.sync();
        const int own = i0 + T < a.mx ? i0 + T : a.mx;
        const int yfirst = i0 == 0 ? -2 : i0, ylast = own == a.mx ? a.mx + 1 : own - 1;
        for (int c0 = yfirst; c0 + lead <= ylast; c0 += LPC) {
            const int line = c0 + mine;
            lean_split_line<RP, 2, T, NT>(a, ctx, H, Qx, i0, j0, line < ylast ? line : ylast, line <= ylast,
                                          line >= 0 && line < own, dtdy, cflm);
        }
    } else {
        int chunk = 0;
        {
            const int first = j0 - 1, last = j0 + T < a.my ? j0 + T : a.my;
            for (int c0 = first; c0 <= last; c0 += LPC, chunk++) {
                const int line = c0 + mine, clast = c0 + LPC - 1 < last ? c0 + LPC - 1 : last;
                lean_chunk<RP, 1, T, NT>(a, ctx, H, Qx, CX + (chunk & 1) * 2 * MEQN * SM::NX, i0, j0, line < last ? line : last,
                                         c0, clast, line <= last, dtdx, dtdy, cflm);
            }
        }
        {
            const int first = i0 - 1, last = i0 + T < a.mx ? i0 + T : a.mx;
            for (int c0 = first; c0 <= last; c0 += LPC, chunk++) {
                const int line = c0 + mine, clast = c0 + LPC - 1 < last ? c0 + LPC - 1 : last;
                lean_chunk<RP, 2, T, NT>(a, ctx, H, Qx, CX + (chunk & 1) * 2 * MEQN * SM::NX, i0, j0, line < last ? line : last,
                                         c0, clast, line <= last, dtdy, dtdx, cflm);
            }
        }
    }
    return cflm;
}

// One warp's look at a tile of a large grid: a tile whose input halo holds one
// state gets its values, ghost images and CFL number here (as in lean_tiles; the
// caller checks that there is no source term), any other is listed for lean_tiles.
// A lane reads a column of the halo, some rows at a time; the first difference ends
// it.  Bound by HBM: 4096^2 cells of shallow water at rest 191 us, 830 MB at 4.3 TB/s.
// Returns the tile's CFL number, infinity for a state that is not finite, 0 for a
// listed tile.
template <class RP, int T>
__device__ __forceinline__ double lean_scan_tile(const StepArgs& a, const double* __restrict__ qin, double* __restrict__ qout,
                                                 int tile, double dtdx, double dtdy)
{
    constexpr int MEQN = RP::MEQN;
    static_assert(T + 4 == 32, "a lane per column");
    const int lane = threadIdx.x & 31, nbx = (a.mx + T - 1) / T, i0 = tile % nbx * T, j0 = tile / nbx * T;
    const int cmax = a.mx + 3 - i0, rmax = a.my + 3 - j0 < 31 ? a.my + 3 - j0 : 31;
    const double* p = qin + (long long)j0 * a.ld + (i0 + (lane < cmax ? lane : cmax));
    double q0[MEQN];
#pragma unroll
    for (int m = 0; m < MEQN; m++) q0[m] = __shfl_sync(0xffffffffu, p[m * a.plane], 0);
    bool keep = true;
    constexpr int ROWS = MEQN == 3 ? 8 : 4;
    for (int r = 0; r <= rmax && keep; r += ROWS) {
        bool same = true;
#pragma unroll
        for (int k = 0; k < ROWS; k++) {
            const long long o = (long long)(r + k < rmax ? r + k : rmax) * a.ld;
#pragma unroll
            for (int m = 0; m < MEQN; m++) same = same & (p[o + m * a.plane] == q0[m]);
        }
        keep = __all_sync(0xffffffffu, same);
    }
    double cu = 0.0;
    if (keep) cu = uniform_cfl<RP>(q0, a.prm, dtdx, dtdy, keep);       // the same in every lane
    if (!keep) {
        if (lane == 0) a.list[atomicAdd(a.ticket + LIST_WORD, 1u)] = tile;
        return 0.0;
    }
    const int i = i0 - 2 + lane, n = a.my - j0 < T ? a.my - j0 : T;
    if (a.custom) write_custom_corners<MEQN>(a, qout, i0, j0, T, T, lane);
    if (lane >= 2 && lane < 2 + T && i < a.mx) {
        double* d = qout + (long long)(j0 + 2) * a.ld + (i + CLAW2_NUM_GHOST);
        for (int r = 0; r < n; r++, d += a.ld) {
#pragma unroll
            for (int m = 0; m < MEQN; m++) d[m * a.plane] = q0[m];
        }
        const bool edge = i0 <= 1 || i0 + T >= a.mx - 2 || j0 <= 1 || j0 + T >= a.my - 2;
        if (a.ghost_fused && edge) {
            for (int j = j0; j < j0 + n; j++)
                if (i <= 1 || i >= a.mx - 2 || j <= 1 || j >= a.my - 2) write_ghosts<MEQN>(a, qout, i, j, q0);
        }
    }
    bool finite = true;
#pragma unroll
    for (int m = 0; m < MEQN; m++) finite = finite && isfinite(q0[m]);
    return finite ? cu : __longlong_as_double(0x7ff0000000000000LL);
}

// The step of a CTA's tiles (the caller checks that the problem has no capacity
// function and no f-waves): tile blockIdx.x of the grid, or with LISTED every
// gridDim.x-th of the list.  LOOK: one-state tiles are passed over.  tm0 / tm1:
// tensor maps of the input state (uncontrolled mode: both of a.qin; controlled
// mode: of a.q0 and a.q1) over the ghosted planes (mx+4 x my+4 x MEQN, row pitch
// ld, boxes of 16 x (T+4) x MEQN, 128-byte swizzle); bar: an mbarrier in shared
// memory.  The halo copy is waited for at most about a second (clock64 cycles); a
// tile whose copy does not arrive reports a timeout instead of a result, and its
// CTA steps no further ones.
constexpr long long kTmaWaitCycles = 2000000000LL;

template <class RP, int T, int NT, bool SPLIT, bool LOOK, bool LISTED, class Ctx>
__device__ __forceinline__ void lean_tiles(const StepArgs& a, Ctx& ctx, const CUtensorMap* tm0, const CUtensorMap* tm1,
                                           uint64_t* bar)
{
    constexpr int MEQN = RP::MEQN;
    using SM = LeanSmem<RP, T, NT, SPLIT>;
    static_assert(RP::MAUX == 0, "the lean body serves the solvers without aux arrays");
    double* H = ctx.smem();
    {
        const uint32_t s0 = smem_addr(H);
        H += ((1024u - (s0 & 1023u)) & 1023u) / 8;       // 1024-byte boundary for the swizzled boxes
    }
    double* Qx = H + SM::HS;
    double* CX = Qx + SM::QX;
    double* red = CX + SM::CX;
    const int tid = ctx.tid();
    double* qout = a.qout;
    double dt = a.dt;
    const CUtensorMap* tm = tm0;
    if (a.ctrl) {
        const int done = a.ctrl->done, cur = a.ctrl->cur;           // loaded together
        dt = a.ctrl->dt;
        if (done) return;                          // uniform across the grid
        tm = cur ? tm1 : tm0;
        qout = cur ? a.q0 : a.q1;
    }
    const int nbx = (a.mx + T - 1) / T, ncta = gridDim.x;
    const int count = LISTED ? *(volatile int*)(a.ticket + LIST_WORD) : ncta;
    // CTAs that report: those with a tile, or the first if there is none
    const int reports = count < ncta ? (count > 0 ? count : 1) : ncta;
    if (LISTED && (int)blockIdx.x >= reports) return;
    const double dtdx = dt / a.dx, dtdy = dt / a.dy;
    if (tid == 0) mbar_init(bar, 1);
    double cflm = 0.0;
    bool bad = false, fault = false;
    uint32_t phase = 0;
    for (int b = blockIdx.x; b < count; b += ncta) {
        const int tile = LISTED ? a.list[b] : b, i0 = tile % nbx * T, j0 = tile / nbx * T;
        // stage the halo: rows j0-2.., columns i0-2.. are ghosted-array indices
        // j0, i0 (x = i0 is even, so the box starts on a 16-byte boundary)
        if (tid == 0) {
            mbar_arrive_expect_tx(bar, (uint32_t)(SM::HS * 8 + a.halo_shortfall));
#pragma unroll
            for (int k = 0; k < SM::NBOX; k++) tma_load_3d(H + k * SM::BOX, tm, bar, i0 + 16 * k, j0, 0);
        }
        ctx.sync();                                // the barrier is initialised
        // the whole CTA takes the same path
        fault = __syncthreads_or(!mbar_wait_bounded(bar, phase, kTmaWaitCycles));
        if (fault) {
            mbar_wait_bounded(bar, phase, kTmaWaitCycles);       // let a late copy land before the CTA moves on
            break;
        }
        bool keep = false;                         // the tile's cells keep their values
        if (LOOK && lean_uniform_halo<RP, SM::TR>(a, H, i0, j0, tid, NT)) {
            // A tile whose input halo holds one state has zero waves and
            // fluctuations at every interface: its cells keep their values (the
            // full step adds only zeros) and only its CFL number is computed.
            double q0[MEQN];
#pragma unroll
            for (int m = 0; m < MEQN; m++) q0[m] = H[lean_hidx<MEQN, SM::TR>(m, 0, 0)];
            keep = true;
            const double cu = uniform_cfl<RP>(q0, a.prm, dtdx, dtdy, keep);
            if (keep) {                            // the same in every thread
                for (int e = tid; e < T * SM::QP; e += NT) {
#pragma unroll
                    for (int m = 0; m < MEQN; m++) Qx[m * T * SM::QP + e] = q0[m];
                }
                cflm = cflm > cu ? cflm : cu;
            }
        }
        if (!keep) {
            const double c = lean_tile_sweeps<RP, T, NT, SPLIT>(a, ctx, H, Qx, CX, i0, j0, dtdx, dtdy);
            cflm = cflm > c || cflm != cflm ? cflm : c;          // a NaN stays
        }
        // (the split sweeps wrote to the halo that the next copy overwrites)
        if (LISTED && SPLIT) asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        ctx.sync();
        bad |= store_tile<MEQN, T, T, NT, SM::QP>(a, ctx, Qx, T * SM::QP, qout, i0, j0, dt);
        if (!LISTED) break;
        phase ^= 1;
    }
    report_cell<NT>(a, ctx, reports, red, cflm, bad, fault);
}

}  // namespace claw2
