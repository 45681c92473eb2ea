// Truncated QDB / non-banded scan of whole windows by diagonals
// (generic_tr_scan, src/cm_dpsearch_trunc.rs:1800-2316), for models with
// cm_from_guide's node topology.
//
// As in diag_scan.cu a warp takes 32 consecutive columns and walks, node by
// node from the bottom up, the spans d of all the node's states at once: for
// one span every column is independent.  A cell has three planes here -- J,
// L, R, and T for bifurcations -- which read cells of spans d-2, d-1 and d
// (the L plane of right emitters and the R plane of left emitters take no
// residue and read span d of states below), so a node computes IR first, then
// IL, then its split states.  Inserts stay in registers; of the next node
// only the split states' planes are loaded, two spans ahead.  Warps run
// skewed by one 16-span phase with one CTA barrier per phase.  (So the last
// warp has finished a phase of a group before the first one reaches the same
// phase of the next group, if a group has at least as many phases as the CTA
// warps; the launch takes fewer warps where it has not.)
//
// ROOT.  The reference never resets its ROOT row: a truncated begin counts
// only if it exceeds the best one of every earlier column of the same parity
// (per plane and span).  Every begin state posts its cells to the column's
// best value and entry state per plane (the smallest state on equal values,
// which is the first the reference reaches); after the last node a warp takes
// the maximum over the earlier columns of its parity -- a scan over the lanes
// by steps of two and a carry from the columns on its left -- and keeps what
// exceeds it.  Of the planes that do, the best score wins, the smaller state
// and then the plane order J, L, R, T on equal scores: the order of the
// reference's comparisons.
//
// Cells of spans beyond a column's own start hold values nobody reads.
//
// Measured on one B200, 200 cut sequences of about 107 nt, non-banded Inside,
// M = 379: 175 ms with the column wavefront of trq_scan.cu, 23 ms here.
// Bound: the latency of one warp's log-sum chains (one to two windows per
// SM, four warps each); DRAM 2%.
#include <climits>
#include <cstring>
#include <type_traits>

#include "cm_internal.h"
#include "devbuf.h"
#include "plan_util.h"
#include "semiring.cuh"
#include "trq_diag.h"

namespace cmx {
namespace trqd {

using dev::Sem;

struct Ctx {
    uint32_t *reg;
    const uint16_t *tbl;
    const uint8_t *ring;
    uint32_t *xch;  // [warps][2][CHUNK][4]: last column's IL J, R and IR J, R
    int nz, rmask, nw, w, lane, col, jrel, ridx, cj, jmax, span, step;
    bool first, last;
    // region
    uint32_t *buf, *begl, *begr, *bnd, *rbm, *rby, *carry;
};

__device__ __forceinline__ void phase(int nthreads) { asm volatile("barrier.sync 1, %0;" ::"r"(nthreads) : "memory"); }

template <class S>
__device__ __forceinline__ typename S::T cmb(typename S::T a, typename S::T b, const Ctx &c) {
    if constexpr (S::ORDERED) return S::comb(a, b, c.tbl, c.nz);
    else return fmaxf(a, b);
}
template <class S>
__device__ __forceinline__ typename S::T mx(typename S::T a, typename S::T b) {
    if constexpr (S::ORDERED) return max(a, b);
    else return fmaxf(a, b);
}
// first term of a fold of n terms whose initial value is init (has) or
// impossible: the impossible value only clamps at zero(), which in Inside
// every later combination does as well
template <class S>
__device__ __forceinline__ typename S::T fold0(bool has, typename S::T init, typename S::T x, const Ctx &c, int n) {
    if (has) return cmb<S>(init, x, c);
    return S::ORDERED && n > 1 ? x : mx<S>(x, S::zero());
}

// region of a CTA: three node buffers, the bifurcations' decks, the ROOT
// row's best values and entry states, the saved last columns, the carries
__host__ __device__ inline int64_t off_begl(const Params &p) { return 3 * (int64_t)p.W1 * ROW; }
__host__ __device__ inline int64_t off_begr(const Params &p) {
    return off_begl(p) + (int64_t)p.nbif * 3 * p.W1 * p.ring_cols;
}
__host__ __device__ inline int64_t off_rbm(const Params &p) { return off_begr(p) + (int64_t)p.nbif * 3 * p.W1 * COLS; }
__host__ __device__ inline int64_t off_rby(const Params &p) { return off_rbm(p) + 4 * (int64_t)p.W1 * COLS; }
__host__ __device__ inline int64_t off_bnd(const Params &p) { return off_rby(p) + 4 * (int64_t)p.W1 * COLS; }
__host__ __device__ inline int64_t off_carry(const Params &p) {
    return off_bnd(p) + (int64_t)p.nnodes * p.W1 * BND;
}
int64_t region_words(const Params &p) { return (off_carry(p) + 8 * (int64_t)p.W1 + 63) & ~(int64_t)63; }

// Posts one state's cell to the node's best begin per plane.
template <class S>
__device__ __forceinline__ void post(typename S::T x, int v, typename S::T &m, int &y) {
    if (x > m || (x == m && v < y)) {
        m = x;
        y = v;
    }
}

template <class S, int NT, int NN>
__device__ __forceinline__ void node(const Params &p, Ctx &c, const Node *np, int nidx) {
    typedef typename S::T T;
    constexpr bool HAS_IL = NT == MATP_ND || NT == MATL_ND || NT == ROOT_ND || NT == BEGR_ND;
    constexpr bool HAS_IR = NT == MATP_ND || NT == MATR_ND || NT == ROOT_ND;
    constexpr bool LEFT = HAS_IR;
    constexpr int NSPLIT = NT == MATP_ND ? 4 : (NT == MATL_ND || NT == MATR_ND) ? 2 : 1;
    constexpr int QIL = NSPLIT, QIR = HAS_IL ? NSPLIT + 1 : NSPLIT;
    constexpr int NI = (HAS_IL ? 1 : 0) + (HAS_IR ? 1 : 0);
    constexpr int CN = NI + NN;
    constexpr int MP = NT == MATP_ND ? 0 : -1, ML = NT == MATP_ND ? 1 : NT == MATL_ND ? 0 : -1,
                  MR = NT == MATP_ND ? 2 : NT == MATR_ND ? 0 : -1;
    const unsigned FULL = 0xffffffffu;
    const T Z = S::zero();
    const bool FL = p.fill_l, FR = p.fill_r;
    const int v0 = np->v0, rhi = min((int)np->rhi, c.span), chi = np->chi;
    const bool cend = np->next_end != 0, need_left = np->need_left != 0;
    const T cbase = S::ld(&np->cbase);
    const int endmask = np->endmask, beginmask = np->beginmask, skip = np->skip;
    // outputs: planes J, L, R of split state q at o + (q * 3 + plane) * oslot
    uint32_t *out;
    int ostride, oslot;
    if (NT == BEGL_ND) {
        out = c.begl + (int64_t)np->deck * 3 * p.W1 * p.ring_cols + c.ridx;
        ostride = p.ring_cols;
        oslot = p.W1 * p.ring_cols;
    } else if (NT == BEGR_ND) {
        out = c.begr + (int64_t)np->deck * 3 * p.W1 * COLS + c.col;
        ostride = COLS;
        oslot = p.W1 * COLS;
    } else {
        out = c.buf + (int64_t)np->buf * p.W1 * ROW + 32 + c.col;
        ostride = ROW;
        oslot = PITCH;
    }
    const uint32_t *in = c.buf + (int64_t)((np->buf + 2) % 3) * p.W1 * ROW + 32 + c.col;
    uint32_t *bnd = c.bnd + (int64_t)nidx * p.W1 * BND;

    // spans the inner step takes
    int ihi = min(rhi, min(p.dx0, min(chi, p.W1 - 1) - 2));
#pragma unroll
    for (int q = 0; q < NSPLIT + NI; q++) ihi = min(ihi, (int)np->dx[q]);
    constexpr int INS = (HAS_IL ? 1 << QIL : 0) | (HAS_IR ? 1 << QIR : 0);
    if (cend || skip || (endmask & ~1) || (beginmask & ~(1 | INS))) ihi = -1;
    const bool end0 = (endmask & 1) != 0, beg0 = (beginmask & 1) != 0;
    const bool begil = HAS_IL && (beginmask >> QIL & 1), begir = HAS_IR && (beginmask >> QIR & 1);
    const T es0 = end0 ? S::ldg(p.endsc + v0) : Z, pen0 = beg0 ? S::ldg(p.pty + v0) : Z,
            penil = begil ? S::ldg(p.pty + v0 + QIL) : Z, penir = begir ? S::ldg(p.pty + v0 + QIR) : Z;

    T ts[NSPLIT][CN], til[HAS_IL ? CN : 1], tir[HAS_IR ? NN + 1 : 1];
#pragma unroll
    for (int q = 0; q < NSPLIT; q++)
#pragma unroll
        for (int k = 0; k < CN; k++) ts[q][k] = S::ldg(p.tsc + (v0 + q) * 6 + k);
    if constexpr (HAS_IL)
#pragma unroll
        for (int k = 0; k < CN; k++) til[k] = S::ldg(p.tsc + (v0 + QIL) * 6 + k);
    if constexpr (HAS_IR)
#pragma unroll
        for (int k = 0; k < NN + 1; k++) tir[k] = S::ldg(p.tsc + (v0 + QIR) * 6 + k);

    // plane pl of split state y of the next node at (j - shift, d)
    auto ldx = [&](int y, int pl, int d, int shift) -> T {
        if (cend) return d == 0 ? cbase : Z;
        if (d < 0 || d > chi || d >= p.W1) return Z;
        return S::ld(in + (int64_t)d * ROW + (y * 3 + pl) * PITCH - shift);
    };
    const uint32_t *esc0 = p.esc + (int64_t)v0 * ESC, *escr = esc0 + c.cj;
    const uint32_t *lm0 = p.lm + v0 * KP, *rm0 = p.rm + v0 * KP + c.cj;

    // child planes: J at d-1, d, d+1 and column j-1 at d-2, d-1, d; L at d-1,
    // d, d+1; R at d, d+1 and column j-1 at d-1, d
    T jp[NN], jc[NN], jn[NN], jl2[NN], jl1[NN], jl0[NN], lp[NN], lc[NN], ln[NN], rc[NN], rn[NN], rl1[NN], rl0[NN];
    T ilJp = Z, ilJ1 = Z, ilJ2 = Z, ilLp = Z, ilR1 = Z, irJp = Z, irJ1 = Z, irJ2 = Z, irLp = Z, irR1 = Z;
#pragma unroll
    for (int y = 0; y < NN; y++) {
        jp[y] = lp[y] = jl1[y] = jl2[y] = rl1[y] = Z;
        jc[y] = ldx(y, 0, 0, 0);
        lc[y] = ldx(y, 1, 0, 0);
        rc[y] = ldx(y, 2, 0, 0);
        jn[y] = ldx(y, 0, 1, 0);
        ln[y] = ldx(y, 1, 1, 0);
        rn[y] = ldx(y, 2, 1, 0);
        jl0[y] = LEFT ? ldx(y, 0, 0, 1) : Z;
        rl0[y] = LEFT ? ldx(y, 2, 0, 1) : Z;
    }
    int ci = 0;
    if (HAS_IL) ci = c.ring[(c.jrel + 1) & c.rmask];  // residue j-d+1 at d = 0: loaded one span ahead
    const int nthreads = c.nw * 32;
    int d = 0;
    for (int r0 = 0; r0 <= rhi; r0 += CHUNK) {
        const int rend = min(r0 + CHUNK - 1, rhi);
        const int dstop = min(rend, c.jmax);
        const int slot = c.step & 1;
        // inserts of the column left of the warp: lane r holds span r0 + r
        T h0 = Z, h1 = Z, h2 = Z, h3 = Z;
        const int hr = c.lane & (CHUNK - 1);
        if constexpr (HAS_IR) {
            const uint32_t *s = nullptr;
            if (c.w > 0) s = c.xch + (((c.w - 1) * 2 + slot) * CHUNK + hr) * 4;
            else if (!c.first && r0 + hr <= rend) s = bnd + (int64_t)(r0 + hr) * BND + SLOTS;
            if (s) h0 = S::ld(s), h1 = S::ld(s + 1), h2 = S::ld(s + 2), h3 = S::ld(s + 3);
        }
        uint32_t *xs = c.xch + (c.w * 2 + slot) * (CHUNK * 4);
        if (NT != ROOT_ND && need_left && c.w == 0 && c.lane < CHUNK && r0 + hr <= dstop) {
            // the column left of the group: planes J and R are read
            const int h = r0 + hr;
#pragma unroll
            for (int q = 0; q < NSPLIT; q++)
#pragma unroll
                for (int pl = 0; pl < 3; pl += 2) {
                    T x = h == 0 && pl == 0 ? S::ld(&np->base[q]) : Z;
                    if (!c.first) x = S::ld(bnd + (int64_t)h * BND + q * 3 + pl);
                    S::st(out - c.lane + (int64_t)h * ROW + (q * 3 + pl) * PITCH - 1, x);
                }
        }
        // One span; px, po: rows d of the child (column j) and of the outputs.
        // The inner version needs no test: every state in band, d >= 2, the
        // child rows stored, at most the first state with a local end, begins
        // in it and the inserts only (where cm_tr_penalties puts them: without
        // the inserts no node with begins took it, and the scan below 35 ms).
        // Planes L and R are computed in every pass; J does not read
        // them, and a pass without one posts no begin from it.
        auto step = [&](auto inner_c, const uint32_t *px, uint32_t *o) {
            constexpr bool INNER = decltype(inner_c)::value;
            T jf[NN], lf[NN], rf[NN], jlf[NN], rlf[NN];
#pragma unroll
            for (int y = 0; y < NN; y++) {
                const uint32_t *x = px + y * 3 * PITCH;
                jf[y] = INNER ? S::ld(x + 2 * ROW) : ldx(y, 0, d + 2, 0);
                lf[y] = INNER ? S::ld(x + 2 * ROW + PITCH) : ldx(y, 1, d + 2, 0);
                rf[y] = INNER ? S::ld(x + 2 * ROW + 2 * PITCH) : ldx(y, 2, d + 2, 0);
                if (LEFT) {
                    jlf[y] = INNER ? S::ld(x + ROW - 1) : ldx(y, 0, d + 1, 1);
                    rlf[y] = INNER ? S::ld(x + ROW + 2 * PITCH - 1) : ldx(y, 2, d + 1, 1);
                }
            }
            // the ROOT row's best begins so far
            const bool post0 = INNER ? beginmask != 0 : beginmask && d >= 1 && d <= p.dx0;
            uint32_t *rb = c.rbm + (int64_t)d * COLS + c.col, *ry = c.rby + (int64_t)d * COLS + c.col;
            T b0 = Z, b1 = Z, b2 = Z;
            if (post0) {
                b0 = S::ld(rb);
                b1 = S::ld(rb + (int64_t)p.W1 * COLS);
                b2 = S::ld(rb + (int64_t)p.W1 * COLS * 2);
            }
            const int cd = ci;  // residue j-d+1
            if (HAS_IL) ci = c.ring[(c.jrel - d) & c.rmask];
            const uint32_t *escd = esc0 + cd;
            T eil = Z, eir = Z, eml = Z, emr = Z, emp = Z, elm = Z, erm = Z;
            if (HAS_IL) eil = S::ldg(escd + QIL * ESC);
            if (HAS_IR) eir = S::ldg(escr + QIR * ESC);
            if (ML >= 0) eml = S::ldg(escd + (ML < 0 ? 0 : ML) * ESC);
            if (MR >= 0) emr = S::ldg(escr + (MR < 0 ? 0 : MR) * ESC);
            if (MP >= 0) {
                emp = S::ldg(escr + cd * KP);
                elm = S::ldg(lm0 + cd);
                erm = S::ldg(rm0);
            }
            const T el0 = S::ldg(p.el + d), el1 = S::ldg(p.el + max(d - 1, 0)), el2 = S::ldg(p.el + max(d - 2, 0));
            auto has = [&](int q) { return INNER ? q == 0 && end0 : (endmask >> q & 1) != 0; };
            auto init = [&](int q, T el) -> T { return S::add(el, INNER ? es0 : S::ldg(p.endsc + v0 + q)); };
            auto in_band = [&](int q) { return INNER || (d >= 1 && d <= np->dx[q] && !(skip >> q & 1)); };
            // best begin of the node's states, per plane
            T mj = Z, ml = Z, mr = Z;
            int yj = INT_MAX, yl = INT_MAX, yr = INT_MAX;
            auto begin = [&](int q, T J, T L, T R) {
                if (INNER) {
                    if (q != 0 && q != QIL && q != QIR) return;
                    if (q == 0 ? !beg0 : q == QIL && HAS_IL ? !begil : !begir) return;
                    const T pen = q == 0 ? pen0 : q == QIL && HAS_IL ? penil : penir;
                    const T xj = S::add(J, pen), xl = S::add(L, pen), xr = S::add(R, pen);
                    if (xj >= mj) mj = xj, yj = v0 + q;
                    if (xl >= ml) ml = xl, yl = v0 + q;
                    if (xr >= mr) mr = xr, yr = v0 + q;
                    return;
                }
                if (!(beginmask >> q & 1)) return;
                const T pen = S::ldg(p.pty + v0 + q);
                post<S>(S::add(J, pen), v0 + q, mj, yj);
                post<S>(S::add(L, pen), v0 + q, ml, yl);
                post<S>(S::add(R, pen), v0 + q, mr, yr);
            };
            // folds of one plane over the node's inserts and the next node's
            // split states, children ascending
            auto fold = [&](int q, const T *t, T el, T i0, T i1, const T *x) -> T {
                T a = Z;
                bool f = true;
                if (HAS_IL) a = fold0<S>(has(q), init(q, el), S::add(i0, t[0]), c, CN), f = false;
                if (HAS_IR) {
                    const T u = S::add(i1, t[HAS_IL ? 1 : 0]);
                    a = f ? fold0<S>(has(q), init(q, el), u, c, CN) : cmb<S>(a, u, c);
                    f = false;
                }
#pragma unroll
                for (int y = 0; y < NN; y++) {
                    const T u = S::add(x[y], t[NI + y]);
                    a = f && y == 0 ? fold0<S>(has(q), init(q, el), u, c, CN) : cmb<S>(a, u, c);
                }
                return a;
            };
            // the larger of two planes of each child
            auto fold2 = [&](int q, const T *t, T el, T i0a, T i0b, T i1a, T i1b, const T *x, const T *z) -> T {
                T a = Z;
                bool f = true;
                if (HAS_IL) {
                    a = fold0<S>(has(q), init(q, el), mx<S>(S::add(i0a, t[0]), S::add(i0b, t[0])), c, CN);
                    f = false;
                }
                if (HAS_IR) {
                    const T k = t[HAS_IL ? 1 : 0], u = mx<S>(S::add(i1a, k), S::add(i1b, k));
                    a = f ? fold0<S>(has(q), init(q, el), u, c, CN) : cmb<S>(a, u, c);
                    f = false;
                }
#pragma unroll
                for (int y = 0; y < NN; y++) {
                    const T u = mx<S>(S::add(x[y], t[NI + y]), S::add(z[y], t[NI + y]));
                    a = f && y == 0 ? fold0<S>(has(q), init(q, el), u, c, CN) : cmb<S>(a, u, c);
                }
                return a;
            };
            T ilJ = Z, ilL = Z, ilR = Z, irJ = Z, irL = Z, irR = Z;
            if constexpr (HAS_IR) {
                if (in_band(QIR)) {
                    T x = fold0<S>(has(QIR), init(QIR, el1), S::add(irJ1, tir[0]), c, NN + 1);
                    T z = fold0<S>(has(QIR), init(QIR, el1), S::add(irR1, tir[0]), c, NN + 1), l = Z;
#pragma unroll
                    for (int y = 0; y < NN; y++) {
                        x = cmb<S>(x, S::add(jl1[y], tir[1 + y]), c);
                        z = cmb<S>(z, S::add(rl1[y], tir[1 + y]), c);
                        const T u = mx<S>(S::add(jc[y], tir[1 + y]), S::add(lc[y], tir[1 + y]));
                        l = y == 0 ? fold0<S>(has(QIR), init(QIR, el0), u, c, NN) : cmb<S>(l, u, c);
                    }
                    irJ = S::add(x, eir);
                    irR = INNER || d >= 2 ? S::add(z, eir) : eir;
                    irL = l;
                    begin(QIR, irJ, irL, irR);
                }
            }
            if constexpr (HAS_IL) {
                if (in_band(QIL)) {
                    T x = fold0<S>(has(QIL), init(QIL, el1), S::add(ilJp, til[0]), c, CN);
                    T z = fold0<S>(has(QIL), init(QIL, el1), S::add(ilLp, til[0]), c, CN), r = Z;
                    if (HAS_IR) {
                        x = cmb<S>(x, S::add(irJp, til[1]), c);
                        z = cmb<S>(z, S::add(irLp, til[1]), c);
                        r = fold0<S>(has(QIL), init(QIL, el0), mx<S>(S::add(irJ, til[1]), S::add(irR, til[1])), c, CN - 1);
                    }
#pragma unroll
                    for (int y = 0; y < NN; y++) {
                        x = cmb<S>(x, S::add(jp[y], til[NI + y]), c);
                        z = cmb<S>(z, S::add(lp[y], til[NI + y]), c);
                        const T u = mx<S>(S::add(jc[y], til[NI + y]), S::add(rc[y], til[NI + y]));
                        r = !HAS_IR && y == 0 ? fold0<S>(has(QIL), init(QIL, el0), u, c, CN - 1) : cmb<S>(r, u, c);
                    }
                    ilJ = S::add(x, eil);
                    ilL = INNER || d >= 2 ? S::add(z, eil) : eil;
                    ilR = r;
                    begin(QIL, ilJ, ilL, ilR);
                }
            }
            if constexpr (NT != ROOT_ND) {
                T J[NSPLIT], L[NSPLIT], R[NSPLIT];
#pragma unroll
                for (int q = 0; q < NSPLIT; q++) {
                    J[q] = !INNER && d == 0 ? S::ld(&np->base[q]) : Z;
                    L[q] = R[q] = Z;
                    if (!in_band(q)) continue;
                    const bool two = INNER || d >= 2;
                    if (q == MP) {
                        L[q] = elm;
                        R[q] = erm;
                        if (two) {
                            J[q] = S::add(fold(q, ts[q], el2, ilJ2, irJ2, jl2), emp);
                            L[q] = S::add(fold2(q, ts[q], el1, ilJp, ilLp, irJp, irLp, jp, lp), elm);
                            R[q] = S::add(fold2(q, ts[q], el1, ilJ1, ilR1, irJ1, irR1, jl1, rl1), erm);
                        }
                    } else if (q == ML) {
                        J[q] = S::add(fold(q, ts[q], el1, ilJp, irJp, jp), eml);
                        L[q] = two ? S::add(fold(q, ts[q], el1, ilLp, irLp, lp), eml) : eml;
                        R[q] = fold2(q, ts[q], el0, ilJ, ilR, irJ, irR, jc, rc);
                    } else if (q == MR) {
                        J[q] = S::add(fold(q, ts[q], el1, ilJ1, irJ1, jl1), emr);
                        R[q] = two ? S::add(fold(q, ts[q], el1, ilR1, irR1, rl1), emr) : emr;
                        L[q] = fold2(q, ts[q], el0, ilJ, ilL, irJ, irL, jc, lc);
                    } else {  // D, S
                        J[q] = fold(q, ts[q], el0, ilJ, irJ, jc);
                        L[q] = fold(q, ts[q], el0, ilL, irL, lc);
                        R[q] = fold(q, ts[q], el0, ilR, irR, rc);
                    }
                    begin(q, J[q], L[q], R[q]);
                }
#pragma unroll
                for (int q = 0; q < NSPLIT; q++) {
                    S::st(o + (q * 3) * oslot, J[q]);
                    S::st(o + (q * 3 + 1) * oslot, L[q]);
                    S::st(o + (q * 3 + 2) * oslot, R[q]);
                }
            }
            // the node's states lie above every state posted before, so an
            // equal value takes their (smaller) entry state
            if (post0) {
                const int64_t pl = (int64_t)p.W1 * COLS;
                if (mj > Z && mj >= b0) S::st(rb, mj), ry[0] = (uint32_t)yj;
                if (FL && ml > Z && ml >= b1) S::st(rb + pl, ml), ry[pl] = (uint32_t)yl;
                if (FR && mr > Z && mr >= b2) S::st(rb + 2 * pl, mr), ry[2 * pl] = (uint32_t)yr;
            }
            // hand the inserts to the column on the right
            if constexpr (HAS_IR) {
                auto left = [&](T x, T h) -> T {
                    const T u = __shfl_up_sync(FULL, x, 1), v = __shfl_sync(FULL, h, d - r0);
                    return c.lane == 0 ? v : u;
                };
                if (HAS_IL) {
                    ilJ2 = ilJ1;
                    ilJ1 = left(ilJ, h0);
                    ilR1 = left(ilR, h1);
                }
                irJ2 = irJ1;
                irJ1 = left(irJ, h2);
                irR1 = left(irR, h3);
                if (c.lane == 31) {
                    uint32_t *x = xs + (d - r0) * 4;
                    S::st(x, ilJ);
                    S::st(x + 1, ilR);
                    S::st(x + 2, irJ);
                    S::st(x + 3, irR);
                }
            }
            ilJp = ilJ;
            ilLp = ilL;
            irJp = irJ;
            irLp = irL;
#pragma unroll
            for (int y = 0; y < NN; y++) {
                jp[y] = jc[y];
                jc[y] = jn[y];
                jn[y] = jf[y];
                lp[y] = lc[y];
                lc[y] = ln[y];
                ln[y] = lf[y];
                rc[y] = rn[y];
                rn[y] = rf[y];
                if (LEFT) {
                    jl2[y] = jl1[y];
                    jl1[y] = jl0[y];
                    jl0[y] = jlf[y];
                    rl1[y] = rl0[y];
                    rl0[y] = rlf[y];
                }
            }
        };
        while (d <= dstop) {
            uint32_t *po = out + (int64_t)d * ostride;
            const int iend = min(dstop, ihi);
            if (NT != ROOT_ND && d >= 2 && d <= iend) {
                const uint32_t *px = in + (int64_t)d * ROW;
#pragma unroll 1
                for (; d <= iend; d++) {
                    step(std::true_type(), px, po);
                    px += ROW;
                    po += ostride;
                }
            } else {
                step(std::false_type(), in, po);
                d++;
            }
        }
        // the group's last column, for the next group
        if (!c.last && c.w == c.nw - 1) {
            __syncwarp();
            if (c.lane < CHUNK && r0 + hr <= dstop) {
                const int h = r0 + hr;
                uint32_t *b = bnd + (int64_t)h * BND;
                if (NT != ROOT_ND && need_left)
#pragma unroll
                    for (int q = 0; q < NSPLIT; q++)
#pragma unroll
                        for (int pl = 0; pl < 3; pl += 2)
                            b[q * 3 + pl] = out[(31 - c.lane) + (int64_t)h * ROW + (q * 3 + pl) * PITCH];
                if (HAS_IR)
#pragma unroll
                    for (int k = 0; k < 4; k++) b[SLOTS + k] = xs[hr * 4 + k];
            }
        }
        c.step++;
        phase(nthreads);
    }
}

// Bifurcation node (src/cm_dpsearch_trunc.rs, B states of generic_tr_scan):
// per span the splits k ascending, J over BEGL.J + BEGR.J, L over BEGL.J +
// BEGR.L, R over BEGL.R + BEGR.J, T over BEGL.R + BEGR.L (1 <= k <= d-1), then
// the whole span in the left (L) or right (R) child.  Two spans at a time
// share the BEGR loads.
template <class S>
__device__ __forceinline__ void bif(const Params &p, Ctx &c, const Node *np, int nidx) {
    typedef typename S::T T;
    const T Z = S::zero();
    const bool FL = p.fill_l, FR = p.fill_r, FT = p.fill_t;
    const int v = np->v0, rhi = min((int)np->rhi, c.span), dx = np->dx[0], dxw = np->dx_w, dxy = np->dx_y;
    const int RC = p.ring_cols;
    const int64_t lpl = (int64_t)p.W1 * RC, ypl = (int64_t)p.W1 * COLS;
    const uint32_t *begl = c.begl + (int64_t)np->deck * 3 * lpl, *begr = c.begr + (int64_t)np->deck * 3 * ypl + c.col;
    const T lbase = S::ld(&np->begl_base);
    const bool has = np->endmask & 1, beg = np->beginmask & 1, need_left = np->need_left != 0;
    const T pen = beg ? S::ldg(p.pty + v) : Z, es = has ? S::ldg(p.endsc + v) : Z;
    uint32_t *out = c.buf + (int64_t)np->buf * p.W1 * ROW + 32 + c.col;
    uint32_t *bnd = c.bnd + (int64_t)nidx * p.W1 * BND;
    constexpr int U = 2;
    for (int r0 = 0; r0 <= rhi; r0 += CHUNK) {
        const int dstop = min(min(r0 + CHUNK - 1, rhi), c.jmax);
#pragma unroll 1
        for (int d0 = r0; d0 <= dstop; d0 += U) {
            T aj[U], al[U], ar[U], at[U];
            int klo[U], khi[U];
            int ka = INT_MAX, kb = -1, ba = 1, bb = INT_MAX;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int d = d0 + u;
                const T a = has ? S::add(S::ldg(p.el + min(d, p.W)), es) : Z;
                aj[u] = a;
                al[u] = FL ? a : Z;
                ar[u] = FR ? a : Z;
                at[u] = FT ? a : Z;
                klo[u] = p.nonbanded ? 0 : max(d - dxw, 0);
                khi[u] = p.nonbanded ? d : min(dxy, d);
                if (d < 1 || d > dx || d > dstop) klo[u] = 0, khi[u] = -1;
                if (khi[u] >= klo[u]) ka = min(ka, klo[u]), kb = max(kb, khi[u]);
                ba = max(ba, klo[u]);
                bb = min(bb, min(khi[u], d - 1));
            }
            auto ring = [&](int k) {
                const int x = c.ridx - k;
                return x < 0 ? x + RC : x;
            };
            auto one = [&](int u, T lj, T lr, T yj, T yl, bool t) {
                aj[u] = cmb<S>(aj[u], S::add(lj, yj), c);
                if (FL) al[u] = cmb<S>(al[u], S::add(lj, yl), c);
                if (FR) ar[u] = cmb<S>(ar[u], S::add(lr, yj), c);
                if (FT && t) at[u] = cmb<S>(at[u], S::add(lr, yl), c);
            };
            auto edge = [&](int k0, int k1) {
#pragma unroll 1
                for (int k = k0; k <= k1; k++) {
                    const T yj = S::ld(begr + (int64_t)k * COLS), yl = FL ? S::ld(begr + ypl + (int64_t)k * COLS) : Z;
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        if (k < klo[u] || k > khi[u]) continue;
                        const int e = d0 + u - k;
                        const uint32_t *l = begl + (int64_t)e * RC + ring(k);
                        const T lj = e == 0 ? lbase : S::ld(l);
                        const T lr = !FR || e == 0 ? Z : S::ld(l + 2 * lpl);
                        one(u, lj, lr, yj, yl, k >= 1 && e >= 1);
                    }
                }
            };
            if (bb < ba) {
                edge(ka, kb);
            } else {
                edge(ka, ba - 1);
#pragma unroll 2
                for (int k = ba; k <= bb; k++) {
                    const T yj = S::ld(begr + (int64_t)k * COLS), yl = FL ? S::ld(begr + ypl + (int64_t)k * COLS) : Z;
                    const uint32_t *l = begl + (int64_t)(d0 - k) * RC + ring(k);
                    T lj[U], lr[U];
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        lj[u] = S::ld(l + (int64_t)u * RC);
                        lr[u] = FR ? S::ld(l + 2 * lpl + (int64_t)u * RC) : Z;
                    }
#pragma unroll
                    for (int u = 0; u < U; u++) one(u, lj[u], lr[u], yj, yl, true);
                }
                edge(bb + 1, kb);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int d = d0 + u;
                if (d > dstop) continue;
                const bool in = d >= 1 && d <= dx;
                const T b0 = d == 0 ? S::ld(&np->base[0]) : Z;
                if (in && FL && klo[u] == 0) {
                    const uint32_t *l = begl + (int64_t)d * RC + c.ridx;
                    al[u] = cmb<S>(al[u], mx<S>(S::ld(l), S::ld(l + lpl)), c);
                }
                if (in && FR && khi[u] == d) {
                    const uint32_t *y = begr + (int64_t)d * COLS;
                    ar[u] = cmb<S>(ar[u], mx<S>(S::ld(y), S::ld(y + 2 * ypl)), c);
                }
                const T J = in ? aj[u] : b0, L = in && FL ? al[u] : Z, R = in && FR ? ar[u] : Z;
                uint32_t *o = out + (int64_t)d * ROW;
                S::st(o, J);
                S::st(o + PITCH, L);
                S::st(o + 2 * PITCH, R);
                if (need_left) {
                    uint32_t *b = bnd + (int64_t)d * BND;
                    if (c.w == 0 && c.lane == 0) {
                        S::st(o - 1, c.first ? b0 : S::ld(b));
                        S::st(o + 2 * PITCH - 1, c.first ? Z : S::ld(b + 2));
                    }
                    __syncwarp();  // (one warp may hold both columns)
                    if (!c.last && c.w == c.nw - 1 && c.lane == 31) {
                        S::st(b, J);
                        S::st(b + 2, R);
                    }
                }
                if (beg && in && d <= p.dx0) {
                    auto rmw = [&](int pl, T x) {
                        const int64_t at2 = ((int64_t)pl * p.W1 + d) * COLS + c.col;
                        const T m = S::add(x, pen);
                        if (m > Z && m >= S::ld(c.rbm + at2)) {
                            S::st(c.rbm + at2, m);
                            c.rby[at2] = (uint32_t)v;
                        }
                    };
                    rmw(0, J);
                    if (FL) rmw(1, L);
                    if (FR) rmw(2, R);
                    if (FT) rmw(3, at[u]);
                }
            }
        }
        c.step++;
        phase(c.nw * 32);
    }
}

// ROOT of the warp's columns: what exceeds the earlier columns of the same
// parity, the column's best begin, the reportable cells and the best cell per
// span (first column on equal scores).
template <class S>
__device__ void root(const Params &p, const Ctx &c, const Win &wn, float *vb, int *vbj, int *vbm, float *s_full) {
    typedef typename S::T T;
    const unsigned FULL = 0xffffffffu;
    const T Z = S::zero();
    const bool fill[4] = {true, p.fill_l != 0, p.fill_r != 0, p.fill_t != 0};
    const int mode[4] = {hb::TRM_J, hb::TRM_L, hb::TRM_R, hb::TRM_T};
    const int j = wn.i0 + c.jrel, par = j & 1;
    const int dmax = min(p.dx0, c.jmax);
#pragma unroll 1
    for (int d = 1; d <= dmax; d++) {
        const bool live = d <= c.jrel + 1 && j <= wn.j0;
        float bs = -1.0e36f;
        int bm = hb::TRM_UNKNOWN, br = INT_MAX;
#pragma unroll
        for (int pl = 0; pl < 4; pl++) {
            if (!fill[pl]) continue;
            const int64_t at = ((int64_t)pl * p.W1 + d) * COLS + c.col;
            const T m = live ? S::ld(c.rbm + at) : Z;
            // maximum over the earlier columns of this parity
            T inc = m;
#pragma unroll
            for (int o = 2; o < 32; o <<= 1) {
                const T x = __shfl_up_sync(FULL, inc, o);
                if (c.lane >= o) inc = mx<S>(inc, x);
            }
            T ex = __shfl_up_sync(FULL, inc, 2);
            uint32_t *cy = c.carry + (int64_t)(pl * 2) * p.W1 + d;
            const T cr = S::ld(cy + (int64_t)par * p.W1);
            ex = c.lane >= 2 ? mx<S>(ex, cr) : cr;
            __syncwarp();
            // lanes 30 and 31 hold the warp's maxima of the two parities
            if (c.lane >= 30) S::st(cy + (int64_t)par * p.W1, mx<S>(inc, cr));
            if (live && m > ex) {
                const float f = S::bits(m);
                const int y = (int)c.rby[at];
                if (f > bs || (f == bs && y < br)) {
                    bs = f;
                    bm = mode[pl];
                    br = y;
                }
            }
        }
        if (br == INT_MAX) br = 0;
        if (live) {
            if (j == wn.j0 && d == wn.j0) *s_full = bs;
            if (bs >= p.cutoff && bs > -1.0e36f) {
                const unsigned long long k = atomicAdd(p.ncand, 1ull);
                if ((int64_t)k < p.cap) p.cand[k] = hb::TrCand{wn.idx, j, d, bs, bm, br};
            }
        }
        // first column with the warp's best
        float best = live ? bs : -1.0e36f;
#pragma unroll
        for (int o = 16; o; o >>= 1) best = fmaxf(best, __shfl_xor_sync(FULL, best, o));
        const unsigned who = __ballot_sync(FULL, live && bs == best);
        if (who && c.lane == __ffs(who) - 1 && bs > vb[d]) {
            vb[d] = bs;
            vbj[d] = j;
            vbm[d] = bm;
        }
    }
}

template <bool INS>
__global__ void __launch_bounds__(32 * MAX_WARPS, 1) kernel(const __grid_constant__ Params p) {
    typedef Sem<INS> S;
    extern __shared__ __align__(16) uint32_t tq_smem[];
    __shared__ int s_win;
    __shared__ float s_full;
    const int tid = threadIdx.x, nthreads = blockDim.x;
    Ctx c;
    c.nw = nthreads >> 5;
    c.w = __shfl_sync(0xffffffffu, tid >> 5, 0);
    c.lane = tid & 31;
    c.col = tid;
    c.reg = p.region + (int64_t)blockIdx.x * p.region_words;
    c.buf = c.reg;
    c.begl = c.reg + off_begl(p);
    c.begr = c.reg + off_begr(p);
    c.rbm = c.reg + off_rbm(p);
    c.rby = c.reg + off_rby(p);
    c.bnd = c.reg + off_bnd(p);
    c.carry = c.reg + off_carry(p);
    c.xch = tq_smem;
    float *vb = reinterpret_cast<float *>(tq_smem + c.nw * 2 * CHUNK * 4);
    int *vbj = reinterpret_cast<int *>(vb + p.W1), *vbm = vbj + p.W1;
    uint8_t *ring = reinterpret_cast<uint8_t *>(vbm + p.W1);
    uint16_t *tbl = reinterpret_cast<uint16_t *>(ring + p.ring_len);
    c.ring = ring;
    c.tbl = tbl;
    c.nz = p.ilog_nz;
    c.rmask = p.ring_len - 1;
    if (INS)
        for (int x = tid; x <= p.ilog_nz; x += nthreads) tbl[x] = p.ilog[x];
    for (int x = tid; x < p.ring_len; x += nthreads) ring[x] = 0;
    const int cols = c.nw * 32;
    for (;;) {
        if (tid == 0) s_win = atomicAdd(p.queue, 1);
        __syncthreads();
        const int it = s_win;
        if (it >= p.nwin) break;
        const Win wn = p.wins[it];
        const int ncols = wn.j0 - wn.i0 + 1;
        c.span = wn.w;
        for (int x = tid; x < p.W1; x += nthreads) {
            vb[x] = -1.0e36f;
            vbj[x] = 0;
            vbm[x] = hb::TRM_UNKNOWN;
        }
        for (int x = tid; x < 8 * p.W1; x += nthreads) S::st(c.carry + x, S::zero());
        if (tid == 0) s_full = -1.0e36f;
        __syncthreads();
        const uint8_t *dsq = p.dsq + wn.dsq_off;
        c.step = 0;
        for (int x = 0; x < c.w; x++) phase(nthreads);
        for (int g0 = 0; g0 < ncols; g0 += cols) {
            c.first = g0 == 0;
            c.last = g0 + cols >= ncols;
            c.jrel = g0 + c.col;
            c.ridx = c.jrel % p.ring_cols;
            const int w0 = g0 + c.w * 32;
            c.jmax = w0 < ncols ? min(wn.w, min(w0 + 32, ncols)) : 0;
            int r = c.jrel < ncols ? __ldg(dsq + wn.i0 + c.jrel) : 0;
            r = r > 17 ? 17 : r;
            ring[c.jrel & c.rmask] = (uint8_t)r;
            c.cj = r;
            __syncwarp();
            for (int d = 1; d <= min(p.dx0, c.jmax); d++)
                for (int pl = 0; pl < 4; pl++)
                    S::st(c.rbm + ((int64_t)pl * p.W1 + d) * COLS + c.col, S::zero());
            for (int n = 0; n < p.nnodes; n++) {
                const Node *np = p.nodes + n;
                switch (np->type * 8 + np->nn) {
                case MATP_ND * 8 + 1: node<S, MATP_ND, 1>(p, c, np, n); break;
                case MATP_ND * 8 + 2: node<S, MATP_ND, 2>(p, c, np, n); break;
                case MATP_ND * 8 + 4: node<S, MATP_ND, 4>(p, c, np, n); break;
                case MATL_ND * 8 + 1: node<S, MATL_ND, 1>(p, c, np, n); break;
                case MATL_ND * 8 + 2: node<S, MATL_ND, 2>(p, c, np, n); break;
                case MATL_ND * 8 + 4: node<S, MATL_ND, 4>(p, c, np, n); break;
                case MATR_ND * 8 + 1: node<S, MATR_ND, 1>(p, c, np, n); break;
                case MATR_ND * 8 + 2: node<S, MATR_ND, 2>(p, c, np, n); break;
                case MATR_ND * 8 + 4: node<S, MATR_ND, 4>(p, c, np, n); break;
                case BEGL_ND * 8 + 1: node<S, BEGL_ND, 1>(p, c, np, n); break;
                case BEGL_ND * 8 + 2: node<S, BEGL_ND, 2>(p, c, np, n); break;
                case BEGL_ND * 8 + 4: node<S, BEGL_ND, 4>(p, c, np, n); break;
                case BEGR_ND * 8 + 1: node<S, BEGR_ND, 1>(p, c, np, n); break;
                case BEGR_ND * 8 + 2: node<S, BEGR_ND, 2>(p, c, np, n); break;
                case BEGR_ND * 8 + 4: node<S, BEGR_ND, 4>(p, c, np, n); break;
                case ROOT_ND * 8 + 1: node<S, ROOT_ND, 1>(p, c, np, n); break;
                case ROOT_ND * 8 + 2: node<S, ROOT_ND, 2>(p, c, np, n); break;
                case ROOT_ND * 8 + 4: node<S, ROOT_ND, 4>(p, c, np, n); break;
                default: bif<S>(p, c, np, n); break;
                }
            }
            if (c.jmax > 0) root<S>(p, c, wn, vb, vbj, vbm, &s_full);
            phase(nthreads);
        }
        for (int x = c.w; x < c.nw - 1; x++) phase(nthreads);
        __syncthreads();
        if (tid == 0) {
            float best = -1.0e36f;
            int bj = INT_MAX, bm = hb::TRM_UNKNOWN;
            for (int d = 1; d <= wn.w; d++)
                if (vb[d] > best || (vb[d] == best && best > -1.0e36f && vbj[d] < bj)) {
                    best = vb[d];
                    bj = vbj[d];
                    bm = vbm[d];
                }
            p.res[wn.idx] = Res{best, bm, s_full, 0};
        }
        __syncthreads();
    }
}

int64_t group_phases(const std::vector<Node> &nodes, int span) {
    int64_t n = 1;  // ROOT's begins
    for (const Node &x : nodes) n += (std::min((int)x.rhi, span) + CHUNK) / CHUNK;
    return n;
}

static size_t smem_bytes(const Params &p, int warps) {
    size_t b = (size_t)warps * 2 * CHUNK * 4 * 4 + (size_t)p.W1 * 12 + (size_t)p.ring_len;
    if (p.inside) b += ((size_t)(p.ilog_nz + 1) * 2 + 15) & ~(size_t)15;
    return b;
}

int occupancy(const Params &p, int warps) {
    int n = 0;
    const size_t smem = smem_bytes(p, warps);
    auto k = p.inside ? kernel<true> : kernel<false>;
    if (allow_max_dynamic_smem(k) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, warps * 32, smem) != cudaSuccess) return 0;
    return n;
}

cudaError_t launch(const Params &p, int ctas, int warps, cudaStream_t s) {
    auto k = p.inside ? kernel<true> : kernel<false>;
    cudaError_t e = allow_max_dynamic_smem(k);
    if (e != cudaSuccess) return e;
    k<<<ctas, warps * 32, smem_bytes(p, warps), s>>>(p);
    return cudaGetLastError();
}

bool build(const cmgpu_cm *cm, bool inside, const std::vector<int32_t> &dxcap, const std::vector<char> &kind_skip,
           const std::vector<uint32_t> &pty, const std::vector<int32_t> &pbeg, const std::vector<uint32_t> &lm,
           const std::vector<uint32_t> &rm, const std::vector<uint32_t> &base, const std::vector<int> &begl_idx,
           bool esc_plain, int64_t esc_best, std::vector<Node> &out, int *nbif) {
    const int M = cm->M, W = cm->W;
    if (W > 32000 || M > 32767) return false;
    std::vector<NodeTopo> topo;
    if (!node_topology(cm, topo, nullptr)) return false;
    if (!inside) {
        auto ok = [](const float *f, size_t n) {
            for (size_t x = 0; x < n; x++)
                if (!plain_float(f[x])) return false;
            return true;
        };
        if (!esc_plain || !ok(cm->tsc, (size_t)M * MAXC) || !ok(cm->endsc, M) ||
            !ok(&cm->el_selfsc, 1) || !ok(reinterpret_cast<const float *>(lm.data()), lm.size()) ||
            !ok(reinterpret_cast<const float *>(rm.data()), rm.size()) ||
            !ok(reinterpret_cast<const float *>(pty.data()), pty.size()))
            return false;
    } else {
        // bits of two different integer scores must differ: below 16,384 bits
        // a thousandth is more than a float's step
        int64_t best = std::max<int64_t>(esc_best, 0);
        for (uint32_t x : lm) best = std::max<int64_t>(best, (int32_t)x);
        for (uint32_t x : rm) best = std::max<int64_t>(best, (int32_t)x);
        if ((best + 1000) * (W + 1) > 16000000) return false;
    }
    std::vector<char> begin(M, 0);
    for (int32_t y : pbeg) {
        if (kind_skip[y] || cm->sttype[y] == E_ST) return false;
        begin[y] = 1;
    }
    const int nn = (int)topo.size();
    std::vector<int> hi(nn, 0);
    for (int n = 0; n < nn; n++)
        for (int q = 0; q < topo[n].nst; q++) {
            const int v = topo[n].v0 + q;
            if (cm->sttype[v] == E_ST || v == 0) continue;
            const int dx = std::max(0, dxcap[v]);
            hi[n] = std::max(hi[n], dx);
            if (cm->sttype[v] != B_ST && n + 1 < nn) hi[n + 1] = std::max(hi[n + 1], dx);
        }
    out.clear();
    *nbif = 0;
    for (int n = 0; n < nn; n++)
        if (topo[n].type == BIF_ND) (*nbif)++;
    std::vector<int> deck(nn, -1);
    int b = 0, t = 0;
    for (int n = 0; n < nn; n++)
        if (topo[n].type == BIF_ND) deck[topo[n].begl] = deck[topo[n].begr] = deck[n] = b++;
    for (int n = nn - 1; n >= 0; n--) {
        if (topo[n].type == END_ND) continue;
        Node d{};
        d.v0 = topo[n].v0;
        d.type = (int16_t)topo[n].type;
        d.nn = n + 1 < nn ? (int16_t)topo[n + 1].nsplit : 1;
        d.next_end = topo[n].type != BIF_ND && topo[n + 1].type == END_ND;
        d.need_left = topo[n].need_left;
        d.rhi = (int16_t)std::min(hi[n], W);
        d.chi = n + 1 < nn ? (int16_t)std::min(hi[n + 1], W) : 0;
        d.buf = (int16_t)(t++ % 3);
        d.deck = (int16_t)deck[n];
        for (int q = 0; q < topo[n].nst; q++) {
            const int v = topo[n].v0 + q;
            d.dx[q] = (int16_t)std::max(0, dxcap[v]);
            if (kind_skip[v]) d.skip |= 1 << q;
            if (begin[v]) d.beginmask |= 1 << q;
            const bool has = inside ? cm->iendsc[v] != -INFTY : cm->endsc[v] > IMPOSSIBLE + 1.0f;
            if (has) d.endmask |= 1 << q;
            if (q < 4 && topo[n].type != BEGL_ND) d.base[q] = base[v];
        }
        if (topo[n].type == BEGL_ND) d.base[0] = base[(size_t)3 * M + begl_idx[topo[n].v0]];
        if (d.next_end) d.cbase = base[topo[n + 1].v0];
        if (topo[n].type == BIF_ND) {
            const int wl = cm->cfirst[d.v0], y = cm->cnum[d.v0];
            d.dx_w = (int16_t)std::min(std::max(dxcap[wl], -1), W);
            d.dx_y = (int16_t)std::min(std::max(dxcap[y], -1), W);
            d.begl_base = base[(size_t)3 * M + begl_idx[wl]];
        }
        out.push_back(d);
    }
    return true;
}

}  // namespace trqd
}  // namespace cmx
