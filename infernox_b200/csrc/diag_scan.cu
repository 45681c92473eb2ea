// QDB-banded CYK / Inside window scan by diagonals, for sm_100a.
//
// Cell (v, j, d) of the scan (generic_scan, src/cm_nohmm.rs:549-763) reads
// cells of shorter spans (d-1, d-2) at columns j and j-1, and cells of the
// same span of states below v.  So for one span d every column j is
// independent, IL's self-loop included (it reads span d-1): a warp takes 32
// consecutive columns, one per lane, and walks d upwards with no serial chain
// across lanes and no divergence -- the state type, the band test and the
// transition scores are the same for all lanes.
//
// Order of work.  A work item is a piece of a window; a CTA takes its columns
// in groups of 32 x warps, left to right.  For a group the nodes run from
// the last one up, and inside a node d runs from the shortest span stored to
// the longest.  All states of a node are computed together: its inserts never
// leave the registers (their left neighbour comes by shuffle), and of the
// next node only the split states are read, once per span: one load and one
// store per split cell, instead of one load per child relaxation.
//   buffers   three node buffers [span][split state][column] used in turn;
//   BEGL      a ring of W + group columns per bifurcation (a split reads
//             columns j-k), BEGR the group's columns;
//   bmax      the ROOT row of local begins (a maximum, so the node order does
//             not matter);
//   boundary  the last column of every node is saved for the first column of
//             the next group, so groups repeat no work.
// All of it is in a per-CTA region of global memory.  A CTA works on two node
// buffers at a time, 0.6 MB each for a MATP node at W = 148, so the 296 CTAs of
// a full GPU hold more than the L2 does: 39% of the sectors hit, and a cell
// moves 7.75 bytes of DRAM.
//
// Warps run skewed.  A step is one node over 16 spans; a warp starts a step
// when the warp on its left has finished it, so the column left of its first
// one is there.  A warp may run ahead of the one on its right by a few steps
// and one node: three node buffers in turn and an exchange ring keep what that
// one still reads.  Warps publish their step counts in shared memory; every
// wait is bounded.  There is no CTA barrier inside an item: with one per step
// every warp waited for the slowest node in flight (a third of the stall
// cycles), with one step of slack the handshake itself was the limit.
//
// Spans beyond a column's own start (d > j - jstart + 1) and columns past the
// item's end hold values nobody reads: a valid cell depends on valid cells
// only.  Rows are addressed by span, residues by a masked ring, so those
// cells stay in bounds.
//
// Measured on one B200 (before: the level kernel of qdb_scan.cu): Inside,
// non-banded, M = 379, W = 148, 296 windows of 512: 219 Gcells/s, CYK 335; two
// 1 kb windows of a 4,629-state model, CYK, whole call: 1,745 -> 51 ms.  Bound:
// the latency of the log-sum chains (LDS and dependent ALU) at 16 warps per SM,
// half of the issue slots; DRAM 26% of the copy bandwidth.
#include <cuda_runtime.h>
#include <cstdint>
#include <type_traits>

#include "devbuf.h"
#include "diag_kernel.h"
#include "report_device.cuh"
#include "cm_internal.h"
#include "semiring.cuh"

namespace cmx {
namespace dev {

// Per-warp view of the group it works on.
struct DgCtx {
    uint32_t *reg;           // the CTA's region
    const uint8_t *ring;     // residues of the item (shared memory)
    uint32_t *xch;           // [warps][DG_XCH][DG_CHUNK][2] last column's inserts (shared memory)
    int nz, rmask;
    int nw, w, lane, col;    // col = 32 w + lane
    int jrel;                // column relative to the item's first
    int ridx;                // jrel modulo the BEGL ring
    int cj;                  // residue of column j
    int jmax;                // longest span any lane of the warp can hold (0: no column)
    int ncols;               // columns of the item
    uint32_t prog;           // shared address of the warps' step counts
    int *err;                // a wait gave up (shared memory)
    int step, step0, gsteps; // steps done, at the item's start, steps of a whole group
    int prev;                // step the previous node began with
    int slack;               // steps a warp may be ahead of its right neighbour, at most DG_XCH
    uint32_t *stg;           // the warp's staged child spans (shared memory)
    bool first, last;        // first / last group of the item
    int item, j, jreport, jend;
};

// Waits between warps: each warp publishes how many steps it has finished.
constexpr int DG_TRIES = 1 << 24;  // polls before a wait gives up (two seconds or so)

__device__ __forceinline__ int dg_seen(uint32_t addr) {
    int v;
    asm volatile("ld.acquire.cta.shared.s32 %0, [%1];" : "=r"(v) : "r"(addr) : "memory");
    return v;
}

// Until warp w has finished `need` steps.  Bounded: past DG_TRIES the error
// is marked, every other wait gives up too, and the call fails.
__device__ __forceinline__ void dg_wait(const DgCtx &c, int w, int need) {
    for (int it = 0; dg_seen(c.prog + w * 4) - need < 0; it++) {
        if (it < 16) continue;
        if (*(volatile int *)c.err || it > DG_TRIES) {
            *(volatile int *)c.err = 1;
            break;
        }
        __nanosleep(20);
    }
}

// Before a node: the warp on the right has finished the node before the
// previous one (prev: the step the previous node began with), so it no longer
// reads the buffer this node writes.  (The plan keeps that so from a group's
// ROOT to the next group's first node.)
__device__ __forceinline__ void dg_begin_node(DgCtx &c) {
    if (c.w < c.nw - 1) dg_wait(c, c.w + 1, c.prev);
    c.prev = c.step;
}

// Before step s: the warp on the left has finished it (this warp reads its
// last column), and the warp on the right step s - slack (it has read the
// exchange slot this step writes).  The first warp's left neighbour is the
// last warp one group earlier.  (The ring holds DG_XCH steps; slack is at most
// that.)
__device__ __forceinline__ void dg_begin_step(const DgCtx &c) {
    if (c.w > 0) dg_wait(c, c.w - 1, c.step + 1);
    else if (c.step - c.step0 >= c.gsteps) dg_wait(c, c.nw - 1, c.step - c.gsteps + 1);
    if (c.w < c.nw - 1) dg_wait(c, c.w + 1, c.step - c.slack + 1);
    __syncwarp();
}

// After a step: every write of the warp, then its count.
__device__ __forceinline__ void dg_end_step(DgCtx &c) {
    c.step++;
    __syncwarp();
    if (c.lane == 0)
        asm volatile("st.release.cta.shared.s32 [%0], %1;" ::"r"(c.prog + c.w * 4), "r"(c.step) : "memory");
}

// 16 and 4 bytes to shared memory, asynchronously
__device__ __forceinline__ void dg_cp16(uint32_t *dst, const uint32_t *src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}
__device__ __forceinline__ void dg_cp4(uint32_t *dst, const uint32_t *src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"((uint32_t)__cvta_generic_to_shared(dst)), "l"(src)
                 : "memory");
}

extern __shared__ __align__(16) uint32_t dg_smem[];  // Inside: the ILogsum table first

// ILogsum as Sem<true>::comb, with the table at a fixed shared-memory
// address; max for CYK (the plan holds no -0 or NaN).
//
// FAST leaves out the rule for impossible operands (at or below -INFTY they
// add nothing, and the result is at least -INFTY).  The table reaches less
// than 2^15, so it cannot matter where one operand is a real score: the other
// one is then out of the table's reach.  Two impossible operands may come out
// up to a table entry too high, which stays impossible (below REAL) and, by
// the same argument, changes no real score it is combined with.  So a fold
// (before its emission score) whose FAST value is a real score is exact.
// |a - b| is the smaller of a - b and b - a as unsigned numbers.
template <class S, bool FAST>
__device__ __forceinline__ typename S::T dg_comb(typename S::T a, typename S::T b, int nz) {
    if constexpr (S::ORDERED) {
        const uint16_t *tbl = reinterpret_cast<const uint16_t *>(dg_smem);
        if (FAST) {
            const uint32_t x = (uint32_t)a - (uint32_t)b, y = (uint32_t)b - (uint32_t)a;
            return (int32_t)((uint32_t)max(a, b) + tbl[min(min(x, y), (uint32_t)nz)]);
        }
        const int32_t mx = max(max(a, b), -INFTY_D), mn = min(a, b);
        const uint32_t i = min((uint32_t)mx - (uint32_t)mn, (uint32_t)nz);
        return (int32_t)((uint32_t)mx + tbl[mn > -INFTY_D ? i : (uint32_t)nz]);
    } else {
        return fmaxf(a, b);
    }
}
constexpr int32_t DG_REAL = -500000000;  // real scores are above, impossible ones (and sums of two) below

// reduce_c_order (src/cm_nohmm.rs:187-242) of CN child terms and, where the
// state has a local end, its initial score.  Without one the initial score is
// -INFTY: combining with it only clamps at -INFTY, which every later
// combination does anyway, so it is left out (with one child it is not).
template <class S, int CN, bool FAST>
__device__ __forceinline__ typename S::T dg_reduce(const typename S::T *t, bool has, typename S::T init,
                                                   int nz) {
    typedef typename S::T T;
    if constexpr (!S::ORDERED) {
        T s = has ? init : S::zero();
#pragma unroll
        for (int k = 0; k < CN; k++) s = fmaxf(s, t[k]);
        return s;
    } else {
        T s;
        if constexpr (CN == 1) {
            s = has ? dg_comb<S, FAST>(init, t[0], nz) : max(t[0], -INFTY_D);
            return s;
        }
        if constexpr (CN == 2) s = t[1];
        if constexpr (CN == 3) s = dg_comb<S, FAST>(t[2], t[1], nz);
        if constexpr (CN == 4 || CN == 5) s = dg_comb<S, FAST>(t[CN - 1], t[CN - 2], nz);
        if constexpr (CN == 6) s = t[5];
        if (has) s = dg_comb<S, FAST>(s, init, nz);
        if constexpr (CN == 4) s = dg_comb<S, FAST>(s, t[1], nz);
        if constexpr (CN == 5) {
            s = dg_comb<S, FAST>(s, t[1], nz);
            s = dg_comb<S, FAST>(s, t[2], nz);
        }
        if constexpr (CN == 6) {
            s = dg_comb<S, FAST>(s, t[4], nz);
            s = dg_comb<S, FAST>(s, t[3], nz);
            s = dg_comb<S, FAST>(s, t[2], nz);
            s = dg_comb<S, FAST>(s, t[1], nz);
        }
        return dg_comb<S, FAST>(s, t[0], nz);
    }
}

// Children in natural order (BEGL_S and ROOT_S, src/cm_nohmm.rs:601-611, :700-719).
template <class S, int CN, bool FAST>
__device__ __forceinline__ typename S::T dg_natural(const typename S::T *t, bool has, typename S::T init,
                                                    int nz) {
    typedef typename S::T T;
    if constexpr (!S::ORDERED) {
        return dg_reduce<S, CN, FAST>(t, has, init, nz);
    } else {
        T s = has ? dg_comb<S, FAST>(init, t[0], nz) : max(t[0], -INFTY_D);
#pragma unroll
        for (int k = 1; k < CN; k++) s = dg_comb<S, FAST>(s, t[k], nz);
        return s;
    }
}

// Local begins: the larger of two ROOT values as begin_less orders them
// (KEY, cmcalibrate's order: -INFTY is held as INT_MIN).
template <class S>
__device__ __forceinline__ typename S::T dg_begin_max(typename S::T a, typename S::T c) {
    return a < c ? c : a;
}
template <class S, bool KEY>
__device__ __forceinline__ typename S::T dg_begin_key(typename S::T c) {
    if constexpr (S::ORDERED && KEY)
        if (c == -INFTY_D) return INT32_MIN;
    return c;
}
template <class S, bool KEY>
__device__ __forceinline__ typename S::T dg_begin_none() {
    if constexpr (S::ORDERED) return KEY ? INT32_MIN : -INFTY_D;
    else return -INFINITY;
}

// One node over the group's columns: NT its type, NN the split states of the
// next node.
//
// Two versions of the same step: `edge` tests every band and row range;
// `inner` runs where nothing needs a test (every state in band, the child
// rows stored, no d = 0) and at most the first state has a local begin or a
// local end, which is how local models are configured.  Child values come
// through shared memory, copied asynchronously eight spans ahead or more.
template <class S, bool KEY, int NT, int NN>
__device__ __forceinline__ void dg_node(const DgParams &p, DgCtx &c, const DgNode *np) {
    typedef typename S::T T;
    constexpr bool HAS_IL = NT == MATP_ND || NT == MATL_ND || NT == ROOT_ND || NT == BEGR_ND;
    constexpr bool HAS_IR = NT == MATP_ND || NT == MATR_ND || NT == ROOT_ND;
    constexpr bool LEFT = HAS_IR;  // MP, MR and IR read column j-1
    constexpr int NSPLIT = NT == MATP_ND ? 4 : (NT == MATL_ND || NT == MATR_ND) ? 2 : 1;
    constexpr int QIL = NSPLIT, QIR = HAS_IL ? NSPLIT + 1 : NSPLIT;  // insert states within the node
    constexpr int NI = (HAS_IL ? 1 : 0) + (HAS_IR ? 1 : 0);
    constexpr int CN = NI + NN;  // children of a split state
    // staged spans: as many stages of four as the warp's share holds
    constexpr int SROW = NN * 36 + 32, SB = NN * 36, NST = DG_STG / (DG_STAGE * SROW);
    constexpr int MP = NT == MATP_ND ? 0 : -1, ML = NT == MATP_ND ? 1 : NT == MATL_ND ? 0 : -1,
                  MR = NT == MATP_ND ? 2 : NT == MATR_ND ? 0 : -1;
    const unsigned FULL = 0xffffffffu;
    const T ZERO = S::zero();
    const int v0 = np->v0, rlo = np->rlo, clo = np->clo, chi = np->chi;
    const int rhi = min(np->rhi, c.ncols);  // no column of the item holds a longer span
    const bool cend = np->next_end != 0;
    const T cinit = S::ld(&np->cinit0);
    const int endmask = np->endmask, beginmask = np->beginmask;
    const bool need_left = np->need_left != 0;
    uint32_t *out = c.reg + np->out_off;
    int ostride;
    if (NT == BEGL_ND) {
        out += c.ridx;
        ostride = p.ring_cols;
    } else if (NT == BEGR_ND) {
        out += c.col;
        ostride = DG_COLS;
    } else {
        out += 32 + c.col;
        ostride = DG_ROW;
    }
    const uint32_t *in = c.reg + np->in_off + 32 + c.col;
    uint32_t *bnd = c.reg + np->bnd_off;
    uint32_t *bndi = bnd + (int64_t)(np->rhi - rlo + 1) * DG_SLOTS;
    T *const bmax = reinterpret_cast<T *>(c.reg + c.col);

    // spans the inner step takes
    int ilo = max(1, p.root_dn), ihi = min(rhi, p.root_dxcap);
#pragma unroll
    for (int q = 0; q < NSPLIT + NI; q++) {
        ilo = max(ilo, (int)np->dn[q]);
        ihi = min(ihi, (int)np->dx[q]);
    }
    ilo = max(ilo, clo);
    ihi = min(ihi, chi);
    if (cend || ((endmask | beginmask) & ~1)) ihi = -1;
    const bool end0 = (endmask & 1) != 0, beg0 = p.local && (beginmask & 1) != 0;
    const T es0 = end0 ? S::ldg(p.endsc + v0) : ZERO;
    const T bs0 = beg0 ? S::ldg(p.bsv + v0) : ZERO;

    // transition scores, in registers
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

    auto ldx = [&](int y, int d, int shift) -> T {  // split state y of the next node at (j - shift, d)
        if (cend) return d == 0 ? cinit : ZERO;
        if (d < clo || d > chi) return ZERO;
        return S::ld(in + (int64_t)(d - clo) * DG_ROW + y * DG_PITCH - shift);
    };
    // Spans h..h+3 of the child (and of the ROOT row of local begins) on their
    // way to shared memory: 8 lanes a span, one copy per split state, and the
    // column on the left.
    const bool begins = p.local && beginmask != 0;
    const int frow = c.lane >> 3, fpart = (c.lane & 7) * 4, hrow = c.lane / NN, hy = c.lane % NN;
    const uint32_t *fsrc = in - c.lane + (int64_t)(rlo + frow - clo) * DG_ROW + fpart;
    const uint32_t *hsrc = in - c.lane + (int64_t)(rlo + hrow - clo) * DG_ROW + hy * DG_PITCH - 1;
    const uint32_t *bsrc = c.reg + c.col - c.lane + fpart + (int64_t)(rlo + frow) * DG_COLS;
    const int flo = cend ? 1 << 30 : clo, blo = begins ? p.root_dn : 1 << 30;
    int fh = rlo;  // first span of the next stage
    auto fetch = [&](int half) {
        uint32_t *dst = c.stg + half * (DG_STAGE * SROW);
        if (fh + frow >= flo && fh + frow <= chi)
#pragma unroll
            for (int y = 0; y < NN; y++) dg_cp16(dst + frow * SROW + y * 36 + 4 + fpart, fsrc + y * DG_PITCH);
        if (LEFT && hrow < DG_STAGE && fh + hrow >= flo && fh + hrow <= chi) dg_cp4(dst + hrow * SROW + hy * 36 + 3, hsrc);
        if (fh + frow >= blo && fh + frow <= p.root_dxcap) dg_cp16(dst + frow * SROW + SB + fpart, bsrc);
        asm volatile("cp.async.commit_group;" ::: "memory");
        fh += DG_STAGE;
        fsrc += DG_STAGE * DG_ROW;
        hsrc += DG_STAGE * DG_ROW;
        bsrc += DG_STAGE * DG_COLS;
    };
    const uint32_t *esc0 = p.esc + (int64_t)v0 * ESC;
    const uint32_t *escr = esc0 + c.cj;

    // xp: column j at d-1; xl2, xl1: column j-1 at d-2, d-1; il*, ir*: the
    // inserts at d-1 (and column j-1, d-1 and d-2)
    T xp[NN], xl2[NN], xl1[NN];
    T ilp = ZERO, irp = ZERO, il1 = ZERO, il2 = ZERO, ir1 = ZERO, ir2 = ZERO;
    int d = rlo;
#pragma unroll
    for (int k = 0; k < NST - 1; k++) fetch(k);
    int half = 0;  // stage of span d
#pragma unroll
    for (int y = 0; y < NN; y++) {
        xp[y] = ldx(y, d - 1, 0);
        if (LEFT) {
            xl2[y] = ldx(y, d - 2, 1);
            xl1[y] = ldx(y, d - 1, 1);
        }
    }
    int ci = HAS_IL ? c.ring[(c.jrel - d + 1) & c.rmask] : 0;  // residue j-d+1
    for (int r0 = rlo; r0 <= rhi; r0 += DG_CHUNK) {
        const int rend = min(r0 + DG_CHUNK - 1, rhi);
        const int dstop = min(rend, c.jmax);
        const int slot = c.step & (DG_XCH - 1);
        dg_begin_step(c);
        // the inserts of the column left of the warp: lane r holds span r0 + r
        T hil = ZERO, hir = ZERO;
        if constexpr (HAS_IR) {
            const int r = c.lane & (DG_CHUNK - 1);
            if (c.w > 0) {
                const uint32_t *lp = c.xch + (((c.w - 1) * DG_XCH + slot) * DG_CHUNK + r) * 2;
                hil = S::ld(lp);
                hir = S::ld(lp + 1);
            } else if (!c.first && r0 + r <= rend) {
                const uint32_t *lp = bndi + (int64_t)(r0 + r - rlo) * 2;
                hil = S::ld(lp);
                hir = S::ld(lp + 1);
            }
        }
        uint32_t *xs = c.xch + (c.w * DG_XCH + slot) * (DG_CHUNK * 2);
        // the column left of the group (its parent reads it)
        if (NT != ROOT_ND && need_left && c.w == 0) {
            const int r = c.lane & (DG_CHUNK - 1), h = r0 + r;
            if (c.lane < DG_CHUNK && h <= dstop) {
#pragma unroll
                for (int q = 0; q < NSPLIT; q++) {
                    T x = h == 0 ? S::ld(&np->init0[q]) : ZERO;
                    if (!c.first) x = S::ld(bnd + (h - rlo) * DG_SLOTS + q);
                    S::st(out - c.lane + (int64_t)(h - rlo) * DG_ROW + q * DG_PITCH - 1, x);
                }
            }
        }

        // one span; px, po: rows d of the child (column j) and of the outputs
        auto step = [&](auto inner_c, const uint32_t *sx, uint32_t *po, T *bp) -> bool {
            constexpr bool INNER = decltype(inner_c)::value;
            T xc[NN], xln[NN];
            const bool stored = INNER || (!cend && d >= clo && d <= chi);
#pragma unroll
            for (int y = 0; y < NN; y++) {
                const T none = !INNER && cend && d == 0 ? cinit : ZERO;
                xc[y] = stored ? S::ld(sx + y * 36 + 4) : none;
                if (LEFT) xln[y] = stored ? S::ld(sx + y * 36 + 3) : none;
            }
            const uint32_t *esci = esc0 + ci;
            T eil, eml, emp;
            if (HAS_IL) eil = S::ldg(esci + QIL * ESC);
            if (ML >= 0) eml = S::ldg(esci + (ML < 0 ? 0 : ML) * ESC);
            if (MP >= 0) emp = S::ldg(escr + ci * KP);
            const int cn = HAS_IL ? c.ring[(c.jrel - d) & c.rmask] : 0;
            const T el0 = INNER && (NT != BEGL_ND && NT != BEGR_ND) ? ZERO : S::ldg(p.el_sca + d);
            const T el1 = INNER && NT == MATP_ND ? ZERO : S::ldg(p.el_sca + max(d - 1, 0));
            const T el2 = NT == MATP_ND ? S::ldg(p.el_sca + max(d - 2, 0)) : ZERO;
            T bc = dg_begin_none<S, KEY>();
            auto begin = [&](int q, T x) {
                if (!INNER && (beginmask >> q & 1))
                    bc = dg_begin_max<S>(bc, dg_begin_key<S, KEY>(S::add(x, S::ldg(p.bsv + v0 + q))));
            };
            auto in_band = [&](int q) { return INNER || (d >= np->dn[q] && d <= np->dx[q]); };
            auto fill = [&](int q) -> T { return !INNER && d == 0 ? S::ld(&np->init0[q]) : ZERO; };
            // (inner: without a local end the first state's initial score is
            // the impossible one, which changes nothing, so no branch)
            auto has = [&](int q) { return INNER ? q == 0 : (endmask >> q & 1) != 0; };
            auto init = [&](int q, T el) -> T {
                return INNER ? (end0 ? S::add(el, es0) : ZERO) : S::add(el, S::ldg(p.endsc + v0 + q));
            };
            T iln = ZERO, irn = ZERO;
            T val[NSPLIT];
            int32_t low = INT32_MAX;  // smallest value before its emission
            // inserts
            if constexpr (HAS_IL) {
                iln = fill(QIL);
                if (in_band(QIL)) {
                    T t[CN];
                    t[0] = S::add(ilp, til[0]);
                    if (HAS_IR) t[1] = S::add(irp, til[1]);
#pragma unroll
                    for (int y = 0; y < NN; y++) t[NI + y] = S::add(xp[y], til[NI + y]);
                    iln = dg_reduce<S, CN, INNER>(t, has(QIL), INNER ? ZERO : init(QIL, el1), c.nz);
                    if constexpr (INNER && S::ORDERED) low = min(low, (int32_t)iln);
                    iln = S::add(iln, eil);
                    begin(QIL, iln);
                }
            }
            if constexpr (HAS_IR) {
                irn = fill(QIR);
                if (in_band(QIR)) {
                    T t[NN + 1];
                    t[0] = S::add(ir1, tir[0]);
#pragma unroll
                    for (int y = 0; y < NN; y++) t[1 + y] = S::add(xl1[y], tir[1 + y]);
                    irn = dg_reduce<S, NN + 1, INNER>(t, has(QIR), INNER ? ZERO : init(QIR, el1), c.nz);
                    if constexpr (INNER && S::ORDERED) low = min(low, (int32_t)irn);
                    irn = S::add(irn, S::ldg(escr + QIR * ESC));
                    begin(QIR, irn);
                }
            }
            // split states
#pragma unroll
            for (int q = 0; q < NSPLIT; q++) {
                val[q] = fill(q);
                if (!in_band(q)) continue;
                T t[CN];
                T x;
                if (q == MP) {
                    t[0] = S::add(il2, ts[q][0]);
                    t[1] = S::add(ir2, ts[q][1]);
#pragma unroll
                    for (int y = 0; y < NN; y++) t[NI + y] = S::add(xl2[y], ts[q][NI + y]);
                    x = dg_reduce<S, CN, INNER>(t, has(q), init(q, el2), c.nz);
                } else if (q == ML) {
                    t[0] = S::add(ilp, ts[q][0]);
                    if (HAS_IR) t[1] = S::add(irp, ts[q][1]);
#pragma unroll
                    for (int y = 0; y < NN; y++) t[NI + y] = S::add(xp[y], ts[q][NI + y]);
                    x = dg_reduce<S, CN, INNER>(t, has(q), init(q, el1), c.nz);
                } else if (q == MR) {
                    t[0] = S::add(HAS_IL ? il1 : ir1, ts[q][0]);
                    if (HAS_IL) t[1] = S::add(ir1, ts[q][1]);
#pragma unroll
                    for (int y = 0; y < NN; y++) t[NI + y] = S::add(xl1[y], ts[q][NI + y]);
                    x = dg_reduce<S, CN, INNER>(t, has(q), init(q, el1), c.nz);
                } else {  // D, S
                    if (HAS_IL) t[0] = S::add(iln, ts[q][0]);
                    if (HAS_IR) t[HAS_IL ? 1 : 0] = S::add(irn, ts[q][HAS_IL ? 1 : 0]);
#pragma unroll
                    for (int y = 0; y < NN; y++) t[NI + y] = S::add(xc[y], ts[q][NI + y]);
                    if (NT == ROOT_ND) x = dg_natural<S, CN, INNER>(t, false, ZERO, c.nz);
                    else if (NT == BEGL_ND) x = dg_natural<S, CN, INNER>(t, has(q), init(q, el0), c.nz);
                    else x = dg_reduce<S, CN, INNER>(t, has(q), init(q, el0), c.nz);
                }
                if constexpr (INNER && S::ORDERED) low = min(low, (int32_t)x);
                if (q == MP) x = S::add(x, emp);
                else if (q == ML) x = S::add(x, eml);
                else if (q == MR) x = S::add(x, S::ldg(escr + q * ESC));
                val[q] = x;
                if (NT != ROOT_ND) begin(q, x);
            }
            if constexpr (INNER && S::ORDERED) {
                // a lane whose span is too long for its column holds anything
                if (__any_sync(FULL, low < DG_REAL && d <= c.jrel + 1)) return false;
            }
            if (NT != ROOT_ND)
#pragma unroll
                for (int q = 0; q < NSPLIT; q++) S::st(po + q * DG_PITCH, val[q]);
            if (INNER) {
                if (beg0) {
                    *bp = dg_begin_max<S>(S::ld(sx + SB), dg_begin_key<S, KEY>(S::add(val[0], bs0)));
                }
            } else if (d >= p.root_dn && d <= p.root_dxcap) {
                if (begins) *bp = dg_begin_max<S>(S::ld(sx + SB), bc);
                if (NT == ROOT_ND) {
                    T a = val[0];
                    if (p.local && dg_begin_key<S, KEY>(a) < *bp) a = *bp;
                    if (p.prefilter) {
                        *bp = a;
                    } else {
                        const float sc = S::bits(a);
                        const bool hit = sc >= p.cutoff && sc > IMPOSSIBLE_D + 1.0f && d <= c.jrel + 1 &&
                                         c.j >= c.jreport && c.j <= c.jend;
                        emit_cand(p, c.lane, hit, c.item, c.j, d, S::u(a));
                    }
                }
            }
            // hand the inserts to the column on the right
            if constexpr (HAS_IR) {
                T li = ZERO, lr, t;
                if (HAS_IL) {
                    li = __shfl_up_sync(FULL, iln, 1);
                    t = __shfl_sync(FULL, hil, d - r0);
                    if (c.lane == 0) li = t;
                }
                lr = __shfl_up_sync(FULL, irn, 1);
                t = __shfl_sync(FULL, hir, d - r0);
                if (c.lane == 0) lr = t;
                if (c.lane == 31) {
                    if (HAS_IL) S::st(xs + (d - r0) * 2, iln);
                    S::st(xs + (d - r0) * 2 + 1, irn);
                }
                il2 = il1;
                il1 = li;
                ir2 = ir1;
                ir1 = lr;
            }
            ilp = iln;
            irp = irn;
#pragma unroll
            for (int y = 0; y < NN; y++) {
                xp[y] = xc[y];
                if (LEFT) {
                    xl2[y] = xl1[y];
                    xl1[y] = xln[y];
                }
            }
            if (HAS_IL) ci = cn;
            return true;
        };
        for (int s0 = r0; s0 <= dstop; s0 += DG_STAGE) {
            const int send = min(s0 + DG_STAGE - 1, dstop);
            __syncwarp();
            fetch(half == 0 ? NST - 1 : half - 1);
            asm volatile("cp.async.wait_group %0;" ::"n"(NST - 1) : "memory");
            __syncwarp();
            const uint32_t *sx = c.stg + half * (DG_STAGE * SROW) + c.lane;
            uint32_t *po = out + (int64_t)(d - rlo) * ostride;
            T *bp = bmax + (int64_t)d * DG_COLS;
            while (d <= send) {
                if (NT != ROOT_ND && d >= ilo && d <= ihi) {
                    const int iend = min(send, ihi);
#pragma unroll 1
                    while (step(std::true_type(), sx, po, bp)) {
                        sx += SROW;
                        po += ostride;
                        bp += DG_COLS;
                        if (++d > iend) break;
                    }
                    if (d > iend) continue;
                }
                step(std::false_type(), sx, po, bp);
                sx += SROW;
                po += ostride;
                bp += DG_COLS;
                d++;
            }
            half = half == NST - 1 ? 0 : half + 1;
        }
        // the group's last column, for the next group
        if (!c.last && c.w == c.nw - 1) {
            __syncwarp();
            const int r = c.lane & (DG_CHUNK - 1), h = r0 + r;
            if (c.lane < DG_CHUNK && h <= dstop) {
                if (NT != ROOT_ND && need_left)
#pragma unroll
                    for (int q = 0; q < NSPLIT; q++)
                        S::st(bnd + (h - rlo) * DG_SLOTS + q,
                              S::ld(out + (31 - c.lane) + (int64_t)(h - rlo) * DG_ROW + q * DG_PITCH));
                if (HAS_IR) {
                    bndi[(int64_t)(h - rlo) * 2] = xs[r * 2];
                    bndi[(int64_t)(h - rlo) * 2 + 1] = xs[r * 2 + 1];
                }
            }
        }
        dg_end_step(c);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncwarp();
}

// Bifurcation node: alpha[v][d] = init (+) over k ascending of
// BEGL(j-k, d-k) + BEGR(j, k) (src/cm_nohmm.rs:578-600).  Four spans at a
// time share the BEGR loads and give four independent chains.
template <class S, bool KEY>
__device__ __forceinline__ void dg_bif(const DgParams &p, DgCtx &c, const DgNode *np) {
    typedef typename S::T T;
    const T ZERO = S::zero();
    const int v0 = np->v0, rlo = np->rlo, rhi = min(np->rhi, c.ncols);
    const int dn = np->dn[0], dx = np->dx[0];
    const int kdn_y = np->kdn_y, kdx_y = np->kdx_y, kdn_w = np->kdn_w, kdx_w = np->kdx_w;
    const uint32_t *begl = c.reg + np->begl_off, *begr = c.reg + np->begr_off + c.col;
    const int llo = np->begl_lo, ylo = np->begr_lo, RC = p.ring_cols;
    const T linit = S::ld(&np->begl_init0);
    const bool need_left = np->need_left != 0, has = (np->endmask & 1) != 0, beg = (np->beginmask & 1) != 0;
    const T bs = beg ? S::ldg(p.bsv + v0) : ZERO, es = has ? S::ldg(p.endsc + v0) : ZERO;
    uint32_t *out = c.reg + np->out_off + 32 + c.col;
    uint32_t *bnd = c.reg + np->bnd_off;
    constexpr int U = 4;
    for (int r0 = rlo; r0 <= rhi; r0 += DG_CHUNK) {
        const int dstop = min(min(r0 + DG_CHUNK - 1, rhi), c.jmax);
        dg_begin_step(c);
        for (int d0 = r0; d0 <= dstop; d0 += U) {
            T acc[U];
            int klo[U], khi[U];
            int ka = 1 << 30, kb = -1, ba = 0, bb = 1 << 30;
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int d = d0 + u;
                acc[u] = has ? S::add(S::ldg(p.el_sca + min(d, p.W)), es) : ZERO;
                klo[u] = max(0, max(kdn_y, d - kdx_w));
                khi[u] = min(kdx_y, d - kdn_w);
                if (d < dn || d > dx || d > dstop) klo[u] = 0, khi[u] = -1;
                if (khi[u] >= klo[u]) {
                    ka = min(ka, klo[u]);
                    kb = max(kb, khi[u]);
                }
                // splits every span has, with a BEGL span of at least 1
                ba = max(ba, klo[u]);
                bb = min(bb, min(khi[u], d - 1));
            }
            auto ring = [&](int k) {
                int x = c.ridx - k;
                return x < 0 ? x + RC : x;
            };
            auto edge = [&](int k0, int k1) {
                for (int k = k0; k <= k1; k++) {
                    const T rv = S::ld(begr + (int64_t)(k - ylo) * DG_COLS);
                    const uint32_t *lc = begl + ring(k) + (int64_t)(d0 - k - llo) * RC;
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        if (k < klo[u] || k > khi[u]) continue;
                        const T lv = k == d0 + u ? linit : S::ld(lc + (int64_t)u * RC);
                        acc[u] = S::ORDERED ? dg_comb<S, false>(acc[u], S::add(lv, rv), c.nz)
                                            : (T)fmaxf((float)acc[u], (float)S::add(lv, rv));
                    }
                }
            };
            if (bb < ba) {
                edge(ka, kb);
            } else {
                edge(ka, ba - 1);
                const uint32_t *rp = begr + (int64_t)(ba - ylo) * DG_COLS;
                int rx = ring(ba);
                const uint32_t *lr = begl + (int64_t)(d0 - ba - llo) * RC;
#pragma unroll 4
                for (int k = ba; k <= bb; k++) {
                    const T rv = S::ld(rp);
#pragma unroll
                    for (int u = 0; u < U; u++) {
                        const T x = S::add(S::ld(lr + rx + (int64_t)u * RC), rv);
                        if constexpr (S::ORDERED) acc[u] = dg_comb<S, false>(acc[u], x, c.nz);
                        else acc[u] = fmaxf(acc[u], x);
                    }
                    rp += DG_COLS;
                    lr -= RC;
                    rx = rx == 0 ? RC - 1 : rx - 1;
                }
                edge(bb + 1, kb);
            }
#pragma unroll
            for (int u = 0; u < U; u++) {
                const int d = d0 + u;
                if (d > dstop) continue;
                const bool in = d >= dn && d <= dx;
                const T fill = d == 0 ? S::ld(&np->init0[0]) : ZERO;
                const T x = in ? acc[u] : fill;
                uint32_t *o = out + (int64_t)(d - rlo) * DG_ROW;
                S::st(o, x);
                if (need_left) {
                    // the column left of the group, and the group's last one,
                    // which takes its place (a warp alone holds both)
                    if (c.w == 0 && c.lane == 0) S::st(o - 1, c.first ? fill : S::ld(bnd + (d - rlo) * DG_SLOTS));
                    if (c.nw == 1) __syncwarp();
                    if (!c.last && c.w == c.nw - 1 && c.lane == 31) S::st(bnd + (d - rlo) * DG_SLOTS, x);
                }
                if (p.local && beg && in && d >= p.root_dn && d <= p.root_dxcap) {
                    T *bm = reinterpret_cast<T *>(c.reg + c.col + (int64_t)d * DG_COLS);
                    *bm = dg_begin_max<S>(*bm, dg_begin_key<S, KEY>(S::add(x, bs)));
                }
            }
        }
        dg_end_step(c);
    }
}

// Report pre-filter of the warp's columns, one column per lane (the rule of
// prefilter_row in qdb_scan.cu: with approximate corrected scores, a cell is
// dropped only when it surely can neither be reported nor raise the running
// maximum of the reported scores).  null3 only lowers a score, so a cell
// whose uncorrected score is already below the running maximum needs none.
template <class S>
__device__ void dg_prefilter(const DgParams &p, const DgCtx &c) {
    const uint32_t *row = c.reg + c.col;
    uint32_t c01 = 0, c23 = 0;  // counts of residues 0,1 / 2,3 in j-d+1..j, 16 bits each
    float run = -INFINITY;
    const bool live = c.j >= c.jreport && c.j <= c.jend;
    const int dmax = min(p.root_dxcap, c.jmax);
    for (int d = 1; d <= dmax; d++) {
        const int r = c.ring[(c.jrel - d + 1) & c.rmask];
        c01 += (r == 0 ? 1u : 0u) | (r == 1 ? 0x10000u : 0u);
        c23 += (r == 2 ? 1u : 0u) | (r == 3 ? 0x10000u : 0u);
        bool hit = false;
        uint32_t raw = 0;
        if (live && d >= p.root_dn && d <= c.jrel + 1) {
            raw = row[(int64_t)d * DG_COLS];
            const float bits = S::bits(S::ld(row + (int64_t)d * DG_COLS));
            const float bar = run == -INFINITY ? -INFINITY : run - pf_margin(run);
            if (bits > IMPOSSIBLE_D + 1.0f && !(bits + pf_margin(bits) <= bar)) {
                float x = bits;
                if (p.do_null3) {
                    const uint32_t n[4] = {c01 & 0xffffu, c01 >> 16, c23 & 0xffffu, c23 >> 16};
                    x = __fsub_rn(x, null3_approx(p, n, d));
                }
                const float m = pf_margin(x);
                hit = x + m >= p.cutoff && (run == -INFINITY || x + m > bar);
                if (x - m >= p.cutoff) run = fmaxf(run, x);
            }
        }
        emit_cand(p, c.lane, hit, c.item, c.j, d, raw);
    }
}

template <bool INS, bool KEY>
__global__ void __launch_bounds__(32 * DG_MAX_WARPS, 1) diag_kernel(const __grid_constant__ DgParams p) {
    typedef Sem<INS> S;
    typedef typename S::T T;
    __shared__ int s_item, s_err, s_prog[DG_MAX_WARPS];
    const int tid = threadIdx.x, nthreads = blockDim.x;
    DgCtx c;
    c.nw = nthreads >> 5;
    c.w = __shfl_sync(0xffffffffu, tid >> 5, 0);  // uniform over the warp
    c.lane = tid & 31;
    c.col = tid;
    c.reg = p.region + (int64_t)blockIdx.x * p.region_words;
    c.stg = dg_smem + (INS ? (p.ilog_nz + 8) / 8 * 4 : 0) + c.w * DG_STG;
    c.xch = dg_smem + (INS ? (p.ilog_nz + 8) / 8 * 4 : 0) + c.nw * DG_STG;
    uint8_t *ring = reinterpret_cast<uint8_t *>(c.xch + c.nw * DG_XCH * DG_CHUNK * 2);
    c.ring = ring;
    c.nz = p.ilog_nz;
    c.rmask = p.ring_len - 1;
    c.prog = (uint32_t)__cvta_generic_to_shared(s_prog);
    c.err = &s_err;
    if (tid == 0) s_err = 0;
    if (tid < DG_MAX_WARPS) s_prog[tid] = 0;
    c.step = c.prev = 0;
    if (INS)
        for (int x = tid; x <= p.ilog_nz; x += nthreads) reinterpret_cast<uint16_t *>(dg_smem)[x] = p.ilog[x];
    for (int x = tid; x < p.ring_len; x += nthreads) ring[x] = 0;
    const T NONE = dg_begin_none<S, KEY>();
    const int cols = c.nw * 32;
    for (;;) {
        if (tid == 0) s_item = s_err ? p.nitems : atomicAdd(p.next_item, 1);
        __syncthreads();
        const int it = s_item;
        if (it >= p.nitems) break;
        const WorkItem wi = p.items[it];
        c.item = p.item_base + it;
        c.jreport = wi.jreport;
        c.jend = wi.jend;
        c.ncols = wi.jend - wi.jstart + 1;
        const uint8_t *dsq = p.dsq + wi.dsq_off;
        c.step0 = c.prev = c.step;
        // steps of a group, the same for every warp
        c.gsteps = 0;
        for (int n = 0; n < p.nnodes; n++) {
            const int rows = min(p.nodes[n].rhi, c.ncols) - p.nodes[n].rlo + 1;
            if (rows > 0) c.gsteps += (rows + DG_CHUNK - 1) / DG_CHUNK;
        }
        c.slack = min(p.slack, c.gsteps);  // never two groups ahead
        for (int g0 = 0; g0 < c.ncols; g0 += cols) {
            if (p.stall && c.w < c.nw - 1) dg_wait(c, c.w + 1, c.step + p.stall);
            c.first = g0 == 0;
            c.last = g0 + cols >= c.ncols;
            c.jrel = g0 + c.col;
            c.j = wi.jstart + c.jrel;
            c.ridx = c.jrel % p.ring_cols;
            const int w0 = g0 + c.w * 32;  // the warp's first column
            c.jmax = w0 < c.ncols ? min(p.W, min(w0 + 32, c.ncols)) : 0;
            int r = c.jrel < c.ncols ? __ldg(dsq + c.j) : 0;  // (j of a later column may wrap)
            r = r > 17 ? 17 : r;
            ring[c.jrel & c.rmask] = (uint8_t)r;
            c.cj = r;
            __syncwarp();
            if (p.local && c.jmax > 0)
                for (int d = p.root_dn; d <= min(p.root_dxcap, c.jmax); d++)
                    S::st(c.reg + c.col + (int64_t)d * DG_COLS, NONE);
            // Before the first node, not only its first step: the node starts with
            // residues the warps on the left have written for this group, and
            // copies the begin row of every lane.
            dg_begin_step(c);
            for (int n = 0; n < p.nnodes; n++) {
                const DgNode *np = p.nodes + n;
                dg_begin_node(c);
                switch (np->type * 8 + np->nn) {
                case MATP_ND * 8 + 1: dg_node<S, KEY, MATP_ND, 1>(p, c, np); break;
                case MATP_ND * 8 + 2: dg_node<S, KEY, MATP_ND, 2>(p, c, np); break;
                case MATP_ND * 8 + 4: dg_node<S, KEY, MATP_ND, 4>(p, c, np); break;
                case MATL_ND * 8 + 1: dg_node<S, KEY, MATL_ND, 1>(p, c, np); break;
                case MATL_ND * 8 + 2: dg_node<S, KEY, MATL_ND, 2>(p, c, np); break;
                case MATL_ND * 8 + 4: dg_node<S, KEY, MATL_ND, 4>(p, c, np); break;
                case MATR_ND * 8 + 1: dg_node<S, KEY, MATR_ND, 1>(p, c, np); break;
                case MATR_ND * 8 + 2: dg_node<S, KEY, MATR_ND, 2>(p, c, np); break;
                case MATR_ND * 8 + 4: dg_node<S, KEY, MATR_ND, 4>(p, c, np); break;
                case BEGL_ND * 8 + 1: dg_node<S, KEY, BEGL_ND, 1>(p, c, np); break;
                case BEGL_ND * 8 + 2: dg_node<S, KEY, BEGL_ND, 2>(p, c, np); break;
                case BEGL_ND * 8 + 4: dg_node<S, KEY, BEGL_ND, 4>(p, c, np); break;
                case BEGR_ND * 8 + 1: dg_node<S, KEY, BEGR_ND, 1>(p, c, np); break;
                case BEGR_ND * 8 + 2: dg_node<S, KEY, BEGR_ND, 2>(p, c, np); break;
                case BEGR_ND * 8 + 4: dg_node<S, KEY, BEGR_ND, 4>(p, c, np); break;
                case ROOT_ND * 8 + 1: dg_node<S, KEY, ROOT_ND, 1>(p, c, np); break;
                case ROOT_ND * 8 + 2: dg_node<S, KEY, ROOT_ND, 2>(p, c, np); break;
                case ROOT_ND * 8 + 4: dg_node<S, KEY, ROOT_ND, 4>(p, c, np); break;
                default: dg_bif<S, KEY>(p, c, np); break;
                }
            }
            if (p.prefilter && c.jmax > 0) dg_prefilter<S>(p, c);
        }
        __syncthreads();
        if (tid == 0 && s_err) atomicExch(p.error, 1);
    }
}

static size_t dg_smem_bytes(const DgParams &p, int warps) {
    size_t b = (size_t)warps * (DG_XCH * DG_CHUNK * 2 + DG_STG) * 4 + (size_t)p.ring_len;
    if (p.inside) b += (size_t)((p.ilog_nz + 8) / 8) * 16;
    return b;
}

}  // namespace dev

int diag_occupancy(const DgParams &p, int warps) {
    int n = 0;
    const size_t smem = dev::dg_smem_bytes(p, warps);
    auto k = !p.inside ? dev::diag_kernel<false, false>
             : p.begin_key ? dev::diag_kernel<true, true> : dev::diag_kernel<true, false>;
    if (allow_max_dynamic_smem(k) != cudaSuccess) return 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, k, warps * 32, smem) != cudaSuccess) return 0;
    return n;
}

cudaError_t diag_launch(const DgParams &p, int ctas, int warps, cudaStream_t s) {
    auto k = !p.inside ? dev::diag_kernel<false, false>
             : p.begin_key ? dev::diag_kernel<true, true> : dev::diag_kernel<true, false>;
    cudaError_t e = allow_max_dynamic_smem(k);
    if (e != cudaSuccess) return e;
    k<<<ctas, warps * 32, dev::dg_smem_bytes(p, warps), s>>>(p);
    return cudaGetLastError();
}

}  // namespace cmx
