// Host plan of the diagonal scan kernel (diag_kernel.h).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "diag_kernel.h"
#include "plan_util.h"

namespace cmx {

namespace {

// A score a floating maximum treats as the reference's `a >= b ? a : b` does
// in every sum and comparison: not NaN, not +inf, not -0 (with none of these
// in the tables no sum yields one).
bool plain_float(uint32_t bits) {
    float f;
    std::memcpy(&f, &bits, 4);
    if (std::isnan(f) || (std::isinf(f) && f > 0)) return false;
    return !(f == 0.0f && std::signbit(f));
}

}  // namespace

bool build_diag_plan(const cmgpu_cm *cm, const Plan &p, int qdbidx, DiagPlan &dp, std::string *why) {
    auto fail = [&](const char *m) {
        if (why) *why = m;
        return false;
    };
    const int M = cm->M, W = cm->W;
    dp = DiagPlan();
    if (p.semiring != CMGPU_INSIDE_I32) {
        for (const auto *t : {&p.tsc, &p.endsc, &p.beginsc_all, &p.esc, &p.el_sca})
            for (uint32_t x : *t)
                if (!plain_float(x)) return fail("score tables hold -0, NaN or +inf");
    }
    // nodes from the unique state ids
    std::vector<NodeShape> shape;
    std::vector<int> v0s, node_of(M, -1);
    for (int v = 0; v < M;) {
        NodeShape ns;
        if (!node_shape(cm->stid[v], ns)) return fail("state list does not start a node where expected");
        if (v + ns.nst > M) return fail("truncated node");
        static const int TYPES[20] = {S_ST, IL_ST, IR_ST, S_ST, S_ST, IL_ST, MP_ST, ML_ST, MR_ST, D_ST,
                                      IL_ST, IR_ST, ML_ST, D_ST, IL_ST, MR_ST, D_ST, IR_ST, B_ST, E_ST};
        for (int q = 0; q < ns.nst; q++) {
            if (cm->stid[v + q] != ns.ids[q] || cm->sttype[v + q] != TYPES[ns.ids[q]])
                return fail("unexpected state inside a node");
            node_of[v + q] = (int)shape.size();
        }
        shape.push_back(ns);
        v0s.push_back(v);
        v += ns.nst;
    }
    const int nn = (int)shape.size();
    if (shape[0].type != ROOT_ND || shape[nn - 1].type != END_ND) return fail("first node is not ROOT or last not END");
    auto is_insert = [&](int v) { return cm->sttype[v] == IL_ST || cm->sttype[v] == IR_ST; };
    std::vector<int> bif_l(nn, -1), bif_r(nn, -1);  // BIF node -> BEGL / BEGR node
    std::vector<char> claimed(nn, 0);               // BEGL / BEGR nodes with their bifurcation
    for (int v = 0; v < M; v++) {
        const int st = cm->sttype[v], n = node_of[v];
        if (st == E_ST) continue;
        if (st == B_ST) {
            const int wl = cm->cfirst[v], y = cm->cnum[v];
            if (wl != v + 1 || cm->stid[wl] != UID_BEGL_S || y <= wl || y >= M || cm->stid[y] != UID_BEGR_S)
                return fail("bifurcation children are not BEGL_S / BEGR_S");
            bif_l[n] = node_of[wl];
            bif_r[n] = node_of[y];
            if (claimed[bif_l[n]] || claimed[bif_r[n]]) return fail("a subtree belongs to two bifurcations");
            claimed[bif_l[n]] = claimed[bif_r[n]] = 1;
            continue;
        }
        if (n + 1 >= nn) return fail("a non-END last node");
        if (shape[n + 1].type == BEGL_ND || shape[n + 1].type == BEGR_ND || shape[n + 1].type == ROOT_ND)
            return fail("a node is followed by a subtree start");
        const int v0 = v0s[n];
        int k = 0;
        bool ok = true;
        auto kid = [&](int u) { ok = ok && k < cm->cnum[v] && cm->cfirst[v] + k == u, k++; };
        for (int q = 0; q < shape[n].nst; q++)
            if (is_insert(v0 + q) && !(is_insert(v) && v0 + q < v)) kid(v0 + q);
        for (int q = 0; q < shape[n + 1].nsplit; q++) kid(v0s[n + 1] + q);
        if (!ok || k != cm->cnum[v]) return fail("children are not the node's inserts and the next node's split states");
    }
    for (int n = 0; n < nn; n++)
        if ((shape[n].type == BEGL_ND || shape[n].type == BEGR_ND) && !claimed[n])
            return fail("a subtree start without its bifurcation");
    // spans a node stores: its states' bands and every span a parent or a
    // bifurcation reads
    Bands b = select_bands(cm, qdbidx);
    std::vector<int> lo(nn, 1 << 30), hi(nn, -1);
    auto cover = [&](int n, int a, int c) {
        if (c < a) return;
        lo[n] = std::min(lo[n], a);
        hi[n] = std::max(hi[n], c);
    };
    for (int v = 0; v < M; v++) {
        const int st = cm->sttype[v], n = node_of[v];
        if (st == E_ST || b.dxcap[v] < b.dn[v]) continue;
        cover(n, b.dn[v], b.dxcap[v]);
        if (st == B_ST) {
            const int wl = cm->cfirst[v], y = cm->cnum[v];
            cover(bif_l[n], std::max(0, std::min(b.dmin[wl], W)), std::min(b.dmax[wl], W));
            cover(bif_r[n], std::max(0, std::min(b.dmin[y], W)), std::min(b.dmax[y], W));
        } else {
            const int sd = v == 0 ? 0 : state_delta(st);
            cover(n + 1, b.dn[v] - sd, b.dxcap[v] - sd);
        }
    }
    for (int n = 0; n < nn; n++) {
        if (hi[n] < lo[n]) lo[n] = 0, hi[n] = -1;
        if (lo[n] < 0) return fail("W too small");
        if (shape[n].type != END_ND) dp.R = std::max(dp.R, hi[n] - lo[n] + 1);
    }
    dp.R = std::max(dp.R, 1);
    // region: ROOT row of local begins, three node buffers (a node's outputs
    // stay until the warp to the right, one phase behind, has read them),
    // the bifurcations' decks, the saved last columns
    dp.ring_cols = (W + DG_COLS + 31) & ~31;
    int64_t off = (int64_t)(W + 1) * DG_COLS;
    const int64_t buf0 = off;
    off += 3 * (int64_t)dp.R * DG_ROW;
    std::vector<int64_t> deck(nn, 0);
    for (int n = 0; n < nn; n++) {
        const int64_t rows = hi[n] - lo[n] + 1;
        if (shape[n].type == BEGL_ND) {
            deck[n] = off;
            off += rows * dp.ring_cols;
        } else if (shape[n].type == BEGR_ND) {
            deck[n] = off;
            off += rows * DG_COLS;
        }
    }
    std::vector<int> buf(nn, 0);
    int t = 0;
    for (int n = nn - 1; n >= 0; n--) {
        if (shape[n].type == END_ND) continue;
        buf[n] = t++ % 3;
        DgNode d{};
        d.v0 = v0s[n];
        d.type = (int16_t)shape[n].type;
        d.nn = n + 1 < nn ? (int16_t)shape[n + 1].nsplit : 1;
        d.next_end = n + 1 < nn && shape[n + 1].type == END_ND;
        const int pt = n > 0 ? shape[n - 1].type : BIF_ND;
        const bool child_of_prev = n > 0 && shape[n].type != BEGL_ND && shape[n].type != BEGR_ND;
        d.need_left = child_of_prev && (pt == MATP_ND || pt == MATR_ND || pt == ROOT_ND);
        d.rlo = lo[n];
        d.rhi = hi[n];
        if (n + 1 < nn) d.clo = lo[n + 1], d.chi = hi[n + 1];
        d.out_kind = shape[n].type == BEGL_ND ? DG_OUT_BEGL : shape[n].type == BEGR_ND ? DG_OUT_BEGR : DG_OUT_BUF;
        d.out_off = d.out_kind == DG_OUT_BUF ? buf0 + buf[n] * (int64_t)dp.R * DG_ROW : deck[n];
        d.in_off = n + 1 < nn ? buf0 + buf[n + 1] * (int64_t)dp.R * DG_ROW : 0;
        d.bnd_off = off;
        off += (int64_t)(hi[n] - lo[n] + 1) * (DG_SLOTS + 2);
        for (int q = 0; q < shape[n].nst; q++) {
            const int v = v0s[n] + q;
            const StateDev &s = p.states[v];
            const bool live = s.dxcap >= s.dn;
            d.dn[q] = live ? s.dn : (int16_t)32767;
            d.dx[q] = live ? s.dxcap : (int16_t)-1;
            d.init0[q] = p.init0[v];
            if (s.flags & SF_ENDSC) d.endmask |= 1 << q;
            if (live && (s.flags & SF_BEGIN)) d.beginmask |= 1 << q;
        }
        if (d.next_end) d.cinit0 = p.init0[v0s[n + 1]];
        if (shape[n].type == BIF_ND) {
            const int wl = cm->cfirst[v0s[n]], y = cm->cnum[v0s[n]];
            d.begl_lo = lo[bif_l[n]];
            d.begr_lo = lo[bif_r[n]];
            d.begl_off = deck[bif_l[n]];
            d.begr_off = deck[bif_r[n]];
            d.kdn_y = std::min(b.dmin[y], W);
            d.kdx_y = std::min(b.dmax[y], W);
            d.kdn_w = std::min(b.dmin[wl], W);
            d.kdx_w = std::min(b.dmax[wl], W);
            d.begl_init0 = p.init0[wl];
        }
        dp.nodes.push_back(d);
    }
    dp.words = (off + 63) & ~(int64_t)63;
    return true;
}

}  // namespace cmx
