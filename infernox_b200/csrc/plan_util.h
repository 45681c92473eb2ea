// Band selection and node shapes shared by the scan plans (qdb_plan.cpp,
// diag_plan.cpp).
#pragma once
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include "../../include/cmscan_gpu.h"
#include "cm_internal.h"

namespace cmx {

struct Bands {
    std::vector<int32_t> dmin, dmax, dn, dxcap;
};

// dn/dxcap as generic_scan selects them (src/cm_nohmm.rs:431-456)
inline Bands select_bands(const cmgpu_cm *cm, int qdbidx) {
    Bands b;
    const int M = cm->M, W = cm->W;
    b.dmin.resize(M);
    b.dmax.resize(M);
    b.dn.resize(M);
    b.dxcap.resize(M);
    for (int v = 0; v < M; v++) {
        if (qdbidx == CMGPU_NOQDB) {
            b.dmin[v] = 0;
            b.dmax[v] = W;
        } else if (qdbidx == CMGPU_QDB1) {
            b.dmin[v] = cm->dmin1[v];
            b.dmax[v] = cm->dmax1[v];
        } else {
            b.dmin[v] = cm->dmin2[v];
            b.dmax[v] = cm->dmax2[v];
        }
        int base = cm->sttype[v] == MP_ST ? 2 : 1;
        int dn = std::max(b.dmin[v], base);
        if (dn > W) dn = W;
        b.dn[v] = dn;
        b.dxcap[v] = std::min(b.dmax[v], W);
    }
    return b;
}

// unique state ids (src/constants.rs:46-81)
enum {
    UID_ROOT_S = 0, UID_ROOT_IL, UID_ROOT_IR, UID_BEGL_S, UID_BEGR_S, UID_BEGR_IL, UID_MATP_MP, UID_MATP_ML,
    UID_MATP_MR, UID_MATP_D, UID_MATP_IL, UID_MATP_IR, UID_MATL_ML, UID_MATL_D, UID_MATL_IL, UID_MATR_MR,
    UID_MATR_D, UID_MATR_IR, UID_BIF_B, UID_END_E
};

struct NodeShape {
    int type, nst, nsplit;  // node type, states, split (non-insert) states
    int ids[6];             // unique state ids in state order
};

// The node a state id starts, with its state list (src/cm_modelmaker.rs:979-1110).
inline bool node_shape(int first_id, NodeShape &ns) {
    switch (first_id) {
    case UID_ROOT_S: ns = {ROOT_ND, 3, 1, {UID_ROOT_S, UID_ROOT_IL, UID_ROOT_IR}}; return true;
    case UID_BEGL_S: ns = {BEGL_ND, 1, 1, {UID_BEGL_S}}; return true;
    case UID_BEGR_S: ns = {BEGR_ND, 2, 1, {UID_BEGR_S, UID_BEGR_IL}}; return true;
    case UID_MATP_MP:
        ns = {MATP_ND, 6, 4, {UID_MATP_MP, UID_MATP_ML, UID_MATP_MR, UID_MATP_D, UID_MATP_IL, UID_MATP_IR}};
        return true;
    case UID_MATL_ML: ns = {MATL_ND, 3, 2, {UID_MATL_ML, UID_MATL_D, UID_MATL_IL}}; return true;
    case UID_MATR_MR: ns = {MATR_ND, 3, 2, {UID_MATR_MR, UID_MATR_D, UID_MATR_IR}}; return true;
    case UID_BIF_B: ns = {BIF_ND, 1, 1, {UID_BIF_B}}; return true;
    case UID_END_E: ns = {END_ND, 1, 1, {UID_END_E}}; return true;
    default: return false;
    }
}

// One node of a CM with cm_from_guide's topology.
struct NodeTopo {
    int v0, type, nst, nsplit;
    int begl = -1, begr = -1;  // BIF: the nodes of its two subtrees
    bool need_left = false;    // the parent node reads column j-1 of the split states
};

// The nodes of `cm` in order, if a state's children are its node's own
// inserts followed by the next node's split states, and a bifurcation's are
// BEGL_S and BEGR_S; else false with the reason in `why`.
inline bool node_topology(const cmgpu_cm *cm, std::vector<NodeTopo> &out, const char **why) {
    auto fail = [&](const char *m) {
        if (why) *why = m;
        return false;
    };
    const int M = cm->M;
    std::vector<NodeShape> shape;
    std::vector<int> node_of(M, -1);
    out.clear();
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
        NodeTopo t;
        t.v0 = v;
        t.type = ns.type;
        t.nst = ns.nst;
        t.nsplit = ns.nsplit;
        out.push_back(t);
        v += ns.nst;
    }
    const int nn = (int)shape.size();
    if (nn < 2 || shape[0].type != ROOT_ND || shape[nn - 1].type != END_ND)
        return fail("first node is not ROOT or last not END");
    auto is_insert = [&](int v) { return cm->sttype[v] == IL_ST || cm->sttype[v] == IR_ST; };
    std::vector<char> claimed(nn, 0);  // BEGL / BEGR nodes with their bifurcation
    for (int v = 0; v < M; v++) {
        const int st = cm->sttype[v], n = node_of[v];
        if (st == E_ST) continue;
        if (st == B_ST) {
            const int wl = cm->cfirst[v], y = cm->cnum[v];
            if (wl != v + 1 || cm->stid[wl] != UID_BEGL_S || y <= wl || y >= M || cm->stid[y] != UID_BEGR_S)
                return fail("bifurcation children are not BEGL_S / BEGR_S");
            out[n].begl = node_of[wl];
            out[n].begr = node_of[y];
            if (claimed[out[n].begl] || claimed[out[n].begr]) return fail("a subtree belongs to two bifurcations");
            claimed[out[n].begl] = claimed[out[n].begr] = 1;
            continue;
        }
        if (n + 1 >= nn) return fail("a non-END last node");
        if (shape[n + 1].type == BEGL_ND || shape[n + 1].type == BEGR_ND || shape[n + 1].type == ROOT_ND)
            return fail("a node is followed by a subtree start");
        const int v0 = out[n].v0;
        int k = 0;
        bool ok = true;
        auto kid = [&](int u) { ok = ok && k < cm->cnum[v] && cm->cfirst[v] + k == u, k++; };
        for (int q = 0; q < shape[n].nst; q++)
            if (is_insert(v0 + q) && !(is_insert(v) && v0 + q < v)) kid(v0 + q);
        for (int q = 0; q < shape[n + 1].nsplit; q++) kid(out[n + 1].v0 + q);
        if (!ok || k != cm->cnum[v])
            return fail("children are not the node's inserts and the next node's split states");
        if (cm->sttype[v] != S_ST || n == 0) {
            const int pt = shape[n].type;
            if (pt == MATP_ND || pt == MATR_ND || pt == ROOT_ND) out[n + 1].need_left = true;
        }
    }
    for (int n = 0; n < nn; n++)
        if ((shape[n].type == BEGL_ND || shape[n].type == BEGR_ND) && !claimed[n])
            return fail("a subtree start without its bifurcation");
    return true;
}

// The largest of `most`, its halves and `least` that get() says it has had
// (0: not even the least).  Scratch is sized by the free memory, which another
// caller may take in between.
template <class F>
size_t most_that_fit(size_t most, size_t least, F get) {
    for (size_t n = std::max(most, least);;) {
        if (get(n)) return n;
        if (n <= least) return 0;
        n = std::max(n / 2, least);
    }
}

// A score a floating maximum treats as the reference's `a >= b ? a : b` does
// in every sum and comparison: not NaN, not +inf, not -0 (with none of these
// in the tables no sum yields one).
inline bool plain_float(float f) {
    if (std::isnan(f) || (std::isinf(f) && f > 0)) return false;
    return !(f == 0.0f && std::signbit(f));
}

}  // namespace cmx
