// Host plan of the diagonal scan kernel (diag_kernel.h).
#include <algorithm>
#include <cmath>
#include <cstring>

#include "diag_kernel.h"
#include "plan_util.h"

namespace cmx {

bool build_diag_plan(const cmgpu_cm *cm, const Plan &p, int qdbidx, DiagPlan &dp, std::string *why) {
    auto fail = [&](const char *m) {
        if (why) *why = m;
        return false;
    };
    const int M = cm->M, W = cm->W;
    dp = DiagPlan();
    if (p.semiring != CMGPU_INSIDE_I32) {
        for (const auto *t : {&p.tsc, &p.endsc, &p.beginsc_all, &p.esc, &p.el_sca})
            for (uint32_t x : *t) {
                float f;
                std::memcpy(&f, &x, 4);
                if (!plain_float(f)) return fail("score tables hold -0, NaN or +inf");
            }
    }
    std::vector<NodeTopo> shape;
    const char *msg = nullptr;
    if (!node_topology(cm, shape, &msg)) return fail(msg);
    const int nn = (int)shape.size();
    std::vector<int> node_of(M, 0);
    for (int n = 0; n < nn; n++)
        for (int q = 0; q < shape[n].nst; q++) node_of[shape[n].v0 + q] = n;
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
            cover(shape[n].begl, std::max(0, std::min(b.dmin[wl], W)), std::min(b.dmax[wl], W));
            cover(shape[n].begr, std::max(0, std::min(b.dmin[y], W)), std::min(b.dmax[y], W));
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
    // the bifurcations' decks, the saved last columns.  A warp begins a group's
    // first node while the one on its right may be in the group before's ROOT,
    // which reads buffer (nodes - 2) % 3: where that is the first one, the first
    // node has a fourth to itself.  (With two nodes ROOT reads that very node.)
    dp.ring_cols = (W + DG_COLS + 31) & ~31;
    int64_t off = (int64_t)(W + 1) * DG_COLS;
    const int64_t buf0 = off;
    int owners = 0;
    for (const NodeTopo &t : shape) owners += t.type != END_ND;
    if (owners < 3) return fail("fewer than three nodes with states of their own");
    const bool fourth = (owners - 2) % 3 == 0;
    off += (fourth ? 4 : 3) * (int64_t)dp.R * DG_ROW;
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
        buf[n] = fourth && t == 0 ? 3 : t % 3;
        t++;
        DgNode d{};
        d.v0 = shape[n].v0;
        d.type = (int16_t)shape[n].type;
        d.nn = n + 1 < nn ? (int16_t)shape[n + 1].nsplit : 1;
        d.next_end = n + 1 < nn && shape[n + 1].type == END_ND;
        d.need_left = shape[n].need_left;
        d.rlo = lo[n];
        d.rhi = hi[n];
        if (n + 1 < nn) d.clo = lo[n + 1], d.chi = hi[n + 1];
        d.out_kind = shape[n].type == BEGL_ND ? DG_OUT_BEGL : shape[n].type == BEGR_ND ? DG_OUT_BEGR : DG_OUT_BUF;
        d.out_off = d.out_kind == DG_OUT_BUF ? buf0 + buf[n] * (int64_t)dp.R * DG_ROW : deck[n];
        d.in_off = n + 1 < nn ? buf0 + buf[n + 1] * (int64_t)dp.R * DG_ROW : 0;
        d.bnd_off = off;
        off += (int64_t)(hi[n] - lo[n] + 1) * (DG_SLOTS + 2);
        for (int q = 0; q < shape[n].nst; q++) {
            const int v = shape[n].v0 + q;
            const StateDev &s = p.states[v];
            const bool live = s.dxcap >= s.dn;
            d.dn[q] = live ? s.dn : (int16_t)32767;
            d.dx[q] = live ? s.dxcap : (int16_t)-1;
            d.init0[q] = p.init0[v];
            if (s.flags & SF_ENDSC) d.endmask |= 1 << q;
            if (live && (s.flags & SF_BEGIN)) d.beginmask |= 1 << q;
        }
        if (d.next_end) d.cinit0 = p.init0[shape[n + 1].v0];
        if (shape[n].type == BIF_ND) {
            const int wl = cm->cfirst[d.v0], y = cm->cnum[d.v0];
            d.begl_lo = lo[shape[n].begl];
            d.begr_lo = lo[shape[n].begr];
            d.begl_off = deck[shape[n].begl];
            d.begr_off = deck[shape[n].begr];
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
