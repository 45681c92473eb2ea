// Band selection and node shapes shared by the scan plans (qdb_plan.cpp,
// diag_plan.cpp).
#pragma once
#include <algorithm>
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

}  // namespace cmx
