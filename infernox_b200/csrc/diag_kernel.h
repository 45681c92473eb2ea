// Plan and launch interface of the diagonal scan kernel (diag_scan.cu).
//
// The kernel walks the CM node by node from the bottom up and, inside a node,
// span by span (d ascending); the lanes of a warp are consecutive columns j.
// It relies on the node topology every CM built by cm_from_guide has
// (src/cm_modelmaker.rs:979-1110), which build_diag_plan checks: a state's
// children are its node's own inserts followed by the split states of the
// next node, and a bifurcation's are BEGL_S and BEGR_S.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <string>
#include <vector>

#include "../../include/cmscan_gpu.h"
#include "qdb_kernel.h"
#include "qdb_plan.h"

namespace cmx {

constexpr int DG_CHUNK = 16;                        // spans per step
constexpr int DG_MAX_WARPS = 16;                    // warps per CTA
constexpr int DG_COLS = 32 * DG_MAX_WARPS;          // columns per group, at most
constexpr int DG_PITCH = DG_COLS + 32;              // one row of a node buffer: halo column at 31
constexpr int DG_SLOTS = 4;                         // split states of a node, at most
constexpr int DG_ROW = DG_SLOTS * DG_PITCH;         // words per span of a node buffer

constexpr int DG_XCH = 8;                           // steps a warp may be ahead of its right neighbour, at most
constexpr int DG_STAGE = 4;                         // spans staged at a time
// words staged per warp: two stages of four split states with a halo and the
// begin row (three or more where the next node has fewer split states)
constexpr int DG_STG = 2 * DG_STAGE * (4 * 36 + 32);

// One node, in the order the kernel runs them (last node first; END nodes
// are constants and have no entry).
struct DgNode {
    int32_t v0;
    int16_t type, nn;          // node type (cm_internal.h), split states of the next node
    int16_t next_end;          // the next node is END
    int16_t need_left;         // the parent node reads column j-1 of this node's split states
    int32_t rlo, rhi;          // spans stored: the states' bands and every span a parent reads
    int32_t clo, chi;          // the next node's rlo, rhi
    int32_t endmask, beginmask;  // states with a local end / a local begin (bit = state within the node)
    int32_t out_kind;          // DG_OUT_*
    int64_t out_off, in_off;   // words from the start of the CTA's region
    int64_t bnd_off;           // saved last column of the split states [span][4], then of the inserts [span][2]
    int16_t dn[6], dx[6];      // band per state
    uint32_t init0[6];         // d = 0 base value per state
    uint32_t cinit0;           // base value of the END child
    // BIF: the two decks (row d - lo) and the split range of generic_scan
    int32_t begl_lo, begr_lo, kdn_y, kdx_y, kdn_w, kdx_w;
    uint32_t begl_init0;
    int64_t begl_off, begr_off;
};

enum { DG_OUT_BUF = 0, DG_OUT_BEGL = 1, DG_OUT_BEGR = 2 };

struct DiagPlan {
    std::vector<DgNode> nodes;
    int R = 0;               // rows of a node buffer
    int ring_cols = 0;       // columns of a BEGL ring
    int64_t words = 0;       // words of one CTA's region
};

// false when the model is outside the kernel's scope (`why`): another node
// topology, a single node between ROOT and END, or (CYK) score tables
// holding -0, NaN or +inf, for which a floating maximum and the reference's
// comparison can differ.
bool build_diag_plan(const cmgpu_cm *cm, const Plan &p, int qdbidx, DiagPlan &dp, std::string *why);

struct DgParams {
    const DgNode *nodes;
    int nnodes;
    const uint32_t *tsc, *endsc, *esc, *el_sca, *bsv;
    int slack;                   // steps a warp may be ahead of its right neighbour
    int stall;                   // 0, or (test hook) steps more than the right neighbour will ever do
    int W, ring_cols, ring_len;  // ring_len: residues kept per CTA (power of two)
    int root_dn, root_dxcap;
    int inside, local, begin_key, prefilter, do_null3;
    float pf_null[4];
    float pf_omega;
    const uint16_t *ilog;
    int ilog_nz;
    const uint8_t *dsq;
    const WorkItem *items;
    int nitems, item_base;
    int *next_item, *error;
    Cand *cands;
    int cand_cap;
    int *cand_count;
    float cutoff;
    uint32_t *region;
    int64_t region_words;
};

// CTAs per SM that a launch of `warps` warps per CTA keeps resident
int diag_occupancy(const DgParams &p, int warps);
cudaError_t diag_launch(const DgParams &p, int ctas, int warps, cudaStream_t s);

}  // namespace cmx
