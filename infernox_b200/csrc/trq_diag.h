// Plan and launch interface of the truncated diagonal scan (trq_diag.cu).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

#include "../../include/cmscan_gpu.h"
#include "trunc_report.h"

namespace cmx {
namespace trqd {

constexpr int CHUNK = 16;                 // spans per phase
constexpr int MAX_WARPS = 8;              // warps per CTA
constexpr int COLS = 32 * MAX_WARPS;      // columns per group, at most
constexpr int PITCH = COLS + 32;          // one row of a node buffer: halo column at 31
constexpr int SLOTS = 12;                 // split states x planes J, L, R
constexpr int ROW = SLOTS * PITCH;        // words per span of a node buffer
constexpr int BND = SLOTS + 4;            // words per span of a node's saved last column

// One node, in the order the kernel runs them (last node first; END nodes
// are constants and have no entry).
struct Node {
    int32_t v0;
    int16_t type, nn, next_end, need_left;
    int16_t rhi;                  // longest span stored: its states' bands and what a parent reads
    int16_t buf;                  // node buffer 0..2
    int16_t deck;                 // BEGL / BEGR: bifurcation
    int16_t skip;                 // insert states that are never computed (detached): bit = state
    int16_t beginmask;            // states with a truncated begin
    int16_t endmask;              // states with a local end
    int16_t chi;                  // the next node's rhi
    int16_t dx[6];                // band 1..dx per state
    uint32_t base[4];             // d = 0 value of the split states (J plane)
    uint32_t cbase;               // ... of the END child (every plane)
    // BIF
    int16_t dx_w, dx_y;           // bands of BEGL_S and BEGR_S
    uint32_t begl_base;
};

struct Win {
    int64_t dsq_off;
    int32_t i0, j0, w, idx;  // idx: the window's index in the caller's batch
};

struct Res {
    float vsc;
    int32_t vmode;
    float bsc_full;
    int32_t pad;
};

struct Params {
    const Node *nodes;
    int nnodes, nbif;
    const uint32_t *tsc, *esc, *lm, *rm, *pty, *endsc, *el;  // semiring words
    int W, W1, dx0, ring_cols, ring_len;  // W1: rows of a buffer (longest window span + 1)
    int inside, fill_l, fill_r, fill_t, nonbanded;
    const uint16_t *ilog;
    int ilog_nz;
    const uint8_t *dsq;
    const Win *wins;
    int nwin;
    int *queue;
    uint32_t *region;
    int64_t region_words;
    float cutoff;
    hb::TrCand *cand;
    int64_t cap;
    unsigned long long *ncand;
    Res *res;
};

// words of one CTA's region for windows spanning at most W1 - 1
int64_t region_words(const Params &p);
int occupancy(const Params &p, int warps);
// phases a warp takes for one group of columns of a window spanning `span`
int64_t group_phases(const std::vector<Node> &nodes, int span);
cudaError_t launch(const Params &p, int ctas, int warps, cudaStream_t s);

// The nodes of a model for band caps dxcap (false: another node topology, or
// scores for which the kernel's maxima could differ from the reference's
// comparisons).  kind_skip[v]: states the scan never computes; esc_plain,
// esc_best: the emission table holds plain floats, its largest integer.
bool build(const cmgpu_cm *cm, bool inside, const std::vector<int32_t> &dxcap, const std::vector<char> &kind_skip,
           const std::vector<uint32_t> &pty, const std::vector<int32_t> &pbeg, const std::vector<uint32_t> &lm,
           const std::vector<uint32_t> &rm, const std::vector<uint32_t> &base, const std::vector<int> &begl_idx,
           bool esc_plain, int64_t esc_best, std::vector<Node> &out, int *nbif);

}  // namespace trqd
}  // namespace cmx
