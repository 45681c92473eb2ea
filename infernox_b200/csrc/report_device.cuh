// Device-side reporting shared by the QDB scan kernels: appending reportable
// cells to the candidate buffer, and the approximate null3 correction of the
// report pre-filter.  P is the kernel's parameter block (cands, cand_cap,
// cand_count, pf_null, pf_omega).
#pragma once
#include <cuda_runtime.h>
#include <cstdint>

#include "qdb_kernel.h"
#include "semiring.cuh"

namespace cmx {
namespace dev {

// Appends the cells of the warp's lanes with hit set to the candidate buffer
// (one atomic per warp); entries past cand_cap are counted, not written.
template <class P>
__device__ __forceinline__ void emit_cand(const P &p, int wl, bool hit, int item, int j, int d,
                                          uint32_t raw) {
    const unsigned m = __ballot_sync(0xffffffffu, hit);
    if (!m) return;
    const int leader = __ffs(m) - 1;
    int base = 0;
    if (wl == leader) base = atomicAdd(p.cand_count, __popc(m));
    base = __shfl_sync(0xffffffffu, base, leader);
    if (hit) {
        const int pos = base + __popc(m & ((1u << wl) - 1));
        if (pos < p.cand_cap) {
            Cand cd;
            cd.item = item;
            cd.j = j;
            cd.d = d;
            cd.raw = raw;
            p.cands[pos] = cd;
        }
    }
}

// Null3 correction of a hit of length len with residue counts n[4]
// (score_correction_null3, src/cp9.rs:6516-6528), computed as the host does
// but with the device's log and, for the final FLogsum(0, x), the exact
// log2(1 + 2^-x) instead of the 0.001-step table: used only to decide which
// cells the host must look at, within a margin that covers both differences.
template <class P>
__device__ float null3_approx(const P &p, const uint32_t *n, int len) {
    float comp[4], sum = 0.0f;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        comp[a] = (float)n[a];
        sum = __fadd_rn(sum, comp[a]);
    }
#pragma unroll
    for (int a = 0; a < 4; a++) comp[a] = sum > 0.0f ? __fdiv_rn(comp[a], sum) : 0.25f;
    float score = 0.0f;
#pragma unroll
    for (int a = 0; a < 4; a++) {
        const double q = (double)__fdiv_rn(comp[a], p.pf_null[a]);
        const double t = (q > 0.0 ? log(q) * 1.44269504 : -1.0e36) * (double)comp[a] * (double)len;
        score = (float)((double)score + t);
    }
    const double om = (double)p.pf_omega;
    score = (float)((double)score + (om > 0.0 ? log(om) * 1.44269504 : -1.0e36));
    const float mx = fmaxf(0.0f, score), mn = fminf(0.0f, score);
    if (mx - mn >= 23.0f) return mx;
    return mx + (float)log2(1.0 + exp2(-(double)(mx - mn)));
}

// Margin of an approximate corrected score: FLogsum's table step (<= 5e-4
// bits) plus the double-precision log differences (relative ~1e-15) plus
// f32 rounding of the sums (a few ulps of |x|), with room to spare.
__device__ __forceinline__ float pf_margin(float x) { return 2.0e-3f + 1.0e-5f * fabsf(x); }

}  // namespace dev
}  // namespace cmx
