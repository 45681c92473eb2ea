// Host-side replay of the reportable cells of a batch: the kernels append
// them in any order, the reference's greedy report wants each window's in
// (j, d) order.
#pragma once
#include <algorithm>
#include <atomic>
#include <cstddef>
#include <cstdint>
#include <exception>
#include <iterator>
#include <map>
#include <thread>
#include <vector>

namespace cmx {

// Runs f(0) .. f(n - 1) on up to one thread per `grain` units of work, at
// most the host's cores; the items are taken in order.  What an item throws
// reaches the caller once every thread has stopped (the first one thrown; the
// items not begun by then are left out).
template <class F>
void on_cores(size_t n, size_t work, size_t grain, F f) {
    const size_t nthr = std::min<size_t>({n, (size_t)std::max(1u, std::thread::hardware_concurrency()),
                                          work / std::max<size_t>(grain, 1) + 1});
    if (nthr <= 1) {
        for (size_t k = 0; k < n; k++) f(k);
        return;
    }
    std::atomic<size_t> next{0};
    std::atomic<bool> failed{false};
    std::exception_ptr thrown;
    auto run = [&]() {
        try {
            for (size_t k; (k = next.fetch_add(1)) < n;) f(k);
        } catch (...) {
            next.store(n);
            if (!failed.exchange(true)) thrown = std::current_exception();
        }
    };
    std::vector<std::thread> pool;
    pool.reserve(nthr);
    try {
        for (size_t t = 1; t < nthr; t++) pool.emplace_back(run);
    } catch (const std::exception &) {
        // no more threads to be had: those there are, and this one, do the work
    }
    run();
    for (auto &th : pool) th.join();
    if (thrown) std::rethrow_exception(thrown);
}

// Cells c[0..n) of windows 0..nwin-1 (field env) -> `out` ordered by (window,
// j, d); first[w] is window w's first cell.  Then report(w, cells, count) for
// every window, several at a time.  One counting sort by window and a small
// sort per window: a single sort of a few hundred thousand cells took longer
// than the scan that found them.
template <class C, class F>
void replay_cells(const C *c, size_t n, size_t nwin, std::vector<C> &out, F report) {
    std::vector<size_t> first(nwin + 1, 0);
    for (size_t k = 0; k < n; k++) first[(size_t)c[k].env + 1]++;
    for (size_t w = 0; w < nwin; w++) first[w + 1] += first[w];
    out.resize(n);
    {
        std::vector<size_t> at(first.begin(), first.end() - 1);
        for (size_t k = 0; k < n; k++) out[at[(size_t)c[k].env]++] = c[k];
    }
    on_cores(nwin, n, 4096, [&](size_t w) {
        C *f = out.data() + first[w], *l = out.data() + first[w + 1];
        std::sort(f, l, [](const C &a, const C &b) { return a.j != b.j ? a.j < b.j : a.d < b.d; });
        report(w, f, (size_t)(l - f));
    });
}

// remove_overlaps_greedy (src/cp9.rs:6544-6574, src/cm_dpsearch_trunc.rs:2470):
// hits by score (descending, stable) then start; a hit is removed when it
// overlaps an earlier hit that was kept.  The kept hits are disjoint.
//
// Lists with a hit per 32 residues or more (150,000 hits of one window: 19 ms
// when they were all sorted): most hits overlap one of the best ones, so only
// the best part is sorted, and what overlaps the hits kept so far is dropped
// before the next part is; a count of covered residues tells an overlap.  That
// takes five bytes per residue between the first and the last hit, so lists
// with fewer hits are sorted whole, and the kept hit with the largest start
// <= j is looked up in a map: memory follows the hits in both.
template <class H>
void remove_overlaps(std::vector<H> &h) {
    if (h.size() < 2) return;
    auto lo = h[0].i, hi = h[0].j;
    for (const H &x : h) {
        lo = std::min(lo, std::min(x.i, x.j));
        hi = std::max(hi, std::max(x.i, x.j));
    }
    if ((size_t)(hi - lo) / 32 > h.size()) {
        std::stable_sort(h.begin(), h.end(), [](const H &a, const H &b) {
            return a.score != b.score ? a.score > b.score : a.i < b.i;
        });
        std::map<decltype(lo), decltype(lo)> kept;  // start -> end
        size_t o = 0;
        for (size_t k = 0; k < h.size(); k++) {
            const auto it = kept.upper_bound(h[k].j);
            if (it != kept.begin() && std::prev(it)->second >= h[k].i) continue;
            kept.emplace(h[k].i, h[k].j);
            h[o++] = h[k];
        }
        h.resize(o);
        return;
    }
    std::vector<char> mark((size_t)(hi - lo + 1), 0);
    std::vector<int32_t> upto((size_t)(hi - lo + 2), 0);  // covered residues before lo + x
    std::vector<uint32_t> rest(h.size());
    for (size_t k = 0; k < rest.size(); k++) rest[k] = (uint32_t)k;
    auto before = [&](uint32_t a, uint32_t b) {
        if (h[a].score != h[b].score) return h[a].score > h[b].score;
        if (h[a].i != h[b].i) return h[a].i < h[b].i;
        return a < b;
    };
    std::vector<H> kept;
    while (!rest.empty()) {
        const size_t part = rest.size() <= 4096 ? rest.size() : std::max<size_t>(2048, rest.size() / 16);
        if (part < rest.size()) std::nth_element(rest.begin(), rest.begin() + (long)part, rest.end(), before);
        std::sort(rest.begin(), rest.begin() + (long)part, before);
        for (size_t k = 0; k < part; k++) {
            const H &x = h[rest[k]];
            bool free_ = true;
            for (auto p = x.i; p <= x.j && free_; p++) free_ = !mark[(size_t)(p - lo)];
            if (!free_) continue;
            for (auto p = x.i; p <= x.j; p++) mark[(size_t)(p - lo)] = 1;
            kept.push_back(x);
        }
        if (part == rest.size()) break;
        for (size_t p = 0; p + 1 < upto.size(); p++) upto[p + 1] = upto[p] + mark[p];
        size_t o = 0;
        for (size_t k = part; k < rest.size(); k++) {
            const H &x = h[rest[k]];
            if (upto[(size_t)(x.j - lo) + 1] == upto[(size_t)(x.i - lo)]) rest[o++] = rest[k];
        }
        rest.resize(o);
    }
    h.swap(kept);
}

}  // namespace cmx
