"""The host-side replay of reportable cells (csrc/replay.h), compiled alone with
the host's C++ compiler: the overlap rule against the pairwise rule and within
memory that follows the hits."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infernox_b200", "csrc")

PRELUDE = r"""
#include <cassert>
#include <cstdio>
#include <cstdlib>
#include <new>
#include <random>
#include "replay.h"
struct Hit { int32_t i, j; float score, bias; };
"""

OVERLAPS = PRELUDE + r"""
static size_t held = 0, peak = 0;
void *operator new(size_t n) {
    size_t *p = (size_t *)std::malloc(n + 16);
    if (!p) throw std::bad_alloc();
    *p = n;
    held += n;
    if (held > peak) peak = held;
    return (char *)p + 16;
}
void operator delete(void *p) noexcept {
    if (!p) return;
    held -= *(size_t *)((char *)p - 16);
    std::free((char *)p - 16);
}
void operator delete(void *p, size_t) noexcept { operator delete(p); }

// the reference's pairwise rule
static std::vector<Hit> pairwise(std::vector<Hit> h) {
    std::stable_sort(h.begin(), h.end(), [](const Hit &a, const Hit &b) {
        return a.score != b.score ? a.score > b.score : a.i < b.i;
    });
    std::vector<Hit> out;
    for (const Hit &x : h) {
        bool clear = true;
        for (const Hit &y : out) clear = clear && (x.j < y.i || y.j < x.i);
        if (clear) out.push_back(x);
    }
    return out;
}

int main() {
    std::mt19937 rng(5);
    for (int32_t n : {0, 1, 2, 3, 50, 700, 5000, 20000})
        for (int32_t span : {1, 30, 2000, 40000, 3000000}) {
            std::vector<Hit> h;
            for (int32_t k = 0; k < n; k++) {
                const int32_t i = 7 + (int32_t)(rng() % span), len = 1 + (int32_t)(rng() % 150);
                h.push_back(Hit{i, i + len - 1, (float)(rng() % 60), (float)k});
            }
            const std::vector<Hit> want = pairwise(h);
            const size_t before = held;
            peak = held;
            cmx::remove_overlaps(h);
            // a few hundred bytes per hit, and a few kB
            if (peak - before > 400 * (size_t)n + 16384) return std::printf("%d %d: %zu bytes\n", n, span, peak - before), 1;
            assert(h.size() == want.size());
            for (size_t k = 0; k < h.size(); k++)
                assert(h[k].i == want[k].i && h[k].j == want[k].j && h[k].bias == want[k].bias);
        }
    std::vector<Hit> far = {{1, 90, 3.0f, 0}, {249999900, 250000000, 4.0f, 1}, {50, 200, 3.5f, 2}};
    peak = held;
    const size_t before = held;
    cmx::remove_overlaps(far);
    assert(far.size() == 2 && far[0].bias == 1 && far[1].bias == 2);
    if (peak - before > 16384) return std::printf("two ends of a window: %zu bytes\n", peak - before), 1;
    return 0;
}
"""


def run(tmp_path, name, source):
    src, exe = tmp_path / (name + ".cpp"), tmp_path / name
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-o", str(exe), str(src)], check=True)
    return subprocess.run([str(exe)], capture_output=True, text=True, timeout=120)


def test_overlap_rule_and_its_memory(tmp_path):
    r = run(tmp_path, "overlaps", OVERLAPS)
    assert r.returncode == 0, r.stdout + r.stderr


THROWS = PRELUDE + r"""
int main() {
    for (int bad : {0, 57, 199}) {
        std::atomic<int> ran{0};
        bool caught = false;
        try {
            cmx::on_cores(200, 200, 1, [&](size_t k) {
                ran++;
                if ((int)k == bad) throw std::bad_alloc();
            });
        } catch (const std::bad_alloc &) {
            caught = true;
        }
        assert(caught && ran > bad);
    }
    std::atomic<int> ran{0};
    cmx::on_cores(1000, 1000, 1, [&](size_t) { ran++; });
    assert(ran == 1000);
    return 0;
}
"""


def test_what_an_item_throws_reaches_the_caller(tmp_path):
    r = run(tmp_path, "throws", THROWS)
    assert r.returncode == 0, r.stdout + r.stderr


FITS = PRELUDE + r"""
#include "plan_util.h"
int main() {
    // the calls made for a limit, and what was had
    auto tries = [](size_t most, size_t least, size_t limit) {
        std::vector<size_t> seen;
        const size_t got = cmx::most_that_fit(most, least, [&](size_t n) {
            seen.push_back(n);
            return n <= limit;
        });
        seen.push_back(got);
        return seen;
    };
    assert((tries(296, 1, 1000) == std::vector<size_t>{296, 296}));
    assert((tries(296, 1, 100) == std::vector<size_t>{296, 148, 74, 74}));
    assert((tries(5, 1, 1) == std::vector<size_t>{5, 2, 1, 1}));
    assert((tries(5, 1, 0) == std::vector<size_t>{5, 2, 1, 0}));
    assert((tries(1, 1, 0) == std::vector<size_t>{1, 0}));
    assert((tries(90, 40, 39) == std::vector<size_t>{90, 45, 40, 0}));
    assert((tries(30, 40, 40) == std::vector<size_t>{40, 40}));
    return 0;
}
"""


def test_scratch_that_fits(tmp_path):
    r = run(tmp_path, "fits", FITS)
    assert r.returncode == 0, r.stdout + r.stderr
