"""Host code that needs no GPU, compiled alone with the host's C++ compiler: the
replay of reportable cells (csrc/replay.h) -- the overlap rule against the
pairwise rule and within memory that follows the hits, exceptions of its
threads -- and the plan of the diagonal kernel (csrc/diag_plan.cpp)."""
import os
import subprocess

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "infernox_b200", "csrc")
CUDA = os.environ.get("CUDA_HOME", "/usr/local/cuda")

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


def run(tmp_path, name, source, files=()):
    src, exe = tmp_path / (name + ".cpp"), tmp_path / name
    src.write_text(source)
    subprocess.run(["g++", "-std=c++17", "-O1", "-pthread", "-I", CSRC, "-I", os.path.join(CUDA, "include"), "-o",
                    str(exe), str(src)] + [os.path.join(CSRC, f) for f in files], check=True)
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


PLAN = PRELUDE + r"""
#include "diag_kernel.h"
namespace cmx {
bool build_plan(const cmgpu_cm *cm, int semiring, int qdbidx, Plan &p);
void set_error(const std::string &) {}
}
// ROOT, `n` MATL nodes, END
struct Model {
    std::vector<int8_t> st{6, 4, 5}, id{0, 1, 2};
    std::vector<int32_t> cf, cn, lo, hi, it, ie, iv;
    std::vector<float> t, e, v;
    cmgpu_cm cm{};
    explicit Model(int n) {
        for (int k = 0; k < n; k++) {
            for (int8_t x : {2, 0, 4}) st.push_back(x);
            for (int8_t x : {12, 13, 14}) id.push_back(x);
        }
        st.push_back(7);
        id.push_back(19);
        const int M = (int)st.size();
        for (int s = 0; s < M; s++) {
            const int node0 = s < 3 ? 0 : s - (s - 3) % 3;               // first state of the node
            const int ins = s == 2 ? 2 : node0 == 0 ? 1 : node0 + 2;     // first insert it reaches
            const int next = node0 == 0 ? 3 : node0 + 3, split = next == M - 1 ? 1 : 2;
            cf.push_back(s == M - 1 ? -1 : ins);
            cn.push_back(s == M - 1 ? 0 : next - ins + split);
        }
        lo.assign(M, 1), hi.assign(M, 40);
        lo[M - 1] = hi[M - 1] = 0;
        t.assign(M * 6, -1.0f), e.assign(M * 324, 0.5f), v.assign(M, -1e36f);
        it.assign(M * 6, -1000), ie.assign(M * 324, 500), iv.assign(M, -987654321);
        cm.M = M, cm.W = 40;
        cm.sttype = st.data(), cm.stid = id.data(), cm.cfirst = cf.data(), cm.cnum = cn.data();
        cm.tsc = t.data(), cm.oesc = e.data(), cm.endsc = cm.beginsc = v.data(), cm.el_selfsc = -0.1f;
        cm.itsc = it.data(), cm.ioesc = ie.data(), cm.iendsc = cm.ibeginsc = iv.data(), cm.iel_selfsc = -100;
        cm.dmin1 = cm.dmin2 = lo.data(), cm.dmax1 = cm.dmax2 = hi.data();
    }
};

int main() {
    for (int n = 1; n <= 14; n++)
        for (int semiring : {0, 1}) {
            Model m(n);
            cmx::Plan p;
            cmx::DiagPlan d;
            std::string why;
            assert(cmx::build_plan(&m.cm, semiring, 1, p));
            const bool ok = cmx::build_diag_plan(&m.cm, p, 1, d, &why);
            if (n < 2) {
                assert(!ok);
                continue;
            }
            if (!ok) return std::printf("%d nodes: %s\n", n, why.c_str()), 1;
            // While a warp writes node k's buffer the one on its right may be in
            // node k - 1 (it has finished those before), the ROOT of the group
            // before for the first node.  It reads that node's child and writes
            // the node's own buffer.
            const int N = (int)d.nodes.size();
            assert(N == n + 1);
            for (int k = 0; k < N - 1; k++) {  // ROOT, the last one, writes no buffer
                const cmx::DgNode &w = d.nodes[k], &r = d.nodes[(k + N - 1) % N];
                const int64_t size = (int64_t)d.R * cmx::DG_ROW;
                auto apart = [&](int64_t a, int64_t b) { return a + size <= b || b + size <= a; };
                assert(w.out_off + size <= d.words);
                if (!r.next_end && !apart(w.out_off, r.in_off)) return std::printf("%d nodes: node %d\n", n, k), 1;
                if (k > 0 && !apart(w.out_off, r.out_off)) return std::printf("%d nodes: node %d, own\n", n, k), 1;
            }
        }
    return 0;
}
"""


def test_node_buffers_of_the_diagonal_plan(tmp_path):
    r = run(tmp_path, "plan", PLAN, ["diag_plan.cpp", "qdb_plan.cpp"])
    assert r.returncode == 0, r.stdout + r.stderr
