"""Plans of the GEMM on CTA pairs (csrc/awq_pair_plan.cuh), built for the host: the pieces that a plan's pairs walk are every
(column tile, unit of 32 token rows) exactly once, and the parts of K that its pairs multiply are all of K."""
import os
import subprocess

import pytest

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "mlir_air_b200", "csrc")

SOURCE = r"""
#include <cstdio>
#include <cstdlib>
#include <initializer_list>
#include <vector>
#include "awq_pair_plan.cuh"
using namespace awq;

static std::vector<int> at;  // length of the piece that starts at a unit
static bool partition(const PairPlan &pl) {
    const int all = pl.R * pl.C;
    at.assign(all + 1, 0);
    long long pieces = 0, seen = 0;
    for (int p = 0; p < pl.P; ++p) {
        PairWalk w(p, pl);
        while (w.next()) {
            if (w.tile < 0 || w.tile >= pl.C || w.unit < 0 || w.units < 1 || w.units > pl.max_units || w.unit + w.units > pl.R) return false;
            int &len = at[w.tile * pl.R + w.unit];
            if (len) return false;
            len = w.units;
            ++pieces;
        }
    }
    for (int u = 0; u < all; u += at[u], ++seen)
        if (!at[u]) return false;
    return seen == pieces;
}
static bool covers_k(const PairPlan &pl, int K) {  // as the kernel cuts it: pairs of k-blocks, none of the parts empty
    const int KB2 = (K + 2 * GP_BK - 1) / (2 * GP_BK);
    for (int s = 0; s < pl.S; ++s)
        if ((s + 1) * KB2 / pl.S <= s * KB2 / pl.S) return false;
    return true;
}
static long long n_plans = 0;
static void check(bool w4, int M, int N, int K, int pairs, bool split, const PairPlan &pl, const char *what) {
    ++n_plans;
    if (pl.P >= 1 && pl.P * pl.S <= pairs && pl.S >= 1 && pl.S <= GP_MAX_PARTS && pl.max_units <= GP_MAX_UNITS &&
        (!w4 || pl.sets == 1 || pl.max_units <= GP_MAX_UNITS / 2) && covers_k(pl, K) && partition(pl))
        return;
    std::printf("%s plan of %s weights, M %d K %d N %d, %d pairs, parts %d: P %d R %d C %d units %d waves %d NT %d base %d snap %d S %d\n", what,
                w4 ? "int4" : "bf16", M, K, N, pairs, split, pl.P, pl.R, pl.C, pl.max_units, pl.waves, pl.NT, pl.base, pl.snap, pl.S);
    std::exit(1);
}

int main(int argc, char **argv) {
    const int w4_kind = std::atoi(argv[1]), C_first = std::atoi(argv[2]), C_step = std::atoi(argv[3]);
    const bool w4 = w4_kind != 0;
    // the plan that is chosen
    for (int C = C_first; C <= 400; C += C_step)
        for (int R = 1; R <= 200; ++R)
            for (int K : {512, 4096, 14336})
                for (int split = 0; split < (R * C < 600 ? 2 : 1); ++split) {  // (parts: fewer than two tiles for a pair)
                    const int M = 32 * R - (C * 7 + R * 3) % 32, N = 256 * C - (C * 5 + R) % 8 * 32;
                    check(w4, M, N, K, 74, split, pair_search(w4, M, N, K, 74, split), "chosen");
                }
    // every plan that is considered, on chips of several sizes
    for (int C = C_first; C <= 120; C += 3 * C_step)
        for (int R = 1; R <= 70; R += R < 24 ? 1 : 5)
            for (int pairs = 60; pairs <= 80; pairs += 1 + C % 3)
            {
                auto consider = [&](const PairPlan &pl) { check(w4, 32 * R, 256 * C, 8192, pairs, true, pl, "considered"); };
                pair_candidates(32 * R, 256 * C, 8192, pairs, w4, true, consider);
                if (w4) pair_even_candidates(32 * R, 256 * C, pairs, consider);
            }
    std::printf("%lld plans\n", n_plans);
}
"""


@pytest.fixture(scope="module")
def checker(tmp_path_factory):
    d = tmp_path_factory.mktemp("pair_plan")
    src, exe = d / "plans.cpp", d / "plans"
    src.write_text(SOURCE)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    return str(exe)


@pytest.mark.parametrize("kind", [0, 1], ids=["bf16", "int4"])
def test_plans_cover_every_unit_once(checker, kind):
    step = 6
    procs = [subprocess.Popen([checker, str(kind), str(first), str(step)], stdout=subprocess.PIPE, text=True) for first in range(1, step + 1)]
    outs = [p.communicate()[0] for p in procs]
    assert all(p.returncode == 0 for p in procs), "".join(o for o, p in zip(outs, procs) if p.returncode)
    assert sum(int(o.split()[0]) for o in outs) > 100000


# The hand-over of k-blocks between the int4 kernel's warp roles, step by step with random durations: barriers are counters of finished
# phases that a waiter sees only as a parity, as mbarrier.test_wait shows them.  Each wait that returns is compared with what
# has really happened.
HANDOVER = r"""
#include <cstdio>
#include <cstdlib>
#include <random>
#include <vector>
#include "awq_pair_plan.cuh"
using namespace awq;

static std::mt19937 rng;
static int upto(int n) { return (int)(rng() % (unsigned)n); }
struct Bars {
    std::vector<int> phases = std::vector<int>(64, 0);
    bool looks_over(int b, int parity) const { return (phases[b] & 1) != parity; }
};
struct Role {
    int i, step, state = 0, until = 0;
};
// `by_stage`: "landed" barriers numbered by the stage
static int run(int stages, int n, int slow, bool by_stage) {
    Bars landed, multiplied;
    std::vector<int> load_end(n, -1), has_landed(n, 0), has_multiplied(n, 0), ready(n, 0);
    auto lb = [&](int i) { return by_stage ? i % stages : pair_bar(i); };
    auto lp = [&](int i) { return by_stage ? i / stages & 1 : pair_bar_parity(i); };
    std::vector<Role> producers, groups;
    for (int p = 0; p < GP_PRODUCERS_INT4; ++p) producers.push_back({p, GP_PRODUCERS_INT4});
    for (int g = 0; g < GP_DEQUANT_GROUPS; ++g) groups.push_back({g, GP_DEQUANT_GROUPS});
    int mma = 0, mma_until = 0;
    for (int t = 0; has_multiplied[n - 1] == 0; ++t) {
        if (t > 4000 * n) return 2;  // nobody moves any more
        for (int i = 0; i < n; ++i)
            if (load_end[i] == t) has_landed[i] = 1, ++landed.phases[lb(i)];
        for (Role &p : producers) {
            if (p.i >= n) continue;
            const int freed = p.i - stages;
            if (freed >= 0) {
                if (!multiplied.looks_over(pair_bar(freed), pair_bar_parity(freed))) continue;
                if (!has_multiplied[freed]) return 1;
            }
            load_end[p.i] = t + 5 + upto(20) + (upto(8) == 0 ? upto(slow) : 0);
            p.i += p.step;
        }
        for (Role &g : groups) {
            if (g.i >= n || t < g.until) continue;
            if (g.state == 0) {  // looks for its k-block, reads and converts it
                if (!landed.looks_over(lb(g.i), lp(g.i))) continue;
                if (!has_landed[g.i]) return 1;
                g.state = 1, g.until = t + 4 + upto(8);
            } else if (g.state == 1) {  // looks for its weight buffer, writes it
                const int freed = g.i - GP_ABUF;
                if (freed >= 0) {
                    if (!multiplied.looks_over(pair_bar(freed), pair_bar_parity(freed))) continue;
                    if (!has_multiplied[freed]) return 1;
                }
                g.state = 2, g.until = t + 1 + upto(3);
            } else {
                ready[g.i] = 1;
                g.i += g.step, g.state = 0;
            }
        }
        if (t >= mma_until && ready[mma] && ready[mma + 1]) {
            for (int k = 0; k < 2; ++k) has_multiplied[mma + k] = 1, ++multiplied.phases[pair_bar(mma + k)];
            mma += 2, mma_until = t + 2 + upto(6);
            if (mma >= n) break;
        }
    }
    return 0;
}
int main(int, char **argv) {
    const bool by_stage = std::atoi(argv[1]) != 0;
    int early = 0, stuck = 0;
    for (int stages = 6; stages <= GP_MAX_STAGES; ++stages)
        for (int seed = 0; seed < 400; ++seed) {
            rng.seed(1000 * stages + seed);
            const int r = run(stages, 64, 10 << seed % 6, by_stage);
            early += r == 1, stuck += r == 2;
        }
    std::printf("%d %d\n", early, stuck);
}
"""


def test_no_wait_for_a_k_block_returns_early(tmp_path):
    src, exe = tmp_path / "handover.cpp", tmp_path / "handover"
    src.write_text(HANDOVER)
    subprocess.run(["g++", "-std=c++17", "-O2", "-Wall", "-I", CSRC, str(src), "-o", str(exe)], check=True)
    run = lambda arg: subprocess.run([str(exe), arg], check=True, stdout=subprocess.PIPE, text=True).stdout.split()
    assert run("0") == ["0", "0"]
    assert int(run("1")[0]) > 0  # the model sees what barriers numbered by the stage would allow
