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
                pair_candidates(32 * R, 256 * C, 8192, pairs, w4, true, [&](const PairPlan &pl) { check(w4, 32 * R, 256 * C, 8192, pairs, true, pl, "considered"); });
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
