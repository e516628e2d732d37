// The schedule of the GEMM on CTA pairs (awq_gemm_pair.cu): what a plan is, how a pair walks it, and how one is chosen.
// Plain arithmetic, the same on the host and on the device, and built by a C++ compiler alone too, so that plans can be checked
// without a GPU.
#pragma once

#include <stddef.h>

#ifdef __CUDACC__
#define GP_HD __host__ __device__
#else
#define GP_HD
#endif

namespace awq {

constexpr int GP_BN = 256, GP_HALF = 128, GP_BK = 64, GP_GROUP = 128;  // weight columns of a pair and of a CTA, k of a block and of a scale
constexpr int GP_UNIT = 32, GP_MAX_UNITS = 8;  // token rows: unit of the schedule, most units per piece
constexpr int GP_MAX_PARTS = 8;                // parts of K

// Hand-over of k-blocks, counted through all pieces of a launch: k-block i lies in stage i % stages, is dequantised (int4) by warp group
// i % 4 into weight buffer i % 8, and has two barriers, "landed" and "multiplied", each in a ring of 16 by its own number.
// A wait for a phase by its parity takes the phase before the last for the one it means, so whoever waits for k-block i must
// know that k-block i - 16's phase of the same barrier is over.  It does: a warp that is at i has waited for "multiplied" of
// i - 12 (a dequant warp, at its step before), which is after "landed" of it, or of i - 3 - stages (a producer; 12 stages at
// most).  The stage's own number would not do for "landed": with 7 stages, k-block i - 7 is another group's, and may still be on
// its way while group i % 4 looks for i; its wait returned at once then, and it dequantised what the stage held before.
constexpr int GP_BAR_RING = 16;
GP_HD inline int pair_bar(int i) { return i & (GP_BAR_RING - 1); }
GP_HD inline int pair_bar_parity(int i) { return (i / GP_BAR_RING) & 1; }
constexpr int GP_MAX_STAGES = 12, GP_ABUF = 8, GP_DEQUANT_GROUPS = 4, GP_PRODUCERS_INT4 = 3, GP_PRODUCERS_BF16 = 2;

// What a launch makes of its shared memory; widths are those of its widest piece.
constexpr int GP_SMEM_MAX = 227 * 1024;
constexpr int GP_X_UNIT_BYTES = GP_UNIT / 2 * GP_BK * 2;  // 2 KB: a CTA's half of a unit of token rows x 64 k
constexpr int GP_STAGING_STRIDE = GP_HALF * 2 + 16;       // bytes of a token row in the staging tile (+16: no bank conflicts)
constexpr int GP_NUM_BARS = 2 * GP_BAR_RING + GP_ABUF / 2 + 4, GP_BAR_BYTES = (GP_NUM_BARS * 8 + 16 + 127) / 128 * 128;
GP_HD constexpr int pair_w_bytes(bool w4) { return w4 ? GP_BK * (GP_HALF / 8) * 4 : GP_HALF * GP_BK * 2; }  // 4 KB of packed words / 16 KB of bf16
GP_HD constexpr int pair_s_bytes(bool w4) { return w4 ? GP_HALF * 2 : 0; }
GP_HD constexpr int pair_z_bytes(bool w4) { return w4 ? GP_HALF / 8 * 4 : 0; }
struct PairLayout {
    int stage_bytes, stages, staging_rows;
};
GP_HD inline PairLayout pair_layout(bool w4, int max_units) {
    PairLayout l;
    // token rows that go through the staging tile at a time: all of a piece (int4: the accumulators must be free again
    // quickly, there may be one set only), or 64 (bf16: two sets, the room goes to stages)
    const int staging_units = w4 ? GP_MAX_UNITS : 2;
    l.stage_bytes = (max_units * GP_X_UNIT_BYTES + pair_w_bytes(w4) + pair_s_bytes(w4) + pair_z_bytes(w4) + 1023) / 1024 * 1024;
    l.staging_rows = GP_UNIT * (max_units < staging_units ? max_units : staging_units);
    const int room = GP_SMEM_MAX - 1024 - GP_BAR_BYTES - l.staging_rows * GP_STAGING_STRIDE;
    l.stages = room / l.stage_bytes < GP_MAX_STAGES ? room / l.stage_bytes : GP_MAX_STAGES;
    return l;
}

// The schedule of a launch.  Token rows are counted in units of 32, R of them per column tile.  First `waves` rounds in
// which the P pairs take neighbouring tiles of the (column tile, token tile) grid, token tiles innermost (N_T nearly equal
// ones per column tile): the pairs of a round share token rows and weights in L2.  What does not fill a round is cut
// evenly: units from `base` on, counted column tile by column tile, one contiguous range per pair, where a cut between two
// ranges that is closer than `snap` units to a column tile's edge moves there.
// With S > 1, P pairs share the plane S times: the pairs of part s multiply the s-th part of K and leave f32 sums, which a
// second kernel adds up (gemm_pair_sum_kernel).
struct PairPlan {
    int P, R, C, max_units, sets, waves, NT, base, snap, S;
    GP_HD int cut(int p) const {
        if (p == 0) return base;  // nobody's range ends here: moved on to an edge, the units up to it would be left out
        const int v = base + (int)((long long)p * ((long long)R * C - base) / P), r = v % R;
        if (r == 0) return v;
        if (r <= snap) return v - r > base ? v - r : base;
        return R - r <= snap ? v + R - r : v;
    }
};

struct PairWalk {
    const PairPlan &pl;
    int p, w = 0, cur, end, seg_tile = 0, seg_a = 0, seg_len = 0, n = 0, i = 0;
    int tile = 0, unit = 0, units = 0;  // the current piece
    GP_HD PairWalk(int p_, const PairPlan &plan) : pl(plan), p(p_), cur(plan.cut(p_)), end(plan.cut(p_ + 1)) {}
    GP_HD bool next() {
        int a, b;
        if (w < pl.waves) {
            const int t = w * pl.P + p, j = t % pl.NT;
            ++w;
            tile = t / pl.NT;
            a = j * pl.R / pl.NT;
            b = (j + 1) * pl.R / pl.NT;
        } else {
            if (i == n) {
                if (cur >= end) return false;
                seg_tile = cur / pl.R;
                seg_a = cur - seg_tile * pl.R;
                seg_len = pl.R - seg_a < end - cur ? pl.R - seg_a : end - cur;
                n = (seg_len + pl.max_units - 1) / pl.max_units;
                i = 0;
                cur += seg_len;
            }
            tile = seg_tile;
            a = seg_a + i * seg_len / n;
            b = seg_a + (i + 1) * seg_len / n;
            ++i;
        }
        unit = a;
        units = b - a;
        return true;
    }
};

// The longest pair's time for a plan, in cycles.  Measured with clock64 per k-block of 64: 69 cycles per unit of 32 token
// rows (64 at the tensor pipe's peak), but not less than about 370 with int4 weights (the chain of a dequant group: fetch
// 240, arithmetic 630, tensor-memory store 200, over four groups) and 280 plus 35 per unit with bf16 ones (its bytes at the
// 59 bytes per cycle and SM that L2 delivers: a narrow piece's stage is mostly weights).  With one accumulator set a piece's drain is
// exposed: what a second and a third piece of 256 rows add beyond their multiplications is 2,700 to 4,000 cycles (74 column tiles,
// K 1024 and 2048), charged as 3,000.  With two sets it overlaps the next piece; the 600 charged for a piece are an estimate.
// Parts of K: their sums cross L2 twice, and the second pass is a launch.
// `ring`: with what the number of stages does to int4 pieces (pair_search says where).  A k-block takes about 4,500 cycles from the
// request of its stage to the end of its MMAs, so no piece takes less than that over the number of stages, which its width
// leaves room for: 7 with eight units, 10 with six, 12 with up to five.
// `limit`: from this figure on (0: nowhere) it need not be exact.
inline size_t pair_parts_bytes(int M, int N, int S) { return (size_t)S * M * ((N + GP_BN - 1) / GP_BN * GP_BN) * 4; }
constexpr size_t GP_PARTS_MAX_BYTES = 64u << 20;  // about half of L2
inline long long pair_cost(const PairPlan &pl, int KB_all, bool w4, int M, bool ring = false, long long limit = 0) {
    const int KB = (KB_all / 2 + pl.S - 1) / pl.S * 2;
    const int turn = ring ? 4500 / pair_layout(w4, pl.max_units).stages : 0;
    const int floor_cycles = ring ? (turn > 420 ? turn : 420) : (w4 ? 370 : 280), floor_unit = w4 ? 0 : 35;
    const int drain = pl.sets == 2 ? (ring ? 1500 : 600) : 3000;
    auto segment = [&](int len, int n) -> long long {  // `len` units of one column tile in n pieces
        const long long least = (long long)n * floor_cycles + (long long)len * floor_unit;
        const long long kblock = 69 * len > least ? 69 * len : least;
        return KB * kblock + (long long)n * drain;
    };
    auto cut_up = [&](int len) -> long long { return len <= 0 ? 0 : segment(len, (len + pl.max_units - 1) / pl.max_units); };
    const long long whole = cut_up(pl.R);
    const long long parts = pl.S > 1 ? 6000 + (long long)pl.S * M * pl.C * GP_BN * 4 / 1000 : 0;
    const long long rounds = pl.waves * segment((pl.R + pl.NT - 1) / pl.NT, 1) + parts;
    long long worst = 0;
    int a = pl.cut(0);
    for (int p = 0; p < pl.P && a < pl.R * pl.C; ++p) {
        const int b = pl.cut(p + 1), ta = a / pl.R, tb = b / pl.R;
        const long long t = ta == tb ? cut_up(b - a) : cut_up((ta + 1) * pl.R - a) + (tb - ta - 1) * whole + cut_up(b - tb * pl.R);
        if (t > worst) worst = t;
        if (limit && worst + rounds >= limit) break;
        a = b;
    }
    return worst + rounds;
}

// Every plan that is considered for a shape, each given to `consider`.
template <typename F>
inline void pair_candidates(int M, int N, int K, int all_pairs, bool w4, bool may_split, F &&consider) {
    PairPlan pl;
    pl.R = (M + GP_UNIT - 1) / GP_UNIT;
    pl.C = (N + GP_BN - 1) / GP_BN;
    const int KB = (K + 2 * GP_BK - 1) / (2 * GP_BK) * 2;
    const int nt_min = (pl.R + GP_MAX_UNITS - 1) / GP_MAX_UNITS;
    // parts of K: of eight k-blocks at least, and not where the plane alone gives every pair two pieces
    for (pl.S = 1; pl.S == 1 || (may_split && pl.S <= GP_MAX_PARTS && KB >= 8 * pl.S && pl.C * nt_min < 2 * all_pairs &&
                                 pair_parts_bytes(M, N, pl.S) <= GP_PARTS_MAX_BYTES);
         pl.S += pl.S < 4 ? 1 : 2) {
        const int pairs = all_pairs / pl.S;
        for (pl.NT = nt_min; pl.NT <= pl.R && pl.NT < nt_min + 4; ++pl.NT) {
            const int tiles = pl.NT * pl.C;
            pl.max_units = (pl.R + pl.NT - 1) / pl.NT;  // of a tile, and of a piece of what is cut evenly
            pl.sets = !w4 || pl.max_units <= GP_MAX_UNITS / 2 ? 2 : 1;
            pl.P = tiles < pairs ? tiles : pairs;
            for (int back = 0; back < 2 && back <= tiles / pl.P; ++back) {  // rounds; the rest is cut evenly
                pl.waves = tiles / pl.P - back;
                const int t = pl.waves * pl.P;
                pl.base = t / pl.NT * pl.R + t % pl.NT * pl.R / pl.NT;
                if (t == tiles) {
                    pl.snap = 0;
                    consider(pl);
                    continue;
                }
                if (pl.S > 1) continue;  // parts of whole tiles only (512 x 8192 x 2048 bf16: 20.8 us so, 23.1 in three parts cut evenly)
                for (int sn : {0, 2, pl.R}) {
                    pl.snap = sn;
                    consider(pl);
                }
            }
            if (pl.S == 1 && tiles < pairs && pl.R * pl.C > tiles) {  // fewer tiles than pairs: cut everything evenly over all pairs
                pl.P = pl.R * pl.C < pairs ? pl.R * pl.C : pairs;
                pl.waves = pl.base = 0;
                for (int sn : {0, 2}) {
                    pl.snap = sn;
                    consider(pl);
                }
            }
        }
    }
}

// The plans considered once more where everything is best cut evenly (int4): pieces of every width, and a round whose tiles are six
// units wide.
template <typename F>
inline void pair_even_candidates(int M, int N, int all_pairs, F &&consider) {
    PairPlan pl;
    pl.S = 1;
    pl.R = (M + GP_UNIT - 1) / GP_UNIT;
    pl.C = (N + GP_BN - 1) / GP_BN;
    const int nt_min = (pl.R + GP_MAX_UNITS - 1) / GP_MAX_UNITS, nt_six = (pl.R + 5) / 6;
    auto with_snaps = [&] {
        pl.sets = pl.max_units <= GP_MAX_UNITS / 2 ? 2 : 1;
        for (int sn : {0, 2}) {
            pl.snap = sn;
            consider(pl);
        }
    };
    for (pl.NT = nt_min; pl.NT <= nt_six || pl.NT < nt_min + 4; ++pl.NT) {
        if (pl.NT > pl.R || (pl.NT >= nt_min + 4 && pl.NT != nt_six)) continue;
        const int tiles = pl.NT * pl.C;
        pl.max_units = (pl.R + pl.NT - 1) / pl.NT;
        pl.P = tiles < all_pairs ? tiles : all_pairs;
        pl.waves = 1;
        pl.base = pl.P / pl.NT * pl.R + pl.P % pl.NT * pl.R / pl.NT;
        with_snaps();
    }
    pl.P = pl.R * pl.C < all_pairs ? pl.R * pl.C : all_pairs;
    pl.waves = pl.base = 0;
    for (pl.max_units = pl.R < GP_MAX_UNITS ? pl.R : GP_MAX_UNITS; pl.max_units >= 3; --pl.max_units) {
        pl.NT = (pl.R + pl.max_units - 1) / pl.max_units;
        with_snaps();
    }
}

// The cheapest of them.  Where that is everything cut evenly, with int4 weights and K uncut, a pair has one or two pieces of very
// different widths, and the widest decides for all how many stages there are: there the choice is made again with the ring's depth in
// the model.  Over 67 such shapes 8 % faster, none slower (4096 x 8192 x 1056 100 -> 78 us, 3000 x 8192 x 2048 93 -> 77; the kernel
// that gave a CTA 160 rows, and whose times these plans had missed: 76 and 77).  Where whole rounds are made, the depth in the model
// changes the choice by less than two runs differ.
inline PairPlan pair_search(bool w4, int M, int N, int K, int all_pairs, bool may_split) {
    const int KB = (K + 2 * GP_BK - 1) / (2 * GP_BK) * 2;
    PairPlan best_plan;
    long long best = -1;
    pair_candidates(M, N, K, all_pairs, w4, may_split, [&](const PairPlan &pl) {
        const long long c = pair_cost(pl, KB, w4, M, false, best > 0 ? best : 0);
        if (best < 0 || c < best) best = c, best_plan = pl;
    });
    if (!w4 || best_plan.S > 1 || best_plan.waves > 0) return best_plan;
    best = pair_cost(best_plan, KB, w4, M, true);
    pair_even_candidates(M, N, all_pairs, [&](const PairPlan &pl) {
        const long long c = pair_cost(pl, KB, w4, M, true, best);
        if (c < best) best = c, best_plan = pl;
    });
    return best_plan;
}

}  // namespace awq
