// Prefill GEMM on CTA pairs: C[M, N] = bf16(A[M, K] @ W) with int4-AWQ or bf16 weights.
//
// Two CTAs of a cluster (two SMs) work on one tile with tcgen05.mma.cta_group::2: 256 weight columns (the MMA's M side,
// 128 per CTA) x up to 256 token rows (its N side, half of them loaded by each CTA).  Each SM then reads half the token
// rows per flop from shared memory, and a dequantised weight serves 256 token rows.  What bounds it: from about 1000 rows on
// the tensor pipe (a k-block of 64 takes 552 cycles where 512 are its peak, the drain of a tile 8 % beside them) and, in a
// long loop, power; below, the dequantisation, 370 cycles per k-block however few the rows.
//
// Measured (us per launch inside a CUDA graph, M x K x N; before = the faster of the one-CTA kernels this one replaced:
// dequantised weights as a shared-memory tile / in tensor memory with 192-row tiles dealt round-robin):
//   128 x 4096 x 14336   35 -> 20      512 x 4096 x 14336   59 -> 50     2048 x 4096 x 14336   202 -> 173 (1.39 PFLOP/s)
//   128 x 14336 x 4096  105 -> 50      777 x 14336 x 4096  106 -> 73     4096 x 8192 x 57344  3350 -> 3090
// These are short bursts; in a loop of seconds at the power cap 2048 x 4096 x 14336 takes 227 -> 200.
// With scratch from the caller, K cut into parts (uncut -> cut, second pass included): 128 x 14336 x 4096 49 -> 23, 256 x 8192 x 2048
// 31 -> 18, 65 x 4096 x 4096 19 -> 13.5; bf16 weights 512 x 8192 x 2048 34 -> 24.  Letting the next launch start early (programmatic
// dependent launch) takes 1 to 2 us off each launch in a row: 96 x 512 x 1024 8.2 -> 6.0.
//
//   int4   the weights are dequantised into tensor memory (ldmatrix.trans -> LOP3 / bf16x2 -> tcgen05.st), each CTA its
//          own 128 columns; four groups of four dequant warps take alternate k-blocks and hold a finished k-block in
//          registers while its tensor-memory buffer is still being multiplied
//   bf16   both operands come from shared memory (K-major, 128-byte swizzle)
//
//   work     token rows are counted in units of 32 and the (column tile, token unit) plane is cut into one contiguous
//            range per pair, so that no pair idles in a partial last wave whatever M and N are; a range is walked in
//            pieces of nearly equal width inside a column tile.  Where the cuts may lie is chosen on the host by a cost
//            model (awq_pair_plan.cuh)
//   TMEM     int4: accumulators at 0 (two sets of 128 columns, or one of 256), eight weight buffers of 32 columns (64 k)
//            from 256 on; bf16: two accumulator sets of 256
//   epilogue accumulators -> bf16 (or f32 + residual -> bf16) -> stmatrix.trans into a staging tile in shared memory ->
//            16-byte row stores; the accumulators are free again after about a thousand cycles, the stores overlap the next piece
//
// Every wait is bounded; on expiry the kernel records an error and all roles drain, so the tensor memory is always released.
#include <cudaTypedefs.h>
#include <cuda_bf16.h>

#include <mutex>

#include "awq_common.cuh"
#include "awq_pair_plan.cuh"
#include "awq_ptx.cuh"
#include "awq_tcgen05.cuh"

namespace awq {

int encode_tensor_map_2d(CUtensorMap *map, int dtype, const void *base, uint64_t dim0, uint64_t dim1,
                         uint64_t stride1_bytes, uint32_t box0, uint32_t box1, int swizzle);

constexpr int GP_EPI_WARPS = 8;
constexpr uint32_t GP_TMEM_COLS = 512;
constexpr int GP_ABUF_COLS = GP_BK / 2, GP_ABUF_COL0 = 256;
static_assert(2 * GP_UNIT * GP_MAX_UNITS <= (int)GP_TMEM_COLS, "two accumulator sets (bf16)");
static_assert(GP_UNIT * GP_MAX_UNITS <= GP_ABUF_COL0 && GP_ABUF_COL0 + GP_ABUF * GP_ABUF_COLS <= (int)GP_TMEM_COLS, "accumulators, then weight buffers (int4)");

template <bool W4>
struct PairCfg {
    static constexpr int W_BYTES = pair_w_bytes(W4), S_BYTES = pair_s_bytes(W4), Z_BYTES = pair_z_bytes(W4);
    // Warps that load, on alternate k-blocks: a k-block costs a loading warp about 430 cycles (a look at a barrier 120, four
    // copies 180, the rest the loop), which one warp alone turned into the launch's time for pieces narrower than 200 rows.
    static constexpr int PRODUCERS = W4 ? GP_PRODUCERS_INT4 : GP_PRODUCERS_BF16;
    static constexpr int DEQUANT_WARPS = W4 ? 4 * GP_DEQUANT_GROUPS : 0;
    static constexpr int EPI_WARP0 = 4 + DEQUANT_WARPS;
    static constexpr int THREADS = (EPI_WARP0 + GP_EPI_WARPS) * 32;
};
// f32 accumulate, bf16 x bf16, both K-major, M 256 over the pair; N is added per piece
constexpr uint32_t GP_IDESC_BASE = (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(256 >> 4) << 24);

struct PairMaps {
    CUtensorMap x[GP_MAX_UNITS];  // token rows: box of 16 (i + 1) rows x 64 k
    CUtensorMap w, s, z;
};

__device__ int g_gemm_pair_error;  // 0 = ok; set when a bounded wait gave up

__device__ __forceinline__ uint32_t gp_cluster_rank() {
    uint32_t r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t gp_mapa(uint32_t addr, uint32_t rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
__device__ __forceinline__ void gp_arrive_cluster(uint32_t mapped_bar) {
    asm volatile("mbarrier.arrive.shared::cluster.b64 _, [%0];" ::"r"(mapped_bar) : "memory");
}
__device__ __forceinline__ void gp_cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ void gp_commit_both(uint32_t bar) {  // arrives at `bar` of both CTAs
    asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar),
                 "h"((uint16_t)3)
                 : "memory");
}
// A load into this CTA's shared memory that counts on a barrier of either CTA of the pair.
__device__ __forceinline__ void gp_tma_load_2d_pair(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t mapped_bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.cta_group::2.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(mapped_bar)
        : "memory");
}
__device__ __forceinline__ void gp_umma_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
__device__ __forceinline__ void gp_umma_ss(uint32_t d_tmem, uint64_t a_desc, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
        ::"r"(d_tmem), "l"(a_desc), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}
// 16 lanes x 32 columns: v[4 i .. 4 i + 3] for columns 8 i .. 8 i + 7, laid out as dg_tmem_st_16x256b's r0..r3
__device__ __forceinline__ void gp_tmem_st_16x256b_x4(uint32_t taddr, const uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x256b.x4.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]),
        "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
// 16 lanes x 16 columns of f32: r[4 i], r[4 i + 1] = columns 8 i + 2 t, + 1 of lane l / 4; r[4 i + 2], r[4 i + 3] of lane l / 4 + 8
__device__ __forceinline__ void gp_tmem_ld_16x256b_x2(uint32_t taddr, uint32_t *r) {
    asm volatile("tcgen05.ld.sync.aligned.16x256b.x2.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}
__device__ __forceinline__ uint32_t gp_cvt_bf16x2(float lo, float hi) {
    uint32_t r;
    asm("cvt.rn.bf16x2.f32 %0, %1, %2;" : "=r"(r) : "f"(hi), "f"(lo));
    return r;
}
__device__ __forceinline__ void gp_stmatrix_x4_trans(uint32_t addr, const uint32_t (&r)[4]) {
    asm volatile("stmatrix.sync.aligned.m8n8.x4.trans.shared.b16 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3])
                 : "memory");
}
__device__ __forceinline__ bool gp_bar_and(int id, int threads, bool ok) {  // named barrier; true if `ok` on every thread
    uint32_t r;
    asm volatile(
        "{\n\t.reg .pred p, q;\n\tsetp.ne.u32 q, %1, 0;\n\t"
        "barrier.cta.red.and.pred p, %2, %3, q;\n\tselp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(r)
        : "r"(ok ? 1u : 0u), "r"(id), "r"(threads)
        : "memory");
    return r != 0;
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t v) { asm volatile("st.shared.u32 [%0], %1;" ::"r"(addr), "r"(v) : "memory"); }

// How many consecutive barriers (lane 0's, lane 1's, ...; 0 = none) have completed their phase, at least MIN: bounded, 0 on expiry.
template <int MIN>
__device__ __forceinline__ int gp_count_ready(uint32_t bar, uint32_t parity, long long limit) {
    const long long t0 = clock64();
    while (true) {
#pragma unroll 1
        for (int i = 0; i < 64; ++i) {
            uint32_t ok = 0;
            if (bar)
                asm volatile(
                    "{\n\t.reg .pred p;\n\t"
                    "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                    "selp.u32 %0, 1, 0, p;\n\t}"
                    : "=r"(ok)
                    : "r"(bar), "r"(parity)
                    : "memory");
            const int n = __ffs(~__ballot_sync(0xffffffffu, ok != 0)) - 1;
            if (n >= MIN) return n;
        }
        if (__any_sync(0xffffffffu, clock64() - t0 > limit)) return 0;
    }
}

template <bool W4>
__global__ void __cluster_dims__(2, 1, 1) __launch_bounds__(PairCfg<W4>::THREADS, 1)
gemm_pair_kernel(const __grid_constant__ PairMaps maps, uint16_t *__restrict__ C, const uint16_t *__restrict__ R, int epi, int M, int N,
                 int K, const __grid_constant__ PairPlan plan, long long wait_limit) {
    using Cfg = PairCfg<W4>;
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t *smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));
    const PairLayout lay = pair_layout(W4, plan.max_units);
    const int stages = lay.stages, acc_sets = plan.sets;
    const int x_bytes = plan.max_units * GP_X_UNIT_BYTES;
    const uint32_t bar_base = smem_base + (uint32_t)(stages * lay.stage_bytes);
    const uint32_t staging = bar_base + GP_BAR_BYTES;
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(smem_gen + stages * lay.stage_bytes + GP_NUM_BARS * 8);
    // k-block i has landed: int4 in this CTA; bf16 in both (leader's)
    auto full_bar = [&](int i) { return bar_base + 8u * pair_bar(i); };
    // int4, leader's: weight buffers 2 b and 2 b + 1 are dequantised in both CTAs
    auto ready_bar = [&](int b) { return bar_base + 8u * (GP_BAR_RING + b); };
    // the pair's MMAs of k-block i are done: frees its stage and its weight buffer
    auto done_bar = [&](int i) { return bar_base + 8u * (GP_BAR_RING + GP_ABUF / 2 + pair_bar(i)); };
    auto acc_full = [&](int a) { return bar_base + 8u * (2 * GP_BAR_RING + GP_ABUF / 2 + a); };
    auto acc_empty = [&](int a) { return bar_base + 8u * (2 * GP_BAR_RING + GP_ABUF / 2 + 2 + a); };  // (leader's)
    auto stage_addr = [&](int s) { return smem_base + (uint32_t)(s * lay.stage_bytes); };

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t rank = gp_cluster_rank();
    const int KB2 = (K + 2 * GP_BK - 1) / (2 * GP_BK);  // k-blocks are multiplied two at a time
    const int pair = (int)(blockIdx.x >> 1), part = pair / plan.P;
    const int kb_first = part * KB2 / plan.S * 2, KB = (part + 1) * KB2 / plan.S * 2 - kb_first;  // this pair's part of K
    constexpr int ACC_STRIDE = W4 ? GP_ABUF_COL0 / 2 : 256;  // columns between two accumulator sets
    PairWalk walk(pair - part * plan.P, plan);

    if (threadIdx.x == 0) {
        for (int b = 0; b < GP_ABUF / 2; ++b) mbar_init(ready_bar(b), 16);  // per k-block four dequant warps in each CTA
        for (int i = 0; i < GP_BAR_RING; ++i) {
            mbar_init(full_bar(i), 1);
            mbar_init(done_bar(i), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full(a), 1);
            mbar_init(acc_empty(a), 2 * GP_EPI_WARPS);
        }
        mbar_fence_init();
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)), "r"(GP_TMEM_COLS) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    }
    dg_fence_before();
    __syncthreads();
    gp_cluster_sync();  // the peer's barriers are initialised
    dg_fence_after();
    const uint32_t tmem_base = *tmem_slot;
    pdl_launch_dependents();
    pdl_wait();

    if (warp == 0 || (warp > 1 && warp <= Cfg::PRODUCERS)) {
        // ------------------------------ producers: k-blocks prod, prod + PRODUCERS, ... ------------------------------
        const int prod = warp == 0 ? 0 : warp - 1;
        if (elect_one()) {
            tma_prefetch_desc(&maps.w);
            if (W4) {
                tma_prefetch_desc(&maps.s);
                tma_prefetch_desc(&maps.z);
            }
        }
        const uint32_t full0 = W4 ? full_bar(0) : gp_mapa(full_bar(0), 0);
        int s = prod % stages, it = prod, kb = prod;  // k-block `it` of the launch is k-block kb of the piece
        bool ok = true;
        while (ok && walk.next()) {
            const int half_rows = walk.units * (GP_UNIT / 2);
            const int m0 = walk.unit * GP_UNIT + (int)rank * half_rows, n0 = walk.tile * GP_BN + (int)rank * GP_HALF;
            const CUtensorMap *mx = &maps.x[walk.units - 1];
            const uint32_t tx = (uint32_t)half_rows * GP_BK * 2 + Cfg::W_BYTES + Cfg::S_BYTES + Cfg::Z_BYTES;
            for (; kb < KB; kb += Cfg::PRODUCERS, it += Cfg::PRODUCERS) {
                const int freed = it - stages;  // the k-block that had the stage before
                if (freed >= 0 && !mbar_wait_bounded_warp(done_bar(freed), pair_bar_parity(freed), wait_limit)) {
                    if (lane == 0) atomicExch(&g_gemm_pair_error, 1);
                    ok = false;
                    break;
                }
                const uint32_t st = stage_addr(s), bar = full0 + 8u * pair_bar(it);
                const int k0 = (kb_first + kb) * GP_BK;
                if (elect_one()) {
                    if (W4) {
                        const int g = k0 / GP_GROUP;
                        mbar_expect_tx(bar, tx);
                        tma_load_2d(st + x_bytes, &maps.w, n0 / 8, k0, bar);
                        tma_load_2d(st + x_bytes + Cfg::W_BYTES, &maps.s, n0, g, bar);
                        tma_load_2d(st + x_bytes + Cfg::W_BYTES + Cfg::S_BYTES, &maps.z, n0 / 8, g, bar);
                        tma_load_2d(st, mx, k0, m0, bar);
                    } else {
                        if (rank == 0) mbar_expect_tx(full_bar(it), 2 * tx);  // both CTAs' copies are counted on the leader's barrier
                        gp_tma_load_2d_pair(st, mx, k0, m0, bar);
                        gp_tma_load_2d_pair(st + x_bytes, &maps.w, k0, n0, bar);
                    }
                }
                __syncwarp();
                for (s += Cfg::PRODUCERS; s >= stages;) s -= stages;
            }
            kb -= KB;
        }
    } else if (warp == 1) {
        // ------------------------------ MMA issuer (leader CTA only) ------------------------------
        if (rank == 0) {
            // What is looked at: int4 the four barriers of the weight buffer pairs, bf16 those of the k-blocks.  Two k-blocks take eight
            // MMAs, two commits and one look at most: a k-block at a time, the issuing warp's own instructions (a look costs
            // a hundred cycles even when it is over at once) took 430 cycles per k-block however narrow the piece.
            constexpr int ring = W4 ? GP_ABUF / 2 : GP_BAR_RING, look = W4 ? ring : 8;  // (every lane that looks costs: 16 of them 2 %)
            constexpr int STEP = W4 ? 1 : 2;  // barriers per two k-blocks
            int s = 0, r = 0, rphase = 0, piece = 0, avail = 0, j = 0;
            bool ok = true;
            while (ok && walk.next()) {
                const int set = acc_sets == 2 ? piece & 1 : 0, use = acc_sets == 2 ? piece >> 1 : piece;
                if (use > 0 && !mbar_wait_bounded(acc_empty(set), (use - 1) & 1, wait_limit)) {
                    if (lane == 0) atomicExch(&g_gemm_pair_error, 2);
                    break;
                }
                dg_fence_after();
                const uint32_t d_tmem = tmem_base + (uint32_t)(set * ACC_STRIDE);
                const uint32_t idesc = GP_IDESC_BASE | ((uint32_t)(walk.units * GP_UNIT >> 3) << 17);
                for (int kb = 0; kb < KB; kb += 2, ++j) {
                    if (avail < STEP) {
                        const int b = r + lane < ring ? r + lane : r + lane - ring;
                        const uint32_t parity = r + lane < ring ? rphase : rphase ^ 1;
                        avail = gp_count_ready<STEP>(lane < look ? (W4 ? ready_bar(b) : full_bar(b)) : 0u, parity, wait_limit);
                        if (avail == 0) {
                            if (lane == 0) atomicExch(&g_gemm_pair_error, 3);
                            ok = false;
                            break;
                        }
                        dg_fence_after();
                    }
                    avail -= STEP;
                    const int s1 = s + 1 == stages ? 0 : s + 1;
                    const uint64_t x_desc[2] = {dg_desc_sw128(stage_addr(s)), dg_desc_sw128(stage_addr(s1))};
                    const uint32_t a_tmem = tmem_base + GP_ABUF_COL0 + (uint32_t)((j & (GP_ABUF / 2 - 1)) * 2 * GP_ABUF_COLS);
                    const uint32_t w_off = (uint32_t)x_bytes >> 4;  // (bf16) descriptor distance of the weights from the token rows
                    const uint32_t acc0 = kb ? 1u : 0u;
                    if (elect_one()) {
#pragma unroll
                        for (int k16 = 0; k16 < 2 * GP_BK / 16; ++k16) {
                            const uint64_t xd = x_desc[k16 >> 2] + (uint64_t)(2 * (k16 & 3));
                            if (W4)
                                gp_umma_ta(d_tmem, a_tmem + 8 * k16, xd, idesc, k16 ? 1u : acc0);
                            else
                                gp_umma_ss(d_tmem, xd + w_off, xd, idesc, k16 ? 1u : acc0);
                            if ((k16 & 3) == 3) gp_commit_both(done_bar(2 * j + (k16 >> 2)));
                        }
                    }
                    __syncwarp();
                    s = s1 + 1 == stages ? 0 : s1 + 1;
                    r += STEP;
                    if (r >= ring) r -= ring, rphase ^= 1;
                }
                if (ok && elect_one()) gp_commit_both(acc_full(set));
                __syncwarp();
                ++piece;
            }
        }
    } else if (W4 && warp >= 4 && warp < Cfg::EPI_WARP0) {
        // ------------------------------ dequant ------------------------------
        // Group grp = (warp - 4) / 4 takes k-blocks grp, grp + 4, ..., k-block i into weight buffer i % 8; in a group warp w owns TMEM lanes
        // 32 (w % 4) .. + 31, i.e. 32 columns: one 16-byte chunk (4 packed words) of a 64-byte row of words.
        const int grp = (warp - 4) >> 2, q = warp & 3;
        const int g = lane >> 2;  // ldmatrix.trans: lane (g, t = lane % 4) gets 16-bit column g of the chunk, rows 2t and 2t + 1
        // Row addresses of the four 8 x 8 matrices of an ldmatrix.x4: matrix m = 2 sp + x serves k16 step sp of the call's
        // 32 k and holds rows k = 16 sp + 4 j + 2 x + {0, 1} (j = 0..3), so that lane (g, t) receives the k pair 2t + x
        const int mi = lane >> 3, rr = lane & 7;
        const int k_lane = 16 * (mi >> 1) + 4 * (rr >> 1) + 2 * (mi & 1) + (rr & 1);  // + 32 for the second call
        const uint32_t w_off = (uint32_t)k_lane * 64 + (uint32_t)((q ^ ((k_lane >> 1) & 3)) << 4);  // 64B swizzle; k + 32 keeps the chunk
        const uint32_t a_tmem0 = tmem_base + ((uint32_t)(32 * q) << 16) + GP_ABUF_COL0;
        const uint32_t ready0 = gp_mapa(ready_bar(0), 0);
        int units = 0;
        while (walk.next()) units += KB;
        int s = grp;
        for (int it = grp; it < units; it += GP_DEQUANT_GROUPS) {
            const int ab = it % GP_ABUF, freed = it - GP_ABUF;  // the k-block that had the buffer before
            if (!mbar_wait_bounded(full_bar(it), pair_bar_parity(it), wait_limit)) {
                if (lane == 0) atomicExch(&g_gemm_pair_error, 4);
                break;
            }
            const uint32_t st = stage_addr(s) + x_bytes;  // packed words, then scales, then zeros
            const uint32_t zw = lds32(st + Cfg::W_BYTES + Cfg::S_BYTES + (4 * q + (g >> 1)) * 4) >> (16 * (g & 1));
            const uint4 sv = lds128(st + Cfg::W_BYTES + (32 * q + 8 * (g >> 1)) * 2);
            const uint32_t sw[4] = {sv.x, sv.y, sv.z, sv.w};
            uint32_t r[2][4];
            ldmatrix_x4_trans(r[0], st + w_off);
            ldmatrix_x4_trans(r[1], st + w_off + 32 * 64);
            uint32_t zz[4], ss[4];
#pragma unroll
            for (int e = 0; e < 4; ++e) {
                zz[e] = ((zw >> (4 * e)) & 0xFu) * 0x00010001u + 0x43004300u;
                asm("prmt.b32 %0, %1, %1, %2;" : "=r"(ss[e]) : "r"(sw[e]), "r"((g & 1) ? 0x3232u : 0x1010u));
            }
            uint32_t lo[16], hi[16];  // TMEM lanes 0-15 and 16-31 of the warp's quarter, 32 columns
#pragma unroll
            for (int c = 0; c < 4; ++c) {  // k16 step c
                const uint32_t p0 = r[c >> 1][2 * (c & 1)], p1 = r[c >> 1][2 * (c & 1) + 1];  // k pairs 2t and 2t + 1
#pragma unroll
                for (int e = 0; e < 4; ++e) {
                    const uint32_t v0 = dg_bf16x2_mul(dg_bf16x2_sub(nib2_to_bf16x2_biased(p0 >> (4 * e)), zz[e]), ss[e]);
                    const uint32_t v1 = dg_bf16x2_mul(dg_bf16x2_sub(nib2_to_bf16x2_biased(p1 >> (4 * e)), zz[e]), ss[e]);
                    uint32_t *d = e < 2 ? lo : hi;
                    d[4 * c + 2 * (e & 1)] = v0;
                    d[4 * c + 2 * (e & 1) + 1] = v1;
                }
            }
            if (freed >= 0 && !mbar_wait_bounded(done_bar(freed), pair_bar_parity(freed), wait_limit)) {
                if (lane == 0) atomicExch(&g_gemm_pair_error, 4);
                break;
            }
            dg_fence_after();
            const uint32_t a_tmem = a_tmem0 + (uint32_t)(ab * GP_ABUF_COLS);
            gp_tmem_st_16x256b_x4(a_tmem, lo);
            gp_tmem_st_16x256b_x4(a_tmem + (16u << 16), hi);
            dg_tmem_st_wait();
            dg_fence_before();
            __syncwarp();
            if (lane == 0) gp_arrive_cluster(ready0 + 8u * (ab >> 1));
            s += GP_DEQUANT_GROUPS;
            if (s >= stages) s -= stages;
        }
    } else if (warp >= Cfg::EPI_WARP0) {
        // ------------------------------ epilogue ------------------------------
        const int q = warp & 3;                            // this warp's 32 TMEM lanes ...
        const int th = (warp - Cfg::EPI_WARP0) >> 2;       // ... of this half of the piece's token rows
        const int tid = threadIdx.x - Cfg::EPI_WARP0 * 32;  // 0 .. 255
        constexpr int ET = GP_EPI_WARPS * 32;
        const uint32_t acc_empty_leader[2] = {gp_mapa(acc_empty(0), 0), gp_mapa(acc_empty(1), 0)};
        int piece = 0;
        while (walk.next()) {
            const int set = acc_sets == 2 ? piece & 1 : 0, use = acc_sets == 2 ? piece >> 1 : piece;
            const int rows = walk.units * GP_UNIT, m_base = walk.unit * GP_UNIT, n0 = walk.tile * GP_BN + (int)rank * GP_HALF;
            const int valid = M - m_base < rows ? M - m_base : rows;
            if (plan.S > 1) {
                // this part's sums as they are: a lane per column, 16 token rows at a time
                const bool full = mbar_wait_bounded(acc_full(set), use & 1, wait_limit);
                if (!__all_sync(0xffffffffu, full)) {
                    if (lane == 0) atomicExch(&g_gemm_pair_error, 5);
                    break;
                }
                dg_fence_after();
                const int n_pad = plan.C * GP_BN;
                float *out = reinterpret_cast<float *>(C) + ((size_t)part * M + m_base) * n_pad + n0 + 32 * q + (W4 ? dg_lane_column(lane) : lane);
                const uint32_t acc = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(set * ACC_STRIDE);
                for (int t = th * (rows / 2); t < (th + 1) * (rows / 2); t += 16) {
                    uint32_t v[16];
                    dg_tmem_ld_32x32b_x16(acc + (uint32_t)t, v);
                    dg_tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 16; ++i)
                        if (t + i < valid) __stcg(out + (size_t)(t + i) * n_pad, __uint_as_float(v[i]));
                }
                dg_fence_before();
                __syncwarp();
                if (lane == 0) gp_arrive_cluster(acc_empty_leader[set]);
                ++piece;
                continue;
            }
            if (epi == GEMM_EPI_RESIDUAL) {
                // the residual tile goes through the staging tile in the order the accumulators will have there
                named_bar_sync(1, ET);  // the previous piece has left the staging tile
                const int c16 = tid & 15, n = n0 + 8 * c16;
                for (int m = tid >> 4; m < valid; m += ET / 16) {
                    if (n >= N) continue;
                    const uint4 v = *reinterpret_cast<const uint4 *>(R + (size_t)(m_base + m) * N + n);
                    const uint32_t a = staging + (uint32_t)(m * GP_STAGING_STRIDE + (c16 >> 2) * 64 + (c16 & 3) * 4);
                    sts32(a, v.x);
                    sts32(a + 16, v.y);
                    sts32(a + 32, v.z);
                    sts32(a + 48, v.w);
                }
            }
            const bool got = mbar_wait_bounded(acc_full(set), use & 1, wait_limit);
            if (!gp_bar_and(1, ET, got)) {  // (also: the previous piece has left the staging tile, the residual is in it)
                if (tid == 0) atomicExch(&g_gemm_pair_error, 5);
                break;
            }
            dg_fence_after();
            const uint32_t t_acc = tmem_base + ((uint32_t)(32 * q) << 16) + (uint32_t)(set * ACC_STRIDE);
            const int mi = lane >> 3, rr = lane & 7;
            for (int c0 = 0; c0 < rows; c0 += lay.staging_rows) {
                const int c_rows = rows - c0 < lay.staging_rows ? rows - c0 : lay.staging_rows;
                if (c0) named_bar_sync(1, ET);  // the previous chunk has left the staging tile
                const int tok1 = (th + 1) * (c_rows / 2);
                // 16 token rows at a time (TMEM lanes 0-15 and 16-31 of the quarter); the next ones are on their way meanwhile
                uint32_t v[2][16];
                int tok = th * (c_rows / 2);
                gp_tmem_ld_16x256b_x2(t_acc + (uint32_t)(c0 + tok), &v[0][0]);
                gp_tmem_ld_16x256b_x2(t_acc + (16u << 16) + (uint32_t)(c0 + tok), &v[0][8]);
                auto put = [&](const uint32_t (&u)[16], int t) {
#pragma unroll
                    for (int blk = 0; blk < 2; ++blk) {  // 8 token rows: four 8 x 8 matrices (TMEM lanes 8 i .. 8 i + 7)
                        const uint32_t addr = staging + (uint32_t)((t + 8 * blk + rr) * GP_STAGING_STRIDE + q * 64 + mi * 16);
                        float f[8];
#pragma unroll
                        for (int j = 0; j < 4; ++j)
                            f[j] = __uint_as_float(u[4 * blk + j]), f[4 + j] = __uint_as_float(u[8 + 4 * blk + j]);
                        if (W4 && epi == GEMM_EPI_RESIDUAL) {
                            uint32_t res[4];
                            ldmatrix_x4_trans(res, addr);
#pragma unroll
                            for (int j = 0; j < 4; ++j) f[2 * j] += bf16x2_lo(res[j]), f[2 * j + 1] += bf16x2_hi(res[j]);
                        }
                        uint32_t o[4];
#pragma unroll
                        for (int j = 0; j < 4; ++j) o[j] = gp_cvt_bf16x2(f[2 * j], f[2 * j + 1]);
                        gp_stmatrix_x4_trans(addr, o);
                    }
                };
                while (true) {
                    dg_tmem_ld_wait();
                    const bool more = tok + 16 < tok1;
                    if (more) {
                        gp_tmem_ld_16x256b_x2(t_acc + (uint32_t)(c0 + tok + 16), &v[1][0]);
                        gp_tmem_ld_16x256b_x2(t_acc + (16u << 16) + (uint32_t)(c0 + tok + 16), &v[1][8]);
                    }
                    put(v[0], tok);
                    tok += 16;
                    if (!more) break;
                    dg_tmem_ld_wait();
                    const bool more2 = tok + 16 < tok1;
                    if (more2) {
                        gp_tmem_ld_16x256b_x2(t_acc + (uint32_t)(c0 + tok + 16), &v[0][0]);
                        gp_tmem_ld_16x256b_x2(t_acc + (16u << 16) + (uint32_t)(c0 + tok + 16), &v[0][8]);
                    }
                    put(v[1], tok);
                    tok += 16;
                    if (!more2) break;
                }
                if (c0 + c_rows == rows) {
                    dg_fence_before();
                    __syncwarp();
                    if (lane == 0) gp_arrive_cluster(acc_empty_leader[set]);
                }
                named_bar_sync(1, ET);
                const int m_chunk = m_base + c0, c_valid = valid - c0 < c_rows ? valid - c0 : c_rows;
                if (W4 && epi == GEMM_EPI_SWIGLU) {
                    const int c8 = tid & 7, n = n0 + 16 * c8;  // 16 interleaved columns -> 8 outputs
                    for (int m = tid >> 3; m < c_valid; m += ET / 8) {
                        if (n >= N) continue;
                        uint32_t o[4];
#pragma unroll
                        for (int j = 0; j < 2; ++j) {
                            uint16_t h[4];
#pragma unroll
                            for (int e = 0; e < 4; ++e) {
                                const uint32_t w = lds32(staging + (uint32_t)(m * GP_STAGING_STRIDE + (c8 >> 1) * 64 + e * 16 + (2 * (c8 & 1) + j) * 4));
                                h[e] = f32_to_bf16_bits(silu_tanh(bf16x2_lo(w)) * bf16x2_hi(w));
                            }
                            o[2 * j] = (uint32_t)h[0] | ((uint32_t)h[1] << 16);
                            o[2 * j + 1] = (uint32_t)h[2] | ((uint32_t)h[3] << 16);
                        }
                        *reinterpret_cast<uint4 *>(C + (size_t)(m_chunk + m) * (N >> 1) + (n >> 1)) = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                } else {
                    const int c16 = tid & 15, n = n0 + 8 * c16;
                    const bool whole = W4 || (N % 8 == 0 && ((size_t)C & 15) == 0);
                    for (int m = tid >> 4; m < c_valid; m += ET / 16) {
                        if (n >= N) continue;
                        uint16_t *out = C + (size_t)(m_chunk + m) * N + n;
                        uint4 v;
                        if (W4) {  // undo dg_lane_column: column 2 e + {0, 1} of the 8 sits in lanes 8 e + 2 (c16 % 4) + {0, 1}
                            const uint32_t a = staging + (uint32_t)(m * GP_STAGING_STRIDE + (c16 >> 2) * 64 + (c16 & 3) * 4);
                            v = make_uint4(lds32(a), lds32(a + 16), lds32(a + 32), lds32(a + 48));
                        } else {
                            v = lds128(staging + (uint32_t)(m * GP_STAGING_STRIDE + c16 * 16));
                        }
                        if (whole) {
                            *reinterpret_cast<uint4 *>(out) = v;
                        } else {
                            const uint32_t vw[4] = {v.x, v.y, v.z, v.w};
                            for (int i = 0; i < 8 && n + i < N; ++i) out[i] = (uint16_t)(vw[i >> 1] >> (16 * (i & 1)));
                        }
                    }
                }
            }
            ++piece;
        }
    }

    dg_fence_before();
    __syncthreads();
    gp_cluster_sync();  // neither CTA leaves while the other may still arrive at its barriers or multiply from its memory
    if (warp == 1) {
        dg_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(tmem_base), "r"(GP_TMEM_COLS) : "memory");
    }
}

// Second pass of a product whose K was cut into S parts: four columns of a token row a thread, the parts' sums in their order, then
// the epilogue (the rounding points of the kernel above).
__global__ void __launch_bounds__(256)
gemm_pair_sum_kernel(const float *__restrict__ parts, int S, uint16_t *__restrict__ C, const uint16_t *__restrict__ R, int epi, int M, int N,
                     int n_pad) {
    pdl_launch_dependents();
    pdl_wait();
    const long long idx = (long long)blockIdx.x * 256 + threadIdx.x;
    const int quads = n_pad >> 2, m = (int)(idx / quads), n = 4 * (int)(idx - (long long)m * quads);
    if (m >= M || n >= N) return;
    const float *src = parts + (size_t)m * n_pad + n;
    float4 v[GP_MAX_PARTS];
#pragma unroll
    for (int s = 0; s < GP_MAX_PARTS; ++s)
        if (s < S) v[s] = __ldcg(reinterpret_cast<const float4 *>(src + (size_t)s * M * n_pad));
    float4 sum = v[0];
#pragma unroll
    for (int s = 1; s < GP_MAX_PARTS; ++s)
        if (s < S) sum.x += v[s].x, sum.y += v[s].y, sum.z += v[s].z, sum.w += v[s].w;
    if (epi == GEMM_EPI_SWIGLU) {  // (N is a multiple of 32)
        *reinterpret_cast<uint32_t *>(C + (size_t)m * (N >> 1) + (n >> 1)) =
            (uint32_t)swiglu_bits(sum.x, sum.y) | ((uint32_t)swiglu_bits(sum.z, sum.w) << 16);
        return;
    }
    uint16_t *out = C + (size_t)m * N + n;
    if (epi == GEMM_EPI_RESIDUAL) {
        const uint2 r = *reinterpret_cast<const uint2 *>(R + (size_t)m * N + n);
        sum.x += bf16x2_lo(r.x), sum.y += bf16x2_hi(r.x), sum.z += bf16x2_lo(r.y), sum.w += bf16x2_hi(r.y);
    }
    const uint2 o = make_uint2(gp_cvt_bf16x2(sum.x, sum.y), gp_cvt_bf16x2(sum.z, sum.w));
    if ((N & 3) == 0 && ((size_t)C & 7) == 0) {
        *reinterpret_cast<uint2 *>(out) = o;
    } else {
        for (int i = 0; i < 4 && n + i < N; ++i) out[i] = (uint16_t)((i < 2 ? o.x : o.y) >> (16 * (i & 1)));
    }
}

// ---------------------------------------------------------------------------------------------
// The cheapest plan for a shape: a pure function of the sizes; the last shapes are remembered, the search takes microseconds.
template <bool W4>
static PairPlan pair_plan(int M, int N, int K, int all_pairs, bool may_split) {
    struct Memo {
        int M = 0, N = 0, K = 0, pairs = 0, split = 0;
        PairPlan plan;
    };
    thread_local Memo memo[64];
    Memo &m = memo[(((unsigned)M * 2654435761u ^ (unsigned)N * 2246822519u ^ (unsigned)K * 3266489917u) >> 27) * 2 + may_split];
    if (m.M != M || m.N != N || m.K != K || m.pairs != all_pairs || m.split != may_split) {
        m.plan = pair_search(W4, M, N, K, all_pairs, may_split);
        m.M = M, m.N = N, m.K = K, m.pairs = all_pairs, m.split = may_split;
    }
    return m.plan;
}

static int pair_count() {
    const int sms = device_sm_count();
    return (sms > 0 ? sms : 148) / 2;
}
// Scratch that lets the plan cut K: 0 where it would not.
template <bool W4>
static size_t pair_workspace_bytes(int M, int K, int N) {
    const PairPlan plan = pair_plan<W4>(M, N, K, pair_count(), true);
    return plan.S > 1 ? pair_parts_bytes(M, N, plan.S) : 0;
}
size_t gemm_pair_workspace_bytes(int M, int K, int N) { return pair_workspace_bytes<true>(M, K, N); }
size_t linear_pair_workspace_bytes(int M, int K, int N) { return pair_workspace_bytes<false>(M, K, N); }

template <bool W4>
static int launch_pair(const uint16_t *A, const void *w, const int32_t *qzeros, const uint16_t *scales, uint16_t *C, int M, int K, int N,
                       cudaStream_t stream, int epilogue, const uint16_t *residual, void *workspace, size_t workspace_bytes) {
    using Cfg = PairCfg<W4>;
    static std::once_flag once;
    static cudaError_t attr_err = cudaSuccess;
    std::call_once(once, [] { attr_err = cudaFuncSetAttribute(gemm_pair_kernel<W4>, cudaFuncAttributeMaxDynamicSharedMemorySize, GP_SMEM_MAX); });
    if (attr_err != cudaSuccess) return check_cuda(attr_err, "pair gemm: shared memory attribute");
    PairPlan plan = pair_plan<W4>(M, N, K, pair_count(), workspace != nullptr);
    if (plan.S > 1 && workspace_bytes < pair_parts_bytes(M, N, plan.S)) plan = pair_plan<W4>(M, N, K, pair_count(), false);
    const PairLayout lay = pair_layout(W4, plan.max_units);
    const size_t smem = 1024 + (size_t)lay.stages * lay.stage_bytes + GP_BAR_BYTES + (size_t)lay.staging_rows * GP_STAGING_STRIDE;
    PairMaps maps;
    int rc;
    for (int u = 1; u <= plan.max_units; ++u)
        if ((rc = encode_tensor_map_2d(&maps.x[u - 1], CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, A, K, M, (uint64_t)K * 2, GP_BK, 16 * u,
                                       CU_TENSOR_MAP_SWIZZLE_128B)))
            return rc;
    if (W4) {
        const int G = K / GP_GROUP, nb = N / 8;
        if ((rc = encode_tensor_map_2d(&maps.w, CU_TENSOR_MAP_DATA_TYPE_INT32, w, nb, K, (uint64_t)nb * 4, GP_HALF / 8, GP_BK,
                                       CU_TENSOR_MAP_SWIZZLE_64B)))
            return rc;
        if ((rc = encode_tensor_map_2d(&maps.s, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, scales, N, G, (uint64_t)N * 2, GP_HALF, 1,
                                       CU_TENSOR_MAP_SWIZZLE_NONE)))
            return rc;
        if ((rc = encode_tensor_map_2d(&maps.z, CU_TENSOR_MAP_DATA_TYPE_INT32, qzeros, nb, G, (uint64_t)nb * 4, GP_HALF / 8, 1,
                                       CU_TENSOR_MAP_SWIZZLE_NONE)))
            return rc;
    } else {
        if ((rc = encode_tensor_map_2d(&maps.w, CU_TENSOR_MAP_DATA_TYPE_BFLOAT16, w, K, N, (uint64_t)K * 2, GP_BK, GP_HALF,
                                       CU_TENSOR_MAP_SWIZZLE_128B)))
            return rc;
    }
    uint16_t *out = plan.S > 1 ? reinterpret_cast<uint16_t *>(workspace) : C;
    const cudaError_t e = launch_pdl(gemm_pair_kernel<W4>, dim3(2 * plan.P * plan.S), dim3(Cfg::THREADS), smem, stream, maps, out, residual,
                                     epilogue, M, N, K, plan, wait_limit_cycles());
    if (e != cudaSuccess || plan.S == 1) return check_cuda(e, "pair gemm launch");
    const int n_pad = plan.C * GP_BN;
    return check_cuda(launch_pdl(gemm_pair_sum_kernel, dim3((unsigned)(((long long)M * (n_pad / 4) + 255) / 256)), dim3(256), 0, stream,
                                 reinterpret_cast<const float *>(workspace), plan.S, C, residual, epilogue, M, N, n_pad),
                      "pair gemm sum launch");
}

bool gemm_pair_supported(int M, int K, int N, int group_size) {
    return group_size == GP_GROUP && K % GP_GROUP == 0 && N % 32 == 0 && M >= 1 && K > 0 && N > 0 && device_is_sm100();
}
int launch_gemm_pair(const uint16_t *A, const int32_t *qweight, const int32_t *qzeros, const uint16_t *scales, uint16_t *C, int M, int K,
                     int N, cudaStream_t stream, int epilogue, const uint16_t *residual, void *workspace, size_t workspace_bytes) {
    return launch_pair<true>(A, qweight, qzeros, scales, C, M, K, N, stream, epilogue, residual, workspace, workspace_bytes);
}
bool linear_pair_supported(int M, int K, int N) { return K % 8 == 0 && M >= 1 && K > 0 && N > 0 && device_is_sm100(); }
int launch_linear_pair(const uint16_t *x, const uint16_t *W, uint16_t *y, int M, int K, int N, cudaStream_t stream, void *workspace,
                       size_t workspace_bytes) {
    return launch_pair<false>(x, W, nullptr, nullptr, y, M, K, N, stream, GEMM_EPI_BF16, nullptr, workspace, workspace_bytes);
}

int gemm_pair_check(cudaStream_t stream) {
    int flag = 0;
    int rc = check_cuda(cudaStreamSynchronize(stream), "gemm_pair_check sync");
    if (rc) return rc;
    rc = check_cuda(cudaMemcpyFromSymbol(&flag, g_gemm_pair_error, sizeof(int)), "gemm_pair_check read");
    if (rc) return rc;
    if (flag != 0) {
        int zero = 0;
        cudaMemcpyToSymbol(g_gemm_pair_error, &zero, sizeof(int));
        return set_error(AWQ_ERR_DEVICE_TIMEOUT,
                         "pair gemm: a device-side wait gave up (role %d: 1 producer, 2/3 MMA issuer, 4 dequant, 5 epilogue)", flag);
    }
    return AWQ_OK;
}

}  // namespace awq
