// The key-switch digit lift as a kernel of its own (lift_word, lift_outputs in
// k5_kernels.cuh). The digit's own limbs are read from their places in the digits' layout
// ([item][digit][Q|P]), where the stage before (K5, or the inverse transform of a
// key switch's input) stores them.
#pragma once
#include "k5_kernels.cuh"

struct LiftJob {
    DevConsts c;
    uint64_t* sd2;
    __device__ __forceinline__ bool bind(int row, LiftDigit& d) const {
        const int item = row / c.dnum, g = row % c.dnum;
        d.lo = g * c.alpha;
        d.n = max(0, min(c.alpha, c.nq - d.lo));  // 0: more digits than primes need
        d.nout = c.npq - d.n;
        d.rows = sd2 + ((size_t)row * c.npq << c.logn);
        d.tab = mma_tab((const uint8_t*)c.mm_lift + (size_t)g * c.mm_lift_stride, mma_groups(d.nout));
        d.mods = c.mods + d.lo;
        d.hatinv = c.dig_hatinv + d.lo;
        d.hatinvs = c.dig_hatinvs + d.lo;
        return true;
    }
};
// a mixed-level batch: rows (item, top level's digits); a level's missing digits are skipped
struct MixedLiftJob {
    Groups G;
    uint64_t* sd2;
    __device__ __forceinline__ bool bind(int row, LiftDigit& d) const {
        const int item = row / G.top_dnum, g = row % G.top_dnum, gr = G.group_of_item(item);
        if (g >= G.dnum[gr]) return false;
        const DevConsts* lv = G.lv[gr];
        d.lo = g * lv->alpha;
        d.n = max(0, min(lv->alpha, lv->nq - d.lo));
        d.nout = lv->npq - d.n;
        d.rows = sd2 + (((size_t)item * G.top_dnum * G.top_npq + (size_t)g * lv->npq) << G.logn);
        d.tab = mma_tab((const uint8_t*)lv->mm_lift + (size_t)g * lv->mm_lift_stride, mma_groups(d.nout));
        d.mods = lv->mods + d.lo;
        d.hatinv = lv->dig_hatinv + d.lo;
        d.hatinvs = lv->dig_hatinvs + d.lo;
        return true;
    }
};

template <int KS, class Job>
static __global__ void __launch_bounds__(256) lift_mma_kernel(Job job, int logn, int alpha, int iters, int stage) {
    constexpr int MT = mma_tiles(KS);
    const MmaPlace pl = mma_place<MT>(logn, iters);
    extern __shared__ uint4 mma_sh[];
    LiftDigit d;
    if (!job.bind(pl.poly, d)) return;  // the whole CTA
    if (stage) {
        mma_stage(mma_sh, d.tab, KS);
        __syncthreads();
    }
    const int first = pl.c * KS;
    size_t k = pl.k;
    for (int it = 0; it < iters; it++, k += pl.each) {
        uint64_t w[MT][2][KS];
        float t[MT][2][KS];
#pragma unroll
        for (int s = 0; s < KS; s++) {
#pragma unroll
            for (int m = 0; m < MT; m++) {
                w[m][0][s] = w[m][1][s] = 0;
                t[m][0][s] = t[m][1][s] = 0.f;
                if (first + s < d.n) {
                    const ulonglong2 x = load2(d.rows + ((size_t)(d.lo + first + s) << logn) + k + 16 * m);
                    w[m][0][s] = x.x;
                    w[m][1][s] = x.y;
                }
            }
        }
#pragma unroll
        for (int s = 0; s < KS; s++)
            if (first + s < d.n)
#pragma unroll
                for (int m = 0; m < MT; m++)
#pragma unroll
                    for (int r = 0; r < 2; r++) lift_word(d, first + s, w[m][r][s], w[m][r][s], t[m][r][s]);
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int r = 0; r < 2; r++) {
                const uint32_t v = lift_quotient<KS>(t[m][r], first, d.n, alpha);
#pragma unroll
                for (int s = 0; s < KS; s++)
                    if (first + s == d.n) w[m][r][s] = v;
            }
        if (stage) lift_outputs<KS, MT>(w, d, mma_tab(mma_sh, d.tab.ng), logn, k, pl);
        else lift_outputs<KS, MT>(w, d, d.tab, logn, k, pl);
    }
}

template <int KS, class Job>
static void lift_mma_launch(const Job& job, size_t table, int rows, int logn, int alpha, int threads, cudaStream_t st) {
    const int each = threads / 2 * mma_tiles(KS);
    constexpr int kStaged = 16 << 10;  // larger tables are read through L1
    const int smem = table <= kStaged ? (int)table : 0;
    // resident CTAs with the largest staged table (registers bound them before that) and with none
    static int res[2][4] = {};
    const int iters = mma_iters(rows, logn, each, resident_ctas_at((const void*)lift_mma_kernel<KS, Job>, threads,
                                                                    smem ? kStaged : 0, res[smem ? 1 : 0]));
    lift_mma_kernel<KS, Job><<<mma_blocks(rows, logn, each, iters), threads, smem, st>>>(job, logn, alpha, iters, smem != 0);
    check_launch("digit_lift");
}
template <class Job>
static void lift_launch_any(const Job& job, size_t table, int rows, int logn, int alpha, int threads, cudaStream_t st) {
    switch (lift_steps(alpha)) {
        case 1: lift_mma_launch<1>(job, table, rows, logn, alpha, threads, st); break;
        case 2: lift_mma_launch<2>(job, table, rows, logn, alpha, threads, st); break;
        case 4: lift_mma_launch<4>(job, table, rows, logn, alpha, threads, st); break;
        case 6: lift_mma_launch<6>(job, table, rows, logn, alpha, threads, st); break;
        default: lift_mma_launch<10>(job, table, rows, logn, alpha, threads, st); break;
    }
}
