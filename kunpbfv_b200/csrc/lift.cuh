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
static __global__ void lift_mma_kernel(Job job, int logn, int alpha, int iters) {
    const MmaPlace pl = mma_place(logn, iters);
    LiftDigit d;
    if (!job.bind(pl.poly, d)) return;
    const int first = pl.c * KS;
    size_t k = pl.k;
    for (int it = 0; it < iters; it++, k += blockDim.x / 2) {
        uint64_t w[2][KS];
        float x0[KS], x1[KS];
#pragma unroll
        for (int s = 0; s < KS; s++) {
            w[0][s] = w[1][s] = 0;
            x0[s] = x1[s] = 0.f;
            if (first + s < d.n) {
                const ulonglong2 v =
                    *reinterpret_cast<const ulonglong2*>(d.rows + ((size_t)(d.lo + first + s) << logn) + k);
                lift_word(d, first + s, v, w[0][s], w[1][s], x0[s], x1[s]);
            }
        }
        lift_outputs<KS>(w, x0, x1, d, logn, alpha, first, k, pl);
    }
}

template <int KS, class Job>
static void lift_mma_launch(const Job& job, int rows, int logn, int alpha, int threads, cudaStream_t st) {
    static int res[4] = {0, 0, 0, 0};
    const int iters =
        mma_iters(rows, logn, threads, resident_ctas_at((const void*)lift_mma_kernel<KS, Job>, threads, 0, res));
    const size_t per = ((size_t)1 << logn) / ((size_t)(threads / 2) * iters);
    lift_mma_kernel<KS, Job><<<(unsigned)(rows * per), threads, 0, st>>>(job, logn, alpha, iters);
    check_launch("digit_lift");
}
template <class Job>
static void lift_launch_any(const Job& job, int rows, int logn, int alpha, int threads, cudaStream_t st) {
    switch (lift_steps(alpha)) {
        case 1: lift_mma_launch<1>(job, rows, logn, alpha, threads, st); break;
        case 2: lift_mma_launch<2>(job, rows, logn, alpha, threads, st); break;
        case 4: lift_mma_launch<4>(job, rows, logn, alpha, threads, st); break;
        case 6: lift_mma_launch<6>(job, rows, logn, alpha, threads, st); break;
        default: lift_mma_launch<10>(job, rows, logn, alpha, threads, st); break;
    }
}
