// Transforms of few rows: one row over a cluster of eight CTAs.
//
// A launch of few rows is bound by the multiply pipes of the SMs it reaches: a
// 2^12-point block on one SM takes 9-10 us (7 of them arithmetic; its twiddles in
// shared memory, copied ahead, changed nothing), a 2^13-point one 16 us, and the
// radix-4 column pass with 2^12-point blocks of a 2^14-point row 14 us in two
// launches. Here each CTA holds an eighth of the row, eight points a thread: the
// three stages across the eighths run on columns (forward: the first pass, read
// from global memory, written into the eighths' shared memory; inverse: the
// last pass, read from there), the others inside the CTA. Distributed shared
// memory replaces the second launch and its round trip through L2. Values and
// results are those of the block kernels (ntt.cuh).
//
// The kernels are launched programmatically dependent: they start while the
// kernel before them still runs and wait for it (pdl_wait) before their first
// access to memory that another kernel uses.
#pragma once
#include "ntt.cuh"

namespace kbfv {

__device__ __forceinline__ void pdl_trigger() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void pdl_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }

__device__ __forceinline__ void cluster_arrive() { asm volatile("barrier.cluster.arrive.aligned;" ::: "memory"); }
__device__ __forceinline__ void cluster_wait() { asm volatile("barrier.cluster.wait.aligned;" ::: "memory"); }
__device__ __forceinline__ uint32_t cluster_rank() {
    uint32_t r;
    asm("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// the address of this CTA's shared word `p` in the CTA of rank `rank`
__device__ __forceinline__ uint32_t remote_shared(const uint64_t* p, uint32_t rank) {
    uint32_t a;
    asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(a) : "r"((uint32_t)__cvta_generic_to_shared(p)), "r"(rank));
    return a;
}
__device__ __forceinline__ void remote_store(uint32_t a, uint64_t v) {
    asm volatile("st.shared::cluster.u64 [%0], %1;" ::"r"(a), "l"(v) : "memory");
}
__device__ __forceinline__ uint64_t remote_load(uint32_t a) {
    uint64_t v;
    asm volatile("ld.shared::cluster.u64 %0, [%1];" : "=l"(v) : "r"(a) : "memory");
    return v;
}

constexpr int kClusterLog = 3;  // eight CTAs a row
template <int LOGN>
struct ClusterShape {
    static constexpr int LOGB = LOGN - kClusterLog, NB = 1 << LOGB, THREADS = NB / 8;
    static constexpr int SMEM_BYTES = (NB + NB / 16) * 8;
};

// the twiddles of one register group of R stages, loaded together (before the
// barrier that the group's points wait for)
template <int R>
struct GroupTw {
    tw_t w[(1 << R) - 1];
    __device__ __forceinline__ GroupTw(const tw_t* tw, int s0, int hi) {
#pragma unroll
        for (int u = 0; u < R; u++)
#pragma unroll
            for (int h = 0; h < (1 << u); h++) w[(1 << u) - 1 + h] = __ldg(tw + (1 << (s0 + u)) + (hi << u) + h);
    }
};
template <int R>
__device__ __forceinline__ void fwd_regs(uint64_t (&x)[1 << R], const GroupTw<R>& g, uint64_t q, uint64_t q4) {
#pragma unroll
    for (int u = 0; u < R; u++)
#pragma unroll
        for (int h = 0; h < (1 << u); h++)
#pragma unroll
            for (int k = 0; k < (1 << (R - 1 - u)); k++) {
                const int a = (h << (R - u)) + k;
                ct_bfly(x[a], x[a + (1 << (R - 1 - u))], g.w[(1 << u) - 1 + h], q, q4);
            }
}
// FOLD: the group's first stage is the transform's (n^-1 applied, fully reduced)
template <int R, bool FOLD>
__device__ __forceinline__ void inv_regs(uint64_t (&x)[1 << R], const GroupTw<R>& g, const tw_t* ftw, uint64_t q,
                                         uint64_t q4) {
    const int last = FOLD ? 1 : 0;
#pragma unroll
    for (int u = R - 1; u >= last; u--)
#pragma unroll
        for (int h = 0; h < (1 << u); h++)
#pragma unroll
            for (int k = 0; k < (1 << (R - 1 - u)); k++) {
                const int a = (h << (R - u)) + k;
                gs_bfly(x[a], x[a + (1 << (R - 1 - u))], g.w[(1 << u) - 1 + h], q, q4);
            }
    if (FOLD) {
        const tw_t n0 = __ldg(ftw), n1 = __ldg(ftw + 1);
#pragma unroll
        for (int k = 0; k < (1 << (R - 1)); k++) {
            const uint64_t a = x[k], b = x[k + (1 << (R - 1))];
            x[k] = reduce_from(shoup4(a + b, n0.x, n0.y, q), q, 2);
            x[k + (1 << (R - 1))] = reduce_from(shoup4(a + q4 - b, n1.x, n1.y, q), q, 2);
        }
    }
}

// one pass of R local stages from S0 over the CTA's points: 8 / 2^R groups a thread
template <int LOGN, int S0, int R, bool FWD>
__device__ __forceinline__ void cluster_pass(uint64_t* sm, const tw_t* tw, int t, int blk, uint64_t q, uint64_t q4) {
    constexpr int LOGB = ClusterShape<LOGN>::LOGB, T = ClusterShape<LOGN>::THREADS, G = 1 << R, NG = 8 / G;
    constexpr int lb = LOGB - S0 - R;
    static_assert(NG == 1 || lb == 0, "only the last stages hold several groups per thread");
#pragma unroll
    for (int g = 0; g < NG; g++) {
        const int gi = g * T + t, lbase = ((gi >> lb) << (lb + R)) | (gi & ((1 << lb) - 1));
        const GroupTw<R> w(tw, kClusterLog + S0, ((blk << LOGB) + lbase) >> (LOGB - S0));
        if (g == 0) __syncthreads();
        uint64_t x[G];
#pragma unroll
        for (int k = 0; k < G; k++) x[k] = sm[spad(lbase + (k << lb))];
        if (FWD) fwd_regs<R>(x, w, q, q4);
        else inv_regs<R, false>(x, w, nullptr, q, q4);
#pragma unroll
        for (int k = 0; k < G; k++) sm[spad(lbase + (k << lb))] = x[k];
    }
}
template <int LOGN, int S0>
__device__ __forceinline__ void cluster_fwd_passes(uint64_t* sm, const tw_t* tw, int t, int blk, uint64_t q, uint64_t q4) {
    constexpr int LOGB = ClusterShape<LOGN>::LOGB;
    if constexpr (S0 < LOGB) {
        constexpr int R = LOGB - S0 < 3 ? LOGB - S0 : 3;
        cluster_pass<LOGN, S0, R, true>(sm, tw, t, blk, q, q4);
        cluster_fwd_passes<LOGN, S0 + R>(sm, tw, t, blk, q, q4);
    }
}
template <int LOGN, int S0>
__device__ __forceinline__ void cluster_inv_passes(uint64_t* sm, const tw_t* tw, int t, int blk, uint64_t q, uint64_t q4) {
    constexpr int LOGB = ClusterShape<LOGN>::LOGB;
    if constexpr (S0 < LOGB) {
        constexpr int R = LOGB - S0 < 3 ? LOGB - S0 : 3;
        cluster_inv_passes<LOGN, S0 + R>(sm, tw, t, blk, q, q4);
        cluster_pass<LOGN, S0, R, false>(sm, tw, t, blk, q, q4);
    }
}

// Forward: outputs as ntt_fwd_block_kernel's (FULL: reduced, else below 8q).
template <int LOGN, class Src, class Dst, bool FULL = true>
static __global__ void __launch_bounds__(ClusterShape<LOGN>::THREADS)
ntt_fwd_cluster_kernel(Src src, Dst dst, const tw_t* __restrict__ tw_all, const uint64_t* __restrict__ mods, int row0) {
    constexpr int LOGB = ClusterShape<LOGN>::LOGB, NB = ClusterShape<LOGN>::NB, T = ClusterShape<LOGN>::THREADS;
    extern __shared__ uint64_t sm[];
    cluster_arrive();  // every CTA of the cluster runs before its shared memory is written
    pdl_trigger();
    const int row = row0 + (int)(blockIdx.x >> kClusterLog), blk = (int)cluster_rank(), t = threadIdx.x;
    const RowTab rt = row_tab(src, row, false, tw_all, mods, LOGN);
    const auto s = src.bind(row);
    const uint64_t q = rt.q, q4 = q << 2;
    const int c = blk * T + t;  // the thread's column
    {
        const GroupTw<3> w(rt.tw, 0, 0);
        pdl_wait();
        uint64_t x[8];
        load_points<8>(s, x, [&](int k) { return c + (k << LOGB); });
        fwd_regs<3>(x, w, q, q4);
        cluster_wait();
#pragma unroll
        for (int k = 0; k < 8; k++) remote_store(remote_shared(sm + spad(c), k), x[k]);
    }
    cluster_arrive();
    cluster_wait();
    cluster_fwd_passes<LOGN, 0>(sm, rt.tw, t, blk, q, q4);
    __syncthreads();
    const auto d = dst.bind(row);
    uint64_t v[8];
    int j[8];
#pragma unroll
    for (int k = 0; k < 8; k++) {
        j[k] = t + k * T;
        v[k] = sm[spad(j[k])];
        j[k] += blk * NB;
    }
    if constexpr (has_store_n<decltype(d)>::value) {
        d.template store_n<8>(j, v);
    } else {
#pragma unroll
        for (int k = 0; k < 8; k++) d.store(j[k], FULL ? reduce_from(v[k], q, 3) : v[k]);
    }
}

// Inverse: n^-1 applied, fully reduced.
template <int LOGN, class Src, class Dst>
static __global__ void __launch_bounds__(ClusterShape<LOGN>::THREADS)
ntt_inv_cluster_kernel(Src src, Dst dst, const tw_t* __restrict__ tw_all, const uint64_t* __restrict__ mods, int row0) {
    constexpr int LOGB = ClusterShape<LOGN>::LOGB, NB = ClusterShape<LOGN>::NB, T = ClusterShape<LOGN>::THREADS;
    extern __shared__ uint64_t sm[];
    pdl_trigger();
    const int row = row0 + (int)(blockIdx.x >> kClusterLog), blk = (int)cluster_rank(), t = threadIdx.x;
    const RowTab rt = row_tab(src, row, true, tw_all, mods, LOGN);
    const auto s = src.bind(row);
    const uint64_t q = rt.q, q4 = q << 2;
    pdl_wait();
    {
        uint64_t x[8];
        load_points<8>(s, x, [&](int k) { return blk * NB + t + k * T; });
#pragma unroll
        for (int k = 0; k < 8; k++) sm[spad(t + k * T)] = x[k];
    }
    cluster_inv_passes<LOGN, 0>(sm, rt.tw, t, blk, q, q4);
    const GroupTw<3> w(rt.tw, 0, 0);
    const int c = blk * T + t;
    cluster_arrive();  // all eighths are done
    cluster_wait();
    uint64_t x[8];
#pragma unroll
    for (int k = 0; k < 8; k++) x[k] = remote_load(remote_shared(sm + spad(c), k));
    cluster_arrive();  // no CTA ends while another reads its shared memory
    inv_regs<3, true>(x, w, fold_tab(dst, row, rt.tw), q, q4);
    const auto d = dst.bind(row);
#pragma unroll
    for (int k = 0; k < 8; k++) d.store(c + (k << LOGB), x[k]);
    cluster_wait();
}

}  // namespace kbfv
