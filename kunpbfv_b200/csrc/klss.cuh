// The reference's key switch over the auxiliary T base (KLSS), for parity with
// kunpBFV at its own parameter sets:
//   lift of Qj blocks into T   modUpQjtoT_23   include/BasisConv.cuh:86-151
//   lift of Ri blocks into T   modUpPQtoT_23   include/BasisConv.cuh:11-79   (key conversion)
//   external product over T    external_product_T  include/ExternalProduct.cuh:11-112 (key_ip.cuh)
//   exact centred T -> P|Q     modUpTtoPQl_23  include/BasisConv.cuh:159-226
// A block of primes B lifts x mod B into each T prime by approximate CRT with a
// single-precision quotient estimate: rb_j = x_j * (B/b_j)^-1 mod b_j,
// v = (int) sum rb_j / b_j (float division and addition in order),
// out_k = sum rb_j * (B/b_j mod t_k) - v * (B mod t_k) mod t_k.
#pragma once
#include "kernels.cuh"

namespace kbfv {

// reference-order index over P|Q -> row in this library's Q|P order (= prime index)
__host__ __device__ __forceinline__ int ref_to_row(int i, int np, int nq) { return i < np ? nq + i : i - np; }

// Lift blocks into T. which = 0: Qj blocks of a Q polynomial (rows 0..nq-1);
// which = 1: Ri blocks of a Q|P polynomial (rows in Q|P order).
// grid: (N/256, blocks, items); out item layout [block][nt].
// Bound by instruction issue (a Barrett reduction of 128 bits per output), so a
// thread takes two points (the constants' loads and the divisor's conversion
// shared) and is compiled for at most W primes a block: with
// one form for all widths the inactive primes' branches were half of the
// instructions. 15 one-prime blocks of 3 items to 4 T primes at N = 32768: 73 -> 33 us (10 for
// the bytes).
template <int W>
static __global__ void __launch_bounds__(128) klss_block_to_t_kernel(DevConsts c, KlssConsts kc, const uint64_t* __restrict__ in,
                                       uint64_t* __restrict__ out, int which, size_t in_item_stride,
                                       size_t out_item_stride) {
    const size_t k = (size_t)blockIdx.x * 256 + threadIdx.x;
    const int b = blockIdx.y;
    const uint64_t* src = in + blockIdx.z * in_item_stride;
    uint64_t* dst = out + blockIdx.z * out_item_stride + (((size_t)b * kc.nt) << c.logn);
    int width, first;
    const uint64_t *hinv, *hinvs, *hat_t, *mod_t;
    if (which == 0) {
        first = b * c.np;
        width = min(c.np, c.nq - first);
        hinv = kc.qj_hatinv + (size_t)b * c.np;
        hinvs = kc.qj_hatinvs + (size_t)b * c.np;
        hat_t = kc.qj_hat_t + (size_t)b * kc.nt * c.np;
        mod_t = kc.qj_mod_t + (size_t)b * kc.nt;
    } else {
        first = b * kc.gamma;
        width = min(kc.gamma, c.np + c.nq - first);
        hinv = kc.ri_hatinv + (size_t)b * kc.gamma;
        hinvs = kc.ri_hatinvs + (size_t)b * kc.gamma;
        hat_t = kc.ri_hat_t + (size_t)b * kc.nt * kc.gamma;
        mod_t = kc.ri_mod_t + (size_t)b * kc.nt;
    }
    const int stride_hat = which == 0 ? c.np : kc.gamma;
    uint64_t rb[2][W];
    float vv[2] = {0.f, 0.f};
#pragma unroll
    for (int j = 0; j < W; j++) {
        if (j < width) {
            const int row = which == 0 ? first + j : ref_to_row(first + j, c.np, c.nq);
            const uint64_t qj = c.mods[row];  // prime index == row in Q|P order
            const float fq = __ull2float_rn(qj);
            uint64_t x[2];
#pragma unroll
            for (int e = 0; e < 2; e++) x[e] = src[((size_t)row << c.logn) + k + 128 * e];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                rb[e][j] = shoup(x[e], hinv[j], hinvs[j], qj);
                vv[e] = __fadd_rn(vv[e], __fdiv_rn(__ull2float_rn(rb[e][j]), fq));
            }
        }
    }
    const uint64_t vf[2] = {(uint64_t)__float2int_rz(vv[0]), (uint64_t)__float2int_rz(vv[1])};
    for (int t = 0; t < kc.nt; t++) {
        const int pt = c.idx_t + t;
        const uint64_t m = c.mods[pt], mh = c.mu_hi[pt], ml = c.mu_lo[pt], bt = mod_t[t];
        u128 acc[2] = {{0, 0}, {0, 0}};
#pragma unroll
        for (int j = 0; j < W; j++)
            if (j < width) {
                const uint64_t h = hat_t[t * stride_hat + j];
                mac(acc[0], rb[0][j], h);
                mac(acc[1], rb[1][j], h);
            }
        uint64_t y[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            sub128(acc[e], vf[e] * bt);
            y[e] = barrett128(acc[e], m, mh, ml);
        }
#pragma unroll
        for (int e = 0; e < 2; e++) dst[((size_t)t << c.logn) + k + 128 * e] = y[e];
    }
}

// Exact centred T -> P|Q: one polynomial's Ri blocks over T (coefficient form)
// to its P|Q limbs (rows in Q|P order). in: [poly][nri][nt]; out: [poly][npq].
// grid: (N/256, nri, polys); two points a thread and at most NT T primes,
// for the reasons above: 6 polynomials of 4 blocks over 4 T primes to 16 limbs at
// N = 32768: 48 -> 34 us (6 for the bytes).
template <int NT>
static __global__ void __launch_bounds__(128) klss_t_to_pq_kernel(DevConsts c, KlssConsts kc, const uint64_t* __restrict__ in,
                                    uint64_t* __restrict__ out) {
    const size_t k = (size_t)blockIdx.x * 256 + threadIdx.x;
    const int b = blockIdx.y;
    const uint64_t* src = in + (((size_t)blockIdx.z * kc.nri + b) * kc.nt << c.logn);
    uint64_t* dst = out + ((size_t)blockIdx.z * c.npq << c.logn);
    uint64_t rb[2][NT];
    float vv[2] = {0.f, 0.f};
#pragma unroll
    for (int t = 0; t < NT; t++) {
        if (t < kc.nt) {
            const uint64_t tt = c.mods[c.idx_t + t];
            const float ft = __ull2float_rn(tt);
            uint64_t x[2];
#pragma unroll
            for (int e = 0; e < 2; e++) x[e] = src[((size_t)t << c.logn) + k + 128 * e];
#pragma unroll
            for (int e = 0; e < 2; e++) {
                // (x + T/2) mod t_k without reduction, as the reference adds before its Shoup product
                rb[e][t] = shoup(x[e] + kc.halft_t[t], kc.thatinv[t], kc.thatinvs[t], tt);
                vv[e] = __fadd_rn(vv[e], __fdiv_rn(__ull2float_rn(rb[e][t]), ft));
            }
        }
    }
    const uint64_t vf[2] = {(uint64_t)__float2int_rz(vv[0]), (uint64_t)__float2int_rz(vv[1])};
    const int first = b * kc.gamma;
    const int width = min(kc.gamma, c.np + c.nq - first);
    for (int j = 0; j < width; j++) {
        const int m = first + j;                    // reference order
        const int row = ref_to_row(m, c.np, c.nq);  // prime index / output row
        const uint64_t ri = c.mods[row], mh = c.mu_hi[row], ml = c.mu_lo[row], tm = kc.t_pq[m], hm = kc.halft_pq[m];
        u128 acc[2] = {{0, 0}, {0, 0}};
#pragma unroll
        for (int t = 0; t < NT; t++)
            if (t < kc.nt) {
                const uint64_t h = kc.that_pq[(size_t)m * kc.nt + t];
                mac(acc[0], rb[0][t], h);
                mac(acc[1], rb[1][t], h);
            }
        uint64_t y[2];
#pragma unroll
        for (int e = 0; e < 2; e++) {
            sub128(acc[e], vf[e] * tm);
            y[e] = csub(barrett128(acc[e], ri, mh, ml) + ri - hm, ri);
        }
#pragma unroll
        for (int e = 0; e < 2; e++) dst[((size_t)row << c.logn) + k + 128 * e] = y[e];
    }
}

}  // namespace kbfv
