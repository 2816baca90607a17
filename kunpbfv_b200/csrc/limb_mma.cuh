// Products of RNS residues with a constant matrix on the int8 tensor cores.
//
// The base conversions of the multiply are contractions: every coefficient's
// nin residues times a fixed [nin][nout] matrix of residues mod the output
// primes. A 64-bit word w is the sum of its bytes w_b 2^(8b), so
//   sum_i w_i c_ij  =  sum_{i,b} w_{i,b} [2^(8b) c_ij mod m_j]   (mod m_j):
// with the bytes of all words as the inner dimension and the eight base-256
// digits of the constants as columns, one u8 matrix product gives, per output,
// eight 24-bit digit sums whose weighted sum is below 2^77 (60-bit constants;
// at most 35 words below 2^60 and a rounding quotient of any 64 bits), and one 17-bit
// quotient reduces it. Against 64-bit
// multiply-accumulates into 128 bits and a 128-bit Barrett reduction that is
// about a third of the multiply-pipe work of a conversion (8 MACs of eight
// 32-bit products each and four high products per output become one wide, one
// low and one high 32-bit product), and the MACs move to a unit that is idle
// otherwise: mma.sync m16n8k32 u8 runs at 5.7e14 MAC/s on the B200, 4096 MACs
// for a coefficient with 8 words and 8 outputs.
//
// mma.sync rather than tcgen05: its fragments are the kernel's own registers.
// A tile is 16 coefficients x 32 bytes = 4 words; the row fragment of lane
// (g = lane / 4, c = lane % 4) is the low and the high half of word
// (step s, c) of coefficients 2g and 2g + 1, i.e. the words as they are loaded
// (16 bytes a lane, whole 128-byte lines), with no packing. A column tile
// holds one digit of eight outputs, so a lane's accumulators over the eight
// digit tiles are all the digits of two outputs of its two coefficients, and
// an output is a word of the next product in the same lane: chained
// conversions (scale-and-round, then R -> Q) never leave the registers. The
// tensor pipe is a fifth busy; the kernels are bound by instruction issue.
//
// Lane c holds the contiguous words c KS .. c KS + KS - 1 of a KS-step product
// and the outputs c 2NG .. c 2NG + 2NG - 1 of an NG-group one (group G: outputs
// 2G, 2G + 1 of those). Floating-point sums over a coefficient's words run in index
// order on one lane per coefficient, which reads the words again (from L1, or
// through shared memory where they are a product's outputs): passing partial
// sums around the quads took 28% of K2's instructions.
#pragma once
#include <cstdint>

#include "arith.cuh"

namespace kbfv {

// Per output: the negated modulus 2^64 - m' with m' = m << sh in [2^59, 2^60)
// (the constants are scaled alike), floor(2^91 / m') and sh.
struct MmaOut {
    uint64_t nm;
    uint32_t mu, sh;
};
static_assert(sizeof(MmaOut) == 16, "one 16-byte load");

// steps (of 4 words) of a table for `words` words and column groups for `nout` outputs
__host__ __device__ constexpr int mma_groups(int nout) { return (nout + 7) / 8; }
// table layout: MmaOut[8 ng], then uint4[ng][ks][4][32] (two digit tiles per entry)
__host__ __device__ constexpr size_t mma_table_bytes(int ks, int ng) {
    return (size_t)ng * 8 * sizeof(MmaOut) + (size_t)ng * ks * 4 * 32 * 16;
}
// The quotient v of a base extension (out = sum_i y_i c_ij - v B) is one more word
// of the product, with the constant -B mod m_j: subtracting it after the
// reduction took a third of the epilogue.
// The step count of a parameter set of nq ciphertext primes: 4 KS words hold
// the nq residues and one more (the scale-and-round's or the base extension's
// quotient), and 2 NG = 2 ceil(KS / 2) words a lane hold the nq + 1 residues over
// R; their quotient takes a step of its own (2 NG + 1 steps).
__host__ __device__ constexpr int mma_steps(int nq) { return nq <= 3 ? 1 : nq <= 7 ? 2 : nq <= 15 ? 4 : nq <= 23 ? 6 : 9; }
__host__ __device__ constexpr int mma_r_groups(int ks) { return (ks + 1) / 2; }

// steps of the lift of digits of alpha primes and the quotient (alpha <= 32);
// for one digit of nq >= 4 primes as many as there are lane words of the product
// R -> Q's outputs, which are then the lift's words
constexpr int lift_steps(int alpha) { return alpha <= 3 ? 1 : alpha <= 7 ? 2 : alpha <= 15 ? 4 : alpha <= 23 ? 6 : 10; }

struct MmaTab {
    const MmaOut* out;
    const uint4* b;
    int ng;
};
__host__ __device__ inline MmaTab mma_tab(const void* p, int ng) {
    return MmaTab{(const MmaOut*)p, (const uint4*)((const uint8_t*)p + (size_t)ng * 8 * sizeof(MmaOut)), ng};
}

// a table copied to shared memory by the CTA (the caller synchronises)
__device__ __forceinline__ void mma_stage(uint4* dst, const MmaTab& t, int ks) {
    const uint4* src = (const uint4*)t.out;
    const int n = (int)(mma_table_bytes(ks, t.ng) / 16);
    for (int i = threadIdx.x; i < n; i += blockDim.x) dst[i] = __ldg(src + i);
}

// c = a * b, and c += a * b
__device__ __forceinline__ void imma_first(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                           uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%10,%10,%10};"
        : "=r"(c[0]), "=r"(c[1]), "=r"(c[2]), "=r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "r"(0));
}
__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                     uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// Digit sums of output group G for MT tiles of 16 coefficients: D[m][h][2 * row
// + e] is digit 2h + 256 * digit 2h + 1 of output (G, e) of the lane's
// coefficient `row` of tile m. A pair of digit tiles is combined as soon as it is
// summed (35 words below 2^60, their top byte below 16, and one full word
// keep the digit sums below 2^24, so the pair fits 32 bits), which keeps
// 16 instead of 32 registers of sums per tile, and one load of the constants
// (tab: in shared memory) serves MT tiles.
template <int KS, int MT>
__device__ __forceinline__ void mma_digits(uint32_t (&D)[MT][4][4], const uint64_t (&w)[MT][2][KS], const MmaTab& tab,
                                           int G, int lane) {
    const uint4* b = tab.b + (size_t)G * KS * 128 + lane;
#pragma unroll
    for (int h = 0; h < 4; h++) {
        int S[MT][2][4];
#pragma unroll
        for (int s = 0; s < KS; s++) {
            const uint4 f = b[(s * 4 + h) * 32];
#pragma unroll
            for (int m = 0; m < MT; m++) {
                const uint32_t a0 = (uint32_t)w[m][0][s], a1 = (uint32_t)w[m][1][s],
                               a2 = (uint32_t)(w[m][0][s] >> 32), a3 = (uint32_t)(w[m][1][s] >> 32);
                if (s == 0) {
                    imma_first(S[m][0], a0, a1, a2, a3, f.x, f.y);
                    imma_first(S[m][1], a0, a1, a2, a3, f.z, f.w);
                } else {
                    imma(S[m][0], a0, a1, a2, a3, f.x, f.y);
                    imma(S[m][1], a0, a1, a2, a3, f.z, f.w);
                }
            }
        }
#pragma unroll
        for (int m = 0; m < MT; m++)
#pragma unroll
            for (int i = 0; i < 4; i++) D[m][h][i] = (uint32_t)S[m][0][i] + ((uint32_t)S[m][1][i] << 8);
    }
}

// sum_h D_h 2^(16h) + (add << sh) mod m, fully reduced. The sum has 96 bits (w2,
// w1, w0); the middle word's first addition does not overflow. The quotient's
// 32-bit estimate (the sum's bits 45..76 times floor(2^91 / m')) is low by at
// most 1. ADD: there is a term add; SH: some output of the table has fewer than
// 60 bits (sh != 0). In 32-bit words with carries: the 64-bit form cost 28
// multiply-pipe instructions per value (register-pair moves) instead of 6.
template <bool ADD, bool SH>
__device__ __forceinline__ uint64_t mma_value(const uint32_t (&D)[4][4], int i, uint64_t add, const MmaOut& o) {
    uint32_t w0, w1, w2;
    asm("{\n\t.reg .u32 a, b, c;\n\t"
        "shl.b32 a, %4, 16;\n\tshr.u32 b, %4, 16;\n\tshl.b32 c, %6, 16;\n\tshr.u32 %2, %6, 16;\n\t"
        "add.cc.u32 %0, %3, a;\n\taddc.u32 %1, %5, b;\n\t"
        "add.cc.u32 %1, %1, c;\n\taddc.u32 %2, %2, 0;\n\t}"
        : "=&r"(w0), "=&r"(w1), "=&r"(w2)
        : "r"(D[0][i]), "r"(D[1][i]), "r"(D[2][i]), "r"(D[3][i]));
    if (ADD) {
        const uint64_t a = SH ? add << o.sh : add;
        asm("add.cc.u32 %0, %0, %3;\n\taddc.cc.u32 %1, %1, %4;\n\taddc.u32 %2, %2, 0;"
            : "+r"(w0), "+r"(w1), "+r"(w2)
            : "r"((uint32_t)a), "r"((uint32_t)(a >> 32)));
    }
    const uint32_t est = __umulhi(__funnelshift_r(w1, w2, 13), o.mu) >> 14;
    uint64_t r = ((uint64_t)w1 << 32) | w0;
    asm("mad.wide.u32 %0, %1, %2, %0;" : "+l"(r) : "r"(est), "r"((uint32_t)o.nm));
    r += (uint64_t)(est * (uint32_t)(o.nm >> 32)) << 32;
    const int64_t t = (int64_t)(r + o.nm);
    const uint64_t x = t < 0 ? r : (uint64_t)t;
    return SH ? x >> o.sh : x;
}

__device__ __forceinline__ MmaOut mma_out(const MmaOut* p) {
    const uint4 x = *(const uint4*)p;
    return MmaOut{((uint64_t)x.y << 32) | x.x, x.z, x.w};
}

// llround of 0 <= x < 2^31: the addition of 2^52 rounds to an integer, ties to
// even; a tie that went down goes up
__device__ __forceinline__ uint32_t round_half_up(double x) {
    const double t = __dadd_rn(x, 4503599627370496.0);
    const double r = __dsub_rn(t, 4503599627370496.0);
    return (uint32_t)__double2loint(t) + (__dsub_rn(x, r) == 0.5 ? 1u : 0u);
}

}  // namespace kbfv
