// Products of RNS residues with a constant matrix on the int8 tensor cores.
//
// The base conversions of the multiply are contractions: every coefficient's
// nin residues times a fixed [nin][nout] matrix of residues mod the output
// primes. A 64-bit word w is the sum of its bytes w_b 2^(8b), so
//   sum_i w_i c_ij  =  sum_{i,b} w_{i,b} [2^(8b) c_ij mod m_j]   (mod m_j):
// with the bytes of all words as the inner dimension and the eight base-256
// digits of the constants as columns, one u8 matrix product gives, per output,
// eight 32-bit digit sums whose weighted sum is below 2^77 (60-bit constants,
// at most 36 words), and one 17-bit quotient reduces it. Against 64-bit
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
// tensor time is hidden under the loads: the kernels run at HBM / issue rate.
//
// Lane c holds the contiguous words c KS .. c KS + KS - 1 of a KS-step product
// and the outputs c 2NG .. c 2NG + 2NG - 1 of an NG-group one (group G: outputs
// 2G, 2G + 1 of those), so floating-point sums over the words in index order
// pass through the quad's lanes once.
#pragma once
#include <cstdint>

#include "arith.cuh"

namespace kbfv {

// Per output: the negated modulus 2^64 - m' with m' = m << sh in [2^59, 2^60)
// (the constants are scaled alike), ((-B mod m) << sh) for the quotient term
// v * B that a base extension subtracts, floor(2^91 / m') and sh.
struct MmaOut {
    uint64_t nm, nb;
    uint32_t mu, sh;
    uint64_t pad;
};
static_assert(sizeof(MmaOut) == 32, "two 16-byte loads");

// steps (of 4 words) of a table for `words` words and column groups for `nout` outputs
__host__ __device__ constexpr int mma_groups(int nout) { return (nout + 7) / 8; }
// table layout: MmaOut[8 ng], then uint4[ng][ks][4][32] (two digit tiles per entry)
__host__ __device__ constexpr size_t mma_table_bytes(int ks, int ng) {
    return (size_t)ng * 8 * sizeof(MmaOut) + (size_t)ng * ks * 4 * 32 * 16;
}
// The step count of a parameter set of nq ciphertext primes: 4 KS words hold
// the nq residues and one more (the scale-and-round's quotient), and 2 NG =
// 2 ceil(KS / 2) words a lane hold the nq + 1 residues over R.
__host__ __device__ constexpr int mma_steps(int nq) { return nq <= 3 ? 1 : nq <= 7 ? 2 : nq <= 15 ? 4 : nq <= 23 ? 6 : 9; }
__host__ __device__ constexpr int mma_r_groups(int ks) { return (ks + 1) / 2; }

// steps of the lift of digits of alpha primes (alpha <= 32); for one digit of
// all nq primes mostly the steps of the product R -> Q, whose outputs are then
// the lift's words
constexpr int lift_steps(int alpha) { return alpha <= 4 ? 1 : alpha <= 8 ? 2 : alpha <= 16 ? 4 : alpha <= 24 ? 6 : 10; }

struct MmaTab {
    const MmaOut* out;
    const uint4* b;
    int ng;
};
__host__ __device__ inline MmaTab mma_tab(const void* p, int ng) {
    return MmaTab{(const MmaOut*)p, (const uint4*)((const uint8_t*)p + (size_t)ng * 8 * sizeof(MmaOut)), ng};
}

__device__ __forceinline__ void imma(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                     uint32_t b1) {
    asm("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
        : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}

// digit sums of output group G: S[t][2 * row + e] is digit t of output (G, e)
// of the lane's coefficient `row`
template <int KS>
__device__ __forceinline__ void mma_digits(int (&S)[8][4], const uint64_t (&w)[2][KS], const MmaTab& tab, int G,
                                           int lane) {
#pragma unroll
    for (int t = 0; t < 8; t++)
#pragma unroll
        for (int i = 0; i < 4; i++) S[t][i] = 0;
    const uint4* b = tab.b + (size_t)G * KS * 128 + lane;
#pragma unroll
    for (int s = 0; s < KS; s++) {
        const uint32_t a0 = (uint32_t)w[0][s], a1 = (uint32_t)w[1][s], a2 = (uint32_t)(w[0][s] >> 32),
                       a3 = (uint32_t)(w[1][s] >> 32);
#pragma unroll
        for (int h = 0; h < 4; h++) {
            const uint4 f = __ldg(b + (s * 4 + h) * 32);
            imma(S[2 * h], a0, a1, a2, a3, f.x, f.y);
            imma(S[2 * h + 1], a0, a1, a2, a3, f.z, f.w);
        }
    }
}

// sum_t S_t 2^(8t) + v * nb + (add << sh) mod m, fully reduced. The sum has 96
// bits (w0, hi): the digit sums stay below 2^24, so S_t + (S_{t+1} << 8) fits
// 32 bits, and the two middle additions do not leave 64. The quotient's 32-bit
// estimate (the sum's bits 45..76 times floor(2^91 / m')) is low by at most 1.
template <bool ADD>
__device__ __forceinline__ uint64_t mma_reduce(int s0, int s1, int s2, int s3, int s4, int s5, int s6, int s7,
                                               uint32_t v, uint64_t add, const MmaOut& o) {
    const uint32_t d0 = (uint32_t)s0 + ((uint32_t)s1 << 8), d1 = (uint32_t)s2 + ((uint32_t)s3 << 8);
    const uint32_t d2 = (uint32_t)s4 + ((uint32_t)s5 << 8), d3 = (uint32_t)s6 + ((uint32_t)s7 << 8);
    uint64_t lo = (((uint64_t)d2 << 32) | d0) + ((uint64_t)d1 << 16);
    lo += (uint64_t)v * (uint32_t)o.nb;
    uint64_t hi = (lo >> 32) + ((uint64_t)d3 << 16);
    hi += (uint64_t)v * (uint32_t)(o.nb >> 32);
    uint32_t w0 = (uint32_t)lo;
    if (ADD) {
        const uint64_t a = add << o.sh;
        const uint64_t t = (uint64_t)w0 + (uint32_t)a;
        w0 = (uint32_t)t;
        hi += (a >> 32) + (t >> 32);
    }
    const uint32_t est = __umulhi((uint32_t)(hi >> 13), o.mu) >> 14;
    const uint64_t r = ((hi << 32) | w0) + (uint64_t)est * o.nm;
    const int64_t t = (int64_t)(r + o.nm);
    return (t < 0 ? r : (uint64_t)t) >> o.sh;
}
template <bool ADD>
__device__ __forceinline__ uint64_t mma_value(const int (&S)[8][4], int i, uint32_t v, uint64_t add, const MmaOut& o) {
    return mma_reduce<ADD>(S[0][i], S[1][i], S[2][i], S[3][i], S[4][i], S[5][i], S[6][i], S[7][i], v, add, o);
}

__device__ __forceinline__ MmaOut mma_out(const MmaOut* p) {
    const ulonglong2 x = __ldg((const ulonglong2*)p);
    const uint2 y = __ldg((const uint2*)p + 2);
    return MmaOut{x.x, x.y, y.x, y.y, 0};
}

// __ull2double_rn from two exact halves and one rounded addition (the
// conversion instruction issues at a quarter of the FP64 rate)
__device__ __forceinline__ double u64_to_double(uint64_t x) {
    const double hi = __hiloint2double(0x45300000, (int)(uint32_t)(x >> 32));  // 2^84 + hi32 * 2^32
    const double lo = __hiloint2double(0x43300000, (int)(uint32_t)x);          // 2^52 + lo32
    return __dadd_rn(__dsub_rn(hi, 19342813118337666422669312.0), lo);         // 2^84 + 2^52
}

// acc = fma(w_i, f_i, acc) for i = 0 .. n-1 in index order, from `init`, where
// lane c of each quad holds words c KS .. c KS + KS - 1 and their factors: the
// partial sum visits the lanes in order (lane c's turn is hop c), the last
// lane's is broadcast.
template <int KS>
__device__ __forceinline__ double quad_fma_sum(const double (&x)[KS], const double (&f)[KS], double init, int first,
                                               int n) {
    double acc = init;
#pragma unroll
    for (int hop = 0; hop < 4; hop++) {
#pragma unroll
        for (int s = 0; s < KS; s++)
            if (first + s < n) acc = __fma_rn(x[s], f[s], acc);
        if (hop < 3) acc = __shfl_up_sync(0xffffffffu, acc, 1, 4);
    }
    return __shfl_sync(0xffffffffu, acc, 3, 4);
}

}  // namespace kbfv
