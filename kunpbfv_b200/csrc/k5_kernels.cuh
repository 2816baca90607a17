// The per-coefficient stages of the multiply pipeline as byte matrix products
// (limb_mma.cuh): K2 (base extension Q -> R), K5 (t/Q scale-and-round Q|R -> R
// and the base extension R -> Q, chained in registers) and the key-switch
// digit lift; and K3 with the Q -> R base extension in its loader
// (q2r_ntt.cuh). Each size of the prime count is instantiated in its own
// translation unit (k5_m<MAXQ>.cu) so that the unrolled variants compile in
// parallel.
//
// A warp takes 16 coefficients of one polynomial per iteration: lane
// (g = lane / 4, c = lane % 4) coefficients 2g and 2g + 1, the words and outputs
// of limb_mma.cuh. A CTA's iterations take consecutive runs of coefficients.
//
// The figures at the kernels are of N = 16384, 7 + 1 primes, 32 pairs (2^21
// coefficients in K2, 1.5 x 2^20 in K5), one launch under ncu, against the same
// stages from 64-bit multiply-accumulates and 128-bit Barrett reductions.
#pragma once
#include "limb_mma.cuh"
#include "mixed.cuh"
#include "q2r_ntt.cuh"

// iterations of a CTA of `threads` threads (threads / 2 coefficients each): as
// few as leave four waves of CTAs, so that small launches cover the SMs and
// large ones load the constants of a lane (held in registers across the
// iterations) rarely
static inline int mma_iters(size_t polys, int logn, int threads, int resident) {
    const size_t per = ((size_t)1 << logn) / (threads / 2);  // iterations that one polynomial takes (a power of two)
    size_t it = 1;
    while (it < per && it < 16 && polys * per / (2 * it) >= (size_t)4 * resident) it *= 2;
    return (int)it;
}

// the CTA's polynomial and first coefficient, the warp's place in an iteration
struct MmaPlace {
    int poly;
    size_t k;    // coefficient of the lane's row 0 in iteration 0
    int lane, c;
};
__device__ __forceinline__ MmaPlace mma_place(int logn, int iters) {
    const unsigned per = (1u << logn) / ((blockDim.x / 2) * iters);
    const int lane = threadIdx.x & 31;
    return MmaPlace{(int)(blockIdx.x / per),
                    (size_t)(blockIdx.x % per) * (blockDim.x / 2) * iters + (threadIdx.x >> 5) * 16 + 2 * (lane >> 2),
                    lane, lane & 3};
}

// ---------------------------------------------------------------------------
// base extension of words y_i = [x_i (B/b_i)^-1]_{b_i} (PREP: of the residues
// x_i): out_j = sum_i y_i (B/b_i) - v B mod m_j, v = round(sum_i y_i / b_i),
// the floating-point sum in index order (BaseConverter::bConv_HPS,
// include/BasisConv_QR.cuh:191-207; include/poly_arithmetic.cuh:1078-1178)
// ---------------------------------------------------------------------------
struct ExtPoly {
    const uint64_t* in;
    uint64_t* out;
    MmaTab tab;
    const double* binv;
    int nin, nout;
    const uint64_t *hatinv, *hatinvs, *mods;  // PREP only
};
struct ExtJob {
    const uint64_t* in;
    uint64_t* out;
    size_t in_stride, out_stride;
    ExtPoly p;
    __device__ __forceinline__ ExtPoly bind(int poly) const {
        ExtPoly e = p;
        e.in = in + poly * in_stride;
        e.out = out + poly * out_stride;
        return e;
    }
};
// K2 of a mixed-level batch: polynomials (item, 4), each with its level's tables
template <int NG>
struct MixedExtJob {
    Groups G;
    const uint64_t* sa;
    uint64_t* sb;
    __device__ __forceinline__ ExtPoly bind(int poly) const {
        const int item = poly / 4, w = poly % 4, g = G.group_of_item(item);
        const DevConsts* lv = G.lv[g];
        ExtPoly e{};
        e.in = sa + (((size_t)item * 4 * G.top_nq + (size_t)w * G.nq[g]) << G.logn);
        e.out = sb + (((size_t)item * 4 * G.top_nr + (size_t)w * G.nr[g]) << G.logn);
        e.tab = mma_tab(lv->mm_q2r, NG);
        e.binv = lv->q2r_inv;
        e.nin = G.nq[g];
        e.nout = G.nr[g];
        return e;
    }
};

// K2, 32 pairs: 179 us with 64-bit multiply-accumulates -> 87 us here
template <int KS, int NG, bool PREP, class Job>
static __global__ void ext_mma_kernel(Job job, int logn, int iters) {
    const MmaPlace pl = mma_place(logn, iters);
    const ExtPoly e = job.bind(pl.poly);
    const int first = pl.c * KS;
    double f[KS];
    MmaOut o[2 * NG];
#pragma unroll
    for (int s = 0; s < KS; s++) f[s] = first + s < e.nin ? e.binv[first + s] : 0.0;
#pragma unroll
    for (int i = 0; i < 2 * NG; i++)
        if (NG <= 2) o[i] = mma_out(e.tab.out + pl.c * 2 * NG + i);
    size_t k = pl.k;
    for (int it = 0; it < iters; it++, k += blockDim.x / 2) {
        uint64_t w[2][KS];
        double x0[KS], x1[KS];
#pragma unroll
        for (int s = 0; s < KS; s++) {
            ulonglong2 v = make_ulonglong2(0, 0);
            if (first + s < e.nin) {
                v = *reinterpret_cast<const ulonglong2*>(e.in + ((size_t)(first + s) << logn) + k);
                if (PREP) {
                    const uint64_t h = e.hatinv[first + s], hs = e.hatinvs[first + s], m = e.mods[first + s];
                    v.x = shoup(v.x, h, hs, m);
                    v.y = shoup(v.y, h, hs, m);
                }
            }
            w[0][s] = v.x;
            w[1][s] = v.y;
        }
#pragma unroll
        for (int s = 0; s < KS; s++) {
            x0[s] = u64_to_double(w[0][s]);
            x1[s] = u64_to_double(w[1][s]);
        }
        const uint32_t v0 = (uint32_t)llround(quad_fma_sum<KS>(x0, f, 0.0, first, e.nin));
        const uint32_t v1 = (uint32_t)llround(quad_fma_sum<KS>(x1, f, 0.0, first, e.nin));
#pragma unroll
        for (int G = 0; G < NG; G++) {
            int S[8][4];
            mma_digits<KS>(S, w, e.tab, G, pl.lane);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int j = pl.c * 2 * NG + 2 * G + i;
                if (j >= e.nout) continue;
                const MmaOut oo = NG <= 2 ? o[2 * G + i] : mma_out(e.tab.out + j);
                ulonglong2 r;
                r.x = mma_value<false>(S, i, v0, 0, oo);
                r.y = mma_value<false>(S, 2 + i, v1, 0, oo);
                *reinterpret_cast<ulonglong2*>(e.out + ((size_t)j << logn) + k) = r;
            }
        }
    }
}

template <int KS, int NG, bool PREP, class Job>
static void ext_mma_launch(const Job& job, int polys, int logn, int threads, cudaStream_t st) {
    if (polys <= 0) return;
    static int res[4] = {0, 0, 0, 0};
    const int iters = mma_iters(polys, logn, threads,
                                resident_ctas_at((const void*)ext_mma_kernel<KS, NG, PREP, Job>, threads, 0, res));
    const size_t per = ((size_t)1 << logn) / ((size_t)(threads / 2) * iters);
    ext_mma_kernel<KS, NG, PREP, Job><<<(unsigned)(polys * per), threads, 0, st>>>(job, logn, iters);
    check_launch("base_extension");
}

// K2: y rows over Q (QHatRowsIO layout) -> R limbs of `polys` polynomials
template <int KS>
void k2_launch_m(const DevConsts& dc, const uint64_t* y, uint64_t* out, int polys, cudaStream_t st) {
    constexpr int NG = mma_r_groups(KS);
    ExtJob job{y, out, (size_t)dc.nq << dc.logn, (size_t)dc.nr << dc.logn, {}};
    job.p.tab = mma_tab(dc.mm_q2r, NG);
    job.p.binv = dc.q2r_inv;
    job.p.nin = dc.nq;
    job.p.nout = dc.nr;
    ext_mma_launch<KS, NG, false>(job, polys, dc.logn, dc.shape.bconv_threads, st);
}
// the standalone conversions, from residues
template <int KS>
void bconv_mma_launch_m(const DevConsts& dc, bool q2r, const uint64_t* in, uint64_t* out, int polys, cudaStream_t st) {
    constexpr int NG = mma_r_groups(KS);
    const BconvTables tb = q2r ? q2r_tables(dc) : r2q_tables(dc);
    ExtJob job{in, out, (size_t)tb.nin << dc.logn, (size_t)tb.nout << dc.logn, {}};
    job.p.tab = mma_tab(q2r ? dc.mm_q2r : dc.mm_r2q, NG);
    job.p.binv = tb.binv;
    job.p.nin = tb.nin;
    job.p.nout = tb.nout;
    job.p.hatinv = tb.hatinv;
    job.p.hatinvs = tb.hatinvs;
    job.p.mods = tb.in_mods;
    if (q2r) ext_mma_launch<KS, NG, true>(job, polys, dc.logn, dc.shape.bconv_threads, st);
    else ext_mma_launch<2 * NG, NG, true>(job, polys, dc.logn, dc.shape.bconv_threads, st);
}

// ---------------------------------------------------------------------------
// key-switch digit lift: digit d of a polynomial over Q (its primes [d alpha,
// (d + 1) alpha) that are live) into every other prime of Q|P, by approximate
// CRT with the single-precision quotient estimate of modUpQjtoT_23
// (include/BasisConv.cuh:86-135):
//   rb_i = [x_i (Q_d/q_i)^-1]_{q_i},  v = (int) sum_i rb_i / q_i (floats, in order),
//   out_m = sum_i rb_i (Q_d/q_i) - v Q_d  mod p_m
// ---------------------------------------------------------------------------
struct LiftDigit {
    uint64_t* rows;  // limb 0 of the digit over Q|P
    MmaTab tab;      // outputs: the primes of Q|P outside the digit, in order
    int lo, n, nout;
    const uint64_t *mods, *hatinv, *hatinvs;  // of the digit's first prime
};
// word i of the digit and its term of the quotient estimate, for the lane's two coefficients
__device__ __forceinline__ void lift_word(const LiftDigit& d, int i, ulonglong2 v, uint64_t& w0, uint64_t& w1, float& x0,
                                          float& x1) {
    const uint64_t h = d.hatinv[i], hs = d.hatinvs[i], q = d.mods[i];
    w0 = shoup(v.x, h, hs, q);
    w1 = shoup(v.y, h, hs, q);
    const float fq = __ull2float_rn(q);
    x0 = __fdiv_rn(__ull2float_rn(w0), fq);
    x1 = __fdiv_rn(__ull2float_rn(w1), fq);
}
// the quotient estimate of one coefficient: the quad's float terms added in index order
template <int KS>
__device__ __forceinline__ int lift_quotient(const float (&x)[KS], int first, int n, int alpha) {
    float acc = 0.f;
#pragma unroll
    for (int hop = 0; hop < 4; hop++) {
#pragma unroll
        for (int s = 0; s < KS; s++)
            if (first + s < n) acc = __fadd_rn(acc, x[s]);
        if (hop < 3) acc = __shfl_up_sync(0xffffffffu, acc, 1, 4);
    }
    return min(__float2int_rz(__shfl_sync(0xffffffffu, acc, 3, 4)), alpha);
}

// the digit's outputs over the primes outside it, stored at d.rows
template <int KS>
__device__ __forceinline__ void lift_outputs(const uint64_t (&w)[2][KS], const float (&x0)[KS], const float (&x1)[KS],
                                             const LiftDigit& d, int logn, int alpha, int first, size_t k,
                                             const MmaPlace& pl) {
    const uint32_t v0 = (uint32_t)lift_quotient<KS>(x0, first, d.n, alpha);
    const uint32_t v1 = (uint32_t)lift_quotient<KS>(x1, first, d.n, alpha);
    const int ng = d.tab.ng;
    for (int G = 0; G < ng; G++) {
        int S[8][4];
        mma_digits<KS>(S, w, d.tab, G, pl.lane);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int j = pl.c * 2 * ng + 2 * G + i;
            if (j >= d.nout) continue;
            const MmaOut o = mma_out(d.tab.out + j);
            ulonglong2 r;
            r.x = mma_value<false>(S, i, v0, 0, o);
            r.y = mma_value<false>(S, 2 + i, v1, 0, o);
            *reinterpret_cast<ulonglong2*>(d.rows + ((size_t)(j < d.lo ? j : j + d.n) << logn) + k) = r;
        }
    }
}

// ---------------------------------------------------------------------------
// K5: t/Q scale-and-round Q|R -> R (scaleAndRound_HPS_QR_R_kernel,
// include/poly_arithmetic.cuh:1263-1307) and the base extension R -> Q of each
// tensor polynomial. K4 stores its R limbs times the scale-and-round constant
// of their own prime and (R/r_j)^-1 (QRFoldRowsIO), the constant matrix carries
// (R/r_j)^-1 too, and the rounded quotient alpha = floor(1/2 + sum_i x_i frac_i)
// is one more word of the product, so that the first product's outputs are the
// second's words:
//   y_j = sum_i x_i (c_ij h_j) + alpha h_j + x'_j   mod r_j
//   out_i = sum_j y_j (R/r_j) - v R                 mod q_i
// ---------------------------------------------------------------------------
struct K5Poly {
    const uint64_t* src;  // limb 0 of Q|R
    uint64_t* dst;        // limb i at i, plus (i / alpha) * digit limbs (a digit's own limbs)
    int alpha, digit;
    int nq, nr;
    MmaTab sr, r2q;
    const double *sr_frac, *r2q_inv;
};
// mode 0: all three outputs over Q to out0 ([item][3][nq]).
// mode 1: a1*a2 to its own limbs of the digits in sd2 ([item][dnum][npq]); cross, b1*b2 to sd ([item][2][nq]).
// mode 2: a1*a2 over Q into sd2 ([item][nq]); cross, b1*b2 to sd (T-base and gadget key switches).
template <int NG>
struct K5Job {
    DevConsts c;
    const uint64_t* sc;
    uint64_t *out0, *sd, *sd2;
    int mode;
    __device__ __forceinline__ K5Poly bind(int poly) const {
        const int item = poly / 3, which = poly % 3;
        K5Poly p;
        p.src = sc + ((size_t)poly * c.nqr << c.logn);
        p.alpha = c.nq;
        p.digit = 0;
        if (mode == 0) {
            p.dst = out0 + ((size_t)poly * c.nq << c.logn);
        } else if (which) {
            p.dst = sd + (((size_t)item * 2 + which - 1) * c.nq << c.logn);
        } else if (mode == 2) {
            p.dst = sd2 + ((size_t)item * c.nq << c.logn);
        } else {
            p.dst = sd2 + ((size_t)item * c.dnum * c.npq << c.logn);
            p.alpha = c.alpha;
            p.digit = c.npq;
        }
        p.nq = c.nq;
        p.nr = c.nr;
        p.sr = mma_tab(c.mm_sr, NG);
        p.r2q = mma_tab(c.mm_r2q, NG);
        p.sr_frac = c.sr_frac;
        p.r2q_inv = c.r2q_inv;
        return p;
    }
    // FUSED: the one digit of a1*a2 (its limbs at p.dst), or nothing to lift
    __device__ __forceinline__ bool lift(int poly, const K5Poly& p, LiftDigit& d) const {
        d.rows = p.dst;
        d.tab = mma_tab(c.mm_lift, mma_groups(c.np));
        d.lo = 0;
        d.n = c.nq;
        d.nout = c.np;
        d.mods = c.mods;
        d.hatinv = c.dig_hatinv;
        d.hatinvs = c.dig_hatinvs;
        return poly % 3 == 0;
    }
};
// mode 1 over a mixed-level batch (scratch with the top level's per-item layout)
template <int NG>
struct MixedK5Job {
    Groups G;
    const uint64_t* sc;
    uint64_t *sd, *sd2;
    __device__ __forceinline__ K5Poly bind(int poly) const {
        const int item = poly / 3, which = poly % 3, g = G.group_of_item(item), logn = G.logn;
        const DevConsts* lv = G.lv[g];
        K5Poly p;
        p.src = sc + (((size_t)item * 3 * G.top_nqr + (size_t)which * G.nqr[g]) << logn);
        p.nq = G.nq[g];
        p.nr = G.nr[g];
        if (which) {
            p.dst = sd + (((size_t)item * 2 * G.top_nq + (size_t)(which - 1) * p.nq) << logn);
            p.alpha = p.nq;
            p.digit = 0;
        } else {
            p.dst = sd2 + (((size_t)item * G.top_dnum * G.top_npq) << logn);
            p.alpha = lv->alpha;
            p.digit = G.npq[g];
        }
        p.sr = mma_tab(lv->mm_sr, NG);
        p.r2q = mma_tab(lv->mm_r2q, NG);
        p.sr_frac = lv->sr_frac;
        p.r2q_inv = lv->r2q_inv;
        return p;
    }
};

// K5, 32 pairs: 163 + 168 us (two kernels of 64-bit multiply-accumulates) -> 117 us here, the lift (lift.cuh) 31 us
// FUSED: the digit lift too, where one digit holds all of Q and the R -> Q
// product's outputs are the lift's words.
template <int KS, int NG, bool FUSED, class Job>
static __global__ void k5_mma_kernel(Job job, int logn, int iters) {
    constexpr int K2 = 2 * NG;  // words a lane holds of the second product
    const MmaPlace pl = mma_place(logn, iters);
    const K5Poly p = job.bind(pl.poly);
    const int first = pl.c * KS, first2 = pl.c * K2;
    double f[KS], f2[K2];
#pragma unroll
    for (int s = 0; s < KS; s++) f[s] = first + s < p.nq ? p.sr_frac[first + s] : 0.0;
#pragma unroll
    for (int s = 0; s < K2; s++) f2[s] = first2 + s < p.nr ? p.r2q_inv[first2 + s] : 0.0;
    size_t k = pl.k;
    for (int it = 0; it < iters; it++, k += blockDim.x / 2) {
        uint64_t y[2][K2];
        {
            uint64_t w[2][KS];
            double x0[KS], x1[KS];
#pragma unroll
            for (int s = 0; s < KS; s++) {
                ulonglong2 v = make_ulonglong2(0, 0);
                if (first + s < p.nq) v = *reinterpret_cast<const ulonglong2*>(p.src + ((size_t)(first + s) << logn) + k);
                w[0][s] = v.x;
                w[1][s] = v.y;
            }
#pragma unroll
            for (int s = 0; s < K2; s++) {
                ulonglong2 v = make_ulonglong2(0, 0);
                if (first2 + s < p.nr)
                    v = *reinterpret_cast<const ulonglong2*>(p.src + ((size_t)(p.nq + first2 + s) << logn) + k);
                y[0][s] = v.x;
                y[1][s] = v.y;
            }
#pragma unroll
            for (int s = 0; s < KS; s++) {
                x0[s] = u64_to_double(w[0][s]);
                x1[s] = u64_to_double(w[1][s]);
            }
            const uint64_t a0 = __double2ull_rz(quad_fma_sum<KS>(x0, f, 0.5, first, p.nq));
            const uint64_t a1 = __double2ull_rz(quad_fma_sum<KS>(x1, f, 0.5, first, p.nq));
#pragma unroll
            for (int s = 0; s < KS; s++) {
                if (first + s == p.nq) {
                    w[0][s] = a0;
                    w[1][s] = a1;
                }
            }
#pragma unroll
            for (int G = 0; G < NG; G++) {
                int S[8][4];
                mma_digits<KS>(S, w, p.sr, G, pl.lane);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const MmaOut o = mma_out(p.sr.out + first2 + 2 * G + i);
                    y[0][2 * G + i] = mma_value<true>(S, i, 0, y[0][2 * G + i], o);
                    y[1][2 * G + i] = mma_value<true>(S, 2 + i, 0, y[1][2 * G + i], o);
                }
            }
        }
        double x0[K2], x1[K2];
#pragma unroll
        for (int s = 0; s < K2; s++) {
            x0[s] = u64_to_double(y[0][s]);
            x1[s] = u64_to_double(y[1][s]);
        }
        const uint32_t v0 = (uint32_t)llround(quad_fma_sum<K2>(x0, f2, 0.0, first2, p.nr));
        const uint32_t v1 = (uint32_t)llround(quad_fma_sum<K2>(x1, f2, 0.0, first2, p.nr));
        ulonglong2 x[FUSED ? K2 : 1];
#pragma unroll
        for (int G = 0; G < NG; G++) {
            int S[8][4];
            mma_digits<K2>(S, y, p.r2q, G, pl.lane);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int j = first2 + 2 * G + i;
                if (FUSED) x[2 * G + i] = make_ulonglong2(0, 0);
                if (j >= p.nq) continue;
                const MmaOut o = mma_out(p.r2q.out + j);
                ulonglong2 r;
                r.x = mma_value<false>(S, i, v0, 0, o);
                r.y = mma_value<false>(S, 2 + i, v1, 0, o);
                *reinterpret_cast<ulonglong2*>(p.dst + ((size_t)(j + j / p.alpha * p.digit) << logn) + k) = r;
                if (FUSED) x[2 * G + i] = r;
            }
        }
        if constexpr (FUSED) {
            LiftDigit d;
            if (job.lift(pl.poly, p, d)) {  // the whole CTA's polynomial
                uint64_t w[2][K2];
                float t0[K2], t1[K2];
#pragma unroll
                for (int s = 0; s < K2; s++) {
                    w[0][s] = w[1][s] = 0;
                    t0[s] = t1[s] = 0.f;
                    if (first2 + s < d.n) lift_word(d, first2 + s, x[s], w[0][s], w[1][s], t0[s], t1[s]);
                }
                lift_outputs<K2>(w, t0, t1, d, logn, p.alpha, first2, k, pl);
            }
        }
    }
}

template <int KS, int NG, bool FUSED, class Job>
static void k5_mma_launch(const Job& job, int polys, int logn, int threads, cudaStream_t st) {
    static int res[4] = {0, 0, 0, 0};
    const int iters = mma_iters(polys, logn, threads,
                                resident_ctas_at((const void*)k5_mma_kernel<KS, NG, FUSED, Job>, threads, 0, res));
    const size_t per = ((size_t)1 << logn) / ((size_t)(threads / 2) * iters);
    k5_mma_kernel<KS, NG, FUSED, Job><<<(unsigned)(polys * per), threads, 0, st>>>(job, logn, iters);
    check_launch("k5");
}
template <int KS>
void k5_launch_m(const DevConsts& dc, int count, const MulScratch& m, uint64_t* out0, int mode, cudaStream_t st) {
    constexpr int NG = mma_r_groups(KS);
    const K5Job<NG> job{dc, m.sc, out0, m.sd, m.sd2, mode};
    // small batches: one launch less on the per-call path; larger ones run the
    // lift, a third of K5's polynomials, as a kernel of fewer registers
    const bool fused = mode == 1 && dc.dnum == 1 && lift_steps(dc.alpha) == 2 * NG && count <= dc.shape.k5_fused_pairs;
    if (fused) k5_mma_launch<KS, NG, true>(job, count * 3, dc.logn, dc.shape.k5_threads, st);
    else k5_mma_launch<KS, NG, false>(job, count * 3, dc.logn, dc.shape.k5_threads, st);
    if (mode == 1 && !fused) lift_launch(dc, m.sd2, count, st);
}

// K2 and K5 of a mixed batch (KS of the top level's prime count, which its levels' tables share)
template <int KS>
void k2_mixed_launch_m(const Groups& G, const LaunchShape& sh, int count, const MulScratch& m, cudaStream_t st) {
    constexpr int NG = mma_r_groups(KS);
    ext_mma_launch<KS, NG, false>(MixedExtJob<NG>{G, m.sa, m.sb}, count * 4, G.logn, sh.bconv_threads, st);
}
template <int KS>
void k5_mixed_launch_m(const Groups& G, const LaunchShape& sh, int count, const MulScratch& m, cudaStream_t st) {
    constexpr int NG = mma_r_groups(KS);
    k5_mma_launch<KS, NG, false>(MixedK5Job<NG>{G, m.sc, m.sd, m.sd2}, count * 3, G.logn, sh.k5_threads, st);
}
