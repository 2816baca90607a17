// The per-coefficient stages of the multiply pipeline as byte matrix products
// (limb_mma.cuh): K2 (base extension Q -> R), K5 (t/Q scale-and-round Q|R -> R
// and the base extension R -> Q, chained in registers) and the key-switch
// digit lift. Each size of the prime count is instantiated in its own
// translation unit (k5_m<MAXQ>.cu) so that the unrolled variants compile in
// parallel.
//
// K2 is a launch of its own at every size. Inside the loader of the NTT over R
// (each row reading all nq words of its coefficients) it saved a launch, but with
// K2 at 5 us for one pair the fused form was the slower one everywhere: one
// captured pair 106 -> 111 us at N = 16384, 84 -> 100 at 4096, 292 -> 357 at 32768.
//
// A warp takes MT tiles of 16 coefficients of one polynomial per iteration: lane
// (g = lane / 4, c = lane % 4) coefficients 2g and 2g + 1 of each, the words and
// outputs of limb_mma.cuh. A CTA's iterations take consecutive runs of coefficients.
//
// The figures at the kernels are of N = 16384, 7 + 1 primes, 32 pairs (2^21
// coefficients in K2, 1.5 x 2^20 in K5), one launch under ncu, against the same
// stages from 64-bit multiply-accumulates and 128-bit Barrett reductions.
#pragma once
#include "limb_mma.cuh"
#include "mixed.cuh"

// Tiles per iteration: two share one load of the constants as long as their
// words and sums fit the registers of at least 16 warps per SM.
constexpr int mma_tiles(int ks) { return ks <= 2 ? 2 : 1; }
// Tables of up to 20 KiB are copied to shared memory by each CTA; larger ones
// (16 primes and more) are read through L1.
constexpr bool mma_staged(int ks) { return ks <= 5; }
constexpr int mma_stage_bytes(int ks, int ng) { return mma_staged(ks) ? (int)mma_table_bytes(ks, ng) : 0; }

// iterations of a CTA that takes `each` coefficients at a time: as few as leave
// four waves of CTAs, so that small launches cover the SMs and large ones load
// a lane's constants rarely
static inline int mma_iters(size_t polys, int logn, int each, int resident) {
    const size_t per = ((size_t)1 << logn) / each;  // iterations that one polynomial takes (a power of two)
    size_t it = 1;
    while (it < per && it < 16 && polys * per / (2 * it) >= (size_t)4 * resident) it *= 2;
    return (int)it;
}
// CTAs of a launch
static inline unsigned mma_blocks(size_t polys, int logn, int each, int iters) {
    return (unsigned)(polys * (((size_t)1 << logn) / ((size_t)each * iters)));
}

// the CTA's polynomial and first coefficient, the lane's place in it; a warp's
// second tile follows its first by 16 coefficients
struct MmaPlace {
    int poly;
    size_t k;    // coefficient of the lane's row 0 in iteration 0
    size_t warp; // first coefficient of the warp in iteration 0
    int own;     // the warp's coefficient whose floating-point sum the lane takes (16 MT lanes; the others repeat)
    int at;      // the lane's row 0 among the warp's coefficients
    int lane, c, each;
};
template <int MT>
__device__ __forceinline__ MmaPlace mma_place(int logn, int iters) {
    const int lane = threadIdx.x & 31, each = blockDim.x / 2 * MT;
    const unsigned per = (1u << logn) / (each * iters);
    const size_t warp = (size_t)(blockIdx.x % per) * each * iters + (threadIdx.x >> 5) * 16 * MT;
    return MmaPlace{(int)(blockIdx.x / per), warp + 2 * (lane >> 2), warp, lane % (16 * MT), 2 * (lane >> 2), lane,
                    lane & 3, each};
}
// the 32-bit value that each coefficient's owner holds as the word of the last step (lane 0 of the quad)
template <int KS, int MT>
__device__ __forceinline__ void put_extra(uint64_t (&w)[MT][2][KS], uint32_t own, const MmaPlace& pl) {
#pragma unroll
    for (int m = 0; m < MT; m++) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const uint32_t v = __shfl_sync(0xffffffffu, own, 16 * m + pl.at + r);
            w[m][r][KS - 1] = pl.c == 0 ? v : 0;
        }
    }
}
// the value that each coefficient's owner holds (T: 32 or 64 bits) as word `word` of the lanes that have it
template <int KS, int MT, class T>
__device__ __forceinline__ void put_word(uint64_t (&w)[MT][2][KS], T own, int word, const MmaPlace& pl) {
#pragma unroll
    for (int m = 0; m < MT; m++) {
#pragma unroll
        for (int r = 0; r < 2; r++) {
            const T v = __shfl_sync(0xffffffffu, own, 16 * m + pl.at + r);
#pragma unroll
            for (int s = 0; s < KS; s++)
                if (pl.c * KS + s == word) w[m][r][s] = v;
        }
    }
}
// The words of a warp's coefficients, copied to a buffer of its own in shared
// memory (rows of 16 MT coefficients, padded by 16 bytes) while it computes the
// iteration before: the copies are asynchronous, the lanes that need a word as a
// fragment and the lane that needs it in a floating-point sum read the same copy
// (loaded to registers when needed, K2 took 88 us at 51% issue, waiting on loads).
template <int MT>
constexpr int kRow = 16 * MT + 2;
template <int MT, int MAXW>
__device__ __forceinline__ void copy_words(uint64_t* buf, const uint64_t* src, int n, int logn, int lane) {
    constexpr int PER = 8 * MT;  // 16-byte pieces of a word's row
    const int piece = lane % PER, w0 = lane / PER;
    const uint64_t* s = src + ((size_t)w0 << logn) + 2 * piece;
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(buf + w0 * kRow<MT> + 2 * piece);
#pragma unroll
    for (int t = 0; t < MAXW; t += 32 / PER)
        if (t + w0 < n)
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d + t * kRow<MT> * 8), "l"(s + ((size_t)t << logn))
                         : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// all copies but the newest group have arrived, for the whole warp
__device__ __forceinline__ void copy_wait() {
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
}
__device__ __forceinline__ ulonglong2 load2(const uint64_t* p) { return *reinterpret_cast<const ulonglong2*>(p); }
__device__ __forceinline__ void store2(uint64_t* p, uint64_t x, uint64_t y) {
    *reinterpret_cast<ulonglong2*>(p) = make_ulonglong2(x, y);
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

// K2, 32 pairs: 179 us with 64-bit multiply-accumulates -> 61 us here (252 MB
// moved: 38 us at the copy rate; issue-bound at 480 instructions per 32 coefficients)
// EXTRA: the quotient word has a step of its own (R -> Q), else it is word nin.
template <int KS, int NG, bool EXTRA, bool PREP, bool SH, class Job>
static __global__ void __maxnreg__(KS <= 4 && !PREP ? 80 : 128) ext_mma_kernel(Job job, int logn, int iters) {
    constexpr int MT = mma_tiles(KS), STEPS = KS + (EXTRA ? 1 : 0), BUF = 4 * KS * kRow<MT>;
    extern __shared__ uint4 mma_sh[];
    const MmaPlace pl = mma_place<MT>(logn, iters);
    const ExtPoly e = job.bind(pl.poly);
    double* binv = (double*)(mma_sh + mma_stage_bytes(STEPS, NG) / 16);
    uint64_t* buf = (uint64_t*)(binv + 4 * KS) + (threadIdx.x >> 5) * 2 * BUF;
    const uint64_t* in = e.in + pl.warp;
    copy_words<MT, 4 * KS>(buf, in, e.nin, logn, pl.lane);
    copy_commit();
    if (mma_staged(STEPS)) mma_stage(mma_sh, e.tab, STEPS);
    if ((int)threadIdx.x < e.nin) binv[threadIdx.x] = __ldg(e.binv + threadIdx.x);
    __syncthreads();
    const MmaTab tab = mma_staged(STEPS) ? mma_tab(mma_sh, NG) : e.tab;
    const int first = pl.c * KS;
    uint64_t* out = e.out + ((size_t)(pl.c * 2 * NG) << logn) + pl.k;
    for (int it = 0; it < iters; it++, out += pl.each) {
        const uint64_t* cur = buf + (it & 1) * BUF;
        in += pl.each;
        if (it + 1 < iters) copy_words<MT, 4 * KS>(buf + (~it & 1) * BUF, in, e.nin, logn, pl.lane);
        copy_commit();
        copy_wait();
        double frac = 0.0;
#pragma unroll
        for (int i = 0; i < 4 * KS; i++) {
            if (i < e.nin) {
                uint64_t y = cur[i * kRow<MT> + pl.own];
                if (PREP) y = shoup(y, __ldg(e.hatinv + i), __ldg(e.hatinvs + i), __ldg(e.mods + i));
                frac = __fma_rn(__ull2double_rn(y), binv[i], frac);
            }
        }
        uint64_t w[MT][2][STEPS];
#pragma unroll
        for (int s = 0; s < STEPS; s++) {
#pragma unroll
            for (int m = 0; m < MT; m++) {
                ulonglong2 x = make_ulonglong2(0, 0);
                if (s < KS && first + s < e.nin) x = load2(cur + (first + s) * kRow<MT> + 16 * m + pl.at);
                w[m][0][s] = x.x;
                w[m][1][s] = x.y;
            }
        }
        if (PREP) {
#pragma unroll
            for (int s = 0; s < KS; s++) {
                if (first + s >= e.nin) continue;
                const uint64_t h = __ldg(e.hatinv + first + s), hs = __ldg(e.hatinvs + first + s),
                               q = __ldg(e.mods + first + s);
#pragma unroll
                for (int m = 0; m < MT; m++)
#pragma unroll
                    for (int r = 0; r < 2; r++) w[m][r][s] = shoup(w[m][r][s], h, hs, q);
            }
        }
        if (EXTRA) put_extra<STEPS>(w, round_half_up(frac), pl);
        else put_word<STEPS>(w, round_half_up(frac), e.nin, pl);
#pragma unroll
        for (int G = 0; G < NG; G++) {
            uint32_t D[MT][4][4];
            mma_digits<STEPS, MT>(D, w, tab, G, pl.lane);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int j = pl.c * 2 * NG + 2 * G + i;
                const MmaOut o = mma_out(tab.out + j);
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    const uint64_t r0 = mma_value<false, SH>(D[m], i, 0, o);
                    const uint64_t r1 = mma_value<false, SH>(D[m], 2 + i, 0, o);
                    if (j < e.nout) store2(out + ((size_t)(2 * G + i) << logn) + 16 * m, r0, r1);
                }
            }
        }
        __syncwarp();  // the buffer is read; the next iteration's copies overwrite it
    }
}

template <int KS, int NG, bool EXTRA, bool PREP, bool SH, class Job>
static void ext_mma_launch_sh(const Job& job, int polys, int logn, int threads, cudaStream_t st) {
    static int res[4] = {0, 0, 0, 0};
    auto smem_of = [](int threads) {
        return mma_stage_bytes(KS + (EXTRA ? 1 : 0), NG) + 4 * KS * 8 +
               threads / 32 * 2 * 4 * KS * kRow<mma_tiles(KS)> * 8;
    };
    const int smem = smem_of(threads);
    allow_smem(ext_mma_kernel<KS, NG, EXTRA, PREP, SH, Job>, smem, smem_of(512));
    const int each = threads / 2 * mma_tiles(KS);
    const int iters = mma_iters(polys, logn, each,
                                resident_ctas_at((const void*)ext_mma_kernel<KS, NG, EXTRA, PREP, SH, Job>, threads, smem, res));
    ext_mma_kernel<KS, NG, EXTRA, PREP, SH, Job><<<mma_blocks(polys, logn, each, iters), threads, smem, st>>>(job, logn, iters);
    check_launch("base_extension");
}
template <int KS, int NG, bool EXTRA, bool PREP, class Job>
static void ext_mma_launch(const Job& job, bool shifted, int polys, int logn, int threads, cudaStream_t st) {
    if (polys <= 0) return;
    if (shifted) ext_mma_launch_sh<KS, NG, EXTRA, PREP, true>(job, polys, logn, threads, st);
    else ext_mma_launch_sh<KS, NG, EXTRA, PREP, false>(job, polys, logn, threads, st);
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
    ext_mma_launch<KS, NG, false, false>(job, dc.mm_shift, polys, dc.logn, dc.shape.bconv_threads, st);
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
    if (q2r) ext_mma_launch<KS, NG, false, true>(job, dc.mm_shift, polys, dc.logn, dc.shape.bconv_threads, st);
    else ext_mma_launch<2 * NG, NG, true, true>(job, dc.mm_shift, polys, dc.logn, dc.shape.bconv_threads, st);
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
// word i of the digit and its term of the quotient estimate
__device__ __forceinline__ void lift_word(const LiftDigit& d, int i, uint64_t x, uint64_t& w, float& t) {
    const uint64_t q = d.mods[i];
    w = shoup(x, d.hatinv[i], d.hatinvs[i], q);
    t = __fdiv_rn(__ull2float_rn(w), __ull2float_rn(q));
}
// the quotient estimate of one coefficient: the quad's float terms added in index order
template <int KS>
__device__ __forceinline__ uint32_t lift_quotient(const float (&x)[KS], int first, int n, int alpha) {
    float acc = 0.f;
#pragma unroll
    for (int hop = 0; hop < 4; hop++) {
#pragma unroll
        for (int s = 0; s < KS; s++)
            if (first + s < n) acc = __fadd_rn(acc, x[s]);
        if (hop < 3) acc = __shfl_up_sync(0xffffffffu, acc, 1, 4);
    }
    return (uint32_t)min(__float2int_rz(__shfl_sync(0xffffffffu, acc, 3, 4)), alpha);
}
// the digit's outputs over the primes outside it, stored at d.rows
template <int KS, int MT>
__device__ __forceinline__ void lift_outputs(const uint64_t (&w)[MT][2][KS], const LiftDigit& d, const MmaTab& tab, int logn, size_t k,
                                             const MmaPlace& pl) {
    const int ng = tab.ng;
    for (int G = 0; G < ng; G++) {
        uint32_t D[MT][4][4];
        mma_digits<KS, MT>(D, w, tab, G, pl.lane);
#pragma unroll
        for (int i = 0; i < 2; i++) {
            const int j = pl.c * 2 * ng + 2 * G + i;
            if (j >= d.nout) continue;
            const MmaOut o = mma_out(tab.out + j);
            uint64_t* row = d.rows + ((size_t)(j < d.lo ? j : j + d.n) << logn);
#pragma unroll
            for (int m = 0; m < MT; m++)
                store2(row + k + 16 * m, mma_value<false, true>(D[m], i, 0, o), mma_value<false, true>(D[m], 2 + i, 0, o));
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

// K5, 32 pairs: 163 + 168 us (two kernels of 64-bit multiply-accumulates) -> 97 us here, the lift (lift.cuh) 26 us
// FUSED: the digit lift too, where one digit holds all of Q and the R -> Q
// product's outputs are the lift's words.
template <int KS, int NG, bool FUSED, bool SH, class Job>
static __global__ void __launch_bounds__(256, KS <= 4 ? 3 : 1) k5_mma_kernel(Job job, int logn, int iters) {
    constexpr int K2 = 2 * NG, MT = mma_tiles(KS);  // K2: words a lane holds of the second product
    extern __shared__ uint4 mma_sh[];
    const MmaPlace pl = mma_place<MT>(logn, iters);
    const K5Poly p = job.bind(pl.poly);
    uint4* sh2 = mma_sh + mma_stage_bytes(KS, NG) / 16;
    // two buffers of the nq + nr input words; the product's nr words go where its input's were
    constexpr int BUF = 4 * (KS + K2) * kRow<MT>, Y0 = 4 * KS * kRow<MT>;
    double* fr = (double*)(sh2 + mma_stage_bytes(K2 + 1, NG) / 16);  // factors of the two floating-point sums
    uint64_t* buf = (uint64_t*)(fr + 4 * (KS + K2)) + (threadIdx.x >> 5) * 2 * BUF;
    if (mma_staged(KS)) mma_stage(mma_sh, p.sr, KS);
    if (mma_staged(K2 + 1)) mma_stage(sh2, p.r2q, K2 + 1);
    for (int i = threadIdx.x; i < p.nq + p.nr; i += blockDim.x)
        fr[i < p.nq ? i : 4 * KS + i - p.nq] = __ldg(i < p.nq ? p.sr_frac + i : p.r2q_inv + (i - p.nq));
    const int first = pl.c * KS, first2 = pl.c * K2;
    const uint64_t* in = p.src + pl.warp;
    auto copy_in = [&](uint64_t* to) {
        copy_words<MT, 4 * KS>(to, in, p.nq, logn, pl.lane);
        copy_words<MT, 4 * K2>(to + Y0, in + ((size_t)p.nq << logn), p.nr, logn, pl.lane);
    };
    copy_in(buf);
    copy_commit();
    __syncthreads();
    const MmaTab sr = mma_staged(KS) ? mma_tab(mma_sh, NG) : p.sr;
    const MmaTab r2q = mma_staged(K2 + 1) ? mma_tab(sh2, NG) : p.r2q;
    size_t k = pl.k;
    for (int it = 0; it < iters; it++, k += pl.each) {
        uint64_t* cur = buf + (it & 1) * BUF;
        in += pl.each;
        if (it + 1 < iters) copy_in(buf + (~it & 1) * BUF);
        copy_commit();
        copy_wait();
        uint64_t y[MT][2][K2 + 1];
        {
            uint64_t w[MT][2][KS];
#pragma unroll
            for (int s = 0; s < KS; s++) {
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    ulonglong2 x = make_ulonglong2(0, 0);
                    if (first + s < p.nq) x = load2(cur + (first + s) * kRow<MT> + 16 * m + pl.at);
                    w[m][0][s] = x.x;
                    w[m][1][s] = x.y;
                }
            }
#pragma unroll
            for (int s = 0; s < K2; s++) {
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    ulonglong2 x = make_ulonglong2(0, 0);
                    if (first2 + s < p.nr) x = load2(cur + Y0 + (first2 + s) * kRow<MT> + 16 * m + pl.at);
                    y[m][0][s] = x.x;
                    y[m][1][s] = x.y;
                }
            }
            double nu = 0.5;
#pragma unroll
            for (int i = 0; i < 4 * KS; i++)
                if (i < p.nq) nu = __fma_rn(__ull2double_rn(cur[i * kRow<MT> + pl.own]), fr[i], nu);
            put_word<KS>(w, (uint64_t)__double2ull_rz(nu), p.nq, pl);
#pragma unroll
            for (int G = 0; G < NG; G++) {
                uint32_t D[MT][4][4];
                mma_digits<KS, MT>(D, w, sr, G, pl.lane);
#pragma unroll
                for (int i = 0; i < 2; i++) {
                    const MmaOut o = mma_out(sr.out + first2 + 2 * G + i);
#pragma unroll
                    for (int m = 0; m < MT; m++) {
#pragma unroll
                        for (int r = 0; r < 2; r++)
                            y[m][r][2 * G + i] =
                                mma_value<true, SH>(D[m], 2 * r + i, y[m][r][2 * G + i], o);
                    }
                }
            }
        }
        // the words of a coefficient to the lane that sums them (each lane overwrites what it read itself)
#pragma unroll
        for (int s = 0; s < K2; s++)
#pragma unroll
            for (int m = 0; m < MT; m++)
                store2(cur + Y0 + (first2 + s) * kRow<MT> + 16 * m + pl.at, y[m][0][s], y[m][1][s]);
        __syncwarp();
        double frac = 0.0;
#pragma unroll
        for (int i = 0; i < 4 * K2; i++)
            if (i < p.nr) frac = __fma_rn(__ull2double_rn(cur[Y0 + i * kRow<MT> + pl.own]), fr[4 * KS + i], frac);
        __syncwarp();  // the buffer is read; the next iteration's copies overwrite it
        put_extra<K2 + 1>(y, round_half_up(frac), pl);
        uint64_t x[FUSED ? MT : 1][2][FUSED ? K2 : 1];
#pragma unroll
        for (int G = 0; G < NG; G++) {
            uint32_t D[MT][4][4];
            mma_digits<K2 + 1, MT>(D, y, r2q, G, pl.lane);
#pragma unroll
            for (int i = 0; i < 2; i++) {
                const int j = first2 + 2 * G + i;
                const MmaOut o = mma_out(r2q.out + j);
                uint64_t* row = p.dst + ((size_t)(p.digit ? j + j / p.alpha * p.digit : j) << logn);
#pragma unroll
                for (int m = 0; m < MT; m++) {
                    const uint64_t r0 = mma_value<false, SH>(D[m], i, 0, o);
                    const uint64_t r1 = mma_value<false, SH>(D[m], 2 + i, 0, o);
                    if (j < p.nq) store2(row + k + 16 * m, r0, r1);
                    if (FUSED) {
                        x[FUSED ? m : 0][0][FUSED ? 2 * G + i : 0] = r0;
                        x[FUSED ? m : 0][1][FUSED ? 2 * G + i : 0] = r1;
                    }
                }
            }
        }
        if constexpr (FUSED) {
            LiftDigit d;
            if (job.lift(pl.poly, p, d)) {  // the whole CTA's polynomial
#pragma unroll
                for (int m = 0; m < MT; m++) {
#pragma unroll
                    for (int r = 0; r < 2; r++) {
                        float t[K2];
#pragma unroll
                        for (int s = 0; s < K2; s++) {
                            t[s] = 0.f;
                            if (first2 + s < d.n) lift_word(d, first2 + s, x[m][r][s], x[m][r][s], t[s]);
                            else x[m][r][s] = 0;
                        }
                        const uint32_t v = lift_quotient<K2>(t, first2, d.n, p.alpha);
#pragma unroll
                        for (int s = 0; s < K2; s++)
                            if (first2 + s == d.n) x[m][r][s] = v;
                    }
                }
                lift_outputs<K2, MT>(x, d, d.tab, logn, k, pl);
            }
        }
    }
}

template <int KS, int NG, bool FUSED, bool SH, class Job>
static void k5_mma_launch_sh(const Job& job, int polys, int logn, int threads, cudaStream_t st) {
    static int res[4] = {0, 0, 0, 0};
    auto smem_of = [](int threads) {
        return mma_stage_bytes(KS, NG) + mma_stage_bytes(2 * NG + 1, NG) + 4 * (KS + 2 * NG) * 8 +
               threads / 32 * 2 * 4 * (KS + 2 * NG) * kRow<mma_tiles(KS)> * 8;
    };
    const int smem = smem_of(threads);
    const int each = threads / 2 * mma_tiles(KS);
    allow_smem(k5_mma_kernel<KS, NG, FUSED, SH, Job>, smem, smem_of(256));
    const int iters = mma_iters(polys, logn, each,
                                resident_ctas_at((const void*)k5_mma_kernel<KS, NG, FUSED, SH, Job>, threads, smem, res));
    k5_mma_kernel<KS, NG, FUSED, SH, Job><<<mma_blocks(polys, logn, each, iters), threads, smem, st>>>(job, logn, iters);
    check_launch("k5");
}
template <int KS, int NG, bool FUSED, class Job>
static void k5_mma_launch(const Job& job, bool shifted, int polys, int logn, int threads, cudaStream_t st) {
    if (shifted) k5_mma_launch_sh<KS, NG, FUSED, true>(job, polys, logn, threads, st);
    else k5_mma_launch_sh<KS, NG, FUSED, false>(job, polys, logn, threads, st);
}
template <int KS>
void k5_launch_m(const DevConsts& dc, int count, const MulScratch& m, uint64_t* out0, int mode, cudaStream_t st) {
    constexpr int NG = mma_r_groups(KS);
    const K5Job<NG> job{dc, m.sc, out0, m.sd, m.sd2, mode};
    // small batches: one launch less on the per-call path; larger ones run the
    // lift, a third of K5's polynomials, as a kernel of fewer registers
    const bool fused = mode == 1 && dc.dnum == 1 && lift_steps(dc.alpha) == 2 * NG && count <= dc.shape.k5_fused_pairs;
    if (fused) k5_mma_launch<KS, NG, true>(job, dc.mm_shift, count * 3, dc.logn, dc.shape.k5_threads, st);
    else k5_mma_launch<KS, NG, false>(job, dc.mm_shift, count * 3, dc.logn, dc.shape.k5_threads, st);
    if (mode == 1 && !fused) lift_launch(dc, m.sd2, count, st);
}

// K2 and K5 of a mixed batch (KS of the top level's prime count, which its levels' tables share)
template <int KS>
void k2_mixed_launch_m(const Groups& G, const LaunchShape& sh, bool shifted, int count, const MulScratch& m, cudaStream_t st) {
    constexpr int NG = mma_r_groups(KS);
    ext_mma_launch<KS, NG, false, false>(MixedExtJob<NG>{G, m.sa, m.sb}, shifted, count * 4, G.logn, sh.bconv_threads, st);
}
template <int KS>
void k5_mixed_launch_m(const Groups& G, const LaunchShape& sh, bool shifted, int count, const MulScratch& m, cudaStream_t st) {
    constexpr int NG = mma_r_groups(KS);
    k5_mma_launch<KS, NG, false>(MixedK5Job<NG>{G, m.sc, m.sd, m.sd2}, shifted, count * 3, G.logn, sh.k5_threads, st);
}
