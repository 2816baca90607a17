// Row functors of the fused multiply pipeline (sources and store targets of
// the NTT kernels that carry the tensor product, key products, mod down and
// output epilogues) and the host functions that launch the pipeline's steps.
#pragma once
#include "internal.cuh"

// Pointer arrays must be device-readable: the batched entry points pass
// PtrBatch by value as a kernel parameter, so functors point into it through
// this wrapper kernel-parameter view.
struct PairQRowsP {
    PtrBatch pb;
    int logn, nq;
    __device__ __forceinline__ int prime(int row) const { return row % nq; }
    __device__ __forceinline__ PtrRow bind(int row) const {
        const int item = row / (4 * nq), w = row % (4 * nq), p = w / nq, l = w % nq;
        const uint64_t* base = p < 2 ? pb.a[item] : pb.b[item];
        return PtrRow{const_cast<uint64_t*>(base) + (((size_t)(p & 1) * nq + l) << logn)};
    }
    __device__ __forceinline__ void prefetch(int row, int off, int n) const { bind(row).prefetch(off, n); }
};

// K1 store target: rows over Q (RowsIO layout) holding the base extension's words y_i = [x_i (Q/q_i)^-1]_{q_i}, the scale folded into
// the inverse transform's last-stage constants
struct QHatRowsIO {
    uint64_t* base;
    int logn, nq;
    const tw_t* fold_base;  // DevConsts::q2r_fold
    __device__ __forceinline__ int prime(int row) const { return row % nq; }
    __device__ __forceinline__ PtrRow bind(int row) const { return PtrRow{base + ((size_t)row << logn)}; }
    __device__ __forceinline__ const tw_t* fold(int row) const { return fold_base + 2 * (row % nq); }
};

// rows of consecutive Q|R polynomials; limb l of Q|R uses prime l (Q) or idx_r + l - nq (R)
// (K4's store target: an R limb times its scale-and-round constant and (R/r_j)^-1, see qr_fold)
struct QRFoldRowsIO {
    uint64_t* base;
    int logn, nq, nqr, idx_r;
    const tw_t* fold_base;  // DevConsts::qr_fold
    __device__ __forceinline__ int prime(int row) const {
        const int l = row % nqr;
        return l < nq ? l : idx_r + (l - nq);
    }
    __device__ __forceinline__ PtrRow bind(int row) const { return PtrRow{base + ((size_t)row << logn)}; }
    __device__ __forceinline__ const tw_t* fold(int row) const { return fold_base + 2 * (row % nqr); }
};

// K4 source: tensor product of the pair at limb l of Q|R, one of three outputs
// values in [0, 4q), as the inverse transform takes them
struct TensorRow {
    static constexpr bool kLoadAdj = true;
    const uint64_t *a1, *b1, *a2, *b2;
    int k;
    template <int K>
    __device__ __forceinline__ void load_adj(int j, uint64_t* x) const {
        const bool wide = wide_ok(a1) && wide_ok(b1) && wide_ok(a2) && wide_ok(b2);
        uint64_t y[K];
        load_adjacent<K>((k == 2 ? b1 : a1) + j, wide, x);
        load_adjacent<K>((k == 0 ? a2 : b2) + j, wide, y);
        if (k == 1) {
            uint64_t u[K], v[K];
            load_adjacent<K>(b1 + j, wide, u);
            load_adjacent<K>(a2 + j, wide, v);
#pragma unroll
            for (int i = 0; i < K; i++) {
                u128 acc = mul_wide(x[i], y[i]);
                mac(acc, u[i], v[i]);  // < 2 q^2
                x[i] = barrett_prod_lazy(acc, q, mh);
            }
        } else {
#pragma unroll
            for (int i = 0; i < K; i++) x[i] = barrett_prod_lazy(mul_wide(x[i], y[i]), q, mh);
        }
    }
    uint64_t q, mh;  // mh: barrett_prod constant (inputs are fully reduced)
    __device__ __forceinline__ uint64_t load(int j) const {
        if (k == 0) return barrett_prod_lazy(mul_wide(a1[j], a2[j]), q, mh);
        if (k == 2) return barrett_prod_lazy(mul_wide(b1[j], b2[j]), q, mh);
        u128 acc = mul_wide(a1[j], b2[j]);
        mac(acc, b1[j], a2[j]);  // < 2 q^2
        return barrett_prod_lazy(acc, q, mh);
    }
    __device__ __forceinline__ void store(int, uint64_t) const {}
};
struct TensorSrc {
    PtrBatch pb;
    const uint64_t* sb;  // NTT-form R limbs: [item][4][nr]
    DevConsts dc;
    __device__ __forceinline__ int prime(int row) const {
        const int l = row % dc.nqr;
        return l < dc.nq ? l : dc.idx_r + (l - dc.nq);
    }
    __device__ __forceinline__ TensorRow bind(int row) const {
        const int nqr = dc.nqr, nq = dc.nq, nr = dc.nr, logn = dc.logn;
        const int item = row / (3 * nqr), w = row % (3 * nqr), k = w / nqr, l = w % nqr;
        TensorRow t;
        t.k = k;
        const int pi = l < nq ? l : dc.idx_r + (l - nq);
        t.q = dc.mods[pi]; t.mh = dc.mu_prod[pi];
        if (l < nq) {
            const uint64_t* A = pb.a[item];
            const uint64_t* B = pb.b[item];
            t.a1 = A + ((size_t)l << logn); t.b1 = A + ((size_t)(nq + l) << logn);
            t.a2 = B + ((size_t)l << logn); t.b2 = B + ((size_t)(nq + l) << logn);
        } else {
            const int r = l - nq;
            const uint64_t* base = sb + (((size_t)item * 4 * nr) << logn);
            t.a1 = base + ((size_t)(0 * nr + r) << logn); t.b1 = base + ((size_t)(1 * nr + r) << logn);
            t.a2 = base + ((size_t)(2 * nr + r) << logn); t.b2 = base + ((size_t)(3 * nr + r) << logn);
        }
        return t;
    }
};

// sum_d digit_d * key_d at K points: [0, 4q) for one digit (fully reduced
// factors), else [0, q). All points' operands of a digit are loaded before they
// are used. (Ordinary loads: a kernel that starts before its predecessor ends must
// not read the predecessor's results through the read-only path.)
template <int K>
__device__ __forceinline__ void key_product(const uint64_t* dig, const uint64_t* key, size_t ds, size_t ks, int ndig,
                                            uint64_t q, uint64_t mh, uint64_t ml, uint64_t mp, const int (&j)[K],
                                            uint64_t* x) {
    uint64_t a[K], b[K];
    if (ndig == 1) {
#pragma unroll
        for (int i = 0; i < K; i++) {
            a[i] = dig[j[i]];
            b[i] = key[j[i]];
        }
#pragma unroll
        for (int i = 0; i < K; i++) x[i] = barrett_prod_lazy(mul_wide(a[i], b[i]), q, mp);
        return;
    }
    u128 acc[K];
#pragma unroll
    for (int i = 0; i < K; i++) acc[i] = u128{0, 0};
    for (int d = 0; d < ndig; d++, dig += ds, key += ks) {
#pragma unroll
        for (int i = 0; i < K; i++) {
            a[i] = dig[j[i]];
            b[i] = key[j[i]];
        }
#pragma unroll
        for (int i = 0; i < K; i++) mac(acc[i], a[i], b[i]);
    }
#pragma unroll
    for (int i = 0; i < K; i++) x[i] = barrett128(acc[i], q, mh, ml);
}

// K6b source: inner product with the relinearisation key over Q|P
struct KeyIPRow {
    static constexpr bool kLoadMany = true;
    const uint64_t* dig;  // limb m of digit 0 (digit stride ds)
    const uint64_t* key;  // limb m, half h of digit 0 (digit stride ks)
    size_t ds, ks;
    int dnum;
    uint64_t q, mh, ml, mp;
    // [0, 4q) (one digit) or [0, q)
    template <int K>
    __device__ __forceinline__ void load_n(const int (&j)[K], uint64_t* x) const {
        key_product<K>(dig, key, ds, ks, dnum, q, mh, ml, mp, j, x);
    }
    __device__ __forceinline__ void store(int, uint64_t) const {}
};
struct KeyIPSrc {
    const uint64_t* sd2;  // [item][ndig][npq]
    const uint64_t* rlk;  // [ndig][2][npq]
    DevConsts dc;
    int ndig;             // digits: dnum (hybrid) or q_count * pieces (gadget)
    int m0 = 0, nm = 0;   // rows cover limbs m0 .. m0+nm-1 of Q|P (nm = 0: all of Q|P)
    __device__ __forceinline__ int prime(int row) const { return m0 + row % (nm ? nm : dc.npq); }
    __device__ __forceinline__ KeyIPRow bind(int row) const {
        const int npq = dc.npq, logn = dc.logn, per = nm ? nm : npq;
        const int item = row / (2 * per), w = row % (2 * per), h = w / per, m = m0 + w % per;
        KeyIPRow r;
        r.dig = sd2 + (((size_t)item * ndig * npq + m) << logn);
        // key limbs: [digit][a|b][Q|P] of the top level; a level reads its live Q limbs and P
        const int km = m < dc.nq ? m : dc.key_nq + (m - dc.nq);
        r.key = rlk + (((size_t)h * dc.key_npq + km) << logn);
        r.ds = (size_t)npq << logn;
        r.ks = (size_t)2 * dc.key_npq << logn;
        r.dnum = ndig;
        r.q = dc.mods[m]; r.mh = dc.mu_hi[m]; r.ml = dc.mu_lo[m]; r.mp = dc.mu_prod[m];
        return r;
    }
};

// Gadget decomposition source: rows (item, digit g = i*J + j, m) -> the j-th
// w-bit piece of limb i of a1*a2 (coefficient form), the same small integer in
// every prime m of Q|P.
struct GadgetRow {
    const uint64_t* x;
    int shift;
    uint64_t mask;
    __device__ __forceinline__ uint64_t load(int j) const { return (x[j] >> shift) & mask; }
    __device__ __forceinline__ void store(int, uint64_t) const {}
};
struct GadgetDigitSrc {
    const uint64_t* sd2;  // [item][nq]
    DevConsts dc;
    int pieces, w;
    __device__ __forceinline__ int prime(int row) const { return row % dc.npq; }
    __device__ __forceinline__ GadgetRow bind(int row) const {
        const int ndig = dc.nq * pieces;
        const int item = row / (ndig * dc.npq), g = (row / dc.npq) % ndig;
        GadgetRow r;
        r.x = sd2 + (((size_t)item * dc.nq + g / pieces) << dc.logn);
        r.shift = w * (g % pieces);
        r.mask = (w >= 64) ? ~0ULL : (((uint64_t)1 << w) - 1);
        return r;
    }
};

// K7 source of the T-base key switch: mod down P|Q -> q_l and add the tensor term
// (coefficient form): add + P^-1 x - sum_k rb_k (P/p_k) P^-1, as lazy Shoup products
// with pinv and md_c (see ModDownKeyRow), rb_k = [x_k (P/p_k)^-1]_{p_k}. Values below
// 8q. Four points' operands are in flight together. (A Barrett reduction of the P limb
// for every prime of Q and exact products: column pass of 90 rows at N = 32768 48 us; 23 us.)
struct ModDownAddRow {
    static constexpr bool kLoadMany = true;
    const uint64_t* x;    // limb l of the Q|P polynomial
    const uint64_t* xp;   // limb 0 of its P part
    const uint64_t* add;  // limb l of the term to add, or null
    const uint64_t* pmods;
    const uint64_t* phatinv;
    const uint64_t* phatinvs;
    const tw_t* c;        // md_c of prime l: [np], with Shoup companions
    size_t limb;
    int np;
    uint64_t q, pinv, pinvs;
    template <int K>
    __device__ __forceinline__ void load_n(const int (&j)[K], uint64_t* v) const {
        uint64_t y[K], z[K];
#pragma unroll
        for (int i = 0; i < K; i++) {
            y[i] = xp[j[i]];
            z[i] = x[j[i]];
            v[i] = add ? add[j[i]] : 0;
        }
#pragma unroll
        for (int i = 0; i < K; i++) v[i] += shoup4(z[i], pinv, pinvs, q);  // below 5q
        for (int k = 0; k < np; k++) {
            if (k) {
#pragma unroll
                for (int i = 0; i < K; i++) y[i] = xp[k * limb + j[i]];
            }
            if (np > 1) {
                const uint64_t h = phatinv[k], hs = phatinvs[k], p = pmods[k];
#pragma unroll
                for (int i = 0; i < K; i++) y[i] = shoup(y[i], h, hs, p);
            }
            const ulonglong2 w = c[k];
#pragma unroll
            for (int i = 0; i < K; i++) v[i] = csub63(v[i], q << 2) + shoup4(y[i], w.x, w.y, q);
        }
    }
    __device__ __forceinline__ void store(int, uint64_t) const {}
};
struct ModDownAddSrc {
    const uint64_t* se;   // [item][2][npq]
    const uint64_t* sd;   // [item][2][nq] or null
    DevConsts dc;
    __device__ __forceinline__ int prime(int row) const { return row % dc.nq; }
    __device__ __forceinline__ ModDownAddRow bind(int row) const {
        const int nq = dc.nq, npq = dc.npq, logn = dc.logn;
        const int item = row / (2 * nq), w = row % (2 * nq), h = w / nq, l = w % nq;
        ModDownAddRow r;
        const uint64_t* poly = se + (((size_t)item * 2 + h) * npq << logn);
        r.x = poly + ((size_t)l << logn);
        r.xp = poly + ((size_t)nq << logn);
        r.add = sd ? sd + (((size_t)(item * 2 + h) * nq + l) << logn) : nullptr;
        r.pmods = dc.mods + dc.idx_p;
        r.phatinv = dc.phatinv_p;
        r.phatinvs = dc.phatinv_ps;
        r.c = dc.md_c + (size_t)l * dc.np;
        r.limb = (size_t)1 << logn;
        r.np = dc.np;
        r.q = dc.mods[l];
        r.pinv = dc.pinv_q[l]; r.pinvs = dc.pinv_qs[l];
        return r;
    }
};

// K7 source of the key-switch tail: add - P^-1 [x_P]_q over Q. K6b stores the P
// limbs as rb_k = [x_k (P/p_k)^-1]_{p_k} (SeFoldRowsP), so that
//   P^-1 [x_P]_q = sum_k rb_k (P/p_k) P^-1  mod q
// is one lazy Shoup product per special prime with the constants
// md_c = -(P/p_k) P^-1 mod q: the reduction of every P limb for every prime of Q
// (and a 128-bit Barrett reduction and a product by P^-1) took 2.5 times the
// multiplies at two special primes. Values below 5q.
struct ModDownKeyRow {
    static constexpr bool kLoadMany = true;
    const uint64_t* xp;   // P limb 0
    const uint64_t* add;  // limb l of the term to add, or null
    const tw_t* c;        // md_c of prime l: [np], with Shoup companions
    size_t limb;
    int np;
    uint64_t q;
    template <int K>
    __device__ __forceinline__ void load_n(const int (&j)[K], uint64_t* x) const {
        uint64_t y[K];
#pragma unroll
        for (int i = 0; i < K; i++) {
            y[i] = xp[j[i]];
            x[i] = add ? add[j[i]] : 0;
        }
        for (int k = 0; k < np; k++) {
            if (k) {
#pragma unroll
                for (int i = 0; i < K; i++) y[i] = xp[k * limb + j[i]];
            }
            const ulonglong2 w = c[k];
#pragma unroll
            for (int i = 0; i < K; i++) x[i] = csub63(x[i], q << 2) + shoup4(y[i], w.x, w.y, q);
        }
    }
    __device__ __forceinline__ void store(int, uint64_t) const {}
};
struct ModDownKeySrc {
    const uint64_t* se;   // [item][2][npq], P limbs scaled
    const uint64_t* sd;   // [item][2][nq] or null
    DevConsts dc;
    __device__ __forceinline__ int prime(int row) const { return row % dc.nq; }
    __device__ __forceinline__ ModDownKeyRow bind(int row) const {
        const int nq = dc.nq, logn = dc.logn;
        const int item = row / (2 * nq), w = row % (2 * nq), h = w / nq, l = w % nq;
        ModDownKeyRow r;
        r.xp = se + ((((size_t)item * 2 + h) * dc.npq + nq) << logn);
        r.add = sd ? sd + (((size_t)(item * 2 + h) * nq + l) << logn) : nullptr;
        r.c = dc.md_c + (size_t)l * dc.np;
        r.limb = (size_t)1 << logn;
        r.np = dc.np;
        r.q = dc.mods[l];
        return r;
    }
};

struct OutCtDst {  // rows: (item, h, l) -> out[item] + (h*nq + l)*N
    PtrBatch pb;
    int logn, nq;
    __device__ __forceinline__ int prime(int row) const { return row % nq; }
    __device__ __forceinline__ PtrRow bind(int row) const {
        const int item = row / (2 * nq), w = row % (2 * nq);
        return PtrRow{pb.o[item] + ((size_t)w << logn)};
    }
};

// rows (item, h, k) -> limb nq + k (P part) of se ([item][2][npq]), stored times
// (P/p_k)^-1 mod p_k (folded into the inverse transform's last-stage constants)
struct SeFoldRowsP {
    uint64_t* se;
    int logn, nq, np, npq;
    const tw_t* fold_base;  // DevConsts::p_fold
    __device__ __forceinline__ int prime(int row) const { return nq + row % np; }
    __device__ __forceinline__ PtrRow bind(int row) const {
        const int item = row / (2 * np), w = row % (2 * np), h = w / np, k = w % np;
        return PtrRow{se + (((size_t)(item * 2 + h) * npq + nq + k) << logn)};
    }
    __device__ __forceinline__ const tw_t* fold(int row) const { return fold_base + 2 * (row % np); }
};

// Output store of the key-switch tail: adds P^-1 * sum_d digit_d * key_d[h] at
// limb l of Q (all NTT form, fully reduced) to the transformed value.
struct OutKeyRow {
    static constexpr bool kStoreMany = true;
    uint64_t* p;
    const uint64_t* dig;  // limb l of digit 0, digit stride ds
    const uint64_t* key;  // limb l of half h of digit 0, digit stride ks
    size_t ds, ks;
    int ndig;
    uint64_t q, mh, ml, mp, pinv, pinvs;
    const uint64_t* extra;  // a term in NTT form to add, or null
    // v below 8q
    template <int K>
    __device__ __forceinline__ void store_n(const int (&j)[K], const uint64_t (&v)[K]) const {
        uint64_t ip[K];
        key_product<K>(dig, key, ds, ks, ndig, q, mh, ml, mp, j, ip);
#pragma unroll
        for (int i = 0; i < K; i++)
            ip[i] = reduce_from(csub63(v[i], q << 2) + shoup4(ip[i], pinv, pinvs, q), q, 3);
        if (extra) {
            uint64_t e[K];
#pragma unroll
            for (int i = 0; i < K; i++) e[i] = extra[j[i]];
#pragma unroll
            for (int i = 0; i < K; i++) ip[i] = add_mod(ip[i], e[i], q);
        }
#pragma unroll
        for (int i = 0; i < K; i++) p[j[i]] = ip[i];
    }
};
// NTT-form terms that the key-switch tail adds to the output halves h >= from:
// base + item * stride + ((h - from) nq + l) N (base null: none)
struct KsExtra {
    const uint64_t* base = nullptr;
    size_t stride = 0;
    int from = 0;
};
struct OutCtKeyDst {  // rows: (item, h, l) -> out[item] + (h*nq + l)*N
    PtrBatch pb;
    const uint64_t* sd2;  // NTT-form digits [item][ndig][npq]
    const uint64_t* rlk;  // [ndig][2][Q|P] of the top level
    DevConsts dc;
    int ndig;
    KsExtra ex;
    __device__ __forceinline__ int prime(int row) const { return row % dc.nq; }
    __device__ __forceinline__ OutKeyRow bind(int row) const {
        const int nq = dc.nq, logn = dc.logn;
        const int item = row / (2 * nq), w = row % (2 * nq), h = w / nq, l = w % nq;
        OutKeyRow r;
        r.p = pb.o[item] + ((size_t)w << logn);
        r.dig = sd2 + (((size_t)item * ndig * dc.npq + l) << logn);
        r.key = rlk + (((size_t)h * dc.key_npq + l) << logn);
        r.ds = (size_t)dc.npq << logn;
        r.ks = (size_t)2 * dc.key_npq << logn;
        r.ndig = ndig;
        r.q = dc.mods[l]; r.mh = dc.mu_hi[l]; r.ml = dc.mu_lo[l]; r.mp = dc.mu_prod[l];
        r.pinv = dc.pinv_q[l]; r.pinvs = dc.pinv_qs[l];
        r.extra = ex.base && h >= ex.from ? ex.base + item * ex.stride + (((size_t)(h - ex.from) * nq + l) << logn) : nullptr;
        return r;
    }
};
// The same over a key product that key_ip.cuh has summed and scaled by P^-1
// (limb l of se's Q part)
struct OutSumRow {
    static constexpr bool kStoreMany = true;
    uint64_t* p;
    const uint64_t* x;
    uint64_t q;
    // v below 8q
    template <int K>
    __device__ __forceinline__ void store_n(const int (&j)[K], const uint64_t (&v)[K]) const {
        uint64_t y[K];
#pragma unroll
        for (int i = 0; i < K; i++) y[i] = x[j[i]];
#pragma unroll
        for (int i = 0; i < K; i++) p[j[i]] = reduce_from(csub63(v[i], q << 2) + y[i], q, 3);
    }
};
struct OutCtSumDst {  // rows: (item, h, l) -> out[item] + (h*nq + l)*N
    PtrBatch pb;
    const uint64_t* se;  // [item][2][npq]
    DevConsts dc;
    __device__ __forceinline__ int prime(int row) const { return row % dc.nq; }
    __device__ __forceinline__ OutSumRow bind(int row) const {
        const int nq = dc.nq, logn = dc.logn;
        const int item = row / (2 * nq), w = row % (2 * nq), h = w / nq, l = w % nq;
        return OutSumRow{pb.o[item] + ((size_t)w << logn), se + (((size_t)(item * 2 + h) * dc.npq + l) << logn), dc.mods[l]};
    }
};
static inline OutCtDst plain_of(const OutCtSumDst& d) { return OutCtDst{d.pb, d.dc.logn, d.dc.nq}; }
// the column pass of a split transform writes plain values; only the block
// kernel's final store runs the epilogue
static inline OutCtDst plain_of(const OutCtKeyDst& d) { return OutCtDst{d.pb, d.dc.logn, d.dc.nq}; }

// rows (item, limb) of the first polynomial of consecutive 3-polynomial tensors
struct TensorA2 {
    const uint64_t* tz;
    int logn, nq;
    __device__ __forceinline__ int prime(int row) const { return row % nq; }
    __device__ __forceinline__ PtrRow bind(int row) const {
        const int item = row / nq, l = row % nq;
        return PtrRow{const_cast<uint64_t*>(tz) + (((size_t)item * 3 * nq + l) << logn)};
    }
};

// decrypt: INTT over Q of (a*s + b), then the rounding
struct DecSrc {
    const uint64_t* ct;
    const uint64_t* sk;
    DevConsts dc;
    struct Row {
        static constexpr bool kLoadAdj = true;
        const uint64_t *a, *b, *s;
        uint64_t q, mh, ml;
        template <int K>
        __device__ __forceinline__ void load_adj(int j, uint64_t* x) const {
            const bool wide = wide_ok(a) && wide_ok(b) && wide_ok(s);
            uint64_t y[K], z[K];
            load_adjacent<K>(a + j, wide, x);
            load_adjacent<K>(s + j, wide, y);
            load_adjacent<K>(b + j, wide, z);
#pragma unroll
            for (int i = 0; i < K; i++)
                x[i] = csub63(barrett_prod_lazy(mul_wide(x[i], y[i]), q, mh), q << 1) + z[i];
        }
        // a and s fully reduced: one-high-product Barrett (mh holds its constant); below 3q
        __device__ __forceinline__ uint64_t load(int j) const {
            return csub63(barrett_prod_lazy(mul_wide(a[j], s[j]), q, mh), q << 1) + b[j];
        }
        __device__ __forceinline__ void store(int, uint64_t) const {}
    };
    __device__ __forceinline__ int prime(int row) const { return row % dc.nq; }
    __device__ __forceinline__ Row bind(int row) const {
        const int item = row / dc.nq, l = row % dc.nq;
        const size_t lq = (size_t)dc.nq << dc.logn;
        Row r;
        r.a = ct + item * 2 * lq + ((size_t)l << dc.logn);
        r.b = r.a + lq;
        r.s = sk + ((size_t)l << dc.logn);
        r.q = dc.mods[l]; r.mh = dc.mu_prod[l]; r.ml = 0;
        return r;
    }
};


// an inverse transform's rows (item, limb of Q) stored at the digits' own limbs
// ([item][dnum][Q|P], limb i in digit i / alpha), or one after the other
struct DigitRowsIO {
    uint64_t* base;
    int logn, nq;
    size_t item, digit;  // strides in rows
    int alpha;
    __device__ __forceinline__ int prime(int row) const { return row % nq; }
    __device__ __forceinline__ PtrRow bind(int row) const {
        const int l = row % nq;
        return PtrRow{base + (((row / nq) * item + (l / alpha) * digit + l) << logn)};
    }
};

// Digits of one prime each need no lift kernel: a digit's word in the prime of
// another limb is x, less q_d where the key switch's single-precision quotient
// estimate x / q_d rounds to 1, and the transform over Q|P takes it as it loads
// (7 digits of 8 ciphertexts at N = 16384: a 29 us launch and its 59 MB less). The
// coefficients then stand in se (free until the tail), which the transforms of the
// digits' own limbs do not overwrite.
static inline bool lift_in_ntt(const DevConsts& dc) { return dc.alpha == 1 && dc.dnum == dc.nq; }
// where the digits' coefficient-form limbs go
static inline DigitRowsIO digit_rows(const DevConsts& dc, const MulScratch& m) {
    if (lift_in_ntt(dc)) return DigitRowsIO{m.se, dc.logn, dc.nq, (size_t)dc.nq, 0, 1};
    return DigitRowsIO{m.sd2, dc.logn, dc.nq, (size_t)dc.dnum * dc.npq, (size_t)dc.npq, dc.alpha};
}
// smallest x whose single-precision value is that of q (x / q then rounds to 1; below it, to less)
__device__ __forceinline__ uint64_t float_equal_from(uint64_t q) {
    const float f = __ull2float_rn(q);
    const uint64_t hi = (uint64_t)f, lo = (uint64_t)__uint_as_float(__float_as_uint(f) - 1);
    if (hi - lo < 2) return hi;  // exact below 2^24
    return ((hi + lo) >> 1) + (__float_as_uint(f) & 1);  // the tie goes to the even one
}
struct LiftOneRow {
    static constexpr bool kLoadMany = true;
    const uint64_t* x;
    uint64_t from, less;  // x >= from: plus less = -q_d mod q
    uint64_t q, mh;       // reduce: x may exceed 4q
    bool reduce;
    // below 5q
    template <int K>
    __device__ __forceinline__ void load_n(const int (&j)[K], uint64_t* v) const {
#pragma unroll
        for (int i = 0; i < K; i++) v[i] = x[j[i]];
#pragma unroll
        for (int i = 0; i < K; i++) {
            const uint64_t add = v[i] >= from ? less : 0;
            if (reduce) v[i] -= __umul64hi(v[i], mh) * q;
            v[i] += add;
        }
    }
    __device__ __forceinline__ void store(int, uint64_t) const {}
};
struct LiftOneSrc {  // rows (item, digit, limb of Q|P)
    const uint64_t* x;  // [item][nq], coefficient form
    DevConsts dc;
    __device__ __forceinline__ int prime(int row) const { return row % dc.npq; }
    __device__ __forceinline__ LiftOneRow bind(int row) const {
        const int m = row % dc.npq, g = row / dc.npq % dc.dnum;
        const uint64_t qd = dc.mods[g], q = dc.mods[m], mh = dc.mu_hi[m];
        LiftOneRow r;
        r.x = x + ((size_t)(row / dc.npq) << dc.logn);  // item * nq + digit
        r.from = m == g ? ~0ULL : float_equal_from(qd);
        r.less = q - barrett64(qd, q, mh);
        r.q = q; r.mh = mh;
        r.reduce = (qd >> 2) > q;
        return r;
    }
};

// INTT over Q of the four input polynomials, Q -> R, NTT over R, fused tensor +
// INTT over Q|R: steps shared by kbfv_mul and the fused multiply-relinearise.
void mul_front(const DevConsts& dc, const PtrBatch& pb, int count, const MulScratch& m, cudaStream_t st);
// K2 and K5 (k5_kernels.cuh), by the steps of the byte matrix products
template <int KS>
void k2_launch_m(const DevConsts& dc, const uint64_t* y, uint64_t* out, int polys, cudaStream_t st);
template <int KS>
void bconv_mma_launch_m(const DevConsts& dc, bool q2r, const uint64_t* in, uint64_t* out, int polys, cudaStream_t st);
template <int KS>
void k5_launch_m(const DevConsts& dc, int count, const MulScratch& m, uint64_t* out0, int mode, cudaStream_t st);
// K5: scale-and-round, R -> Q and (mode 1) the key-switch digit lift
void k5_launch(const DevConsts& dc, int count, const MulScratch& m, uint64_t* out0, int mode, cudaStream_t st);
// the key-switch lift of the digits' own limbs in sd2 ([item][dnum][npq]) into every other prime of Q|P (lift.cu)
void lift_launch(const DevConsts& dc, uint64_t* sd2, int count, cudaStream_t st);
// K6a: the digits' limbs (digit_rows) lifted and transformed over Q|P, into sd2
// ([item][dnum][npq]), fully reduced; `lift`: the lift is still to do
void digits_ntt(const DevConsts& dc, const MulScratch& m, int count, bool lift, cudaStream_t st);
// key-switch tail: key product, mod down and add, written to the outputs of pb
void ks_tail(const DevConsts& dc, const uint64_t* sd2, const uint64_t* key, int ndig, uint64_t* se,
             const uint64_t* add, const PtrBatch& pb, int count, cudaStream_t st, const KsExtra& ex = {});
// the auxiliary streams and fork / join events of the sub-batches (created once)
void ensure_branch_streams(Context& c);
// the whole multiply + relinearise of one sub-batch: K1..K5, the lift, K6a, K6b and K7
// (one launch less where the lift is inside K5 or K6a, one more for key products
// apart, and for each transform that takes two)
void mul_relin_chunk(const DevConsts& dc, const uint64_t* rlk, const PtrBatch& pb, int count, const MulScratch& m,
                     cudaStream_t st);
// the constants of a sub-batch beside another on a sibling stream
static inline DevConsts sibling_consts(const Context& c) {
    DevConsts d = c.dc;
    d.shape.tail_sms = 0;
    return d;
}
// The constants with the launch shapes of a multiply that runs as one stream
// (no sibling sub-batch on another stream to fill the SMs): 2^14-point
// transforms of up to shape.split_rows_alone rows run split.
static inline DevConsts alone_consts(const Context& c) {
    DevConsts d = c.dc;
    d.shape.split_rows14 = d.shape.split_rows_alone;
    return d;
}
