// libkbfv: the reference's key switch over the auxiliary T base (KLSS) and its
// pieces as entry points.
#include "key_ip.cuh"
#include "pipeline.cuh"

// blocks of at most 1, 2, 4, 8 or 16 primes; 4, 8 or 12 T primes
static void klss_block_to_t(const DevConsts& dc, const KlssConsts& kc, const uint64_t* in, uint64_t* out, int which,
                            size_t in_stride, size_t out_stride, unsigned items, cudaStream_t st) {
    const dim3 grid((1u << dc.logn) / 256, (unsigned)(which == 0 ? kc.nqj : kc.nri), items);
    const int w = which == 0 ? dc.np : kc.gamma;
#define L_BT(W) klss_block_to_t_kernel<W><<<grid, 128, 0, st>>>(dc, kc, in, out, which, in_stride, out_stride)
    if (w <= 1) L_BT(1);
    else if (w <= 2) L_BT(2);
    else if (w <= 4) L_BT(4);
    else if (w <= 8) L_BT(8);
    else L_BT(kMaxBlk);
#undef L_BT
    check_launch("klss_block_to_t");
}
static void klss_t_to_pq(const DevConsts& dc, const KlssConsts& kc, const uint64_t* in, uint64_t* out, unsigned polys,
                         cudaStream_t st) {
    const dim3 grid((1u << dc.logn) / 256, (unsigned)kc.nri, polys);
#define L_TP(N) klss_t_to_pq_kernel<N><<<grid, 128, 0, st>>>(dc, kc, in, out)
    if (kc.nt <= 4) L_TP(4);
    else if (kc.nt <= 8) L_TP(8);
    else L_TP(kMaxT);
#undef L_TP
    check_launch("klss_t_to_pq");
}

// External product over T of `count` items, NTT form: out[item][h][block][t] =
// sum over digits i of dig[item][i][t] * key[h][i][block][t] mod t_t.
// Inside the inverse transform's loads, 8 rows of every T prime read each digit again
// and 6 each key limb, 755 MB of L2 reads for 3 items of 15 digits and 4 blocks at N
// = 32768: 147 us with the transform's block pass. Summed apart (key_ip.cuh) 63 + 37
// us, 27 of the 63 for the multiply-accumulates and 19 for the key from HBM. Four
// outputs a thread: with two, every digit is read four times (13 us more).
static void klss_ext_product(const DevConsts& dc, const KlssConsts& kc, const uint64_t* dig, const uint64_t* key,
                             uint64_t* out, int count, cudaStream_t st) {
    const size_t n = (size_t)1 << dc.logn, row = (size_t)kc.nt * n;
    KeyIpJob J{};
    J.dig = dig; J.key = key; J.out = out;
    J.dig_d = row; J.dig_item = kc.nqj * row;
    J.key_d = kc.nri * row;
    J.key_o = row; J.key_half = kc.nqj * J.key_d; J.per_half = kc.nri;
    J.out_o = row; J.out_item = (size_t)2 * kc.nri * row;
    J.ndig = kc.nqj; J.items = count; J.outputs = 2 * kc.nri; J.limbs = kc.nt;
    J.prime0 = dc.idx_t; J.nq = kc.nt;
    key_ip_launch<4>(dc, J, st);
}

// The lift of a block of one prime (klss_block_to_t_kernel at width 1) as the
// transform over T loads it: x where the quotient estimate is 0. (15 blocks of 3 items
// to 4 T primes at N = 32768: a 33 us launch and 94 MB less.)
struct BlockOneRow {
    static constexpr bool kLoadMany = true;
    const uint64_t* x;
    uint64_t from, q, mh, ml, bt;
    bool reduce;
    // below 5q
    template <int K>
    __device__ __forceinline__ void load_n(const int (&j)[K], uint64_t* v) const {
#pragma unroll
        for (int i = 0; i < K; i++) v[i] = x[j[i]];
#pragma unroll
        for (int i = 0; i < K; i++) {
            if (v[i] >= from) {  // quotient 1: one word in 2^24
                u128 acc{v[i], 0};
                sub128(acc, bt);
                v[i] = barrett128(acc, q, mh, ml);
            } else if (reduce) {
                v[i] -= __umul64hi(v[i], mh) * q;
            }
        }
    }
    __device__ __forceinline__ void store(int, uint64_t) const {}
};
struct BlockOneSrc {  // rows (item, block, T prime)
    const uint64_t* x;  // [item][nq], coefficient form; block b is limb b
    DevConsts dc;
    KlssConsts kc;
    __device__ __forceinline__ int prime(int row) const { return dc.idx_t + row % kc.nt; }
    __device__ __forceinline__ BlockOneRow bind(int row) const {
        const int t = row % kc.nt, b = row / kc.nt % kc.nqj, item = row / kc.nt / kc.nqj, p = dc.idx_t + t;
        const uint64_t qd = dc.mods[b];
        BlockOneRow r;
        r.x = x + (((size_t)item * dc.nq + b) << dc.logn);
        r.from = float_equal_from(qd);
        r.q = dc.mods[p]; r.mh = dc.mu_hi[p]; r.ml = dc.mu_lo[p];
        r.bt = kc.qj_mod_t[(size_t)b * kc.nt + t];
        r.reduce = (qd >> 2) > r.q;
        return r;
    }
};

// T-base key switch (the reference's KLSS, include/KeySwitch_23.cuh:244-330) of
// a1*a2 given in coefficient form over Q (sd2, [item][nq]); writes the P|Q
// results into se ([item][2][npq]).
static void klss_keyswitch(Context& c, const uint64_t* rlk_t, int count, const MulScratch& m, cudaStream_t st) {
    const DevConsts& dc = c.dc;
    const KlssConsts& kc = c.kc;
    // Qj blocks -> T (modUpQjtoT_23) and NTT over T
    const RowsIO digits = rows_io(dc, m.st1, dc.idx_t, c.nt);
    if (dc.np == 1) {
        ntt_fwd<BlockOneSrc, RowsIO, true>(dc, BlockOneSrc{m.sd2, dc, kc}, digits, count * kc.nqj * c.nt, st);
    } else {
        klss_block_to_t(dc, kc, m.sd2, m.st1, 0, (size_t)c.nq << c.logn, (size_t)kc.nqj * c.nt << c.logn, (unsigned)count, st);
        ntt_fwd<RowsIO, RowsIO, true>(dc, digits, digits, count * kc.nqj * c.nt, st);
    }
    // external product over T (external_product_T) and INTT over T
    klss_ext_product(dc, kc, m.st1, rlk_t, m.st2, count, st);
    ntt_inv(dc, rows_io(dc, m.st2, dc.idx_t, c.nt), rows_io(dc, m.st2, dc.idx_t, c.nt), count * 2 * kc.nri * c.nt, st);
    // centred T -> P|Q (modUpTtoPQl_23)
    klss_t_to_pq(dc, kc, m.st2, m.se, (unsigned)(count * 2), st);
}

static void mul_relin_klss_chunk(Context& c, const uint64_t* rlk_t, const PtrBatch& pb, int count,
                                 const MulScratch& m, cudaStream_t st) {
    const DevConsts& dc = c.dc;
    mul_front(c.dc, pb, count, m, st);
    k5_launch(c.dc, count, m, nullptr, 2, st);
    klss_keyswitch(c, rlk_t, count, m, st);
    ntt_fwd(dc, ModDownAddSrc{m.se, m.sd, dc}, OutCtDst{pb, dc.logn, dc.nq}, count * 2 * dc.nq, st);
}

extern "C" {

// ---- T-base key switch (the reference's KLSS) ------------------------------
int kbfv_context_klss(const kbfv_context* ctx, uint32_t* ri_blocks, uint32_t* qj_blocks, uint64_t* key_words) {
    return guarded([&] {
        const Context& c = CX(const_cast<kbfv_context*>(ctx));
        require_klss(c);
        if (ri_blocks) *ri_blocks = (uint32_t)c.kc.nri;
        if (qj_blocks) *qj_blocks = (uint32_t)c.kc.nqj;
        if (key_words) *key_words = (uint64_t)2 * c.kc.nqj * c.kc.nri * c.nt * c.n;
    });
}

int kbfv_rlk_to_klss(kbfv_context* ctx, const uint64_t* d_rlk, uint64_t* d_rlk_t, kbfv_stream stream) {
    return guarded([&] {
        Context& c = CX(ctx);
        require_batchable(c);
        require_klss(c);
        KB_REQUIRE(d_rlk && d_rlk_t, KBFV_ERR_INVALID, "null key pointer");
        cudaStream_t st = S(stream);
        const DevConsts& dc = c.dc;
        const KlssConsts& kc = c.kc;
        const int npq = dc.npq;
        uint64_t* coef = (uint64_t*)ensure_scratch(c, (size_t)c.dnum * 2 * npq * c.n * 8);
        // key [digit][a|b][Q|P] in NTT form -> coefficient form
        ntt_inv(dc, rows_io(dc, const_cast<uint64_t*>(d_rlk), 0, npq), rows_io(dc, coef, 0, npq),
                c.dnum * 2 * npq, st);
        // Ri blocks -> T (modUpPQtoT_23), written as [a|b][digit][Ri][T]
        for (int h = 0; h < 2; h++) {
            klss_block_to_t(dc, kc, coef + ((size_t)h * npq << c.logn),
                            d_rlk_t + ((size_t)h * c.dnum * kc.nri * c.nt << c.logn), 1, (size_t)2 * npq << c.logn,
                            (size_t)kc.nri * c.nt << c.logn, (unsigned)c.dnum, st);
        }
        RowsIO io = rows_io(dc, d_rlk_t, dc.idx_t, c.nt);
        ntt_fwd(dc, io, io, 2 * c.dnum * kc.nri * c.nt, st);
    });
}

int kbfv_klss_modup_qj_to_t(kbfv_context* ctx, const uint64_t* d_in, uint64_t* d_out, uint32_t polys,
                            kbfv_stream stream) {
    return guarded([&] {
        Context& c = CX(ctx);
        require_batchable(c);
        require_klss(c);
        KB_REQUIRE(polys <= 65535, KBFV_ERR_INVALID, "at most 65535 polynomials per call");
        if (!polys) return;
        klss_block_to_t(c.dc, c.kc, d_in, d_out, 0, (size_t)c.nq << c.logn, (size_t)c.kc.nqj * c.nt << c.logn, polys,
                        S(stream));
    });
}

int kbfv_klss_modup_pq_to_t(kbfv_context* ctx, const uint64_t* d_in, uint64_t* d_out, uint32_t polys,
                            kbfv_stream stream) {
    return guarded([&] {
        Context& c = CX(ctx);
        require_batchable(c);
        require_klss(c);
        KB_REQUIRE(polys <= 65535, KBFV_ERR_INVALID, "at most 65535 polynomials per call");
        if (!polys) return;
        klss_block_to_t(c.dc, c.kc, d_in, d_out, 1, (size_t)c.dc.npq << c.logn, (size_t)c.kc.nri * c.nt << c.logn, polys,
                        S(stream));
    });
}

int kbfv_klss_external_product(kbfv_context* ctx, const uint64_t* d_digits, const uint64_t* d_rlk_t,
                               uint64_t* d_out, uint32_t count, kbfv_stream stream) {
    return guarded([&] {
        Context& c = CX(ctx);
        require_batchable(c);
        require_klss(c);
        KB_REQUIRE(d_rlk_t, KBFV_ERR_NO_KEY, "T-base relinearisation key missing");
        const KlssConsts& kc = c.kc;
        klss_ext_product(c.dc, kc, d_digits, d_rlk_t, d_out, (int)count, S(stream));
        ntt_inv(c.dc, rows_io(c.dc, d_out, c.dc.idx_t, c.nt), rows_io(c.dc, d_out, c.dc.idx_t, c.nt),
                (int)count * 2 * kc.nri * c.nt, S(stream));
    });
}

int kbfv_klss_t_to_pq(kbfv_context* ctx, const uint64_t* d_in, uint64_t* d_out, uint32_t polys, kbfv_stream stream) {
    return guarded([&] {
        Context& c = CX(ctx);
        require_batchable(c);
        require_klss(c);
        KB_REQUIRE(polys <= 65535, KBFV_ERR_INVALID, "at most 65535 polynomials per call");
        if (!polys) return;
        klss_t_to_pq(c.dc, c.kc, d_in, d_out, polys, S(stream));
    });
}

int kbfv_relinearize_klss(kbfv_context* ctx, const uint64_t* d_rlk_t, const uint64_t* d_tensor, uint64_t* d_ct,
                          uint32_t count, kbfv_stream stream) {
    return guarded([&] {
        Context& c = CX(ctx);
        require_batchable(c);
        require_klss(c);
        KB_REQUIRE(d_rlk_t, KBFV_ERR_NO_KEY, "T-base relinearisation key missing");
        cudaStream_t st = S(stream);
        const DevConsts& dc = c.dc;
        const size_t lq = (size_t)c.nq * c.n;
        for (uint32_t off = 0; off < count; off += kMaxBatch) {
            const int cnt = (int)std::min<uint32_t>(kMaxBatch, count - off);
            uint8_t* base = ensure_scratch(c, mul_scratch_layout(c, cnt, nullptr).bytes);
            MulScratch m = mul_scratch_layout(c, cnt, base);
            const uint64_t* tz = d_tensor + (size_t)off * 3 * lq;
            uint64_t* out = d_ct + (size_t)off * 2 * lq;
            ntt_inv(dc, TensorA2{tz, dc.logn, dc.nq}, rows_io(dc, m.sd2, 0, dc.nq), cnt * dc.nq, st);
            klss_keyswitch(c, d_rlk_t, cnt, m, st);
            std::vector<uint64_t*> O(cnt);
            std::vector<const uint64_t*> Z(cnt);
            for (int i = 0; i < cnt; i++) { O[i] = out + (size_t)i * 2 * lq; Z[i] = nullptr; }
            PtrBatch pb = make_batch(Z.data(), Z.data(), O.data(), cnt);
            ntt_fwd(dc, ModDownAddSrc{m.se, nullptr, dc}, OutCtDst{pb, dc.logn, dc.nq}, cnt * 2 * dc.nq, st);
            launch_add(dc, out, 2 * lq, tz + lq, 3 * lq, out, 2 * lq, (size_t)cnt, 2 * dc.nq, dc.nq, st);
        }
    });
}

int kbfv_mul_relin_klss(kbfv_context* ctx, const uint64_t* d_rlk_t, const uint64_t* d_ct_a, const uint64_t* d_ct_b,
                        uint64_t* d_out, uint32_t count, kbfv_stream stream) {
    return guarded([&] {
        Context& c = CX(ctx);
        require_batchable(c);
        require_klss(c);
        KB_REQUIRE(d_rlk_t, KBFV_ERR_NO_KEY, "T-base relinearisation key missing");
        cudaStream_t st = S(stream);
        const size_t lq = (size_t)c.nq * c.n;
        for (uint32_t off = 0; off < count; off += kMaxBatch) {
            const int cnt = (int)std::min<uint32_t>(kMaxBatch, count - off);
            std::vector<const uint64_t*> A(cnt), B(cnt);
            std::vector<uint64_t*> O(cnt);
            for (int i = 0; i < cnt; i++) {
                A[i] = d_ct_a + (size_t)(off + i) * 2 * lq;
                B[i] = d_ct_b + (size_t)(off + i) * 2 * lq;
                O[i] = d_out + (size_t)(off + i) * 2 * lq;
            }
            PtrBatch pb = make_batch(A.data(), B.data(), O.data(), cnt);
            uint8_t* base = ensure_scratch(c, mul_scratch_layout(c, cnt, nullptr).bytes);
            MulScratch m = mul_scratch_layout(c, cnt, base);
            mul_relin_klss_chunk(c, d_rlk_t, pb, cnt, m, st);
        }
    });
}

}  // extern "C"
