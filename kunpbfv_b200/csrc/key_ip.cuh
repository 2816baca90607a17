// The products of a polynomial's digits with a key switch key, summed over the
// digits, as a kernel of its own:
//   out[i][o][m] = sum_d dig[i][d][m] key[o][d][m]  mod the prime of limb m,
// for items i, outputs o (the key's halves; over the T base its blocks too) and
// limbs m, all in NTT form.
//
// Memory bounds it: with the sums inside a transform's load or store every output
// row reads all digits and all of the key again, 16 bytes a multiply-accumulate,
// and a transform's CTA keeps too few loads in flight for the L2's rate. Here a
// thread holds one point of C items and O outputs, C + O loads for C O
// multiply-accumulates, and its sums (four registers each) are the only state.
// N = 16384, 8 items of 7 digits over 8 limbs: 36 us from HBM (14 for the bytes; 2.3
// waves of CTAs), and the transforms around it 27 -> 12 and 98 -> 37 us.
#pragma once
#include "internal.cuh"

struct KeyIpJob {
    const uint64_t* dig;  // item 0, digit 0, limb 0; limbs adjacent
    const uint64_t* key;  // output 0, digit 0, limb 0
    uint64_t* out;
    size_t dig_item, dig_d, key_o, key_half, key_d, out_item, out_o;  // strides in words
    int per_half;         // output o is number o % per_half of key half o / per_half
    int ndig, items, outputs, limbs;
    int prime0;           // limb m uses prime prime0 + m
    int nq, key_gap;      // limbs from nq on lie key_gap limbs further in the key (a level's key is the top's)
    // limbs below nq of the hybrid key switch: times scale (with companions), plus extra
    const uint64_t *scale, *scales;
    const uint64_t* extra;  // term added to outputs o >= extra_from, or null
    size_t extra_item, extra_o;
    int extra_from;
};

template <int C, int O>
static __global__ void __launch_bounds__(256, C * O > 8 ? 2 : 3) key_ip_kernel(KeyIpJob J, DevConsts c) {
    const int j = blockIdx.x * 256 + threadIdx.x;
    const int m = (int)blockIdx.y % J.limbs, o0 = (int)blockIdx.y / J.limbs * O, i0 = (int)blockIdx.z * C;
    // an item or output beyond the last one repeats it and is not stored
    const uint64_t* dig[C];
    const uint64_t* key[O];
    const size_t at = ((size_t)m << c.logn) + j;
    const size_t kat = ((size_t)(m < J.nq ? m : m + J.key_gap) << c.logn) + j;
#pragma unroll
    for (int i = 0; i < C; i++) dig[i] = J.dig + (size_t)min(i0 + i, J.items - 1) * J.dig_item + at;
#pragma unroll
    for (int o = 0; o < O; o++) {
        const int w = min(o0 + o, J.outputs - 1);
        key[o] = J.key + (size_t)(w / J.per_half) * J.key_half + (size_t)(w % J.per_half) * J.key_o + kat;
    }
    u128 acc[C][O];
#pragma unroll
    for (int i = 0; i < C; i++)
#pragma unroll
        for (int o = 0; o < O; o++) acc[i][o] = u128{0, 0};
#pragma unroll 2
    for (int d = 0; d < J.ndig; d++) {
        uint64_t a[C], b[O];
#pragma unroll
        for (int i = 0; i < C; i++) a[i] = dig[i][(size_t)d * J.dig_d];
#pragma unroll
        for (int o = 0; o < O; o++) b[o] = key[o][(size_t)d * J.key_d];
#pragma unroll
        for (int i = 0; i < C; i++)
#pragma unroll
            for (int o = 0; o < O; o++) mac(acc[i][o], a[i], b[o]);
    }
    const int p = J.prime0 + m;
    const uint64_t q = c.mods[p], mh = c.mu_hi[p], ml = c.mu_lo[p];
    const bool scaled = J.scale && m < J.nq;
    const uint64_t w = scaled ? J.scale[m] : 0, ws = scaled ? J.scales[m] : 0;
#pragma unroll
    for (int i = 0; i < C; i++)
#pragma unroll
        for (int o = 0; o < O; o++) {
            if (i0 + i >= J.items || o0 + o >= J.outputs) continue;
            uint64_t v = barrett128(acc[i][o], q, mh, ml);
            if (scaled) {
                v = shoup(v, w, ws, q);
                if (J.extra && o0 + o >= J.extra_from)
                    v = add_mod(v, J.extra[(size_t)(i0 + i) * J.extra_item + (size_t)(o0 + o - J.extra_from) * J.extra_o + at], q);
            }
            J.out[(size_t)(i0 + i) * J.out_item + (size_t)(o0 + o) * J.out_o + at] = v;
        }
}

template <int O>
static void key_ip_launch(const DevConsts& dc, KeyIpJob J, cudaStream_t st) {
    // a launch takes up to 65535 groups of four items
    constexpr int kItems = 65535 * 4;
    for (; J.items > kItems; J.items -= kItems) {
        KeyIpJob part = J;
        part.items = kItems;
        key_ip_launch<O>(dc, part, st);
        J.dig += kItems * J.dig_item;
        J.out += kItems * J.out_item;
        if (J.extra) J.extra += kItems * J.extra_item;
    }
    if (J.items <= 0) return;
    const int groups = (J.items + 3) / 4, per = (J.items + groups - 1) / groups;
    const dim3 grid((1u << dc.logn) / 256, (unsigned)(J.limbs * ((J.outputs + O - 1) / O)),
                    (unsigned)((J.items + per - 1) / per));
    switch (per) {
        case 1: key_ip_kernel<1, O><<<grid, 256, 0, st>>>(J, dc); break;
        case 2: key_ip_kernel<2, O><<<grid, 256, 0, st>>>(J, dc); break;
        case 3: key_ip_kernel<3, O><<<grid, 256, 0, st>>>(J, dc); break;
        default: key_ip_kernel<4, O><<<grid, 256, 0, st>>>(J, dc);
    }
    check_launch("key_ip");
}
