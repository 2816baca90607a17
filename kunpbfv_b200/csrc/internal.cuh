// Host-side plumbing shared by the library's translation units: errors and
// status codes, launch helpers of the NTT kernels, the dispatch of
// per-coefficient kernels, and the batch / scratch descriptors of the batched
// multiply.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <initializer_list>
#include <map>
#include <memory>
#include <mutex>
#include <stdexcept>
#include <string>
#include <vector>

#include "../../include/kbfv.h"
#include "context.cuh"
#include "host_math.hpp"
#include "kernels.cuh"
#include "ntt.cuh"
#include "ntt_cluster.cuh"
#include "klss.cuh"

using namespace kbfv;
namespace H = kbfv::host;

// ===========================================================================
// errors
// ===========================================================================
// last error message of the calling thread (kbfv_last_error)
extern thread_local std::string g_last_error;

struct KbfvError : std::runtime_error {
    int code;
    KbfvError(int c, const std::string& m) : std::runtime_error(m), code(c) {}
};

#define KB_CHECK_CUDA(call)                                                                        \
    do {                                                                                           \
        cudaError_t e_ = (call);                                                                   \
        if (e_ != cudaSuccess)                                                                     \
            throw KbfvError(e_ == cudaErrorMemoryAllocation ? KBFV_ERR_NOMEM : KBFV_ERR_CUDA,      \
                            std::string(#call) + ": " + cudaGetErrorString(e_));                   \
    } while (0)

#define KB_REQUIRE(cond, code, msg) \
    do {                            \
        if (!(cond)) throw KbfvError((code), (msg)); \
    } while (0)

template <class F>
static int guarded(F&& f) {
    try {
        f();
        return KBFV_OK;
    } catch (const KbfvError& e) {
        g_last_error = e.what();
        return e.code;
    } catch (const std::exception& e) {
        g_last_error = e.what();
        return KBFV_ERR_INVALID;
    }
}

static inline void check_launch(const char* what) {
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw KbfvError(KBFV_ERR_CUDA, std::string(what) + ": " + cudaGetErrorString(e));
}
// ===========================================================================
// launch helpers
// ===========================================================================
static inline cudaStream_t S(kbfv_stream s) { return (cudaStream_t)s; }
static inline unsigned blocks_for(size_t total, unsigned threads) { return (unsigned)((total + threads - 1) / threads); }
// grid of a grid-stride kernel: enough blocks to cover `total`, at most 2^20
static inline unsigned stride_blocks(size_t total, unsigned threads) {
    return (unsigned)std::min<size_t>((total + threads - 1) / threads, (size_t)1 << 20);
}

static inline bool aligned16(std::initializer_list<const void*> ps) {
    uintptr_t x = 0;
    for (const void* p : ps) x |= (uintptr_t)p;
    return (x & 15) == 0;
}
// out = x + y over `items` items of `per` rows of N words (limb = row % limbs), item strides in words
static inline void launch_add(const DevConsts& dc, const uint64_t* x, size_t xs, const uint64_t* y, size_t ys,
                              uint64_t* out, size_t os, size_t items, int per, int limbs, cudaStream_t st) {
    if (aligned16({x, y, out}))
        add_kernel<2><<<row_blocks<2>(items * per, dc.logn), 256, 0, st>>>(dc, x, xs, y, ys, out, os, per, limbs);
    else
        add_kernel<1><<<row_blocks<1>(items * per, dc.logn), 256, 0, st>>>(dc, x, xs, y, ys, out, os, per, limbs);
    check_launch("add");
}

// CTAs of `kernel` that fit on the device at once (SMs x CTAs per SM)
static inline int resident_ctas(const void* kernel, int threads, int smem) {
    int dev = 0, sms = 0, per = 0;
    KB_CHECK_CUDA(cudaGetDevice(&dev));
    KB_CHECK_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    KB_CHECK_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, threads, smem));
    return sms * std::max(per, 1);
}

// the same for launch shapes chosen at run time: cached per CTA size (64..512)
static inline int resident_ctas_at(const void* kernel, int threads, int smem, int (&cache)[4]) {
    const int i = std::min(3, std::max(0, __builtin_ctz((unsigned)threads) - 6));
    if (!cache[i]) cache[i] = resident_ctas(kernel, threads, smem);
    return cache[i];
}

// Allows `kernel` the dynamic shared memory of a launch of `bytes` (without it a launch
// may take 48 KB). The permission belongs to the kernel in one CUDA context, so it is
// asked for at each such launch (53 ns) instead of remembered per process, where
// another GPU's context would go without; and always for the same value, the kernel's
// largest at any CTA size (`most`), so that threads with different CTA sizes do not
// lower it for one another.
constexpr int kPlainSmem = 48 << 10;
template <class K>
static inline void allow_smem(K kernel, int bytes, int most) {
    if (bytes > kPlainSmem)
        KB_CHECK_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, most));
}

// A launch of clusters of `cluster` CTAs. `early`: it may start while the kernel
// before it on the stream still runs (programmatic dependent launch; the kernel
// waits before it touches memory that other kernels use).
template <class... P, class... A>
static void launch_clusters(bool early, void (*kernel)(P...), unsigned grid, unsigned threads, size_t smem,
                            unsigned cluster, cudaStream_t st, A... args) {
    cudaLaunchAttribute at[2]{};
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cfg.attrs = at;
    cfg.numAttrs = early ? 2 : 1;
    KB_CHECK_CUDA(cudaLaunchKernelEx(&cfg, kernel, P(args)...));
}

// Whether a launch of `rows` rows runs on clusters (ntt_cluster.cuh): where that
// takes less time than the other forms. The limits are measured on 148 SMs and for
// that chip only (us, cluster / other):
//   2^12: 128 rows 9.3 / 10.4, 148 rows 13.1 / 10.4      2^13: 128 rows 15.2 / 16.6, 148 rows 17.8 / 16.6
//   2^14: 8 rows 9.5 / 14.4, 26 rows 17 / 14.4 (the split form's single wave of up to
//         148 quarter-row CTAs, against more than one cluster CTA per SM),
//         40 rows 17 / 21.6, 64 rows 17 / 29, 112 rows 28 / 29, 128 rows 31 / 29
//   2^15: 8 rows 11 / 18, 16 rows 17-22 / 17             2^16: never (4 rows 19 / 17)
// Beside a sibling sub-batch the SMs that few rows leave idle are partly used and
// the limits lie lower, at 2^14 most of all (8 pairs, 7 digits: 447 us with a
// limit of 32, 469 with 96); a launch that waits early there holds SMs that the
// sibling could use, so only launches alone on the GPU start early.
static inline bool cluster_rows(const DevConsts& dc, int rows) {
    const bool alone = dc.shape.tail_sms > 0;
    switch (dc.logn) {
        case 12:
        case 13: return rows <= (alone ? 128 : 96);
        case 14: return alone ? rows <= 18 || (rows > 37 && rows <= 112) : rows <= 32;
        case 15: return rows <= 8;
        default: return false;
    }
}
template <int LOGN, class Src, class Dst, bool FULL>
static void launch_fwd_cluster(const DevConsts& dc, Src s, Dst d, int rows, cudaStream_t st, int row0 = 0) {
    using SH = ClusterShape<LOGN>;
    static_assert(SH::SMEM_BYTES <= kPlainSmem, "no permission needed");
    launch_clusters(dc.shape.tail_sms > 0, ntt_fwd_cluster_kernel<LOGN, Src, Dst, FULL>, (unsigned)rows << kClusterLog,
                    SH::THREADS, SH::SMEM_BYTES, 1u << kClusterLog, st, s, d, dc.tw_fwd, dc.mods, row0);
}
template <int LOGN, class Src, class Dst>
static void launch_inv_cluster(const DevConsts& dc, Src s, Dst d, int rows, cudaStream_t st, int row0 = 0) {
    using SH = ClusterShape<LOGN>;
    launch_clusters(dc.shape.tail_sms > 0, ntt_inv_cluster_kernel<LOGN, Src, Dst>, (unsigned)rows << kClusterLog,
                    SH::THREADS, SH::SMEM_BYTES, 1u << kClusterLog, st, s, d, dc.tw_inv, dc.mods, row0);
}

template <int LOGB, class Src, class Dst, bool FULL = true>
static void launch_fwd_block(const DevConsts& dc, Src s, Dst d, int rows, int logn, cudaStream_t st) {
    constexpr int SMEM = BlockShape<LOGB>::SMEM_BYTES;
    allow_smem(ntt_fwd_block_kernel<LOGB, Src, Dst, FULL>, SMEM, SMEM);
    // CTAs of this kernel resident at once on the device
    static const int resident = resident_ctas((const void*)ntt_fwd_block_kernel<LOGB, Src, Dst, FULL>,
                                              BlockShape<LOGB>::THREADS, SMEM);
    const int nblk = 1 << (logn - LOGB);
    ntt_fwd_block_kernel<LOGB, Src, Dst, FULL><<<rows * nblk, BlockShape<LOGB>::THREADS, SMEM, st>>>(
        s, d, dc.tw_fwd, dc.mods, logn, dc.shape.l2_prefetch ? resident : 0);
}

template <int LOGB, class Src, class Dst, bool WHOLE>
static void launch_inv_block(const DevConsts& dc, Src s, Dst d, int rows, int logn, cudaStream_t st) {
    constexpr int SMEM = BlockShape<LOGB>::SMEM_BYTES;
    allow_smem(ntt_inv_block_kernel<LOGB, Src, Dst, WHOLE>, SMEM, SMEM);
    // CTAs of this kernel resident at once on the device
    static const int resident = resident_ctas((const void*)ntt_inv_block_kernel<LOGB, Src, Dst, WHOLE>,
                                              BlockShape<LOGB>::THREADS, SMEM);
    const int nblk = 1 << (logn - LOGB);
    ntt_inv_block_kernel<LOGB, Src, Dst, WHOLE><<<rows * nblk, BlockShape<LOGB>::THREADS, SMEM, st>>>(
        s, d, dc.tw_inv, dc.mods, logn, dc.shape.l2_prefetch ? resident : 0);
}

// The view of a store target that the column pass of a split transform writes
// and the block kernel reads back: the target itself, unless its store adds an
// epilogue (an overload for that target returns its plain rows).
template <class Dst>
static inline Dst plain_of(const Dst& d) { return d; }

// At N = 2^14, launches of at most this many rows that do not run on clusters
// (cluster_rows) run as a radix-4 column pass and 2^12-point blocks: four times the
// CTAs cover the SMs, 12-17 us instead of 25 us for 19-45 rows on the B200. At 64
// rows the split alone is still faster, but beside a concurrent sub-batch it cost the
// batched multiply ~1%, so 64-row launches keep the whole-ring blocks. The
// default of LaunchShape::split_rows14 (KBFV_TUNE_SPLIT_ROWS).
constexpr int kSplitRows14Default = 48;
// The same threshold for a multiply that runs as one stream (batches below two
// sub-batches, the tensor-only multiply), where no sibling sub-batch fills the SMs
// that few whole-ring CTAs leave idle. Clusters take up to 112 of these rows; from there
// to 148 the split form is the slower one (33 us, whole rows 27), and a caller may set
// fewer. The default of LaunchShape::split_rows_alone (KBFV_TUNE_SPLIT_ROWS_ALONE).
constexpr int kSplitRowsAloneDefault = 148;

// A wave of whole-ring CTAs of 2^14 points (one per SM) takes 25 us however few
// rows it has. A launch that has the GPU to itself (tail_sms > 0; beside a sibling
// sub-batch the last wave's idle SMs are not idle) leaves the rows of a short last
// wave to a launch of clusters behind it: at most one cluster CTA per SM (18 rows,
// 8-13 us), or 64 rows (17 us) from the fourth wave on, where the other form of a
// short wave, the split of all rows below, has lost its lead. Us, with / without:
// forward 150 rows 33 / 39, 310: 57 / 63, 448: 80 / 86, 508: 88 / 95, 600: 104 / 113,
// 800: 144 / 150, 900: 160 / 170; inverse 150: 34 / 40, 448: 82 / 93, 900: 162 / 183.
static inline int tail_rows14(const LaunchShape& sh, int rows) {
    if (sh.tail_sms <= 0 || rows <= sh.split_rows14 || rows <= sh.tail_sms) return 0;
    const int full = rows / sh.tail_sms, rest = rows % sh.tail_sms;
    return rest << kClusterLog <= sh.tail_sms || (full >= 3 && rest <= 64) ? rest : 0;
}
// Whether `rows` transforms of 2^14 points run split: few rows, or two and three
// waves of which the last one holds at most 96 - 14 (waves - 1) rows; the split form
// takes 12 us plus 0.17 us a row (180 rows: 50 us whole, 39 split; 231: 52, 50; 333:
// 72, 64; but 256: 49, 52 and 370: 72, 71 not split).
static inline bool split14(const LaunchShape& sh, int rows) {
    if (rows <= sh.split_rows14) return true;
    if (sh.tail_sms <= 0) return false;
    const int waves = (rows + sh.tail_sms - 1) / sh.tail_sms;
    return waves >= 2 && waves <= 3 && rows - (waves - 1) * sh.tail_sms <= 96 - 14 * (waves - 1);
}

// Forward NTT of `rows` rows read through `s` and written through `d`. Few rows of
// 2^12..2^15 points run on clusters (cluster_rows). Else, for logn <= 14 one block
// kernel (N = 2^14: or as tail_rows14 and split14 say); for 15/16 a radix-8/16 column pass
// (s -> plain_of(d)) then 2^12-point block kernels from plain_of(d) to d in
// place (d must also be readable): several 256-thread CTAs per SM run faster
// than one 1024-thread CTA per 2^14-point block. FULL = false leaves outputs in [0, 8q) for consumers that reduce
// anyway (pipeline stages only).
template <class Src, class Dst, bool FULL = true>
static void ntt_fwd(const DevConsts& dc, Src s, Dst d, int rows, cudaStream_t st) {
    if (rows <= 0) return;
    if (cluster_rows(dc, rows)) {
        switch (dc.logn) {
            case 12: launch_fwd_cluster<12, Src, Dst, FULL>(dc, s, d, rows, st); break;
            case 13: launch_fwd_cluster<13, Src, Dst, FULL>(dc, s, d, rows, st); break;
            case 14: launch_fwd_cluster<14, Src, Dst, FULL>(dc, s, d, rows, st); break;
            default: launch_fwd_cluster<15, Src, Dst, FULL>(dc, s, d, rows, st); break;
        }
        check_launch("ntt_fwd");
        return;
    }
    switch (dc.logn) {
        case 10: launch_fwd_block<10, Src, Dst, FULL>(dc, s, d, rows, 10, st); break;
        case 11: launch_fwd_block<11, Src, Dst, FULL>(dc, s, d, rows, 11, st); break;
        case 12: launch_fwd_block<12, Src, Dst, FULL>(dc, s, d, rows, 12, st); break;
        case 13: launch_fwd_block<13, Src, Dst, FULL>(dc, s, d, rows, 13, st); break;
        case 14: {
            if (const int tail = tail_rows14(dc.shape, rows)) {
                launch_fwd_block<14, Src, Dst, FULL>(dc, s, d, rows - tail, 14, st);
                launch_fwd_cluster<14, Src, Dst, FULL>(dc, s, d, tail, st, rows - tail);
                break;
            }
            if (!split14(dc.shape, rows)) {
                launch_fwd_block<14, Src, Dst, FULL>(dc, s, d, rows, 14, st);
                break;
            }
            const size_t total = (size_t)rows << 12;
            using DP = decltype(plain_of(d));
            const DP dp = plain_of(d);
            ntt_fwd_col_kernel<2, Src, DP><<<stride_blocks(total, 256), 256, 0, st>>>(s, dp, dc.tw_fwd, dc.mods, 14, total);
            launch_fwd_block<12, DP, Dst, FULL>(dc, dp, d, rows, 14, st);
            break;
        }
        case 15: {
            const size_t total = (size_t)rows << 12;
            using DP = decltype(plain_of(d));
            const DP dp = plain_of(d);
            ntt_fwd_col_kernel<3, Src, DP><<<stride_blocks(total, 256), 256, 0, st>>>(s, dp, dc.tw_fwd, dc.mods, 15, total);
            launch_fwd_block<12, DP, Dst, FULL>(dc, dp, d, rows, 15, st);
            break;
        }
        case 16: {
            const size_t total = (size_t)rows << 12;
            using DP = decltype(plain_of(d));
            const DP dp = plain_of(d);
            ntt_fwd_col16_kernel<4, Src, DP><<<stride_blocks(total, 256), 256, 0, st>>>(s, dp, dc.tw_fwd, dc.mods, 16, total);
            launch_fwd_block<12, DP, Dst, FULL>(dc, dp, d, rows, 16, st);
            break;
        }
        default: throw KbfvError(KBFV_ERR_INVALID, "unsupported ring degree");
    }
    check_launch("ntt_fwd");
}

template <class Src, class Dst>
static void ntt_inv(const DevConsts& dc, Src s, Dst d, int rows, cudaStream_t st) {
    if (rows <= 0) return;
    if (cluster_rows(dc, rows)) {
        switch (dc.logn) {
            case 12: launch_inv_cluster<12>(dc, s, d, rows, st); break;
            case 13: launch_inv_cluster<13>(dc, s, d, rows, st); break;
            case 14: launch_inv_cluster<14>(dc, s, d, rows, st); break;
            default: launch_inv_cluster<15>(dc, s, d, rows, st); break;
        }
        check_launch("ntt_inv");
        return;
    }
    switch (dc.logn) {
        case 10: launch_inv_block<10, Src, Dst, true>(dc, s, d, rows, 10, st); break;
        case 11: launch_inv_block<11, Src, Dst, true>(dc, s, d, rows, 11, st); break;
        case 12: launch_inv_block<12, Src, Dst, true>(dc, s, d, rows, 12, st); break;
        case 13: launch_inv_block<13, Src, Dst, true>(dc, s, d, rows, 13, st); break;
        case 14: {
            if (const int tail = tail_rows14(dc.shape, rows)) {
                launch_inv_block<14, Src, Dst, true>(dc, s, d, rows - tail, 14, st);
                launch_inv_cluster<14, Src, Dst>(dc, s, d, tail, st, rows - tail);
                break;
            }
            if (!split14(dc.shape, rows)) {
                launch_inv_block<14, Src, Dst, true>(dc, s, d, rows, 14, st);
                break;
            }
            launch_inv_block<12, Src, Dst, false>(dc, s, d, rows, 14, st);
            const size_t total = (size_t)rows << 12;
            ntt_inv_col_kernel<2, Dst, Dst><<<stride_blocks(total, 256), 256, 0, st>>>(d, d, dc.tw_inv, dc.mods, 14, total);
            break;
        }
        case 15: {
            launch_inv_block<12, Src, Dst, false>(dc, s, d, rows, 15, st);
            const size_t total = (size_t)rows << 12;
            ntt_inv_col_kernel<3, Dst, Dst><<<stride_blocks(total, 256), 256, 0, st>>>(d, d, dc.tw_inv, dc.mods, 15, total);
            break;
        }
        case 16: {
            launch_inv_block<12, Src, Dst, false>(dc, s, d, rows, 16, st);
            const size_t total = (size_t)rows << 12;
            ntt_inv_col16_kernel<4, Dst, Dst><<<stride_blocks(total, 256), 256, 0, st>>>(d, d, dc.tw_inv, dc.mods, 16, total);
            break;
        }
        default: throw KbfvError(KBFV_ERR_INVALID, "unsupported ring degree");
    }
    check_launch("ntt_inv");
}

static inline RowsIO rows_io(const DevConsts& dc, uint64_t* base, int p0, int period) {
    return RowsIO{base, dc.logn, p0, period};
}
// bucketed MAX template dispatch for per-coefficient kernels
#define DISPATCH_MAXQ(nq, MACRO) \
    do {                         \
        if ((nq) <= 8) { MACRO(8); }       \
        else if ((nq) <= 16) { MACRO(16); } \
        else if ((nq) <= 24) { MACRO(24); } \
        else { MACRO(33); }                 \
    } while (0)

// the same by the steps of the byte matrix products (DevConsts::mm_ks)
#define DISPATCH_KS(ks, MACRO)          \
    do {                                \
        if ((ks) == 1) { MACRO(1); }    \
        else if ((ks) == 2) { MACRO(2); } \
        else if ((ks) == 4) { MACRO(4); } \
        else if ((ks) == 6) { MACRO(6); } \
        else { MACRO(9); }              \
    } while (0)

// context construction from a parameter set (tables in one device pool)
void build_context(Context& c, const kbfv_params& prm);
// pieces of a 60-bit residue in base 2^w
static inline int gadget_pieces(int w) { return (60 + w - 1) / w; }

// The context's scratch arena: grown to at least `bytes` (at least 64 MiB;
// never shrinks while the context lives). Synchronises the device when it grows.
uint8_t* ensure_scratch(Context& c, size_t bytes);

// ===========================================================================
// batch and scratch descriptors of the batched multiply
// ===========================================================================
constexpr int kMaxBatch = 128;  // pointer tables ride in kernel parameters
struct PtrBatch {
    const uint64_t* a[kMaxBatch];
    const uint64_t* b[kMaxBatch];
    uint64_t* o[kMaxBatch];
};

struct MulScratch {
    uint64_t *sa, *sb, *sc, *sd, *sd2, *se;
    uint64_t *st1, *st2;  // T-base key switch: digits [item][nqj][nt], products [item][2][nri][nt]
    size_t bytes;
};

static inline MulScratch mul_scratch_layout(const Context& c, int count, uint8_t* base) {
    const size_t limb = c.n * 8;
    const int npq = c.nq + c.np, nqr = c.nq + c.nr;
    size_t off = 0;
    MulScratch m{};
    auto take = [&](size_t limbs) {
        uint64_t* p = (uint64_t*)(base ? base + off : nullptr);
        off += limbs * limb;
        return p;
    };
    m.sa = take((size_t)count * 4 * c.nq);
    m.sb = take((size_t)count * 4 * c.nr);
    m.sc = take((size_t)count * 3 * nqr);
    m.sd = take((size_t)count * 2 * c.nq);
    m.sd2 = take((size_t)count * c.dnum * npq);
    m.se = take((size_t)count * 2 * npq);
    if (c.klss_ok) {
        m.st1 = take((size_t)count * c.kc.nqj * c.nt);
        m.st2 = take((size_t)count * 2 * c.kc.nri * c.nt);
    }
    m.bytes = off;
    return m;
}
// Sub-batches of a batched multiply hold at least Context::min_branch_pairs
// pairs (default 1; KBFV_TUNE_MIN_BRANCH_PAIRS). Two of them on two streams fill
// the SMs that one batch's launches leave idle, unless the whole batch is a few rows
// of a small ring: those launches run on clusters, last a few microseconds each and
// start early behind one another on one stream (ntt_cluster.cuh), and a second
// sequence of them costs more than its overlap gives. One / two sub-batches, us:
//   N = 4096, 2 primes: 2 pairs 59 / 73, 10 pairs 89 / 91, 16 pairs 109 / 107, 32 pairs 164 / 148
//   N = 8192, 3 primes: 2 pairs 70 / 82, 5 pairs 99 / 100, 8 pairs 133 / 119
//   N = 16384, 7 primes: 2 pairs 122 / 125, 3 pairs 183 / 168, 8 pairs 349 / 326
//   N = 32768, 14 primes: 2 pairs 466 / 409
// so up to 80 rows over Q and 2^19 points a batch is one sub-batch, until the caller
// chooses a number of sub-batches or their least size.
static inline int branch_count(const Context& c, int cnt) {
    const size_t rows = (size_t)4 * c.nq * cnt;
    if (!c.branches_chosen && rows <= 80 && (rows << c.logn) <= (size_t)1 << 19) return 1;
    return std::max(1, std::min(c.branches, cnt / std::max(1, c.min_branch_pairs)));
}
static inline size_t branch_region_bytes(const Context& c, int per) {
    return (mul_scratch_layout(c, per, nullptr).bytes + 255) & ~(size_t)255;
}
static inline size_t mul_scratch_need(const Context& c, int cnt) {
    const int nb = branch_count(c, cnt);
    const size_t whole = mul_scratch_layout(c, cnt, nullptr).bytes;
    return nb == 1 ? whole : std::max(whole, branch_region_bytes(c, (cnt + nb - 1) / nb) * nb);
}
static inline PtrBatch make_batch(const uint64_t* const* a, const uint64_t* const* b, uint64_t* const* o, int cnt) {
    PtrBatch pb;
    std::memset(&pb, 0, sizeof pb);
    for (int i = 0; i < cnt; i++) {
        pb.a[i] = a[i];
        pb.b[i] = b[i];
        pb.o[i] = o ? o[i] : nullptr;
    }
    return pb;
}

// Fused stages run as one block kernel for N <= 2^14; for split transforms
// (N = 2^15, 2^16, and launches of few rows at 2^14) the fused loader feeds
// the column pass and the store target is read back by the block kernel, which
// every functor here supports.
static inline void require_batchable(const Context& c) {
    KB_REQUIRE(c.logn >= 10 && c.logn <= 16, KBFV_ERR_UNSUPPORTED, "ring degree outside 2^10..2^16");
}
static inline void require_top(const Context& c) {
    KB_REQUIRE(!c.parent, KBFV_ERR_LEVEL, "keys and encryptions are made on the top-level context");
}
static inline void require_klss(const Context& c) {
    KB_REQUIRE(c.klss_ok, KBFV_ERR_INVALID,
               "context has no T-base key switch (needs T primes, q_count divisible by p_count, dnum = q_count / p_count)");
}

// opaque handle of the C ABI
struct kbfv_context {
    Context c;
};

static inline Context& CX(kbfv_context* h) {
    if (!h) throw KbfvError(KBFV_ERR_INVALID, "null context");
    return h->c;
}
