// Split-precision ("Ozaki scheme") block-pair contraction on the B200 5th
// generation tensor cores (tcgen05.mma, accumulators in tensor memory).
//
// Same schedule and task list as the plain FP64 path (one work item per
// (C block, 128 x nt) tile, all coalesced pairs of the C block accumulated
// before the single FP64 write), but the products run on integer-valued
// low-precision slices:
//
//  1. split (oz_split_kernel): every matricised operand row r of a block is
//     scaled by its own power of two 2^-e_r (e_r: exponent of the row's
//     largest magnitude) and cut into S slices of integers by round-to-nearest,
//       x = 2^(e_r - b0) * sum_s sigma_s * 2^(-b*s),  |sigma_s| <= 2^(b0) or 2^(b-1),
//     exactly, up to the dropped tail (Ozaki, Ogita, Oishi, Rump 2012; the
//     per-row power-of-two scaling of Mukunoki et al. 2020).  The permutation
//     of the block pair is applied here, so the slices are GEMM-ready.
//  2. slice products (oz_gemm_kernel): the products sigma_sa x sigma_sb with
//     sa + sb = l (a "level") share one scale, so each level accumulates in its
//     own TMEM accumulator.  INT8 slices accumulate exactly in INT32; BF16 and
//     FP8 E4M3 slices accumulate in FP32, exact while every partial sum stays
//     below 2^24, which the host guarantees by draining every chunk_kb k blocks.
//  3. recombination: after each pair (or chunk) the epilogue warps read the
//     level accumulators from TMEM and add
//       coeff * 2^(e_r + e_c - 2 b0) * sum_l 2^(-b l) * acc_l
//     into FP64 registers; the C tile is written once, in FP64.
// Only levels l <= S-1 are formed: S(S+1)/2 slice products per k step.
//
// The accumulator of level l sits in the nt tensor-memory columns from l * nt,
// and the N-side image of a k block holds its S slices one after the other, so
// the products of M-side slice sa with N-side slices 0 .. S-1-sa are one
// (S - sa) * nt columns wide product into levels sa .. S-1 (issued in pieces of
// at most 256 columns, the widest MMA).  One MMA per slice pair (nt = 64)
// reads the M-side slice from shared memory for every 64 columns: 6 KB per
// 32 clocks of products against 128 B per clock, which held the kernel to a
// third of the MMA rate (ladder o=40 v=240, BF16 x 4: 8.58 ms).
//
// Warp roles (320 threads): warps 0-7 epilogue (two per TMEM lane quarter, one
// tile row and half of the tile's columns per thread), warp 8 bulk-copy
// producer, warp 9 MMA issuer.  Operand tiles are stored in global memory as
// the exact shared-memory images the MMA reads (K-major core matrices, no
// swizzle), so each one moves with a single 1-D cp.async.bulk copy completing
// on the stage's mbarrier (no tensor maps, no multicast); one or two MMA k
// steps per pipeline stage, so even 8 slices leave room for 4 stages.
// Every mbarrier wait is bounded in time and reports through *err.
#include <cuda_bf16.h>
#include <cuda_fp8.h>

#include "ltg_device.cuh"

namespace ltg {

// k elements per 32-byte k block: 32 for 8-bit slices, 16 for BF16.
#ifndef LTG_OZ_KIND
void oz_kind_params(int kind, int *beta0, int *beta, int *esz, int *kbe, int64_t *maxprod) {
    switch (kind) {
    case kOzInt8: *beta0 = 6; *beta = 7; *esz = 1; *kbe = 32; *maxprod = 64 * 64; break;
    case kOzBf16: *beta0 = 6; *beta = 7; *esz = 2; *kbe = 16; *maxprod = 64 * 64; break;
    default:      *beta0 = 4; *beta = 5; *esz = 1; *kbe = 32; *maxprod = 16 * 16; break;
    }
}
#endif

// What one slice-products launch takes besides its template arguments.
struct OzGemmArgs {
    const DPanel *panels;
    const uint8_t *slices;
    const DOzTask *tasks;
    const DCBlock *cblks;
    const DOzItem *items;
    int32_t nitems;
    const int32_t *exps;
    double *c;
    int32_t add, swap, chunk_kb, max_nt;
    int32_t *err;
    uint64_t wait_ns;
    cudaStream_t s;
    const int2 *drange;
    const DCBlock *dests;
};

// The kernels of one kind.  Each kind is a translation unit of its own (compiled
// with LTG_OZ_KIND set to it), as this file's 51 kernels take several minutes
// one after the other; the unit without LTG_OZ_KIND holds the entry points.
template<int KIND> cudaError_t oz_launch_gemm(int S, const OzGemmArgs &a);
template<int KIND> cudaError_t oz_launch_split(int S, const DPanel *panels, const int4 *units, int32_t nunits,
                                               const double *a, const double *b, uint8_t *slices, int32_t *exps,
                                               cudaStream_t s);

namespace {

constexpr int kBM = 128;              // tile rows (TMEM lanes)
constexpr int kRowBytes = 32;         // k-block row length in shared memory (one MMA k step)
constexpr int kXTile = kBM * kRowBytes;   // 4 KB per M-side slice per stage
constexpr int kEpiWarps = 8;          // two per TMEM lane quarter
constexpr int kThreads = 32 * (kEpiWarps + 2);
// Widest N tile: S level accumulators in 512 tensor-memory columns, and at
// most 64 FP64 sums per epilogue thread.
__host__ __device__ constexpr int oz_max_nt(int S) { return 512 / S / 16 * 16 < 128 ? 512 / S / 16 * 16 : 128; }
// Whether the products of M-side slice sa take two MMAs (one is at most 256
// columns wide; fixed per slice count, so that the issuing loop has no branch).
template<int S>
__host__ __device__ constexpr bool two_pieces(int sa) { return (S - sa) * oz_max_nt(S) > 256; }
constexpr int kMaxStages = 8;
constexpr int kStageSmem = 200 * 1024;    // shared memory of all stages
constexpr uint64_t kWaitNs = 2000000000ull;   // 2 s: the drain waits after an abort
// Rows with a NaN or an infinity: a slice is the low word of an integer and a
// level sum is joined as integers, so neither can carry one.  The split pass marks
// the row where its exponent stands, and the products give NaN in what reads it.
constexpr uint32_t kInfHi = 0x7ff00000u;      // high word of an infinity
constexpr int32_t kNonFinite = 2000;          // exponent of a marked row (others: -1073 .. 1024)

__device__ __forceinline__ int64_t mixed_offset(int32_t lin, int n, const int32_t *ext,
                                                const int32_t *str) {
    int64_t off = 0;
    for (int i = n - 1; i >= 0; i--) {
        int32_t e = ext[i];
        int32_t q = lin / e;
        off += (int64_t)(lin - q * e) * str[i];
        lin = q;
    }
    return off;
}

// ---------------------------------------------------------------- split

// Four consecutive integer slice values packed for one store.  Integers become
// floats by bits (1.5 * 2^23 + i, exact); BF16 is then the float's high half
// (at most 7 significant bits), E4M3 one conversion per pair.
__device__ __forceinline__ float small_float(int i) { return __int_as_float(0x4B400000 + i) - 12582912.0f; }

template<int KIND> struct Pack4;
template<> struct Pack4<kOzInt8> {
    typedef uint32_t T;
    __device__ __forceinline__ static T pack(const int *v) {
        return __byte_perm(__byte_perm(v[0], v[1], 0x0040), __byte_perm(v[2], v[3], 0x0040), 0x5410);
    }
};
template<> struct Pack4<kOzE4m3> {
    typedef uint32_t T;
    __device__ __forceinline__ static T pack(const int *v) {
        const uint32_t lo = __nv_cvt_float2_to_fp8x2(make_float2(small_float(v[0]), small_float(v[1])), __NV_SATFINITE, __NV_E4M3);
        const uint32_t hi = __nv_cvt_float2_to_fp8x2(make_float2(small_float(v[2]), small_float(v[3])), __NV_SATFINITE, __NV_E4M3);
        return lo | (hi << 16);
    }
};
template<> struct Pack4<kOzBf16> {
    typedef uint2 T;
    __device__ __forceinline__ static T pack(const int *v) {
        uint2 r;
        r.x = __byte_perm(__float_as_uint(small_float(v[0])), __float_as_uint(small_float(v[1])), 0x7632);
        r.y = __byte_perm(__float_as_uint(small_float(v[2])), __float_as_uint(small_float(v[3])), 0x7632);
        return r;
    }
};

// Byte offset of (row r, byte kb_byte of k block kb, slice s) in the tile
// images of a panel.  Panels are stored as the exact shared-memory images
// the MMA reads: per (row tile, k block, slice) one TR x 32-byte tile,
// K-major without swizzle (8-row x 16-byte core matrices, the two 16-byte k
// halves 128 bytes apart, 8-row groups 256 bytes apart), so one pipeline
// stage is a single contiguous bulk copy per operand.
__device__ __forceinline__ int64_t tile_image_offset(int r, int TR, int nkb, int kb, int s, int S,
                                                     int kb_byte) {
    const int tile = r / TR, rr = r % TR;
    return ((int64_t)(tile * nkb + kb) * S + s) * (TR * 32) + (rr >> 3) * 256 + (kb_byte >> 4) * 128 +
           (rr & 7) * 16 + (kb_byte & 15);
}

// Units (panel, first row, rows, unused): a multiple of 8 rows of one panel,
// all of its k, as core tiles of 8 rows x 16 k spread over the CTA's warps (lane l
// takes row l / 4 and the four consecutive k of group l % 4, so that a warp
// stores whole 128- or 256-byte runs of the tile images).  Two passes over the
// unit: the rows' largest magnitudes, then the slices.  Bound by HBM: the
// operand in once, S slices out.  So that the second pass reads L2, a unit of
// long rows is 8 rows and two CTAs of 512 threads share an SM: 296 units of
// 8 x 4096 doubles are 78 MB of the 126 MB L2; with 32-row units and eight
// CTAs per SM both passes went to HBM.  Ladder o=40 v=240, BF16 x 4 (3.6 GB in,
// 3.7 GB out): 2.37 ms to 1.82; o=30 v=150, FP8 x 8: 0.59 to 0.37 ms.
// Slice s of t = x 2^(beta0 - e) is rint(t 2^(beta s)) of what the slices before
// it left: t + 1.5 * 2^(52 - beta s) rounds to it and holds it in its low word;
// what it leaves is exact.
constexpr int kSplitThreads = 512;
constexpr int kSplitWarps = kSplitThreads / 32;
constexpr int kKoffMax = 4096;        // k offsets tabulated per unit
constexpr int kUnitRowsMax = 256;

template<int KIND, int S>
__global__ void __launch_bounds__(kSplitThreads, 2)
oz_split_kernel(const DPanel *__restrict__ panels, const int4 *__restrict__ units,
                const double *__restrict__ A, const double *__restrict__ B,
                uint8_t *__restrict__ slices, int32_t *__restrict__ exps) {
    typedef typename Pack4<KIND>::T PT;
    constexpr int kEsz = KIND == kOzBf16 ? 2 : 1;
    constexpr int kKbe = 32 / kEsz;                  // elements per 32-byte k block
    constexpr int kBeta0 = KIND == kOzE4m3 ? 4 : 6, kBeta = kBeta0 + 1;
    __shared__ int32_t koff[kKoffMax];
    __shared__ int64_t roff[kUnitRowsMax];
    __shared__ uint32_t rhi[kUnitRowsMax], rlo[kUnitRowsMax];   // largest high word of |x|, all low words or'ed
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, lrow = lane >> 2, kq = lane & 3;
    const int4 un = units[blockIdx.x];
    const DPanel &P = panels[un.x];
    const double *src = (P.src ? B : A) + P.src_off;
    // k offsets: contiguous, tabulated, or computed per element (in 64 bits)
    const int K = P.K, mode = P.nk == 0 || (P.nk == 1 && P.kstr[0] == 1) ? 0 : (K <= kKoffMax && !P.wide ? 1 : 2);
    if (mode == 1)
        for (int k = threadIdx.x; k < K; k += kSplitThreads) koff[k] = (int32_t)mixed_offset(k, P.nk, P.kext, P.kstr);
    for (int i = threadIdx.x; i < un.z; i += kSplitThreads) {
        rhi[i] = 0;
        rlo[i] = 0;
        roff[i] = un.y + i < P.rows ? mixed_offset(un.y + i, P.nr, P.rext, P.rstr) : -1;
    }
    __syncthreads();
    const int nkt = (K + 15) >> 4, ngroups = un.z >> 3;
    // This warp's core tiles: every kSplitWarps-th of the unit's, row group by
    // row group.
    struct Walk {
        int rg, kt;
        __device__ __forceinline__ void wrap(int nkt) { while (kt >= nkt) { kt -= nkt; rg++; } }
    };
    // four elements of this lane's row and k group in tile w (zero outside)
    auto load4 = [&](const Walk &w, double *x) {
        const int64_t ro = w.rg < ngroups ? roff[w.rg * 8 + lrow] : -1;
        const int k0 = w.kt * 16 + kq * 4;
        const double *row = src + ro;
        if (ro >= 0 && mode == 0 && ((uintptr_t)row & 15) == 0 && k0 + 3 < K) {
            const double2 a = *reinterpret_cast<const double2 *>(row + k0);
            const double2 b = *reinterpret_cast<const double2 *>(row + k0 + 2);
            x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
            return;
        }
#pragma unroll
        for (int j = 0; j < 4; j++) {
            const int k = k0 + j;
            x[j] = ro >= 0 && k < K ? row[mode == 0 ? k : mode == 1 ? koff[k] : mixed_offset(k, P.nk, P.kext, P.kstr)]
                                    : 0.0;
        }
    };
    {
        // largest magnitudes, kept while the warp stays on its rows
        uint32_t hi = 0, lo = 0;
        int cur = -1;
        auto flush = [&]() {
            uint32_t h = hi, l = lo;
            h = max(h, __shfl_xor_sync(0xffffffffu, h, 1));
            h = max(h, __shfl_xor_sync(0xffffffffu, h, 2));
            l |= __shfl_xor_sync(0xffffffffu, l, 1);
            l |= __shfl_xor_sync(0xffffffffu, l, 2);
            if (kq == 0) {
                atomicMax(&rhi[cur * 8 + lrow], h);
                atomicOr(&rlo[cur * 8 + lrow], l);
            }
            hi = lo = 0;
        };
        Walk w{0, warp};
        w.wrap(nkt);
        while (w.rg < ngroups) {
            constexpr int kAhead = 4;                 // tiles loaded together
            double x[kAhead][4];
            Walk q[kAhead];
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                q[u] = w;
                load4(w, x[u]);
                w.kt += kSplitWarps;
                w.wrap(nkt);
            }
#pragma unroll
            for (int u = 0; u < kAhead; u++) {
                if (q[u].rg >= ngroups) break;        // uniform over the warp
                if (q[u].rg != cur) {
                    if (cur >= 0) flush();
                    cur = q[u].rg;
                }
#pragma unroll
                for (int j = 0; j < 4; j++) {
                    hi = max(hi, (uint32_t)__double2hiint(x[u][j]) & 0x7fffffffu);
                    lo |= (uint32_t)__double2loint(x[u][j]);
                }
            }
        }
        if (cur >= 0) flush();
    }
    __syncthreads();
    const int TR = P.tr, nkb = P.K_pad / kKbe, sstep = TR * kRowBytes;
    int cur = -1;
    uint8_t *rowdst = nullptr;
    double s1 = 1.0, s2 = 1.0;
    bool one = true;
    Walk w{0, warp};
    w.wrap(nkt);
    double nx[4];
    load4(w, nx);
    while (w.rg < ngroups) {
        const Walk q = w;
        double x[4];
#pragma unroll
        for (int j = 0; j < 4; j++) x[j] = nx[j];
        w.kt += kSplitWarps;
        w.wrap(nkt);
        load4(w, nx);                                 // the next tile's, while this one is cut
        const int i = q.rg * 8 + lrow, r = un.y + i, k0 = q.kt * 16 + kq * 4;
        if (q.rg != cur) {
            cur = q.rg;
            // exponent of the row's largest element (|x| < 2^e): its high word
            // has it, or, below 2^-1042, the highest low bit of the row; a row
            // with a NaN or an infinity is marked and its slices mean nothing
            int e = 0;
            const bool finite = rhi[i] < kInfHi;
            if (finite && (rhi[i] | rlo[i])) frexp(__hiloint2double((int)rhi[i], (int)rlo[i]), &e);
            if (r < P.rows && q.kt == 0 && kq == 0) exps[P.exp_off + r] = finite ? e : kNonFinite;
            // 2^(beta0 - e), as two finite factors where one would not do
            const int sh = kBeta0 - e;
            one = sh >= -1000 && sh <= 1000;
            s1 = ldexp(1.0, one ? sh : sh / 2);
            s2 = one ? 1.0 : ldexp(1.0, sh - sh / 2);
            rowdst = slices + P.slice_off + tile_image_offset(r, TR, nkb, 0, 0, S, 0);
        }
        if (r >= P.rows || k0 >= K) continue;
#pragma unroll
        for (int j = 0; j < 4; j++) x[j] *= s1;       // |x| < 2^beta0, exact
        if (!one)
#pragma unroll
            for (int j = 0; j < 4; j++) x[j] *= s2;
        const int byte = (k0 % kKbe) * kEsz;
        uint8_t *dst = rowdst + (int64_t)(k0 / kKbe) * S * sstep + (byte >> 4) * 128 + (byte & 15);
#pragma unroll
        for (int s = 0; s < S; s++) {
            const double magic = 6755399441055744.0 / (double)(1ll << (kBeta * s));   // 1.5 * 2^(52 - beta s)
            int v[4];
#pragma unroll
            for (int j = 0; j < 4; j++) {
                const double y = x[j] + magic;
                v[j] = __double2loint(y);
                x[j] -= y - magic;
            }
            *reinterpret_cast<PT *>(dst + s * sstep) = Pack4<KIND>::pack(v);
        }
    }
}

// ---------------------------------------------------------------- tcgen05 helpers

__device__ __forceinline__ uint32_t smem_u32(const void *p) {
    return (uint32_t)__cvta_generic_to_shared(p);
}

__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_u32(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.shared::cta.b64 st, [%0]; }" :: "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void mbar_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("{ .reg .b64 st; mbarrier.arrive.expect_tx.shared::cta.b64 st, [%0], %1; }"
                 :: "r"(smem_u32(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Wait for the phase with the given parity to complete, for at most
// limit_ns of wall time (try_wait itself may suspend the thread, so the bound
// is on time, not on iterations); false on timeout or when another role
// aborted.  limit_ns == 0 tests the phase once and does not wait.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, volatile int *abort,
                                          uint64_t limit_ns) {
    const uint32_t a = smem_u32(bar);
    if (limit_ns == 0) {                 // no time at all: one non-blocking test
        uint32_t done;
        asm volatile("{ .reg .pred p; mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(a), "r"(parity) : "memory");
        return done != 0;
    }
    uint64_t t0 = 0;
    for (uint32_t i = 0;; i++) {
        uint32_t done;
        asm volatile("{ .reg .pred p; mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2; selp.u32 %0, 1, 0, p; }"
                     : "=r"(done) : "r"(a), "r"(parity) : "memory");
        if (done) return true;
        if ((i & 63) == 63) {
            if (*abort) return false;
            const uint64_t t = global_ns();
            if (t0 == 0) t0 = t;
            else if (t - t0 > limit_ns) return false;
        }
    }
}

// One contiguous global -> shared bulk copy (16-byte aligned, size a
// multiple of 16), completing on the stage's mbarrier.  No multicast.
__device__ __forceinline__ void bulk_load(uint32_t dst, const void *src, uint32_t bytes, uint32_t bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        :: "r"(dst), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// K-major shared-memory matrix descriptor without swizzle (layout type 0):
// 8-row x 16-byte core matrices, the two k halves 128 bytes apart (leading
// byte offset), 8-row groups 256 bytes apart (stride byte offset), descriptor
// version 1 (sm_100).  Low word: start address and leading offset in 16-byte
// units; high word: stride offset and version.
constexpr uint32_t kDescHi = (256u >> 4) | (1u << 14);
__device__ __forceinline__ uint32_t desc_lo(uint32_t addr) { return ((addr >> 4) & 0x3FFF) | ((128u >> 4) << 16); }

template<int KIND>
__device__ __forceinline__ uint32_t instr_desc(int n) {
    // D format: S32 for int8, F32 otherwise; A/B formats; K-major A and B;
    // N = n (a multiple of 16, at most 256), M = 128.
    uint32_t c_fmt = KIND == kOzInt8 ? 2u : 1u;
    uint32_t ab_fmt = KIND == kOzInt8 ? 1u : (KIND == kOzBf16 ? 1u : 0u);
    return (c_fmt << 4) | (ab_fmt << 7) | (ab_fmt << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(kBM >> 4) << 24);
}

// D (+)= A B^T; x and y are the low words of the operands' descriptors (the
// high word is the same for every tile: kDescHi).  Formed by 32-bit adds from
// one word per stage and with the instruction descriptors ready, an MMA costs
// the issuing thread less than its run time; descriptors and piece widths
// worked out per MMA cost it 260 clocks each (BF16 x 4, 6 MMAs of 112-224
// columns per k block: 4.9 ms against 1.7 of products).
template<int KIND>
__device__ __forceinline__ void umma(uint32_t tmem_d, uint32_t x, uint32_t y, uint32_t idesc, uint32_t accumulate) {
    if (KIND == kOzInt8) {
        asm volatile("{ .reg .pred p; .reg .b64 a, b; mov.b64 a, {%1, %5}; mov.b64 b, {%2, %5};\n"
                     "setp.ne.b32 p, %4, 0;\n"
                     "tcgen05.mma.cta_group::1.kind::i8 [%0], a, b, %3, p; }"
                     :: "r"(tmem_d), "r"(x), "r"(y), "r"(idesc), "r"(accumulate), "n"(kDescHi) : "memory");
    } else if (KIND == kOzBf16) {
        asm volatile("{ .reg .pred p; .reg .b64 a, b; mov.b64 a, {%1, %5}; mov.b64 b, {%2, %5};\n"
                     "setp.ne.b32 p, %4, 0;\n"
                     "tcgen05.mma.cta_group::1.kind::f16 [%0], a, b, %3, p; }"
                     :: "r"(tmem_d), "r"(x), "r"(y), "r"(idesc), "r"(accumulate), "n"(kDescHi) : "memory");
    } else {
        asm volatile("{ .reg .pred p; .reg .b64 a, b; mov.b64 a, {%1, %5}; mov.b64 b, {%2, %5};\n"
                     "setp.ne.b32 p, %4, 0;\n"
                     "tcgen05.mma.cta_group::1.kind::f8f6f4 [%0], a, b, %3, p; }"
                     :: "r"(tmem_d), "r"(x), "r"(y), "r"(idesc), "r"(accumulate), "n"(kDescHi) : "memory");
    }
}

__device__ __forceinline__ void umma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 :: "r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ void tmem_ld8(uint32_t taddr, uint32_t *v) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]),
                   "=r"(v[6]), "=r"(v[7])
                 : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_wait_ld() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---------------------------------------------------------------- slice products

// 2^e f (|e| < 2044), by two normal powers of two: a test for one that fits,
// with ldexp for the others, cost the epilogue 9,400 clocks per drain of
// 128 x 112 elements.
__device__ __forceinline__ double scale_exp(double f, int e) {
    const int e1 = e >> 1, e2 = e - e1;
    return (f * __hiloint2double((e1 + 1023) << 20, 0)) * __hiloint2double((e2 + 1023) << 20, 0);
}

// sum_l 2^(-beta l) acc_l of column j, acc_l the integer level sums v[l][j].
// The levels are joined as integers, kGroup at a time, and only the groups
// become doubles: with one FP32 -> FP64 conversion and one FMA per level the
// epilogue took 34,000 clocks per drain of 57,000 sums, and takes 6,000 now.  FP32 sums (at most
// (l + 1) / S 2^24 in magnitude, so two neighbours fit 32 bits: 2^beta (S - 1) /
// S 2^24 + 2^24 < 2^31) are joined in fours, |.| < 2^46; INT32 sums in threes,
// |.| < 2^46.  Every step is exact up to the final rounding.
template<int KIND, int S>
__device__ __forceinline__ double level_sum(const uint32_t (&v)[S][8], int j) {
    constexpr int kBeta = KIND == kOzE4m3 ? 5 : 7;
    constexpr int kGroup = KIND == kOzInt8 ? 3 : 4;
    auto level = [&](int l) { return KIND == kOzInt8 ? (int)v[l][j] : __float2int_rn(__uint_as_float(v[l][j])); };
    double sum = 0.0;
#pragma unroll
    for (int l0 = (S - 1) / kGroup * kGroup; l0 >= 0; l0 -= kGroup) {
        const int l1 = l0 + kGroup < S ? l0 + kGroup : S;      // levels l0 .. l1 - 1
        long long g;
        if (KIND == kOzInt8) {
            g = level(l0);
#pragma unroll
            for (int l = l0 + 1; l < l1; l++) g = (g << kBeta) + level(l);
        } else if (l1 - l0 == 1) {
            g = level(l0);
        } else {
            g = level(l0) * (1 << kBeta) + level(l0 + 1);
            if (l1 - l0 == 3) g = g * (1 << kBeta) + level(l0 + 2);
            if (l1 - l0 == 4) g = g * (1 << (2 * kBeta)) + (level(l0 + 2) * (1 << kBeta) + level(l0 + 3));
        }
        // int64 -> double by bits (|g| < 2^51)
        const double d = __longlong_as_double(g + 0x4338000000000000ll) - 6755399441055744.0;
        sum = fma(d, 1.0 / (double)(1ll << (kBeta * (l1 - 1))), sum);
    }
    return sum;
}

// SCATTER: each finished tile row goes, by atomic adds into a zeroed
// result, to the destinations dests[drange[cblk]] of its C block (blocks of
// another tensor with their own index mappings and scales: the terms of a
// symmetrizer over the contraction) instead of the C block itself.
template<int KIND, int S, bool SCATTER = false>
__global__ void __launch_bounds__(kThreads, 1)
oz_gemm_kernel(const DPanel *__restrict__ panels, const uint8_t *__restrict__ slices,
               const DOzTask *__restrict__ tasks, const DCBlock *__restrict__ cblks,
               const DOzItem *__restrict__ items, int32_t nitems, const int32_t *__restrict__ exps,
               double *__restrict__ Cp, int32_t add, int32_t swap, int32_t stages, int32_t stage_bytes, int32_t kps,
               int32_t chunk_kb, int32_t beta0, int32_t kbe, int32_t *err, uint64_t wait_ns,
               const int2 *__restrict__ drange = nullptr, const DCBlock *__restrict__ dests = nullptr) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    // 1024-byte aligned stage buffers of kps k blocks: [stage][M-side slices | N-side slices]
    uint8_t *smem = reinterpret_cast<uint8_t *>(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    constexpr int kHalf = oz_max_nt(S) / 2;         // columns per epilogue thread, at most
    __shared__ __align__(8) uint64_t full_bar[kMaxStages], empty_bar[kMaxStages], accf_bar, acce_bar, drain_bar;
    __shared__ uint32_t tmem_base_s;
    __shared__ volatile int abort_s;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < stages; i++) { mbar_init(&full_bar[i], 1); mbar_init(&empty_bar[i], 1); }
        mbar_init(&accf_bar, 1);
        mbar_init(&acce_bar, kEpiWarps);
        mbar_init(&drain_bar, 1);
        abort_s = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;"
                     :: "r"(smem_u32(&tmem_base_s)) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_base_s;
    const uint32_t smem0 = smem_u32(smem);

    if (warp == kEpiWarps) {
        // ------------------------------------------------ bulk-copy producer (1-D cp.async.bulk)
        if (lane == 0) {
            int st = 0;
            uint32_t ph = 0;
            bool ok = true;
            int armed_parity[kMaxStages];
            for (int i = 0; i < kMaxStages; i++) armed_parity[i] = -1;
            for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
                const DOzItem item = items[it];
                const DCBlock &cb = cblks[item.cblk];
                const int ytile = item.nt * kRowBytes;
                for (int ti = cb.t_begin; ti < cb.t_end && ok; ti++) {
                    const DOzTask t = tasks[ti];
                    const int nkb = panels[t.px].K_pad / kbe;
                    // tile images of this (row tile, k block): all S slices contiguous
                    const uint8_t *gx = slices + panels[t.px].slice_off + (int64_t)(item.x0 / kBM) * nkb * S * kXTile;
                    const uint8_t *gy = slices + panels[t.py].slice_off + (int64_t)(item.y0 / item.nt) * nkb * S * ytile;
                    for (int kb = 0; kb < nkb; kb += kps) {
                        if (!mbar_wait(&empty_bar[st], ph ^ 1, &abort_s, wait_ns)) { ok = false; break; }
                        const uint32_t sx = smem0 + st * stage_bytes;
                        const uint32_t fb = smem_u32(&full_bar[st]);
                        const uint32_t slabs = (uint32_t)(min(kps, nkb - kb) * S);
                        mbar_expect_tx(&full_bar[st], slabs * (uint32_t)(kXTile + ytile));
                        bulk_load(sx, gx + (int64_t)kb * S * kXTile, slabs * kXTile, fb);
                        bulk_load(sx + kps * S * kXTile, gy + (int64_t)kb * S * ytile, slabs * (uint32_t)ytile, fb);
                        armed_parity[st] = (int)ph;
                        if (++st == stages) { st = 0; ph ^= 1; }
                    }
                }
            }
            if (!ok) {
                abort_s = 1;
                atomicExch(err, 7);
            }
            // let the copies already in flight land before the CTA exits (after
            // an abort the MMA warp no longer consumes them; in a normal run
            // each stage's last phase has completed already)
            volatile int never = 0;
            for (int i = 0; i < stages; i++)
                if (armed_parity[i] >= 0) (void)mbar_wait(&full_bar[i], (uint32_t)armed_parity[i], &never, kWaitNs);
        }
    } else if (warp == kEpiWarps + 1) {
        // ------------------------------------------------ MMA issuer
        if (lane == 0) {
            int st = 0;
            uint32_t ph = 0, accph = 0;
            int ndrain = 0;
            bool ok = true;
            for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
                const DOzItem item = items[it];
                const DCBlock &cb = cblks[item.cblk];
                // per M-side slice: its columns in one piece, or in two (the
                // first of w columns) where the widest tile needs them
                uint32_t id0[S], id1[S];
                int w[S];
#pragma unroll
                for (int sa = 0; sa < S; sa++) {
                    const int cols = (S - sa) * item.nt;
                    w[sa] = two_pieces<S>(sa) ? (cols / 2 + 15) / 16 * 16 : cols;
                    id0[sa] = instr_desc<KIND>(w[sa]);
                    id1[sa] = instr_desc<KIND>(cols - w[sa]);
                }
                for (int ti = cb.t_begin; ti < cb.t_end && ok; ti++) {
                    const int nkb = panels[tasks[ti].px].K_pad / kbe;
                    for (int kb0 = 0; kb0 < nkb && ok; kb0 += chunk_kb) {
                        // the accumulators are free once the previous drain was read
                        if (ndrain > 0) {
                            if (!mbar_wait(&acce_bar, accph, &abort_s, wait_ns)) { ok = false; break; }
                            accph ^= 1;
                        }
                        tc_fence_after();
                        const int kb1 = min(nkb, kb0 + chunk_kb);
                        uint32_t acc = 0;
                        for (int kb = kb0; kb < kb1; kb += kps) {
                            if (!mbar_wait(&full_bar[st], ph, &abort_s, wait_ns)) { ok = false; break; }
                            tc_fence_after();
                            const int nsub = min(kps, kb1 - kb);
                            uint32_t dx = desc_lo(smem0 + st * stage_bytes);
                            uint32_t dy = dx + (uint32_t)((kps * S * kXTile) >> 4);
                            for (int j = 0; j < nsub; j++) {
#pragma unroll
                                for (int sa = 0; sa < S; sa++) {
                                    const uint32_t xa = dx + (uint32_t)((sa * kXTile) >> 4);
                                    const uint32_t da = tmem + (uint32_t)(sa * item.nt);
                                    umma<KIND>(da, xa, dy, id0[sa], sa == 0 ? acc : 1u);
                                    if (two_pieces<S>(sa))
                                        umma<KIND>(da + (uint32_t)w[sa], xa, dy + (uint32_t)((w[sa] * kRowBytes) >> 4),
                                                   id1[sa], sa == 0 ? acc : 1u);
                                }
                                acc = 1;
                                dx += (uint32_t)((S * kXTile) >> 4);
                                dy += (uint32_t)((S * item.nt * kRowBytes) >> 4);
                            }
                            umma_commit(&empty_bar[st]);       // frees the stage when these MMAs finish
                            if (++st == stages) { st = 0; ph ^= 1; }
                        }
                        umma_commit(&accf_bar);                // accumulators ready for the epilogue
                        ndrain++;
                    }
                }
            }
            if (!ok) {
                abort_s = 1;
                atomicExch(err, 7);
                // the MMAs already issued must finish before TMEM is freed
                volatile int never = 0;
                umma_commit(&drain_bar);
                (void)mbar_wait(&drain_bar, 0, &never, kWaitNs);
            }
        }
    } else {
        // ------------------------------------------------ epilogue (warps 0-7)
        // warp w reads TMEM lanes 32 (w % 4) .. + 31 and the first or second
        // half of the tile's columns
        const int row = (warp & 3) * 32 + lane;           // TMEM lane == tile row
        const uint32_t lane_base = tmem + ((uint32_t)((warp & 3) * 32) << 16);
        uint32_t accph = 0;
        bool ok = true;
        for (int it = blockIdx.x; it < nitems && ok; it += gridDim.x) {
            const DOzItem item = items[it];
            const DCBlock &cb = cblks[item.cblk];
            const int hc = item.nt >> 1, c0 = (warp >> 2) * hc;    // nt is a multiple of 16
            double acc[kHalf];
#pragma unroll
            for (int j = 0; j < kHalf; j++) acc[j] = 0.0;
            const int x = item.x0 + row;
            for (int ti = cb.t_begin; ti < cb.t_end && ok; ti++) {
                const DOzTask t = tasks[ti];
                const DPanel &px = panels[t.px];
                const DPanel &py = panels[t.py];
                const int nkb = px.K_pad / kbe;
                const double nan = __longlong_as_double(0x7ff8000000000000ll);
                const int ex = exps[px.exp_off + x];
                const double f = ex == kNonFinite ? nan : ldexp(t.coeff, ex - 2 * beta0);
                // the columns' exponents, one or two per lane
                const int32_t *ey = exps + py.exp_off + item.y0 + c0;
                const int e_lo = lane < hc ? ey[lane] : 0, e_hi = kHalf > 32 && lane + 32 < hc ? ey[lane + 32] : 0;
                for (int kb0 = 0; kb0 < nkb; kb0 += chunk_kb) {
                    // warp-uniform outcome: tcgen05.ld below is .sync.aligned
                    ok = __all_sync(0xffffffffu, mbar_wait(&accf_bar, accph, &abort_s, wait_ns));
                    if (!ok) break;
                    accph ^= 1;
                    tc_fence_after();
#pragma unroll
                    for (int c = 0; c < kHalf / 8; c++) {
                        if (c * 8 >= hc) continue;        // uniform over the CTA
                        uint32_t v[S][8];
#pragma unroll
                        for (int l = 0; l < S; l++) tmem_ld8(lane_base + (uint32_t)(l * item.nt + c0 + c * 8), v[l]);
                        tmem_wait_ld();
#pragma unroll
                        for (int j = 0; j < 8; j++) {
                            const int e = __shfl_sync(0xffffffffu, c * 8 + j < 32 ? e_lo : e_hi, (c * 8 + j) & 31);
                            acc[c * 8 + j] += scale_exp(f, e) * level_sum<KIND, S>(v, j);
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&acce_bar);
                }
                if (ok && __any_sync(0xffffffffu, e_lo == kNonFinite || e_hi == kNonFinite)) {
#pragma unroll
                    for (int j = 0; j < kHalf; j++) {
                        const int e = __shfl_sync(0xffffffffu, j < 32 ? e_lo : e_hi, j & 31);
                        if (e == kNonFinite) acc[j] = nan;
                    }
                }
            }
            if (!ok) break;
            // FP64 write of the finished tile row: a C row, or with the sides
            // swapped a C column
            const int xe = swap ? cb.N : cb.M, ye = swap ? cb.M : cb.N;
            auto offset = [&](const DCBlock &b, bool xside, int i) {
                return xside != (swap != 0) ? mixed_offset(i, b.nm, b.mext, b.mc_str)
                                            : mixed_offset(i, b.nn, b.next, b.nc_str);
            };
            if (x < xe) {
                if constexpr (SCATTER) {
                    const int2 dr = drange[item.cblk];
                    for (int d = dr.x; d < dr.y; d++) {
                        const DCBlock &db = dests[d];
                        const int64_t drow = db.c_off + offset(db, true, x);
#pragma unroll
                        for (int j = 0; j < kHalf; j++) {
                            const int y = item.y0 + c0 + j;
                            if (j < hc && y < ye) atomicAdd(Cp + drow + offset(db, false, y), db.scale * acc[j]);
                        }
                    }
                } else {
                    const int64_t orow = cb.c_off + offset(cb, true, x);
#pragma unroll
                    for (int j = 0; j < kHalf; j++) {
                        const int y = item.y0 + c0 + j;
                        if (j < hc && y < ye) {
                            double *dst = Cp + orow + offset(cb, false, y);
                            const double val = cb.scale * acc[j];
                            if (add) *dst += val;
                            else *dst = val;
                        }
                    }
                }
            }
            __syncwarp();
        }
        if (!ok) { abort_s = 1; atomicExch(err, 7); }
    }

    tc_fence_before();
    __syncthreads();
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" :: "r"(tmem) : "memory");
    }
}

int g_nsm = 0;

template<int KIND, int S, bool SCATTER = false>
cudaError_t launch_gemm_s(const OzGemmArgs &a) {
    int beta0, beta, esz, kbe;
    int64_t mp;
    oz_kind_params(KIND, &beta0, &beta, &esz, &kbe, &mp);
    // two k blocks per stage while three such stages fit (half the barriers and
    // copies per product); a chunk is then a whole number of stages
    int stage_bytes = S * (kXTile + a.max_nt * kRowBytes), kps = 1;
    if (a.chunk_kb >= 2 && 3 * 2 * stage_bytes <= kStageSmem) { kps = 2; stage_bytes *= 2; }
    const int chunk_kb = a.chunk_kb / kps * kps;
    int stages = kStageSmem / stage_bytes;
    if (stages > kMaxStages) stages = kMaxStages;
    if (stages < 2) return cudaErrorInvalidValue;
    // At least 120 KB so that a second CTA never shares the SM: each CTA
    // holds all 512 TMEM columns.
    size_t smem = (size_t)stages * stage_bytes + 1024;
    if (smem < 120 * 1024) smem = 120 * 1024;
    cudaError_t e = cudaFuncSetAttribute(oz_gemm_kernel<KIND, S, SCATTER>,
                                         cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (e != cudaSuccess) return e;
    if (g_nsm == 0) {
        int dev = 0;
        cudaGetDevice(&dev);
        cudaDeviceGetAttribute(&g_nsm, cudaDevAttrMultiProcessorCount, dev);
    }
    int grid = a.nitems < g_nsm ? a.nitems : g_nsm;
    if (grid < 1) return cudaSuccess;
    oz_gemm_kernel<KIND, S, SCATTER><<<grid, kThreads, smem, a.s>>>(
        a.panels, a.slices, a.tasks, a.cblks, a.items, a.nitems, a.exps, a.c, SCATTER ? 0 : a.add, a.swap, stages,
        stage_bytes, kps, chunk_kb, beta0, kbe, a.err, a.wait_ns, a.drange, a.dests);
    return cudaGetLastError();
}

// Clocks per k block of one 128 x nt tile: its S(S+1)/2 products at nt / 2
// clocks each, or its operand images from L2 at kL2Bytes per clock and SM
// (about 11.6 TB/s over the chip), whichever is longer.  The rule takes nt = 112
// for 400 rows and 4 slices (4 tiles, 89 % of their columns used), 64 for 7
// and 8.  Ladder o=40 v=240, BF16 x 4: products 8.58 ms with 128 x 64 tiles and
// one MMA per slice pair, 3.38 now; o=30 v=150, FP8 x 8: 0.99 to 0.60 ms.
constexpr double kL2Bytes = 42.0;
double oz_tile_clocks(int nt, int S) {
    const double mma = 0.25 * S * (S + 1) * nt, copy = S * (kXTile + nt * kRowBytes) / kL2Bytes;
    return mma > copy ? mma : copy;
}

}  // namespace

#ifdef LTG_OZ_KIND

template<int KIND>
cudaError_t oz_launch_gemm(int S, const OzGemmArgs &a) {
    // the scattering form for the kind's default slice count only
    constexpr int kScatter = KIND == kOzE4m3 ? 8 : 7;
    if (a.dests) return S == kScatter ? launch_gemm_s<KIND, kScatter, true>(a) : cudaErrorNotSupported;
    switch (S) {
#define CASE_S(n) case n: return launch_gemm_s<KIND, n>(a);
    CASE_S(1) CASE_S(2) CASE_S(3) CASE_S(4) CASE_S(5) CASE_S(6) CASE_S(7) CASE_S(8)
#undef CASE_S
    default: return cudaErrorInvalidValue;
    }
}

template<int KIND>
cudaError_t oz_launch_split(int S, const DPanel *panels, const int4 *units, int32_t nunits, const double *a,
                            const double *b, uint8_t *slices, int32_t *exps, cudaStream_t s) {
    switch (S) {
#define CASE_S(n) case n: oz_split_kernel<KIND, n><<<nunits, kSplitThreads, 0, s>>>(panels, units, a, b, slices, exps); break;
    CASE_S(1) CASE_S(2) CASE_S(3) CASE_S(4) CASE_S(5) CASE_S(6) CASE_S(7) CASE_S(8)
#undef CASE_S
    default: return cudaErrorInvalidValue;
    }
    return cudaGetLastError();
}

template cudaError_t oz_launch_gemm<LTG_OZ_KIND>(int, const OzGemmArgs &);
template cudaError_t oz_launch_split<LTG_OZ_KIND>(int, const DPanel *, const int4 *, int32_t, const double *,
                                                  const double *, uint8_t *, int32_t *, cudaStream_t);

#else

int32_t oz_tile_width(int64_t rows, int S) {
    int32_t best = 16;
    double cost = 1e300;
    for (int32_t nt = 16; nt <= oz_max_nt(S); nt += 16) {
        const double c = (double)((rows + nt - 1) / nt) * oz_tile_clocks(nt, S);
        if (c <= cost) { cost = c; best = nt; }
    }
    return best;
}

double oz_product_cost(int64_t x, int64_t y, int S) {
    const int32_t nt = oz_tile_width(y, S);
    return (double)((x + kBM - 1) / kBM) * (double)((y + nt - 1) / nt) * oz_tile_clocks(nt, S);
}

int oz_split_unit_rows(int K) {
    // about 64 core tiles (8 rows x 16 k) per unit of short rows, else 8 rows
    const int nkt = (K + 15) / 16;
    const int g = 64 / nkt;
    return 8 * (g < 1 ? 1 : g > kUnitRowsMax / 8 ? kUnitRowsMax / 8 : g);
}

cudaError_t launch_oz_split(int kind, const DPanel *panels, const int4 *units, int32_t nunits, const double *a,
                            const double *b, uint8_t *slices, int32_t *exps, int32_t S, cudaStream_t s) {
    if (nunits <= 0) return cudaSuccess;
    if (kind == kOzInt8) return oz_launch_split<kOzInt8>(S, panels, units, nunits, a, b, slices, exps, s);
    if (kind == kOzBf16) return oz_launch_split<kOzBf16>(S, panels, units, nunits, a, b, slices, exps, s);
    return oz_launch_split<kOzE4m3>(S, panels, units, nunits, a, b, slices, exps, s);
}

cudaError_t launch_oz_gemm(int kind, const DPanel *panels, const uint8_t *slices, const DOzTask *tasks,
                           const DCBlock *cblks, const DOzItem *items, int32_t nitems, const int32_t *exps,
                           double *c, int32_t add, int32_t S, int32_t swap, int32_t chunk_kb, int32_t max_nt,
                           int32_t *err, uint64_t wait_ns, cudaStream_t s, const int2 *drange, const DCBlock *dests) {
    if (S < 1 || S > 8 || max_nt > oz_max_nt(S)) return cudaErrorInvalidValue;
    const OzGemmArgs a{panels, slices, tasks, cblks, items, nitems, exps, c, add, swap, chunk_kb, max_nt,
                       err, wait_ns, s, drange, dests};
    if (kind == kOzInt8) return oz_launch_gemm<kOzInt8>(S, a);
    if (kind == kOzBf16) return oz_launch_gemm<kOzBf16>(S, a);
    return oz_launch_gemm<kOzE4m3>(S, a);
}

#endif

}  // namespace ltg
