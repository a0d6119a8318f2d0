// FP64 complex GEMM on the 5th-generation tensor cores by error-free splitting
// into 8-bit integers (Ozaki, Ogita, Oishi, Rump, Numer. Algorithms 59 (2012)
// 95; INT8 form: Ootomo, Ozaki, Yokota, IJHPCA 38 (2024) 297).
//
// B200 has no tcgen05 kind for FP64: mma.sync m8n8k4 .f64 is its only FP64
// tensor path (about 40 TFLOP/s), while tcgen05 kind::i8 multiplies 8-bit
// integers about 100 times faster and accumulates them exactly in INT32.
//
//   * Each row (and each K chunk of it) is scaled by a power of two and rounded
//     to a 62-bit integer X (|x| < 2^E becomes |X| <= 2^61, so the spacing is
//     2^-61 of the row's largest part), written in eight signed base-256
//     digits, X = sum_i d_i 256^(7-i).  A row's own 53 bits survive for every
//     element above 2^-8 of its largest.
//   * X Y = sum_{i,j} d_i e_j 256^(14-i-j); the 36 products with i + j <= 7
//     are kept, those of one i + j in one INT32 accumulator: eight accumulators
//     of 64 columns fill the 512 TMEM columns of an SM.  8 products x 2^14 x 8192
//     terms < 2^31.
//   * Complex products in the three-multiplication form of the DMMA kernels,
//     the parts of (re, im, re -+ im) sliced as integers:
//       conj(a) b: T1 = ar br, T2 = ai bi, T3 = (ar - ai)(br + bi)
//       a b:       T1, T2 as above,        T3 = (ar + ai)(br + bi)
//   * The sums over K inside a chunk are exact.  What remains, in units of 2^(EA +
//     EB): the products with i + j = 8, seven of at most 2^14 256^6, and the
//     rounding of the digits, together at most 2^-57 per term of T1 and T2 and
//     2^-55 of the complex product; over random digits about 2^-59 sqrt(K) in
//     all.  That is below K 2^-53 |a||b| (2-norms of the rows) always, and measured
//     below the FP64 accumulation it replaces (i8_cn_pays), but it is relative to
//     the rows' largest parts: where the large elements of one row meet only small
//     ones of the other, FP64 keeps more.  A caller whose result is to hold
//     element by element has that looked at (`unresolved`): a fourth part
//     multiplies the magnitudes, the top 7 bits of max(|re|, |im|), in one digit;
//     sum |a||b| is at least that sum, so that from a quarter of 2^(EA + EB) on
//     the error is at most K 2^-53 sum |a||b|, FP64's own bound.  Costs 7 %
//     of a launch (rotation, 576 x 173,925 x 576: 4.89 -> 5.25 ms).
//
// Kernel (one persistent CTA per SM, work items = 128 x 64 output tile x K
// chunk, three parts each): warp 8 copies operand blocks, warp 9 issues the
// MMAs, warps 0-7 turn the eight accumulators into FP64.  The digits lie in
// global memory as the shared-memory image of one stage (K-major core
// matrices without swizzle), so a stage is two contiguous bulk copies (32 KB
// and 16 KB).  One A digit is multiplied by up to eight B digits in a row and
// stays in the collector buffer meanwhile (collector::a::fill / use): at N =
// 64 re-reading A from shared memory would cost 4 KB per 32 clocks of MMA.
#include "gemm_i8.hpp"
#include "gemm.hpp"
#include "launch_count.hpp"
#include "smem_limit.hpp"
#include "tcgen05.cuh"

#include <algorithm>
#include <atomic>

namespace chfsi {

namespace {

constexpr int kTM = kI8RowTile, kTN = kI8ColTile;
constexpr int kDig = 8;                       // digits per part
constexpr int kSlab = 32;                     // K per MMA and per stage
constexpr int kABytes = kDig * kTM * kSlab;   // one A block
constexpr int kBBytes = kDig * kTN * kSlab;   // one B block
constexpr int kStageBytes = kABytes + kBBytes;
constexpr int kRing = 4;
constexpr int kEpiThreads = 256, kThreads = 320;
constexpr int kMaxSpc = kI8MaxK / kSlab;
constexpr int kNonFinite = 1 << 20;           // exponent mark of a row with inf or NaN
constexpr int kZeroRow = -2000;               // and of one of zeros

constexpr size_t kSmemBytes = 1024 + (size_t)kRing * kStageBytes + 128;

// magnitudes: 2^7 per side, a quarter of the product of the two
constexpr int kResolved = 1 << 12;
constexpr int kParts = 3, kMagPart = 3;       // re, im, re -+ im; magnitudes

struct I8Side {
    const int8_t *data, *mag;
    const int* exps;
    int tiles, rows_pad, nslab, slab0, chunk0;
};

// the error word may lie in host memory: a plain store, no atomic
__device__ __forceinline__ void report(int* err, int code) {
    *(volatile int*)err = code;
    __threadfence_system();
}

__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
            smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

// K-major operand without swizzle: core matrices of 8 rows x 16 bytes; the two
// core columns of a 32-byte K step are rows * 16 bytes apart, row groups 128.
__device__ __forceinline__ uint64_t i8_desc(uint32_t saddr, uint32_t rows) {
    uint64_t d = 0;
    d |= (uint64_t)((saddr >> 4) & 0x3FFF);
    d |= (uint64_t)((rows * 16) >> 4) << 16;  // leading byte offset: along K
    d |= (uint64_t)(128 >> 4) << 32;          // stride byte offset: along rows
    d |= (uint64_t)1 << 46;                   // descriptor version (sm_100)
    return d;
}

// kind::i8 instruction descriptor: S8 x S8 -> S32, K-major A and B
__host__ __device__ constexpr uint32_t idesc_i8(int m, int n) {
    return (2u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) |
           ((uint32_t)(m >> 4) << 24);
}

// COL: 0 single use of A, 1 first of a run, 2 inside, 3 last
#define CHFSI_UMMA_I8(COLLECTOR)                                                               \
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"                             \
                 "tcgen05.mma.cta_group::1.kind::i8" COLLECTOR " [%0], %1, %2, %3, p;\n\t}" ::     \
                     "r"(d), "l"(a), "l"(b), "r"(idesc), "r"(accumulate))
template <int COL>
__device__ __forceinline__ void umma_i8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                        uint32_t accumulate) {
    if constexpr (COL == 1) CHFSI_UMMA_I8(".collector::a::fill");
    else if constexpr (COL == 2) CHFSI_UMMA_I8(".collector::a::use");
    else if constexpr (COL == 3) CHFSI_UMMA_I8(".collector::a::lastuse");
    else CHFSI_UMMA_I8("");
}
#undef CHFSI_UMMA_I8

// true in one lane of a converged warp; the compiler keeps the operands of what
// runs under it in uniform registers (under a lane test the moves into them took
// 60 clocks per MMA)
__device__ __forceinline__ bool elect_one() {
    uint32_t pred = 0;
    asm volatile(
        "{\n\t.reg .b32 r;\n\t.reg .pred q;\n\telect.sync r|q, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, q;\n\t}"
        : "=r"(pred));
    return pred != 0;
}

// products of the A digits I0 .. I1 - 1 of one slab
template <int I0, int I1>
__device__ __forceinline__ void slab_products(uint32_t tmem, uint64_t da, uint64_t db, uint32_t more) {
    constexpr uint32_t idesc = idesc_i8(kTM, kTN);
#pragma unroll
    for (int i = I0; i < I1; ++i) {
        const uint64_t ad = da + (uint64_t)(i * (kTM * kSlab / 16));
        const uint32_t acc = i > 0 ? 1u : more;
#pragma unroll
        for (int j = 0; j < kDig - i; ++j) {
            const uint64_t bd = db + (uint64_t)(j * (kTN * kSlab / 16));
            const uint32_t td = tmem + (uint32_t)((i + j) * kTN);
            if (kDig - i == 1) umma_i8<0>(td, ad, bd, idesc, acc);
            else if (j == 0) umma_i8<1>(td, ad, bd, idesc, acc);
            else if (j == kDig - i - 1) umma_i8<3>(td, ad, bd, idesc, acc);
            else umma_i8<2>(td, ad, bd, idesc, acc);
        }
    }
}

__device__ __forceinline__ void tmem_ld4(uint32_t taddr, int* r) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
                 : "r"(taddr));
}

// 2^p for -1022 <= p <= 1023
__device__ __forceinline__ double pow2(int p) { return __longlong_as_double((long long)(p + 1023) << 52); }
// Scales of a sum v, |v| < 2^80: 2^(EA + EB - 66) v = v side.x fb side.y, in that
// order.  A's exponent goes in two halves where it is large, so that no step leaves
// the range of the exponents where the product does not, whatever the other row's:
// with |a| <= 400 the second half is 1, beyond it the half still to come would have
// to be outweighed by an EB past 2^1024 or 2^-1074.  NaN for a row with an inf or
// NaN, 1 for a row of zeros.
__device__ __forceinline__ double2 side_a(int e) {
    if (e == kNonFinite) return make_double2(__longlong_as_double(0x7ff8000000000000LL), 1.0);
    if (e == kZeroRow) return make_double2(1.0, 1.0);
    const int a = e - 65, h = a > 400 || a < -400 ? a >> 1 : a;
    return make_double2(pow2(h), pow2(a - h));
}
__device__ __forceinline__ double side_b(int e) {
    if (e == kNonFinite) return __longlong_as_double(0x7ff8000000000000LL);
    return e == kZeroRow ? 1.0 : pow2(e - 1);
}

// x as a double, |x| < 2^51: through the exponent bits of 2^52 + 2^51, one add
// on the FP64 pipe (I2F.F64 runs at a small fraction of that pipe's rate: with
// it the accumulators of a part took 13-20k clocks to convert instead of 4k)
__device__ __forceinline__ double small_int(long long x) {
    return __longlong_as_double(0x4338000000000000LL + x) - 6755399441055744.0;
}

// sum of the eight accumulators (each below 2^30) of one element
__device__ __forceinline__ double i8_value(const int* I) {
    const long long a = (long long)I[0] * 65536 + ((long long)I[1] * 256 + I[2]);
    const long long b = (long long)I[3] * 65536 + ((long long)I[4] * 256 + I[5]);
    const long long c = (long long)I[6] * 256 + I[7];
    return fma(small_int(a), 1099511627776.0, fma(small_int(b), 65536.0, small_int(c)));
}

// item -> chunk and tiles; Hermitian products keep the tiles that reach the
// diagonal: row tiles tm <= tn / 2 for the column tile tn
__device__ __forceinline__ void i8_item(int item, int per_chunk, int mt, int nt, bool herm, int& chunk,
                                        int& tm, int& tn) {
    chunk = item / per_chunk;
    int t = item - chunk * per_chunk;
    if (!herm) {
        tm = t / nt;  // neighbours share the row tile, the larger operand block
        tn = t - tm * nt;
        return;
    }
    tn = 0;
    for (int w = min(mt, 1); t >= w; w = min(mt, tn / 2 + 1)) { t -= w; ++tn; }
    tm = t;
}

// The parts of every item, with CHECK the magnitudes behind them (their loads are
// in flight while the third part is converted: in front of the others 1 % slower);
// only_mag: the magnitudes alone.  Nothing when *gate is set.
template <bool CHECK>
__global__ void __launch_bounds__(kThreads, 1)
k_umma_i8(I8Side a, I8Side b, bool only_mag, int M, int N, int mt, int per_chunk, int items, int nslab, int spc,
          int conj, int herm, double2* __restrict__ out, long long ldo, long long chunk_stride,
          double alpha, double beta, int* err, int* unresolved, const int* gate,
          unsigned long long wait_ns, int no_loads) {
    if (gate && *gate) return;
    const int p0 = CHECK && only_mag ? kMagPart : 0, p1 = CHECK ? kMagPart + 1 : kParts;
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    uint64_t* full = (uint64_t*)(base + kRing * kStageBytes);
    uint64_t* empty = full + kRing;
    uint64_t* acc_full = empty + kRing;
    uint64_t* acc_free = acc_full + 1;
    uint64_t* drain = acc_free + 1;
    uint32_t* tmem_slot = (uint32_t*)(drain + 1);
    volatile int* abort_flag = (volatile int*)(tmem_slot + 1);
    const int warp = __shfl_sync(0xffffffffu, (int)(threadIdx.x >> 5), 0);
    const int lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int s = 0; s < kRing; ++s) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], 1);
        }
        mbar_init(acc_full, 1);
        mbar_init(acc_free, kEpiThreads / 32);
        mbar_init(drain, 1);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 9) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                         smem_u32(tmem_slot)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = *tmem_slot;

    if (warp == 8) {
        if (lane == 0 && !no_loads) {
            // ---- copies: the blocks of one part and tile are contiguous along K
            int issued = 0;
            bool ok = true;
            for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
                int c, tm, tn;
                i8_item(item, per_chunk, mt, b.tiles, herm, c, tm, tn);
                const int s0 = c * spc, s1 = min(nslab, s0 + spc);
                for (int part = p0; part < p1 && ok; ++part) {
                    // magnitudes: one digit, kDig slabs to a stage
                    const bool mag = CHECK && part == kMagPart;
                    const int step = mag ? kDig : 1;
                    const size_t ta = (size_t)tm * a.nslab + a.slab0 + s0, tb = (size_t)tn * b.nslab + b.slab0 + s0;
                    const int8_t* pa = mag ? a.mag + ta * (kABytes / kDig)
                                           : a.data + ((size_t)part * a.tiles * a.nslab + ta) * kABytes;
                    const int8_t* pb = mag ? b.mag + tb * (kBBytes / kDig)
                                           : b.data + ((size_t)part * b.tiles * b.nslab + tb) * kBBytes;
                    for (int s = s0; s < s1; s += step, ++issued, pa += kABytes, pb += kBBytes) {
                        const int slot = issued % kRing;
                        if (!mbar_wait_or(&empty[slot], ((issued / kRing) & 1) ^ 1, wait_ns, abort_flag)) {
                            report(err, 1);
                            *abort_flag = 1;
                            ok = false;
                            break;
                        }
                        unsigned char* dst = base + (size_t)slot * kStageBytes;
                        const int planes = mag ? min(kDig, s1 - s) : kDig;
                        mbar_expect_tx(&full[slot], planes * (kStageBytes / kDig));
                        bulk_load(dst, pa, planes * (kABytes / kDig), &full[slot]);
                        bulk_load(dst + kABytes, pb, planes * (kBBytes / kDig), &full[slot]);
                    }
                }
            }
            if (!ok)  // retire the copies still in flight before shared memory goes
                for (int j = issued > kRing ? issued - kRing : 0; j < issued; ++j)
                    if (!mbar_wait(&full[j % kRing], (j / kRing) & 1, wait_ns)) {
                        report(err, 4);
                        break;
                    }
        }
    } else if (warp == 9) {
        // ---- MMAs: 36 digit products per slab, accumulator i + j.  The wait
        // for a slab's operands is taken in the middle of the slab before it:
        // the few queued MMAs do not outlast the latency of the wait itself.
        int total = 0;
        for (int item = blockIdx.x; item < items; item += gridDim.x) {
            int c, tm, tn;
            i8_item(item, per_chunk, mt, b.tiles, herm, c, tm, tn);
            const int n = min(nslab, (c + 1) * spc) - c * spc;
            total += (kParts - p0) * n + (CHECK ? (n + kDig - 1) / kDig : 0);
        }
        // the whole warp waits, and goes on or gives up together
        auto wait = [&](uint64_t* bar, uint32_t parity) {
            return __all_sync(0xffffffffu, mbar_wait_or(bar, parity, wait_ns, abort_flag)) != 0;
        };
        int it = 0, pc = 0;
        bool ok = wait(&full[0], 0);
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
            int c, tm, tn;
            i8_item(item, per_chunk, mt, b.tiles, herm, c, tm, tn);
            const int n = min(nslab, (c + 1) * spc) - c * spc;
            for (int part = p0; part < p1 && ok; ++part, ++pc) {
                if (!(ok = wait(acc_free, (pc & 1) ^ 1))) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (CHECK && part == kMagPart) {
                    for (int s = 0; s < n && ok; s += kDig, ++it) {
                        const int slot = it % kRing;
                        const uint32_t sa = smem_u32(base + (size_t)slot * kStageBytes);
                        const uint64_t da = i8_desc(sa, kTM), db = i8_desc(sa + kABytes, kTN);
                        const int planes = min(kDig, n - s);
                        if (elect_one()) {
#pragma unroll
                            for (int j = 0; j < kDig; ++j)
                                if (j < planes)
                                    umma_i8<0>(tmem, da + (uint64_t)(j * (kTM * kSlab / 16)),
                                               db + (uint64_t)(j * (kTN * kSlab / 16)), idesc_i8(kTM, kTN),
                                               s + j > 0 ? 1u : 0u);
                            umma_commit(&empty[slot]);
                        }
                        if (it + 1 < total) ok = wait(&full[(it + 1) % kRing], ((it + 1) / kRing) & 1);
                    }
                    if (ok && elect_one()) umma_commit(acc_full);
                    continue;
                }
                for (int s = 0; s < n && ok; ++s, ++it) {
                    const int slot = it % kRing;
                    const uint32_t sa = smem_u32(base + (size_t)slot * kStageBytes);
                    const uint64_t da = i8_desc(sa, kTM), db = i8_desc(sa + kABytes, kTN);
                    const uint32_t more = s > 0 ? 1u : 0u;
                    if (elect_one()) slab_products<0, 2>(tmem, da, db, more);
                    if (it + 1 < total) ok = wait(&full[(it + 1) % kRing], ((it + 1) / kRing) & 1);
                    if (elect_one()) {
                        slab_products<2, kDig>(tmem, da, db, more);
                        umma_commit(&empty[slot]);
                    }
                }
                if (ok && elect_one()) umma_commit(acc_full);
            }
        }
        if (!ok && elect_one()) {
            report(err, 2);
            *abort_flag = 1;
            umma_commit(drain);  // arrives once every MMA issued above has completed
            if (!mbar_wait(drain, 0, wait_ns)) report(err, 5);
        }
    } else {
        // ---- accumulators -> FP64: thread = one tile row, 32 of its columns.
        // The real part is written after the second part, the imaginary one
        // after the third, so one value per element is kept between parts.
        const int lq = warp & 3, half = warp >> 2;
        const uint32_t tl = tmem + ((uint32_t)(lq * 32) << 16) + (uint32_t)(half * 32);
        const double sgn = conj ? 1.0 : -1.0;
        double keep[32];
#pragma unroll
        for (int j = 0; j < 32; ++j) keep[j] = 0.0;
        int pc = 0;
        bool ok = true;
        for (int item = blockIdx.x; item < items && ok; item += gridDim.x) {
            int c, tm, tn;
            i8_item(item, per_chunk, mt, b.tiles, herm, c, tm, tn);
            const int i = tm * kTM + lq * 32 + lane, j0 = tn * kTN + half * 32;
            // X = x 2^(61 - E) and the digits' 256^7: products carry 2^(EA + EB - 66)
            const int ea = a.exps[(size_t)(a.chunk0 + c) * a.rows_pad + i];
            const int eb_lane = b.exps[(size_t)(b.chunk0 + c) * b.rows_pad + j0 + lane];
            const double2 fa = side_a(ea);
            const double fb_lane = side_b(eb_lane);
            double2* o = out + (long long)c * chunk_stride + (long long)j0 * ldo + i;
            const int cols = i < M ? N - j0 : 0;
#pragma unroll 1
            for (int part = p0; part < p1; ++part, ++pc) {
                if (lane == 0) ok = mbar_wait_or(acc_full, pc & 1, wait_ns, abort_flag);
                ok = __shfl_sync(0xffffffffu, ok, 0);  // tcgen05.ld is warp-collective
                if (!ok) break;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                if (CHECK && part == kMagPart) {
                    // rows of zeros give exact zeros, rows with an inf or NaN give NaN
                    const bool row = i < M && ea != kZeroRow && ea != kNonFinite;
                    const unsigned colm = __ballot_sync(0xffffffffu, j0 + lane < N && eb_lane != kZeroRow &&
                                                                         eb_lane != kNonFinite);
                    int L[8][4];
#pragma unroll
                    for (int g = 0; g < 8; ++g) tmem_ld4(tl + (uint32_t)(g * 4), L[g]);
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                    __syncwarp();
                    if (lane == 0) mbar_arrive(acc_free);
                    bool low = false;
#pragma unroll
                    for (int j = 0; j < 32; ++j) low |= L[j >> 2][j & 3] < kResolved && ((colm >> j) & 1u);
                    if (__any_sync(0xffffffffu, row && low) && lane == 0) *(volatile int*)unresolved = 1;
                    continue;
                }
                int I[2][kDig][4];
#pragma unroll
                for (int d = 0; d < kDig; ++d) tmem_ld4(tl + (uint32_t)(d * kTN), I[0][d]);
#pragma unroll
                for (int g = 0; g < 8; ++g) {
                    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
                    if (g < 7) {
#pragma unroll
                        for (int d = 0; d < kDig; ++d)
                            tmem_ld4(tl + (uint32_t)(d * kTN + (g + 1) * 4), I[(g + 1) & 1][d]);
                    } else {
                        asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                        __syncwarp();
                        if (lane == 0) mbar_arrive(acc_free);
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int jj = g * 4 + q;
                        int v[kDig];
#pragma unroll
                        for (int d = 0; d < kDig; ++d) v[d] = I[g & 1][d][q];
                        const double t = i8_value(v) * fa.x * __shfl_sync(0xffffffffu, fb_lane, jj) * fa.y;
                        // conj: re = T1 + T2, im = T3 + (T2 - T1); else re = T1 - T2,
                        // im = T3 + (-T2 - T1)
                        const double r = fma(part == 1 ? sgn : 1.0, t, keep[jj]);
                        keep[jj] = part == 0 ? t : fma(sgn, t, -keep[jj]);
                        double* e = reinterpret_cast<double*>(o + (long long)jj * ldo) + (part - 1);
                        const bool put = part > 0 && jj < cols;
                        double old = 0.0;
                        if (put && beta != 0.0) old = *e;
                        if (put) *e = fma(beta, old, alpha * r);
                    }
                }
            }
        }
        if (!ok && lane == 0) {
            report(err, 3);
            *abort_flag = 1;
        }
    }
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    if (warp == 9)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512));
}

// ---- digits
// X in eight signed digits: adding 128 to each of the seven low bytes and
// flipping their top bits turns base-256 bytes into digits of [-128, 127].
__device__ __forceinline__ unsigned long long digits(long long x) {
    return ((unsigned long long)x + 0x0080808080808080ULL) ^ 0x0080808080808080ULL;
}
// 4 x 4 byte transpose: w[p] = bytes p of a, b, c, d
__device__ __forceinline__ void bytes4(uint32_t a, uint32_t b, uint32_t c, uint32_t d, uint32_t* w) {
    const uint32_t ab0 = __byte_perm(a, b, 0x5140), ab1 = __byte_perm(a, b, 0x7362);
    const uint32_t cd0 = __byte_perm(c, d, 0x5140), cd1 = __byte_perm(c, d, 0x7362);
    w[0] = __byte_perm(ab0, cd0, 0x5410);
    w[1] = __byte_perm(ab0, cd0, 0x7632);
    w[2] = __byte_perm(ab1, cd1, 0x5410);
    w[3] = __byte_perm(ab1, cd1, 0x7632);
}
// 16 values along K of one row -> 16 bytes of each digit plane
__device__ __forceinline__ void store16(const long long* x, int8_t* dst, int plane_bytes) {
    uint32_t w[kDig][4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        unsigned long long y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) y[j] = digits(x[4 * g + j]);
        uint32_t lo[4], hi[4];
        bytes4((uint32_t)y[0], (uint32_t)y[1], (uint32_t)y[2], (uint32_t)y[3], lo);
        bytes4((uint32_t)(y[0] >> 32), (uint32_t)(y[1] >> 32), (uint32_t)(y[2] >> 32), (uint32_t)(y[3] >> 32), hi);
#pragma unroll
        for (int p = 0; p < 4; ++p) {
            w[7 - p][g] = lo[p];
            w[3 - p][g] = hi[p];
        }
    }
#pragma unroll
    for (int p = 0; p < kDig; ++p)
        *reinterpret_cast<uint4*>(dst + (size_t)p * plane_bytes) = make_uint4(w[p][0], w[p][1], w[p][2], w[p][3]);
}

// high word without the sign; its last bit is set for any number but zero
__device__ __forceinline__ unsigned int top_word(double2 v) {
    const unsigned x = ((unsigned)__double2hiint(v.x) & 0x7fffffffu) | (__double2loint(v.x) != 0);
    const unsigned y = ((unsigned)__double2hiint(v.y) & 0x7fffffffu) | (__double2loint(v.y) != 0);
    return max(x, y);
}
// largest top word of a row part -> exponent E with |x| < 2^E
__device__ __forceinline__ int row_exponent(unsigned int top) {
    const int f = (int)(top >> 20);
    return f == 2047 ? kNonFinite : top == 0 ? kZeroRow : max(f, 1) - 1022;
}

// round to nearest of v, |v| < 2^61, in two 31-bit steps on the FP64 pipe
__device__ __forceinline__ long long round61(double v) {
    const double magic = 6755399441055744.0;  // 2^52 + 2^51
    const double th = fma(v, 4.656612873077393e-10, magic);  // v 2^-31
    const double h = th - magic;
    const double tl = fma(h, -2147483648.0, v) + magic;      // the rest, exact, at most 2^30
    return ((__double_as_longlong(th) - 0x4338000000000000LL) << 31) +
           (__double_as_longlong(tl) - 0x4338000000000000LL);
}

// top 7 of the 61 bits of the larger part, rounded down (the complement of a
// negative part's high word is at most its magnitude's)
__device__ __forceinline__ uint32_t magnitude(long long xr, long long xi) {
    const int r = (int)(xr >> 32), i = (int)(xi >> 32);
    return (uint32_t)max(r ^ (r >> 31), i ^ (i >> 31)) >> 22;
}

// One block cuts 8 rows (or 32 of a transposed source, whose rows lie side by
// side) of one K chunk: a first read finds each row's exponent, the second,
// from L2, writes the digits.  HBM-bound (16 bytes read, 24 written per
// complex element).
template <bool TRANS, bool MAG>
__global__ void __launch_bounds__(256)
k_i8_slice(const double2* __restrict__ x, long long ld, int sign, int rows, int K, int nslab, int spc,
           int tile, int tiles, int8_t* __restrict__ data, int8_t* __restrict__ mag, int* __restrict__ exps) {
    constexpr int R = TRANS ? 32 : 8;
    __shared__ unsigned int top[8][32];
    __shared__ int ex[32];
    const int r0 = blockIdx.x * R, chunk = blockIdx.y;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int k0 = chunk * spc * kSlab;
    const int sl0 = chunk * spc, sl1 = min(nslab, sl0 + spc);
    const int k1 = min(K, sl1 * kSlab);
    if (TRANS) {
        unsigned int m = 0;
        const int r = r0 + lane;
        if (r < rows)
            for (int k = k0 + warp; k < k1; k += 8) m = max(m, top_word(x[(long long)k * ld + r]));
        top[warp][lane] = m;
        __syncthreads();
        if (warp == 0) {
#pragma unroll
            for (int w = 1; w < 8; ++w) m = max(m, top[w][lane]);
            ex[lane] = row_exponent(m);
        }
    } else {
        unsigned int m = 0;
        const int r = r0 + warp;
        if (r < rows)
            for (int k = k0 + lane; k < k1; k += 32) m = max(m, top_word(x[(long long)r * ld + k]));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
        if (lane == 0) ex[warp] = row_exponent(m);
    }
    __syncthreads();
    if (threadIdx.x < R) exps[(size_t)chunk * tiles * tile + r0 + threadIdx.x] = ex[threadIdx.x];
    const int rl = threadIdx.x % R, r = r0 + rl;
    const int e = ex[rl];
    const bool live = r < rows && e != kNonFinite;
    // x 2^(61 - e) in two factors: 61 - e reaches 1083
    const int s = e == kNonFinite ? 0 : 61 - e;
    const double f1 = pow2(min(s, 1000)), f2 = pow2(s - min(s, 1000));
    const int plane_bytes = tile * kSlab;
    const size_t block_bytes = (size_t)kDig * plane_bytes;
    for (int kc = 2 * sl0 + threadIdx.x / R; kc < 2 * sl1; kc += 256 / R) {
        long long xr[16], xi[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const int k = kc * 16 + j;
            double2 v = make_double2(0.0, 0.0);
            if (live && k < k1) v = TRANS ? x[(long long)k * ld + r] : x[(long long)r * ld + k];
            xr[j] = round61(v.x * f1 * f2);
            xi[j] = round61(v.y * f1 * f2);
        }
        int8_t* dst = data + ((size_t)(r / tile) * nslab + (kc >> 1)) * block_bytes +
                      (size_t)(kc & 1) * tile * 16 + (size_t)(r % tile) * 16;
        const size_t part = (size_t)tiles * nslab * block_bytes;
        store16(xr, dst, plane_bytes);
        store16(xi, dst + part, plane_bytes);
        if constexpr (MAG) {
            uint32_t w[4];
#pragma unroll
            for (int g = 0; g < 4; ++g)
                w[g] = magnitude(xr[4 * g], xi[4 * g]) | magnitude(xr[4 * g + 1], xi[4 * g + 1]) << 8 |
                       magnitude(xr[4 * g + 2], xi[4 * g + 2]) << 16 | magnitude(xr[4 * g + 3], xi[4 * g + 3]) << 24;
            *reinterpret_cast<uint4*>(mag + ((size_t)(r / tile) * nslab + (kc >> 1)) * plane_bytes +
                                      (size_t)(kc & 1) * tile * 16 + (size_t)(r % tile) * 16) =
                make_uint4(w[0], w[1], w[2], w[3]);
        }
#pragma unroll
        for (int j = 0; j < 16; ++j) xr[j] += sign > 0 ? xi[j] : -xi[j];
        store16(xr, dst + 2 * part, plane_bytes);
    }
}

// partials part[chunk][n][m] -> out[m][n], summed in chunk order; accumulate:
// added to out; herm: elements on and above the diagonal, mirrored
__global__ void __launch_bounds__(256)
k_i8_reduce(const double2* __restrict__ part, int chunks, int M, int N, int herm, int accumulate,
            double2* __restrict__ out) {
    __shared__ double2 t[16][17];
    const int m0 = blockIdx.x * 16, n0 = blockIdx.y * 16;
    if (herm && m0 > n0 + 15) return;
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const size_t mn = (size_t)M * N;
    double2 s = make_double2(0.0, 0.0);
    if (m0 + tx < M && n0 + ty < N) {
        const double2* p = part + (size_t)(n0 + ty) * M + m0 + tx;
        for (int c = 0; c < chunks; ++c, p += mn) {
            s.x += p->x;
            s.y += p->y;
        }
    }
    t[ty][tx] = s;
    __syncthreads();
    const int m = m0 + ty, n = n0 + tx;
    if (m >= M || n >= N || (herm && m > n)) return;
    s = t[tx][ty];
    double2* o = out + (size_t)m * N + n;
    if (accumulate) {
        s.x += o->x;
        s.y += o->y;
    }
    *o = s;
    if (herm && m < n) out[(size_t)n * N + m] = make_double2(s.x, -s.y);
}

int ceil_div(int a, int b) { return (a + b - 1) / b; }

int herm_tiles(int mt, int nt) {
    int t = 0;
    for (int tn = 0; tn < nt; ++tn) t += std::min(mt, tn / 2 + 1);
    return t;
}

// Clocks of one launch: waves of items, each three parts of spc slabs plus the
// pipeline fill and the conversion of the accumulators.  36 MMAs of N = 64 take
// 44.6 clocks each (measured: 48 without the collector, against 32 at the full
// INT8 rate, which needs N >= 128 and then TMEM for 16 accumulators).
constexpr int kSms = 148;
constexpr double kSlabClk = 1620.0, kPartClk = 5500.0, kHbmBytesPerClk = 3400.0;
// slicing runs at about 4 TB/s (16 bytes read, 24 written per element)
constexpr double kSliceBytesPerClk = 2100.0, kSliceClk = 9000.0, kReduceClk = 10000.0;
double launch_clk(int tiles, int chunks, int spc) {
    return (double)ceil_div(tiles * chunks, kSms) * 3.0 * (spc * kSlabClk + kPartClk);
}
double slice_clk(double elems) { return kSliceClk + 40.0 * elems / kSliceBytesPerClk; }

// K slabs per chunk: the split of nslab that takes the fewest clocks with its
// partials (M x N written and read per chunk)
int best_spc(int tiles, int nslab, double mn) {
    int best = std::min(nslab, kMaxSpc);
    double best_clk = 1e300;
    for (int chunks = ceil_div(nslab, kMaxSpc); chunks <= std::max(1, nslab / 8); ++chunks) {
        const int spc = ceil_div(nslab, chunks);
        const int used = ceil_div(nslab, spc);
        const double clk = launch_clk(tiles, used, spc) + used * mn * 32.0 / kHbmBytesPerClk;
        if (clk < best_clk) {
            best_clk = clk;
            best = spc;
        }
    }
    return best;
}

struct CnPlan {
    int mt, nt, tiles, nslab, spc, groups, slabs_per_group;
    double clk;
};

size_t align256(size_t n) { return (n + 255) & ~(size_t)255; }

size_t cn_bytes(const CnPlan& p, int M, int N, bool cached_a, bool check) {
    const int K = p.slabs_per_group * kSlab;
    return (cached_a ? 0 : i8_operand_bytes(M, kTM, K, p.spc, check)) + i8_operand_bytes(N, kTN, K, p.spc, check) +
           align256((size_t)ceil_div(p.slabs_per_group, p.spc) * M * N * sizeof(double2));
}

CnPlan cn_plan(int M, int N, int K, bool herm, int fixed_spc, size_t bytes, bool check = false) {
    CnPlan p{};
    p.mt = ceil_div(M, kTM);
    p.nt = ceil_div(N, kTN);
    p.tiles = herm ? herm_tiles(p.mt, p.nt) : p.mt * p.nt;
    p.nslab = ceil_div(K, kSlab);
    for (int g = 1; g <= p.nslab; ++g) {
        p.groups = g;
        p.slabs_per_group = ceil_div(p.nslab, g);
        if (fixed_spc > 0) {
            p.spc = fixed_spc;
            p.slabs_per_group = ceil_div(p.slabs_per_group, p.spc) * p.spc;
            p.groups = ceil_div(p.nslab, p.slabs_per_group);
        } else {
            p.spc = best_spc(p.tiles, p.slabs_per_group, (double)M * N);
        }
        const int chunks = ceil_div(p.slabs_per_group, p.spc);
        p.clk = p.groups * (launch_clk(p.tiles, chunks, p.spc) + chunks * (double)M * N * 32.0 / kHbmBytesPerClk);
        if (cn_bytes(p, M, N, fixed_spc > 0, check) <= bytes) return p;
        if (p.slabs_per_group <= std::max(8, fixed_spc)) break;
    }
    p.groups = 0;
    return p;
}

// Test hook (i8_inject_no_loads): launches left before the one without loads.
std::atomic<long long> g_no_loads_in{-1};
constexpr unsigned long long kInjectedWaitNs = 20000000ULL;
struct Waits { unsigned long long ns; int no_loads; };
Waits launch_waits() {
    if (g_no_loads_in.load() >= 0 && g_no_loads_in.fetch_sub(1) == 0) return {kInjectedWaitNs, 1};
    return {kWaitNs, 0};
}

I8Side side_of(const I8Operand& op, int slab0) {
    return {op.data, op.mag, op.exps, op.tiles, op.tiles * op.tile, op.nslab, slab0, slab0 / op.spc};
}

}  // namespace

void i8_inject_no_loads(long long launches) { g_no_loads_in.store(launches < 0 ? -1 : launches); }

size_t i8_operand_bytes(int rows, int tile, int K, int spc, bool mag) {
    const size_t tiles = ceil_div(rows, tile), nslab = ceil_div(K, kSlab);
    return align256(kParts * tiles * nslab * tile * kSlab * kDig) + (mag ? align256(tiles * nslab * tile * kSlab) : 0) +
           align256((size_t)ceil_div((int)nslab, spc) * tiles * tile * sizeof(int));
}

size_t i8_operand_place(I8Operand& op, void* buf, int rows, int tile, int K, int spc, bool mag) {
    op.rows = rows;
    op.tile = tile;
    op.tiles = ceil_div(rows, tile);
    op.K = K;
    op.nslab = ceil_div(K, kSlab);
    op.spc = spc;
    op.data = (int8_t*)buf;
    const size_t plane = (size_t)op.tiles * op.nslab * tile * kSlab;
    char* at = (char*)buf + align256(kParts * plane * kDig);
    op.mag = mag ? (int8_t*)at : nullptr;
    op.exps = (int*)(at + (mag ? align256(plane) : 0));
    return i8_operand_bytes(rows, tile, K, spc, mag);
}

void i8_slice(const double2* x, long long ld, bool transposed, int sign, const I8Operand& op,
              cudaStream_t st) {
    count_launch();
    // whole tiles are cut: the rows past the matrix as zeros
    const int rp = op.tiles * op.tile;
    auto cut = [&](auto kernel, int rows_per_block) {
        kernel<<<dim3(rp / rows_per_block, op.chunks()), 256, 0, st>>>(
            x, ld, sign, op.rows, op.K, op.nslab, op.spc, op.tile, op.tiles, op.data, op.mag, op.exps);
    };
    if (transposed) cut(op.mag ? k_i8_slice<true, true> : k_i8_slice<true, false>, 32);
    else cut(op.mag ? k_i8_slice<false, true> : k_i8_slice<false, false>, 8);
}

int i8_cn_chunk_slabs(int M, int N, int K) {
    return best_spc(ceil_div(M, kTM) * ceil_div(N, kTN), ceil_div(K, kSlab), (double)M * N);
}

size_t i8_cn_scratch_bytes(int M, int N, int K, bool cached_a, bool check) {
    const CnPlan p = cn_plan(M, N, K, false, cached_a ? i8_cn_chunk_slabs(M, N, K) : 0, (size_t)-1);
    return cn_bytes(p, M, N, cached_a, check);
}

size_t i8_tn_scratch_bytes(int M, int N, int K, bool cached_x, bool check) {
    const int spc = ceil_div(K, kSlab);
    return i8_operand_bytes(M, kTN, K, spc, check) + (cached_x ? 0 : i8_operand_bytes(N, kTM, K, spc, check));
}

// The DMMA kernels: one 64 x 64 tile per SM at 264 clocks per 1 K; the INT8
// path is taken when its clocks, cutting included, are 5 % fewer.  Measured
// (us, INT8 / DMMA): beta^H psi 256 x 160 x 37,073 with beta cut once 213 / 426,
// 1,728 x 576 x 173,925 both cut 17,400 / 38,800; psi V 160 x 37,073 x 160
// 202 / 282, 576 x 173,925 x 576 5,720 / 12,770 (with the check of single elements
// 2-5 % more: 6,550, 19,500 and 232 us a call against 6,340, 19,000 and 220 for 576 x
// 173,925 x 576, 1,728 x 576 x 173,925 and 261 x 77 x 23,847); below the line 20 x 20 x 2,945
// 55 / 47, 160 x 160 x 8,000 94 / 75, 20 x 37,073 x 64 65 / 39.
// Relative error (2-norm over the result) against 64-bit sums of the same
// inputs, INT8 / DMMA: 1,728 x 576 x 173,925 1.1e-14 / 1.5e-14, 261 x 77 x 23,847
// 1.8e-15 / 2.3e-15, 576 x 173,925 x 576 1.1e-15 / 1.6e-15 (what is left is the
// rounding of the 64-bit sums themselves).
bool i8_cn_pays(int M, int N, int K, bool herm, bool cached_a) {
    const CnPlan p = cn_plan(M, N, K, herm, 0, (size_t)-1);
    const double i8 = p.clk + slice_clk((double)N * K) + (cached_a ? 0.0 : slice_clk((double)M * K)) + kReduceClk;
    const int t = ceil_div(M, 64), u = ceil_div(N, 64);
    const int tiles = herm ? u * (u + 1) / 2 : t * u;
    const int splits = splitk_count_tiles(tiles, K);
    const double dmma = (double)ceil_div(tiles * splits, kSms) * ceil_div(K, splits) * 264.0 + 14000.0;
    return i8 < 0.95 * dmma;
}

bool i8_tn_pays(int M, int N, int K, bool cached_x) {
    if (K > kI8MaxK) return false;
    const double i8 = launch_clk(ceil_div(N, kTM) * ceil_div(M, kTN), 1, ceil_div(K, kSlab)) +
                      slice_clk((double)M * K) + (cached_x ? 0.0 : slice_clk((double)N * K));
    const double dmma = (double)ceil_div(ceil_div(M, 64) * ceil_div(N, 64), kSms) * K * 264.0 + 6000.0;
    return i8 < 0.95 * dmma;
}

bool gemm_cn_i8(const double2* A, int lda, const I8Operand* pre, const double2* B, int ldb, int M,
                int N, int K, bool herm, void* scratch, size_t bytes, double2* out, int* err,
                cudaStream_t st, int* unresolved) {
    const bool check = unresolved != nullptr;  // not with digits cut before or herm
    const CnPlan p = cn_plan(M, N, K, herm, pre ? pre->spc : 0, bytes, check);
    const auto umma = check ? k_umma_i8<true> : k_umma_i8<false>;
    if (p.groups == 0 || raise_smem_limit(umma, kSmemBytes) != cudaSuccess) return false;
    for (int g = 0; g < p.groups; ++g) {
        const int slab0 = g * p.slabs_per_group, k0 = slab0 * kSlab;
        if (slab0 >= p.nslab) break;
        const int kg = std::min(K - k0, p.slabs_per_group * kSlab);
        char* at = (char*)scratch;
        I8Operand oa, ob;
        if (pre) {
            oa = *pre;
        } else {
            at += i8_operand_place(oa, at, M, kTM, kg, p.spc, check);
            i8_slice(A + k0, lda, false, -1, oa, st);
        }
        at += i8_operand_place(ob, at, N, kTN, kg, p.spc, check);
        i8_slice(B + k0, ldb, false, 1, ob, st);
        double2* part = (double2*)at;
        const int chunks = ob.chunks(), items = p.tiles * chunks;
        const Waits w = launch_waits();
        count_launch(2);
        umma<<<std::min(items, kSms), kThreads, kSmemBytes, st>>>(
            side_of(oa, pre ? slab0 : 0), side_of(ob, 0), false, M, N, p.mt, p.tiles, items, ob.nslab, p.spc, 1,
            herm ? 1 : 0, part, M, (long long)M * N, 1.0, 0.0, err, unresolved, nullptr, w.ns, w.no_loads);
        k_i8_reduce<<<dim3(ceil_div(M, 16), ceil_div(N, 16)), 256, 0, st>>>(part, chunks, M, N,
                                                                            herm ? 1 : 0, g > 0, out);
    }
    return true;
}

bool gemm_tn_i8(const double2* W, int ldw, const double2* X, int ldx, const I8Operand* pre,
                double2* O, int ldo, int M, int N, int K, double alpha, double beta, void* scratch,
                size_t bytes, int* err, cudaStream_t st, int* unresolved) {
    const bool check = unresolved != nullptr;  // not with digits cut before
    // O += ... cannot be taken back: everything is looked at before any of it is
    // added, and added only if `unresolved` stayed clear
    const bool first_look = check && beta != 0.0;
    if (K > kI8MaxK ||
        (check && raise_smem_limit(k_umma_i8<true>, kSmemBytes) != cudaSuccess) ||
        raise_smem_limit(k_umma_i8<false>, kSmemBytes) != cudaSuccess)
        return false;
    const int spc = ceil_div(K, kSlab), mt = ceil_div(M, kTN);
    const size_t wb = i8_operand_bytes(M, kTN, K, spc, check);
    // rows of X^T per group: what the rest of the scratch holds
    int rows = N;
    if (bytes < wb) return false;
    if (!pre && wb + i8_operand_bytes(N, kTM, K, spc, check) > bytes) {
        const size_t one = i8_operand_bytes(kTM, kTM, K, spc, check);
        const size_t fit = (bytes - wb) / one;
        if (fit < 1) return false;
        const int groups = ceil_div(ceil_div(N, kTM), (int)std::min<size_t>(fit, 1 << 20));
        rows = ceil_div(ceil_div(N, kTM), groups) * kTM;
    }
    I8Operand ow, ox;
    char* at = (char*)scratch;
    at += i8_operand_place(ow, at, M, kTN, K, spc, check);
    i8_slice(W, ldw, true, 1, ow, st);
    for (int pass = first_look ? 0 : 1; pass < 2; ++pass)
        for (int n0 = 0; n0 < N; n0 += rows) {
            const int n = std::min(rows, N - n0);
            if (pre) {
                ox = *pre;
            } else if (pass == 0 || !first_look || rows < N) {
                i8_operand_place(ox, at, n, kTM, K, spc, check);
                i8_slice(X + n0, ldx, true, 1, ox, st);
            }
            const int nt = ceil_div(n, kTM), items = nt * mt;
            const Waits w = launch_waits();
            count_launch();
            const auto umma = check && !(first_look && pass == 1) ? k_umma_i8<true> : k_umma_i8<false>;
            umma<<<std::min(items, kSms), kThreads, kSmemBytes, st>>>(
                side_of(ox, 0), side_of(ow, 0), pass == 0, n, M, nt, items, items, ox.nslab, spc,
                0, 0, O + n0, ldo, 0, alpha, beta, err, unresolved,
                first_look && pass == 1 ? unresolved : nullptr, w.ns, w.no_loads);
        }
    return true;
}

}  // namespace chfsi
