// Local Hamiltonian H_loc|psi> = T psi + FFT^-1[V(r) FFT[psi]] on the
// G-sphere, as three pruned passes over a band batch (role of the reference's
// init_kinetic / zero / scatter / cuFFT Z2Z / veff_multiply / cuFFT /
// gather_add_kinetic sequence, src/eigensolver/chebyshev.rs:279-365):
//
//   pass 1  z-sticks:  scatter the sphere coefficients of a group of (x,y)
//           columns into smem z-lines, inverse FFT along z, write the sticks
//           plane-major: work[b][z][column]
//   pass 2  xy-planes: unpack one z-plane (only the columns that carry
//           plane waves), inverse FFT along y (active x lines only) and x,
//           multiply by V(r), forward FFT along x and y (active x lines),
//           pack the columns back in place
//   pass 3  z-sticks:  forward FFT along z, gather the sphere, add the
//           kinetic and non-local terms and run the Chebyshev-recurrence
//           epilogue, reducing |psi_k|^2 for the norm guard
//
// HBM traffic per band: 4 x (ncol x nz) complex words plus the sphere
// vectors, versus ~14 N^3 words for the unpruned zero/scatter/FFT/multiply/
// FFT/gather sequence.
#include "kernels.hpp"
#include "launch_count.hpp"
#include "smem_limit.hpp"

#include <algorithm>
#include <cstdio>

namespace chfsi {

namespace {

template <typename C> __device__ __forceinline__ C czero() {
    using R = typename RealOf<C>::type;
    return mk((R)0, (R)0);
}

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Block-wide sum; result valid in thread 0.  red needs blockDim/32 doubles.
__device__ __forceinline__ double block_sum(double v, double* red) {
    v = warp_sum(v);
    const int w = threadIdx.x >> 5, l = threadIdx.x & 31;
    __syncthreads();
    if (l == 0) red[w] = v;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x < 32) {
        s = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
        s = warp_sum(s);
    }
    return s;
}

template <typename C> __host__ __device__ __forceinline__ size_t align16(size_t n) {
    return (n * sizeof(C) + 15) & ~(size_t)15;
}

// ---- two-radix line transforms with compile-time plans (N = R0 R1; DIF
// stage 0: radix R0 with span R1; stage 1: radix R1 on blocks of R1
// consecutive elements, all twiddles 1), used by the z-stick and plane passes.
// tw[m] = w^(n1 m), w = exp(2 pi i / N), for the span n1
// DIT stage 0: twiddle, radix-R0 DFT (sign +1)
template <int R0, typename C>
__device__ __forceinline__ void span_inverse(C* x, const C* tw) {
#pragma unroll
    for (int m = 1; m < R0; ++m) x[m] = cmul(tw[m], x[m]);
    dft_r<R0, 1>(x);
}
// DIF stage 0: radix-R0 DFT (sign -1), twiddle
template <int R0, typename C>
__device__ __forceinline__ void span_forward(C* x, const C* tw) {
    dft_r<R0, -1>(x);
#pragma unroll
    for (int m = 1; m < R0; ++m) x[m] = cmulc(tw[m], x[m]);
}
// tables w^j of the x and z axes
__device__ __forceinline__ const double2* xtable(const HGeom& g, double2) { return g.twd_x; }
__device__ __forceinline__ const float2* xtable(const HGeom& g, float2) { return g.twf_x; }
__device__ __forceinline__ const double2* ztable(const HGeom& g, double2) { return g.twd_z; }
__device__ __forceinline__ const float2* ztable(const HGeom& g, float2) { return g.twf_z; }

// ---------------------------------------------------------------- pass 1
// z lines of a block of columns, generic plans (one lane group per line)
template <typename C, int kColsPerBlock>
__global__ void __launch_bounds__(256)
k_zsticks_inverse(const C* __restrict__ psi, int ldp, C* __restrict__ work, HGeom g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* tw = reinterpret_cast<C*>(smem_raw);
    C* lines = reinterpret_cast<C*>(smem_raw + align16<C>(g.nz));
    const int b = blockIdx.y;
    const int c0 = blockIdx.x * kColsPerBlock;
    const int c1 = min(c0 + kColsPerBlock, g.ncol);
    const int nl = c1 - c0;
    copy_twiddles(tw, g.twd_z, g.twf_z, g.nz);
    for (int i = threadIdx.x; i < kColsPerBlock * g.lsz; i += blockDim.x) lines[i] = czero<C>();
    __syncthreads();
    const int g0 = g.col_start[c0], g1 = g.col_start[c1];
    const C* pb = psi + (size_t)b * ldp;
    for (int q = g0 + threadIdx.x; q < g1; q += blockDim.x)
        lines[(g.pw_col[q] - c0) * g.lsz + swz(g.pw_zpos[q], g.nz)] = pb[q];
    __syncthreads();
    fft_lines_grouped<false>(lines, nl, LinesStrided{g.lsz}, 1, g.az, tw);
    C* wb = work + (size_t)b * g.nz * g.ncol;
    for (int u = threadIdx.x; u < g.nz * kColsPerBlock; u += blockDim.x) {
        const int z = u / kColsPerBlock, cl = u - z * kColsPerBlock;
        if (cl < nl) wb[(size_t)z * g.ncol + c0 + cl] = lines[cl * g.lsz + swz(z, g.nz)];
    }
}

// Two-radix plans: 32 columns per block, a lane per column and a warp per
// butterfly of the stage (R0 warps with blocks, R1 with spans), lines stored
// [position][column].  The work array is [z][column] as well, so the stage that
// meets it moves between registers and global memory in 512-byte rows without a
// pass through shared memory; a butterfly's twiddles are the same for the whole
// warp, and every shared access is one row.  The column is XORed with the low
// bits of the position's block, which spreads the plane waves of one column
// (consecutive frequencies, a block apart) over the banks for the scatter and the
// gather.  Against lane groups along each line (which spent 81 % of the
// shared-memory wavefronts, 6.2 per access, half of them on twiddles and
// conflicts), 160 bands on 72^3, us a launch, with the bands in turn below and the
// epilogue's batches: FP64 inverse 138 -> 97, H apply 190 -> 109, Chebyshev step
// 227 -> 128; FP32 100 -> 48 and 195 -> 85.
template <int R0, int R1> struct ZTwo {
    static constexpr int N = R0 * R1, warps = R0 > R1 ? R0 : R1, threads = 32 * warps;
    static constexpr int min_blocks = 65536 / (80 * threads) > 0 ? 65536 / (80 * threads) : 1;
};
template <int R1> __device__ __forceinline__ int zslot(int p, int c) { return p * 32 + (c ^ ((p / R1) & 7)); }

template <typename C> __device__ __forceinline__ void cp_async_elem(C* dst, const C* src) {
    const uint32_t d = (uint32_t)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(C) == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}

// A block takes the same columns of bpb bands.  With more than one band the plane
// waves of the next are copied to a second buffer while this one is transformed:
// with a band per block the pass waited for its loads (registers allow two or
// three blocks an SM, DRAM was 35 % busy): 160 bands on 72^3 122 -> 97 us, 576 on
// 108^3 1,654 -> 1,584.  The last stage leaves zeros behind for the band after the
// next.
template <typename C, int R0, int R1>
__global__ void __launch_bounds__(ZTwo<R0, R1>::threads, ZTwo<R0, R1>::min_blocks)
k_zsticks_inverse2(const C* __restrict__ psi, int ldp, C* __restrict__ work, int nb, int bpb, HGeom g) {
    constexpr int N = R0 * R1, kSlots = 4, T = ZTwo<R0, R1>::threads;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* lines = reinterpret_cast<C*>(smem_raw);
    const int b0 = blockIdx.y * bpb, b1 = min(b0 + bpb, nb);
    const int c0 = blockIdx.x * 32, nl = min(32, g.ncol - c0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < N * 32 * (bpb > 1 ? 2 : 1); i += T) lines[i] = czero<C>();
    const int g0 = g.col_start[c0] + threadIdx.x, g1 = g.col_start[c0 + nl];
    int slot[kSlots];
#pragma unroll
    for (int k = 0; k < kSlots; ++k) {
        const int q = g0 + k * T;
        slot[k] = q < g1 ? zslot<R1>(g.pw_zpos[q], g.pw_col[q] - c0) : 0;
    }
    auto fetch = [&](C* dst, int b) {
        const C* pb = psi + (size_t)b * ldp;
#pragma unroll
        for (int k = 0; k < kSlots; ++k)
            if (g0 + k * T < g1) cp_async_elem(dst + slot[k], pb + g0 + k * T);
        for (int q = g0 + kSlots * T; q < g1; q += T)
            cp_async_elem(dst + zslot<R1>(g.pw_zpos[q], g.pw_col[q] - c0), pb + q);
    };
    __syncthreads();
    fetch(lines, b0);
    for (int b = b0; b < b1; ++b) {
        C* cur = lines + ((b - b0) & 1) * N * 32;
        asm volatile("cp.async.wait_all;\n" ::: "memory");
        __syncthreads();
        if (b + 1 < b1) fetch(lines + ((b + 1 - b0) & 1) * N * 32, b + 1);
        if (warp < R0) {
            C* l = cur + warp * R1 * 32 + (lane ^ (warp & 7));
            C x[R1];
#pragma unroll
            for (int j = 0; j < R1; ++j) x[j] = l[j * 32];
            dft_r<R1, 1>(x);
#pragma unroll
            for (int j = 0; j < R1; ++j) l[j * 32] = x[j];
        }
        __syncthreads();
        if (warp < R1) {
            C x[R0];
#pragma unroll
            for (int j = 0; j < R0; ++j) x[j] = cur[(warp + j * R1) * 32 + (lane ^ (j & 7))];
            if (b + 2 < b1)
#pragma unroll
                for (int j = 0; j < R0; ++j) cur[(warp + j * R1) * 32 + (lane ^ (j & 7))] = czero<C>();
            C tw[R0];
#pragma unroll
            for (int m = 1; m < R0; ++m) tw[m] = __ldg(ztable(g, C{}) + warp * m);
            span_inverse<R0>(x, tw);
            C* wb = work + ((size_t)b * N + warp) * g.ncol + c0 + lane;
            if (lane < nl)
#pragma unroll
                for (int j = 0; j < R0; ++j) wb[(size_t)(j * R1) * g.ncol] = x[j];
        }
    }
}

// ---------------------------------------------------------------- pass 2
// 256 threads with 2 (FP64) or 3 (FP32) resident blocks per SM: the
// global-memory phases of one plane overlap the FFT stages of another.
// Variant 0: 256 threads, 1: 128 threads, 2: 512 threads per block, with as
// many resident blocks per SM as the registers of each precision allow.
template <typename C, int V>
struct PlanesCfg {
    static constexpr int threads = V == 0 ? 256 : (V == 1 ? 128 : 512);
    static constexpr int min_blocks =
        V == 0 ? (sizeof(C) == 16 ? 2 : 3) : (V == 1 ? (sizeof(C) == 16 ? 4 : 6) : 1);
};

template <typename C, int V>
__global__ void __launch_bounds__(PlanesCfg<C, V>::threads, PlanesCfg<C, V>::min_blocks)
k_planes_vloc(C* __restrict__ work, const double* __restrict__ veff, HGeom g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* twx = reinterpret_cast<C*>(smem_raw);
    C* twy = reinterpret_cast<C*>(smem_raw + align16<C>(g.nx));
    C* plane = reinterpret_cast<C*>(smem_raw + align16<C>(g.nx) + align16<C>(g.ny));
    int* xl = reinterpret_cast<int*>(plane + (size_t)g.ny * g.lsx);
    const int z = blockIdx.x, b = blockIdx.y;
    copy_twiddles(twx, g.twd_x, g.twf_x, g.nx);
    copy_twiddles(twy, g.twd_y, g.twf_y, g.ny);
    for (int i = threadIdx.x; i < g.nxact; i += blockDim.x) xl[i] = g.xact[i];
    for (int i = threadIdx.x; i < g.ny * g.lsx; i += blockDim.x) plane[i] = czero<C>();
    __syncthreads();
    C* wp = work + ((size_t)b * g.nz + z) * g.ncol;
    for (int c = threadIdx.x; c < g.ncol; c += blockDim.x) plane[g.col_pos[c]] = wp[c];
    __syncthreads();
    fft_lines_grouped<false>(plane, g.nxact, LinesListed{xl}, g.lsx, g.ay, twy);
    // x rows: inverse, x V(r), forward, all inside one lane group per row
    const double* vz = veff + (size_t)z * g.nx * g.ny;
    using R = typename RealOf<C>::type;
    {
        const LaneGroups lg(g.ax.tpl);
        const int rounds = (g.ny + lg.total - 1) / lg.total;
        for (int rd = 0; rd < rounds; ++rd) {
            const int y = rd * lg.total + lg.id;
            const bool act = lg.in_group && y < g.ny;
            C* row = plane + (act ? swz(y, g.ny) * g.lsx : 0);
            line_fft_group<false>(row, act, lg.i, 1, g.ax, twx);
            if (act) {
                const double* vr = vz + (size_t)y * g.nx;
                for (int x = lg.i; x < g.nx; x += g.ax.tpl) {
                    C& e = row[swz(x, g.nx)];
                    e = cscale(e, (R)vr[x]);
                }
            }
            __syncwarp();
            line_fft_group<true>(row, act, lg.i, 1, g.ax, twx);
        }
    }
    __syncthreads();
    fft_lines_grouped<true>(plane, g.nxact, LinesListed{xl}, g.lsx, g.ay, twy);
    for (int c = threadIdx.x; c < g.ncol; c += blockDim.x) wp[c] = plane[g.col_pos[c]];
}

// ------------------------------------------ pass 2, two-radix compile-time plans
// Square planes on a two-radix plan.  The plane's columns are read and written in
// place of a scatter and a gather: the first inverse y stage of every active x
// line loads its inputs from the column array (zero where (x, y) holds no column),
// the last forward y stage stores its outputs straight to the columns, the first
// inverse x stage takes zero for x positions without columns, and the last
// forward x stage stores only the positions the forward y stage reads; nothing is
// zeroed.  Along x the last inverse stage, the V(r) multiply and the first forward
// stage share registers.
// Bound by shared-memory wavefronts and the FP64 pipe.  A warp takes 8 lines x 4
// butterflies of a stage: the 8 lanes of an access phase hold the same element of
// 8 neighbouring lines, a bank group each (rows are an odd number of 16-byte
// elements long; active x lines come in the order of x, which the digit reversal, with
// positions XOR-swizzled for even R1, spreads over the groups, and whose columns lie
// side by side in memory), a lane's span index is the same
// throughout, so that its twiddles stay in registers, and every lane works in most rounds whatever the radices (with a lane group per
// line a 12 x 9 plan left a quarter of the lanes idle and took 3.7 times the
// wavefronts of its data).  Stages are separated by block barriers and the blocks of
// one SM overlap; on planes up to 50 x 50 a warp keeps its lines instead (40 x 40,
// 200 bands: 134 us a local H against 153; 72 x 72: 815 against 811).  Local H in
// all, us, before / with this kernel: 40^3 x 200 bands 183 / 134, 64^3 x 160 577 /
// 508, 72^3 x 160 820 / 811, 80^3 x 100 1,840 / 746 (generic kernel before),
// 108^3 x 576 17,880 / 11,550.
// NB bands per 16-byte element: 1 in FP64; in FP32 bands 2p and 2p + 1, so that
// each twiddle and V(r) load serves both (an odd last band runs alone: its
// partner's loads repeat it and are not stored).
template <int R0, int R1> struct PlaneTwo {
    static constexpr int N = R0 * R1, LS = N | 1, G = (N + 7) / 8;
    static constexpr int Q0 = (R0 + 3) / 4, Q1 = (R1 + 3) / 4;
    static constexpr int bytes = N * LS * 16 + ((N + 3) & ~3) * 4 + (R0 - 1) * R1 * 16;
    static constexpr int fit = 227 * 1024 / (bytes + 1024);  // blocks by shared memory
    // warps: near 9 (14 where one block fills the SM), a multiple of Q1 so that a
    // warp keeps its spans, wasting the fewest warp rounds of the x stages
    static constexpr int pick() {
        const int lo = fit > 1 ? 8 : 12, hi = fit > 1 ? 10 : 16;
        int best = lo, waste = 1 << 30;
        for (int w = lo; w <= hi; ++w) {
            if (w % Q1) continue;
            const int r = w * (2 * ((G * Q0 + w - 1) / w) + (G + w / Q1 - 1) / (w / Q1));
            if (r <= waste) {
                waste = r;
                best = w;
            }
        }
        return best;
    }
    // small planes (up to 50 x 50): a warp takes a group of lines through all its
    // stages, without block barriers between them
    static constexpr bool own = fit >= 5;
    static constexpr int shared_warps = pick(), warps = own ? G : shared_warps, threads = 32 * warps;
    // 96 registers: what 9 x 8 and 8 x 5 need.  Not fitted plan by plan: -Xptxas -v
    // shows 336 bytes of spill stores for 15 x 5 and (at 80 registers) 10 x 5, 68 for
    // 9 x 5, 28 for 10 x 8, 16 or less for the others
    static constexpr int by_regs = 65536 / (threads * 96);
    static constexpr int min_blocks = fit < by_regs ? fit : by_regs > 0 ? by_regs : 1;
    // place of x position p in a row
    __device__ __forceinline__ static int at(int p) { return R1 % 2 ? p : swz(p, N); }
};

__device__ __forceinline__ void unpack(double2 e, double2 (&x)[1]) { x[0] = e; }
__device__ __forceinline__ void unpack(float4 e, float2 (&x)[2]) {
    x[0] = make_float2(e.x, e.y);
    x[1] = make_float2(e.z, e.w);
}
__device__ __forceinline__ double2 pack(const double2 (&x)[1]) { return x[0]; }
__device__ __forceinline__ float4 pack(const float2 (&x)[2]) { return make_float4(x[0].x, x[0].y, x[1].x, x[1].y); }
template <int NB> struct PlaneElem { using type = double2; };
template <> struct PlaneElem<2> { using type = float4; };

// values of a butterfly, band by band
template <typename C, int NB, int R> struct Bfly {
    C x[NB][R];
    template <typename S> __device__ __forceinline__ void set(int j, S e) {
        C v[NB];
        unpack(e, v);
#pragma unroll
        for (int b = 0; b < NB; ++b) x[b][j] = v[b];
    }
    __device__ __forceinline__ typename PlaneElem<NB>::type get(int j) const {
        C v[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) v[b] = x[b][j];
        return pack(v);
    }
    template <int SIGN> __device__ __forceinline__ void dft() {
#pragma unroll
        for (int b = 0; b < NB; ++b) dft_r<R, SIGN>(x[b]);
    }
};

template <typename C, int NB, int R0, int R1>
__global__ void __launch_bounds__(PlaneTwo<R0, R1>::threads, PlaneTwo<R0, R1>::min_blocks)
k_planes_vloc2(C* __restrict__ work, const double* __restrict__ veff, int nb, HGeom g) {
    using P = PlaneTwo<R0, R1>;
    using S = typename PlaneElem<NB>::type;
    using R = typename RealOf<C>::type;
    constexpr int N = P::N, LS = P::LS, W = P::warps;
    constexpr bool own = P::own;          // a warp takes its lines through all stages
    extern __shared__ __align__(16) unsigned char smem_raw[];
    S* plane = reinterpret_cast<S*>(smem_raw);
    int* xl = reinterpret_cast<int*>(plane + (size_t)N * LS);
    const int z = blockIdx.x, b0 = NB * blockIdx.y, nxact = g.nxact;
    for (int i = threadIdx.x; i < nxact; i += blockDim.x) xl[i] = P::at(g.xline[i]);
    C* wp[NB];
    bool live[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) {
        live[b] = b0 + b < nb;
        wp[b] = work + ((size_t)(live[b] ? b0 + b : b0) * g.nz + z) * g.ncol;
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane & 7, t = lane >> 3;
    const int gy = (nxact + 7) >> 3;
    // twiddles w^(n1 m) of this lane's spans: one span where a warp keeps to its
    // quad, else from the lane-ordered table in shared memory
    C* twm = reinterpret_cast<C*>(xl + ((N + 3) & ~3));
    C tw[R0];
    if constexpr (own) {
        for (int i = threadIdx.x; i < (R0 - 1) * R1; i += blockDim.x) {
            const int m = i / R1 + 1;
            twm[i] = xtable(g, C{})[(i - (m - 1) * R1) * m];
        }
    } else {
        const int n1 = (warp % P::Q1) * 4 + t;
#pragma unroll
        for (int m = 1; m < R0; ++m) tw[m] = n1 < R1 ? __ldg(xtable(g, C{}) + n1 * m) : czero<C>();
    }
    __syncthreads();
    auto stage_sync = [&]() {
        if constexpr (own) __syncwarp();
        else __syncthreads();
    };
    // the butterflies of one stage over `groups` groups of 8 lines: f(line, index)
    auto blocks = [&](int groups, int grp, auto&& f) {
        if constexpr (own) {
#pragma unroll
            for (int q = 0; q < P::Q0; ++q)
                if (q * 4 + t < R0) f(grp * 8 + r, q * 4 + t);
        } else {
            for (int it = warp; it < groups * P::Q0; it += W)
                if ((it % P::Q0) * 4 + t < R0) f((it / P::Q0) * 8 + r, (it % P::Q0) * 4 + t);
        }
    };
    auto spans = [&](int groups, int grp, auto&& f) {
        if constexpr (own) {
#pragma unroll
            for (int q = 0; q < P::Q1; ++q) {
                const int n1 = q * 4 + t;
                if (n1 < R1) {
#pragma unroll
                    for (int m = 1; m < R0; ++m) tw[m] = twm[(m - 1) * R1 + n1];
                    f(grp * 8 + r, n1);
                }
            }
        } else {
            const int n1 = (warp % P::Q1) * 4 + t;
            if (n1 < R1)
                for (int it = warp / P::Q1; it < groups; it += W / P::Q1) f(it * 8 + r, n1);
        }
    };
    auto y_blocks_in = [&](int l, int blk) {  // inverse, from the columns
        if (l >= nxact) return;
        Bfly<C, NB, R1> v;
        const int* ci = g.colidx_t + (size_t)blk * R1 * nxact + l;
#pragma unroll
        for (int j = 0; j < R1; ++j) {
            const int c = __ldg(ci + j * nxact);
#pragma unroll
            for (int b = 0; b < NB; ++b) v.x[b][j] = c >= 0 ? wp[b][c] : czero<C>();
        }
        v.template dft<1>();
        S* p = plane + (size_t)blk * R1 * LS + xl[l];
#pragma unroll
        for (int j = 0; j < R1; ++j) p[j * LS] = v.get(j);
    };
    auto y_span = [&](int l, int n1, bool fwd) {
        if (l >= nxact) return;
        Bfly<C, NB, R0> v;
        S* p = plane + (size_t)n1 * LS + xl[l];
#pragma unroll
        for (int j = 0; j < R0; ++j) v.set(j, p[j * R1 * LS]);
#pragma unroll
        for (int b = 0; b < NB; ++b) {
            if (fwd) span_forward<R0>(v.x[b], tw);
            else span_inverse<R0>(v.x[b], tw);
        }
#pragma unroll
        for (int j = 0; j < R0; ++j) p[j * R1 * LS] = v.get(j);
    };
    auto y_blocks_out = [&](int l, int blk) {  // forward, to the columns
        if (l >= nxact) return;
        Bfly<C, NB, R1> v;
        const S* p = plane + (size_t)blk * R1 * LS + xl[l];
#pragma unroll
        for (int j = 0; j < R1; ++j) v.set(j, p[j * LS]);
        v.template dft<-1>();
        const int* ci = g.colidx_t + (size_t)blk * R1 * nxact + l;
#pragma unroll
        for (int j = 0; j < R1; ++j) {
            const int c = __ldg(ci + j * nxact);
            if (c >= 0)
#pragma unroll
                for (int b = 0; b < NB; ++b)
                    if (live[b]) wp[b][c] = v.x[b][j];
        }
    };
    auto x_blocks_in = [&](int y, int blk) {
        if (y >= N) return;
        Bfly<C, NB, R1> v;
        S* row = plane + y * LS;
#pragma unroll
        for (int j = 0; j < R1; ++j) {
            const int px = blk * R1 + j;
            const bool on = (g.xbits[px >> 5] >> (px & 31)) & 1u;
            v.set(j, on ? row[P::at(px)] : S{});
        }
        v.template dft<1>();
#pragma unroll
        for (int j = 0; j < R1; ++j) row[P::at(blk * R1 + j)] = v.get(j);
    };
    const double* vz = veff + (size_t)z * N * N;
    auto x_spans = [&](int y, int n1) {  // last inverse stage, V(r), first forward stage
        if (y >= N) return;
        Bfly<C, NB, R0> v;
        S* row = plane + y * LS;
        const double* vr = vz + (size_t)y * N + n1;
#pragma unroll
        for (int j = 0; j < R0; ++j) v.set(j, row[P::at(n1 + j * R1)]);
#pragma unroll
        for (int b = 0; b < NB; ++b) span_inverse<R0>(v.x[b], tw);
#pragma unroll
        for (int j = 0; j < R0; ++j) {
            const R s = (R)__ldg(vr + j * R1);
#pragma unroll
            for (int b = 0; b < NB; ++b) v.x[b][j] = cscale(v.x[b][j], s);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) span_forward<R0>(v.x[b], tw);
#pragma unroll
        for (int j = 0; j < R0; ++j) row[P::at(n1 + j * R1)] = v.get(j);
    };
    auto x_blocks_out = [&](int y, int blk) {
        if (y >= N) return;
        Bfly<C, NB, R1> v;
        S* row = plane + y * LS;
#pragma unroll
        for (int j = 0; j < R1; ++j) v.set(j, row[P::at(blk * R1 + j)]);
        v.template dft<-1>();
#pragma unroll
        for (int j = 0; j < R1; ++j) {
            const int px = blk * R1 + j;
            if ((g.xbits[px >> 5] >> (px & 31)) & 1u) row[P::at(px)] = v.get(j);
        }
    };
    for (int grp = warp; grp < (own ? gy : warp + 1); grp += W) {
        blocks(gy, grp, y_blocks_in);
        stage_sync();
        spans(gy, grp, [&](int l, int n1) { y_span(l, n1, false); });
    }
    __syncthreads();
    for (int grp = warp; grp < (own ? P::G : warp + 1); grp += W) {
        blocks(P::G, grp, x_blocks_in);
        stage_sync();
        spans(P::G, grp, x_spans);
        stage_sync();
        blocks(P::G, grp, x_blocks_out);
    }
    __syncthreads();
    for (int grp = warp; grp < (own ? gy : warp + 1); grp += W) {
        spans(gy, grp, [&](int l, int n1) { y_span(l, n1, true); });
        stage_sync();
        blocks(gy, grp, y_blocks_out);
    }
}

// ------------------------- pass 2, FP32, two bands per CTA (compile-time plans)
// The same pipeline with a lane group per line and whole lines per warp, for the
// FP32 filter on planes of which two blocks fit an SM: without the FP64 pipe as a
// second limit its fewer V(r) wavefronts win (72 x 72, 160 bands: 326 us a launch
// against 351 for k_planes_vloc2).
__device__ __forceinline__ float4 pair4(float2 a, float2 b) { return make_float4(a.x, a.y, b.x, b.y); }
__device__ __forceinline__ float2 lo2(float4 v) { return make_float2(v.x, v.y); }
__device__ __forceinline__ float2 hi2(float4 v) { return make_float2(v.z, v.w); }

// lane-ordered span twiddles: twm[(m - 1) R1 + n1] = w^(n1 m)
template <int R0, int R1>
__device__ __forceinline__ void lane_twiddles(float2* twm, const float2* tab) {
    for (int i = threadIdx.x; i < (R0 - 1) * R1; i += blockDim.x) {
        const int m = i / R1 + 1, n1 = i - (m - 1) * R1;
        twm[i] = tab[n1 * m];
    }
}
template <int R0, int R1>
__device__ __forceinline__ void lane_tw(float2* tw, const float2* twm, int n1) {
#pragma unroll
    for (int m = 1; m < R0; ++m) tw[m] = twm[(m - 1) * R1 + n1];
}

// Lane -> (group, index in group) of the two-radix line transforms with T
// lanes per line and PW lines per warp.  Indices 0-7 of every group fill
// whole 8-lane phases (one line per phase), the higher indices follow
// packed: the 16-byte shared-memory accesses of a phase then fall on one
// line, whose XOR-swizzled elements span all eight bank groups.
template <int T, int PW>
__device__ __forceinline__ void p2_lane(int lane, int& gi, int& li) {
    if constexpr (T <= 8) {
        gi = lane / T;
        li = lane - gi * T;
    } else {
        if (lane < PW * 8) {
            gi = lane >> 3;
            li = lane & 7;
        } else {
            const int r = lane - PW * 8;
            gi = r / (T - 8);
            li = 8 + (r - gi * (T - 8));
        }
    }
}
template <int V, int R0, int R1>
__global__ void __launch_bounds__(PlanesCfg<double2, V>::threads, PlanesCfg<double2, V>::min_blocks)
k_planes_vloc_p3x2(float2* __restrict__ work, const double* __restrict__ veff, int nb, HGeom g) {
    constexpr int N = R0 * R1, LS = N | 1, T = R0 > R1 ? R0 : R1, PW = 32 / T;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* twx = reinterpret_cast<float2*>(smem_raw);
    float2* twy = reinterpret_cast<float2*>(smem_raw + align16<float2>(N));
    float4* plane = reinterpret_cast<float4*>(smem_raw + 2 * align16<float2>(N));
    int* xl = reinterpret_cast<int*>(plane + (size_t)N * LS);
    const int z = blockIdx.x, b0 = 2 * blockIdx.y;
    const bool two = b0 + 1 < nb;
    const int nxact = g.nxact;
    lane_twiddles<R0, R1>(twx, g.twf_x);
    lane_twiddles<R0, R1>(twy, g.twf_y);
    for (int i = threadIdx.x; i < nxact; i += blockDim.x) xl[i] = swz(g.xline[i], N);
    __syncthreads();
    float2* wa = work + ((size_t)b0 * g.nz + z) * g.ncol;
    float2* wb = two ? work + ((size_t)(b0 + 1) * g.nz + z) * g.ncol : wa;
    const int lane = threadIdx.x & 31;
    int gi, li;
    p2_lane<T, PW>(lane, gi, li);
    const bool ing = gi < PW;
    const int groups = (blockDim.x >> 5) * PW, gid = (threadIdx.x >> 5) * PW + gi;
    const float2 zero = make_float2(0.f, 0.f);
    // y lines through the active x positions: inverse, inputs from the columns
    for (int l0 = 0; l0 < nxact; l0 += groups) {
        const int l = l0 + gid;
        const bool act = ing && l < nxact;
        float4* line = plane + (act ? xl[l] : 0);
        if (act && li < R0) {
            const int* ci = g.colidx_t + (size_t)li * R1 * nxact + l;
            float2 xa[R1], xb[R1];
#pragma unroll
            for (int j = 0; j < R1; ++j) {
                const int c = __ldg(ci + j * nxact);
                xa[j] = c >= 0 ? wa[c] : zero;
                xb[j] = c >= 0 ? wb[c] : zero;
            }
            dft_r<R1, 1>(xa);
            dft_r<R1, 1>(xb);
#pragma unroll
            for (int m = 0; m < R1; ++m) line[swz(li * R1 + m, N) * LS] = pair4(xa[m], xb[m]);
        }
        __syncwarp();
        if (act && li < R1) {
            float2 xa[R0], xb[R0];
#pragma unroll
            for (int j = 0; j < R0; ++j) {
                const float4 v = line[swz(li + j * R1, N) * LS];
                xa[j] = lo2(v);
                xb[j] = hi2(v);
            }
            float2 tw[R0];
            lane_tw<R0, R1>(tw, twy, li);
            span_inverse<R0>(xa, tw);
            span_inverse<R0>(xb, tw);
#pragma unroll
            for (int j = 0; j < R0; ++j) line[swz(li + j * R1, N) * LS] = pair4(xa[j], xb[j]);
        }
        __syncwarp();
    }
    __syncthreads();
    // x rows: inverse (x positions without columns read as zero), x V(r),
    // forward (only x positions with columns stored)
    const double* vz = veff + (size_t)z * N * N;
    for (int y0 = 0; y0 < N; y0 += groups) {
        const int y = y0 + gid;
        const bool act = ing && y < N;
        float4* row = plane + (act ? swz(y, N) * LS : 0);
        if (act && li < R0) {
            float2 xa[R1], xb[R1];
#pragma unroll
            for (int j = 0; j < R1; ++j) {
                const int px = li * R1 + j;
                const bool on = (g.xbits[px >> 5] >> (px & 31)) & 1u;
                const float4 v = on ? row[swz(px, N)] : make_float4(0.f, 0.f, 0.f, 0.f);
                xa[j] = lo2(v);
                xb[j] = hi2(v);
            }
            dft_r<R1, 1>(xa);
            dft_r<R1, 1>(xb);
#pragma unroll
            for (int m = 0; m < R1; ++m) row[swz(li * R1 + m, N)] = pair4(xa[m], xb[m]);
        }
        __syncwarp();
        if (act && li < R1) {
            float2 xa[R0], xb[R0];
#pragma unroll
            for (int j = 0; j < R0; ++j) {
                const float4 v = row[swz(li + j * R1, N)];
                xa[j] = lo2(v);
                xb[j] = hi2(v);
            }
            float2 tw[R0];
            lane_tw<R0, R1>(tw, twx, li);
            span_inverse<R0>(xa, tw);
            span_inverse<R0>(xb, tw);
            const double* vr = vz + (size_t)y * N + li;
#pragma unroll
            for (int m = 0; m < R0; ++m) {
                const float s = (float)vr[m * R1];
                xa[m] = cscale(xa[m], s);
                xb[m] = cscale(xb[m], s);
            }
            span_forward<R0>(xa, tw);
            span_forward<R0>(xb, tw);
#pragma unroll
            for (int j = 0; j < R0; ++j) row[swz(li + j * R1, N)] = pair4(xa[j], xb[j]);
        }
        __syncwarp();
        if (act && li < R0) {
            float2 xa[R1], xb[R1];
#pragma unroll
            for (int j = 0; j < R1; ++j) {
                const float4 v = row[swz(li * R1 + j, N)];
                xa[j] = lo2(v);
                xb[j] = hi2(v);
            }
            dft_r<R1, -1>(xa);
            dft_r<R1, -1>(xb);
#pragma unroll
            for (int m = 0; m < R1; ++m) {
                const int px = li * R1 + m;
                if ((g.xbits[px >> 5] >> (px & 31)) & 1u) row[swz(px, N)] = pair4(xa[m], xb[m]);
            }
        }
        __syncwarp();
    }
    __syncthreads();
    // y lines forward, outputs to the columns
    for (int l0 = 0; l0 < nxact; l0 += groups) {
        const int l = l0 + gid;
        const bool act = ing && l < nxact;
        float4* line = plane + (act ? xl[l] : 0);
        if (act && li < R1) {
            float2 xa[R0], xb[R0];
#pragma unroll
            for (int j = 0; j < R0; ++j) {
                const float4 v = line[swz(li + j * R1, N) * LS];
                xa[j] = lo2(v);
                xb[j] = hi2(v);
            }
            float2 tw[R0];
            lane_tw<R0, R1>(tw, twy, li);
            span_forward<R0>(xa, tw);
            span_forward<R0>(xb, tw);
#pragma unroll
            for (int j = 0; j < R0; ++j) line[swz(li + j * R1, N) * LS] = pair4(xa[j], xb[j]);
        }
        __syncwarp();
        if (act && li < R0) {
            float2 xa[R1], xb[R1];
#pragma unroll
            for (int j = 0; j < R1; ++j) {
                const float4 v = line[swz(li * R1 + j, N) * LS];
                xa[j] = lo2(v);
                xb[j] = hi2(v);
            }
            dft_r<R1, -1>(xa);
            dft_r<R1, -1>(xb);
            const int* ci = g.colidx_t + (size_t)li * R1 * nxact + l;
#pragma unroll
            for (int m = 0; m < R1; ++m) {
                const int c = __ldg(ci + m * nxact);
                if (c >= 0) {
                    wa[c] = xa[m];
                    if (two) wb[c] = xb[m];
                }
            }
        }
        __syncwarp();
    }
}

// ---------------------------------------------------------------- pass 3
// gather + kinetic + non-local + epilogue over the plane waves of columns c0 ..
// c1 - 1; slot(position, column) is the place of a value in `lines`
template <typename C, int MODE, typename Slot>
__device__ __forceinline__ void z_epilogue(const C* lines, Slot slot, int c0, int c1,
                                           const C* __restrict__ psi, int ldp, C* out, int ldo,
                                           const HGeom& g, const Epilogue& e) {
    __shared__ double red[32];
    using R = typename RealOf<C>::type;
    const int b = blockIdx.y;
    const int g0 = g.col_start[c0], g1 = g.col_start[c1];
    const C* pb = psi + (size_t)b * ldp;
    C* ob = out + (size_t)b * ldo;
    const C* nlb = e.nl ? reinterpret_cast<const C*>(e.nl) + (size_t)b * ldp : nullptr;
    R ie = 0, nc = 0;
    if (MODE == kEpiChebFirst || MODE == kEpiCheb) {
        ie = (R)e.coef[4];
        nc = (R)e.coef[5];
    }
    R ra = 0, rb = 0, rcc = 0, rly = 0;
    const C* yb = nullptr;
    if (MODE == kEpiResid) {
        ra = (R)e.rc[0];
        rb = (R)e.rc[1];
        rcc = (R)e.rc[2];
        rly = (R)(e.rc[0] * e.lam[b]);
        yb = reinterpret_cast<const C*>(e.yres) + (size_t)b * ldp;
    }
    const R inv_n = (R)e.inv_n;
    // the Lanczos vector carried in the batch: plain H x, no recurrence
    const bool plain = b == e.plain_band;
    C* pob = plain ? reinterpret_cast<C*>(e.plain_out) : nullptr;
    double nacc = 0.0;
    if constexpr (sizeof(C) == 8) {
        // FP32 keeps one plane wave at a time: with the batches below the compiler
        // contracts the sums the other way round, another rounding of the filtered
        // bands (3e-8), for 1 % of a mixed pass
        for (int q = g0 + threadIdx.x; q < g1; q += blockDim.x) {
            const C v = lines[slot(g.pw_zpos[q], g.pw_col[q] - c0)];
            const C p = pb[q];
            const R k = (R)e.kin[q];
            C h = mk(p.x * k, p.y * k);
            h = mk(h.x + v.x * inv_n, h.y + v.y * inv_n);
            if (nlb) h = cadd(h, nlb[q]);
            if (plain) {
                pob[q] = h;
            } else if (MODE == kEpiApply) {
                ob[q] = h;
            } else if (MODE == kEpiResid) {
                const C prev = ob[q];
                const C y = yb[q];
                ob[q] = mk(ra * h.x + rb * p.x + rcc * prev.x + rly * y.x,
                           ra * h.y + rb * p.y + rcc * prev.y + rly * y.y);
            } else {
                C s = mk(h.x * ie + nc * p.x, h.y * ie + nc * p.y);
                C o;
                if (MODE == kEpiChebFirst) o = s;
                else {
                    const C prev = ob[q];
                    o = mk((R)2 * s.x - prev.x, (R)2 * s.y - prev.y);
                }
                ob[q] = o;
                nacc += (double)o.x * (double)o.x + (double)o.y * (double)o.y;
            }
        }
        if (MODE != kEpiApply && e.norm_acc) {
            double s = block_sum(nacc, red);
            if (threadIdx.x == 0) atomicAdd(e.norm_acc, s);
        }
        return;
    }
    // the loads of kU plane waves before their arithmetic: one at a time, with
    // `out` both read and written, each waits for the one before (160 bands on 72^3,
    // Chebyshev step 172 -> 128 us)
    constexpr int kU = MODE == kEpiResid ? 2 : 4;
    for (int q0 = g0 + threadIdx.x; q0 < g1; q0 += kU * blockDim.x) {
        C p[kU], nv[kU], prev[kU], y[kU];
        R k[kU];
        int at[kU];
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int q = q0 + u * blockDim.x;
            if (q >= g1) continue;
            p[u] = pb[q];
            k[u] = (R)e.kin[q];
            if (nlb) nv[u] = nlb[q];
            if ((MODE == kEpiCheb || MODE == kEpiResid) && !plain) prev[u] = ob[q];
            if (MODE == kEpiResid && !plain) y[u] = yb[q];
            at[u] = slot(g.pw_zpos[q], g.pw_col[q] - c0);
        }
#pragma unroll
        for (int u = 0; u < kU; ++u) {
            const int q = q0 + u * blockDim.x;
            if (q >= g1) continue;
            const C v = lines[at[u]];
            C h = mk(p[u].x * k[u], p[u].y * k[u]);
            h = mk(h.x + v.x * inv_n, h.y + v.y * inv_n);
            if (nlb) h = cadd(h, nv[u]);
            if (plain) {
                pob[q] = h;
            } else if (MODE == kEpiApply) {
                ob[q] = h;
            } else if (MODE == kEpiResid) {
                ob[q] = mk(ra * h.x + rb * p[u].x + rcc * prev[u].x + rly * y[u].x,
                           ra * h.y + rb * p[u].y + rcc * prev[u].y + rly * y[u].y);
            } else {
                const C c = mk(h.x * ie + nc * p[u].x, h.y * ie + nc * p[u].y);
                C o;
                if (MODE == kEpiChebFirst) o = c;
                else o = mk((R)2 * c.x - prev[u].x, (R)2 * c.y - prev[u].y);
                ob[q] = o;
                nacc += (double)o.x * (double)o.x + (double)o.y * (double)o.y;
            }
        }
    }
    if (MODE != kEpiApply && e.norm_acc) {
        double s = block_sum(nacc, red);
        if (threadIdx.x == 0) atomicAdd(e.norm_acc, s);
    }
}

template <typename C, int MODE, int kColsPerBlock>
__global__ void __launch_bounds__(256)
k_zsticks_forward(const C* __restrict__ work, const C* __restrict__ psi, int ldp, C* out, int ldo,
                  HGeom g, Epilogue e) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* tw = reinterpret_cast<C*>(smem_raw);
    C* lines = reinterpret_cast<C*>(smem_raw + align16<C>(g.nz));
    const int b = blockIdx.y;
    const int c0 = blockIdx.x * kColsPerBlock;
    const int c1 = min(c0 + kColsPerBlock, g.ncol);
    const int nl = c1 - c0;
    copy_twiddles(tw, g.twd_z, g.twf_z, g.nz);
    const C* wb = work + (size_t)b * g.nz * g.ncol;
    for (int u = threadIdx.x; u < g.nz * kColsPerBlock; u += blockDim.x) {
        const int z = u / kColsPerBlock, cl = u - z * kColsPerBlock;
        lines[cl * g.lsz + swz(z, g.nz)] = cl < nl ? wb[(size_t)z * g.ncol + c0 + cl] : czero<C>();
    }
    __syncthreads();
    fft_lines_grouped<true>(lines, nl, LinesStrided{g.lsz}, 1, g.az, tw);
    z_epilogue<C, MODE>(lines, [&](int p, int c) { return c * g.lsz + swz(p, g.nz); }, c0, c1, psi, ldp,
                        out, ldo, g, e);
}

// two-radix plans, laid out as k_zsticks_inverse2
template <typename C, int MODE, int R0, int R1>
__global__ void __launch_bounds__(ZTwo<R0, R1>::threads, ZTwo<R0, R1>::min_blocks)
k_zsticks_forward2(const C* __restrict__ work, const C* __restrict__ psi, int ldp, C* out, int ldo,
                   HGeom g, Epilogue e) {
    constexpr int N = R0 * R1;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* lines = reinterpret_cast<C*>(smem_raw);
    const int b = blockIdx.y, c0 = blockIdx.x * 32, nl = min(32, g.ncol - c0);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (warp < R1) {
        const C* wb = work + ((size_t)b * N + warp) * g.ncol + c0 + lane;
        C x[R0];
#pragma unroll
        for (int j = 0; j < R0; ++j) x[j] = lane < nl ? wb[(size_t)(j * R1) * g.ncol] : czero<C>();
        C tw[R0];
#pragma unroll
        for (int m = 1; m < R0; ++m) tw[m] = __ldg(ztable(g, C{}) + warp * m);
        span_forward<R0>(x, tw);
#pragma unroll
        for (int j = 0; j < R0; ++j) lines[(warp + j * R1) * 32 + (lane ^ (j & 7))] = x[j];
    }
    __syncthreads();
    if (warp < R0) {
        C* l = lines + warp * R1 * 32 + (lane ^ (warp & 7));
        C x[R1];
#pragma unroll
        for (int j = 0; j < R1; ++j) x[j] = l[j * 32];
        dft_r<R1, -1>(x);
#pragma unroll
        for (int j = 0; j < R1; ++j) l[j * 32] = x[j];
    }
    __syncthreads();
    z_epilogue<C, MODE>(lines, [](int p, int c) { return zslot<R1>(p, c); }, c0, c0 + nl, psi, ldp, out,
                        ldo, g, e);
}

// ------------------------------------------------------ density (pass 2')
template <int MAXPT>
__global__ void __launch_bounds__(512)
k_planes_density(const double2* __restrict__ work, const double* __restrict__ occ, int nb, int bpg,
                 double scale, double* part, HGeom g) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* twx = reinterpret_cast<double2*>(smem_raw);
    double2* twy = reinterpret_cast<double2*>(smem_raw + align16<double2>(g.nx));
    double2* plane = reinterpret_cast<double2*>(smem_raw + align16<double2>(g.nx) + align16<double2>(g.ny));
    int* xl = reinterpret_cast<int*>(plane + (size_t)g.ny * g.lsx);
    const int z = blockIdx.x;
    const int b0 = blockIdx.y * bpg, b1 = min(b0 + bpg, nb);
    copy_twiddles(twx, g.twd_x, g.twf_x, g.nx);
    copy_twiddles(twy, g.twd_y, g.twf_y, g.ny);
    for (int i = threadIdx.x; i < g.nxact; i += blockDim.x) xl[i] = g.xact[i];
    double acc[MAXPT];
#pragma unroll
    for (int k = 0; k < MAXPT; ++k) acc[k] = 0.0;
    const int npl = g.nx * g.ny;
    for (int b = b0; b < b1; ++b) {
        const double f = occ[b] * scale;
        if (f == 0.0) continue;
        for (int i = threadIdx.x; i < g.ny * g.lsx; i += blockDim.x) plane[i] = czero<double2>();
        __syncthreads();
        const double2* wp = work + ((size_t)b * g.nz + z) * g.ncol;
        for (int c = threadIdx.x; c < g.ncol; c += blockDim.x) plane[g.col_pos[c]] = wp[c];
        __syncthreads();
        fft_lines_grouped<false>(plane, g.nxact, LinesListed{xl}, g.lsx, g.ay, twy);
        fft_lines_grouped<false>(plane, g.ny, LinesStridedSwz{g.lsx, g.ny}, 1, g.ax, twx);
#pragma unroll
        for (int k = 0; k < MAXPT; ++k) {
            const int i = threadIdx.x + k * blockDim.x;
            if (i < npl) {
                const int y = i / g.nx, x = i - y * g.nx;
                const double2 v = plane[swz(y, g.ny) * g.lsx + swz(x, g.nx)];
                acc[k] += f * (v.x * v.x + v.y * v.y);
            }
        }
        __syncthreads();
    }
    double* rz = part + ((size_t)blockIdx.y * g.nz + z) * npl;
#pragma unroll
    for (int k = 0; k < MAXPT; ++k) {
        const int i = threadIdx.x + k * blockDim.x;
        if (i < npl) rz[i] = acc[k];
    }
}

// Two-radix square planes: the inverse half of k_planes_vloc2 for each band of the
// group, f |psi|^2 summed in the registers of the last x stage.  128 bands on 72^3:
// 440 us, 959 with the generic kernel; 16 bands on 40^3: 20 and 58.  Bound as
// k_planes_vloc2 is.  The parts are added by k_sum_parts (5 us).
template <int R0, int R1>
__global__ void __launch_bounds__(32 * PlaneTwo<R0, R1>::shared_warps, 1)
k_planes_density2(const double2* __restrict__ work, const double* __restrict__ occ, int nb, int bpg,
                  double scale, double* part, HGeom g) {
    using P = PlaneTwo<R0, R1>;
    constexpr int N = P::N, LS = P::LS, W = P::shared_warps, WS = W / P::Q1, kItems = (P::G + WS - 1) / WS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    double2* plane = reinterpret_cast<double2*>(smem_raw);
    int* xl = reinterpret_cast<int*>(plane + (size_t)N * LS);
    const int z = blockIdx.x, nxact = g.nxact;
    const int b0 = blockIdx.y * bpg, b1 = min(b0 + bpg, nb);
    for (int i = threadIdx.x; i < nxact; i += blockDim.x) xl[i] = P::at(g.xline[i]);
    __syncthreads();
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, r = lane & 7, t = lane >> 3;
    const int gy = (nxact + 7) >> 3, n1 = (warp % P::Q1) * 4 + t, gs = warp / P::Q1;
    const double2* wt = g.twd_x;
    double acc[kItems][R0];
#pragma unroll
    for (int k = 0; k < kItems; ++k)
#pragma unroll
        for (int j = 0; j < R0; ++j) acc[k][j] = 0.0;
    for (int b = b0; b < b1; ++b) {
        const double f = occ[b] * scale;
        if (f == 0.0) continue;
        const double2* wp = work + ((size_t)b * g.nz + z) * g.ncol;
        for (int it = warp; it < gy * P::Q0; it += W) {
            const int l = (it / P::Q0) * 8 + r, blk = (it % P::Q0) * 4 + t;
            if (l >= nxact || blk >= R0) continue;
            double2 x[R1];
            const int* ci = g.colidx_t + (size_t)blk * R1 * nxact + l;
#pragma unroll
            for (int j = 0; j < R1; ++j) {
                const int c = __ldg(ci + j * nxact);
                x[j] = c >= 0 ? wp[c] : czero<double2>();
            }
            dft_r<R1, 1>(x);
            double2* p = plane + (size_t)blk * R1 * LS + xl[l];
#pragma unroll
            for (int j = 0; j < R1; ++j) p[j * LS] = x[j];
        }
        __syncthreads();
        for (int it = gs; it < gy; it += WS) {
            const int l = it * 8 + r;
            if (l >= nxact || n1 >= R1) continue;
            double2 x[R0], tw[R0];
            double2* p = plane + (size_t)n1 * LS + xl[l];
#pragma unroll
            for (int j = 0; j < R0; ++j) x[j] = p[j * R1 * LS];
#pragma unroll
            for (int m = 1; m < R0; ++m) tw[m] = __ldg(wt + n1 * m);
            span_inverse<R0>(x, tw);
#pragma unroll
            for (int j = 0; j < R0; ++j) p[j * R1 * LS] = x[j];
        }
        __syncthreads();
        for (int it = warp; it < P::G * P::Q0; it += W) {
            const int y = (it / P::Q0) * 8 + r, blk = (it % P::Q0) * 4 + t;
            if (y >= N || blk >= R0) continue;
            double2 x[R1];
            double2* row = plane + y * LS;
#pragma unroll
            for (int j = 0; j < R1; ++j) {
                const int px = blk * R1 + j;
                const bool on = (g.xbits[px >> 5] >> (px & 31)) & 1u;
                x[j] = on ? row[P::at(px)] : czero<double2>();
            }
            dft_r<R1, 1>(x);
#pragma unroll
            for (int j = 0; j < R1; ++j) row[P::at(blk * R1 + j)] = x[j];
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const int y = (gs + k * WS) * 8 + r;
            if (y >= N || n1 >= R1) continue;
            double2 x[R0], tw[R0];
            const double2* row = plane + y * LS;
#pragma unroll
            for (int j = 0; j < R0; ++j) x[j] = row[P::at(n1 + j * R1)];
#pragma unroll
            for (int m = 1; m < R0; ++m) tw[m] = __ldg(wt + n1 * m);
            span_inverse<R0>(x, tw);
#pragma unroll
            for (int j = 0; j < R0; ++j) acc[k][j] += f * (x[j].x * x[j].x + x[j].y * x[j].y);
        }
        __syncthreads();
    }
    double* rz = part + ((size_t)blockIdx.y * g.nz + z) * N * N;
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int y = (gs + k * WS) * 8 + r;
        if (y >= N || n1 >= R1) continue;
#pragma unroll
        for (int j = 0; j < R0; ++j) rz[(size_t)y * N + n1 + j * R1] = acc[k][j];
    }
}

// rho = sum of the band groups' parts, in group order (the same bits every time:
// with atomics an SCF run that is restarted took another path at the level of
// rounding, which the mixing amplifies)
__global__ void k_sum_parts(const double* __restrict__ part, int groups, size_t n, double* __restrict__ rho) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        double s = part[i];
        for (int q = 1; q < groups; ++q) s += part[q * n + i];
        rho[i] = s;
    }
}

// ------------------------------------------------------ full-grid axis FFT
template <typename C, bool FWD>
__global__ void __launch_bounds__(256)
k_axis_fft(C* data, int nx, int ny, int nz, int axis, AxisPlan P, int lb) {
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int n = P.n;
    const int ls = n | 1;
    C* tw = reinterpret_cast<C*>(smem_raw);
    C* lines = reinterpret_cast<C*>(smem_raw + align16<C>(n));
    load_twiddles(tw, n);
    // line-batch decomposition
    size_t base;      // offset of element 0 of line 0 of the batch
    size_t lstride;   // offset between consecutive lines of the batch
    size_t estride;   // offset between consecutive elements of a line
    int nl;
    if (axis == 0) {
        const int nlines = ny * nz;
        const int l0 = blockIdx.x * lb;
        nl = min(lb, nlines - l0);
        base = (size_t)l0 * nx; lstride = nx; estride = 1;
    } else {
        const int nxb = (nx + lb - 1) / lb;
        const int x0 = (blockIdx.x % nxb) * lb;
        const int other = blockIdx.x / nxb;  // z for axis 1, y for axis 2
        nl = min(lb, nx - x0);
        lstride = 1;
        if (axis == 1) { base = (size_t)other * nx * ny + x0; estride = nx; }
        else { base = (size_t)other * nx + x0; estride = (size_t)nx * ny; }
    }
    for (int u = threadIdx.x; u < lb * n; u += blockDim.x) {
        int l, j;
        if (axis == 0) { l = u / n; j = u - l * n; }
        else { j = u / lb; l = u - j * lb; }
        lines[l * ls + swz(j, n)] = l < nl ? data[base + l * lstride + j * estride] : czero<C>();
    }
    __syncthreads();
    if (FWD) fft_lines_grouped<true>(lines, nl, LinesStrided{ls}, 1, P, tw);
    else fft_lines_grouped<false>(lines, nl, LinesStrided{ls}, 1, P, tw);
    for (int u = threadIdx.x; u < lb * n; u += blockDim.x) {
        int l, j;
        if (axis == 0) { l = u / n; j = u - l * n; }
        else { j = u / lb; l = u - j * lb; }
        if (l < nl) data[base + l * lstride + j * estride] = lines[l * ls + swz(j, n)];
    }
}

// ------------------------------------------------------ potential kernels
__device__ __forceinline__ void lda_pz(double rho, double& exc, double& vxc) {
    // Perdew-Zunger 1981 parametrisation of Ceperley-Alder, unpolarised.
    if (rho < 1e-30) { exc = 0.0; vxc = 0.0; return; }
    const double rs = cbrt(3.0 / (4.0 * 3.14159265358979323846 * rho));
    const double ex = -0.4581652932831429 / rs;
    const double vx = 4.0 / 3.0 * ex;
    double ec, vc;
    if (rs >= 1.0) {
        const double gm = -0.1423, b1 = 1.0529, b2 = 0.3334;
        const double sr = sqrt(rs);
        const double den = 1.0 + b1 * sr + b2 * rs;
        ec = gm / den;
        vc = ec * (1.0 + 7.0 / 6.0 * b1 * sr + 4.0 / 3.0 * b2 * rs) / den;
    } else {
        const double A = 0.0311, B = -0.048, Cc = 0.0020, D = -0.0116;
        const double lr = log(rs);
        ec = A * lr + B + Cc * rs * lr + D * rs;
        vc = A * lr + (B - A / 3.0) + 2.0 / 3.0 * Cc * rs * lr + (2.0 * D - Cc) / 3.0 * rs;
    }
    exc = ex + ec;
    vxc = vx + vc;
}

__global__ void k_real_to_complex(const double* r, double2* c, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        c[i] = make_double2(r[i], 0.0);
}

__global__ void k_take_real(const double2* c, double* r, size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        r[i] = c[i].x;
}

__global__ void __launch_bounds__(256)
k_hartree_gspace(double2* c, GridRecip gr, double omega, double* eh_acc) {
    __shared__ double red[32];
    const size_t n = (size_t)gr.nx * gr.ny * gr.nz;
    const double inv_n = 1.0 / (double)n;
    const double four_pi = 4.0 * 3.14159265358979323846;
    double eh = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const int ix = (int)(i % gr.nx);
        const int iy = (int)((i / gr.nx) % gr.ny);
        const int iz = (int)(i / ((size_t)gr.nx * gr.ny));
        int h = gr.idr_x[ix], k = gr.idr_y[iy], l = gr.idr_z[iz];
        if (h >= (gr.nx + 1) / 2) h -= gr.nx;
        if (k >= (gr.ny + 1) / 2) k -= gr.ny;
        if (l >= (gr.nz + 1) / 2) l -= gr.nz;
        const double gx = h * gr.b[0] + k * gr.b[3] + l * gr.b[6];
        const double gy = h * gr.b[1] + k * gr.b[4] + l * gr.b[7];
        const double gz = h * gr.b[2] + k * gr.b[5] + l * gr.b[8];
        const double g2 = gx * gx + gy * gy + gz * gz;
        if (h == 0 && k == 0 && l == 0) { c[i] = make_double2(0.0, 0.0); continue; }
        const double2 rg = make_double2(c[i].x * inv_n, c[i].y * inv_n);
        eh += 0.5 * omega * four_pi * (rg.x * rg.x + rg.y * rg.y) / g2;
        c[i] = make_double2(four_pi * rg.x / g2, four_pi * rg.y / g2);
    }
    double s = block_sum(eh, red);
    if (threadIdx.x == 0) atomicAdd(eh_acc, s);
}

__global__ void __launch_bounds__(256)
k_assemble_veff(const double* vloc, const double2* vh, const double* rho, double* veff, size_t n,
                double dv, double* exc_acc) {
    __shared__ double red[32];
    double e = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        double ex, vx;
        const double r = rho[i];
        lda_pz(r > 0.0 ? r : 0.0, ex, vx);
        veff[i] = vloc[i] + vh[i].x + vx;
        e += r * ex;
    }
    double s = block_sum(e, red);
    if (threadIdx.x == 0 && exc_acc) atomicAdd(exc_acc, s * dv);
}

__global__ void __launch_bounds__(256)
k_energy_terms(const double* rho_out, const double* veff, const double* vloc, size_t n, double dv,
               double* exc_acc, double* dc_acc) {
    __shared__ double red[32];
    double e = 0.0, d = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        double ex, vx;
        const double r = rho_out[i];
        lda_pz(r > 0.0 ? r : 0.0, ex, vx);
        e += r * ex;
        d += (veff[i] - vloc[i]) * r;
    }
    double s = block_sum(e, red);
    if (threadIdx.x == 0) atomicAdd(exc_acc, s * dv);
    s = block_sum(d, red);
    if (threadIdx.x == 0) atomicAdd(dc_acc, s * dv);
}

int grid_for(size_t n, int threads) {
    size_t b = (n + threads - 1) / threads;
    return (int)(b < 148 * 8 ? b : 148 * 8);
}

}  // namespace

// ------------------------------------------------------------------ launchers
// Two-radix plans with compile-time kernels.  FP32 keeps to the first six.
// clang-format off
#define CHFSI_ZPLANS32(X) X(9, 8) X(12, 9) X(8, 5) X(12, 12) X(8, 8) X(8, 6)
#define CHFSI_ZPLANS64(X) CHFSI_ZPLANS32(X) X(6, 5) X(8, 4) X(6, 6) X(9, 5) X(10, 5) X(9, 6) X(10, 6) \
    X(15, 5) X(10, 8) X(9, 9) X(10, 9) X(12, 8) X(10, 10) X(12, 10)
// planes up to 108 x 108 fit an SM's shared memory in 16-byte elements
#define CHFSI_PLANES32(X) X(9, 8) X(12, 9) X(8, 5) X(8, 8) X(8, 6)
#define CHFSI_PLANES64(X) CHFSI_PLANES32(X) X(6, 5) X(8, 4) X(6, 6) X(9, 5) X(10, 5) X(9, 6) X(10, 6) \
    X(15, 5) X(10, 8) X(9, 9) X(10, 9) X(12, 8) X(10, 10)
// clang-format on

// The plan's key, and whether the kernels for it are built for C
template <typename C> bool two_radix(const AxisPlan& P, int& key) {
    key = P.nst == 2 ? P.r[0] * 100 + P.r[1] : 0;
    switch (key) {
#define CHFSI_KEY(A, B) case A * 100 + B:
        CHFSI_ZPLANS32(CHFSI_KEY) return true;
    default: break;
    }
    if constexpr (sizeof(C) == 16) {
        switch (key) {
            CHFSI_ZPLANS64(CHFSI_KEY) return true;
        default: break;
        }
    }
#undef CHFSI_KEY
    return false;
}

template <typename C, int R0, int R1>
void zsticks_inverse2_launch(const C* psi, int ldp, C* work, int nb, const HGeom& g, cudaStream_t st) {
    // bands per block: as many as leave three waves of blocks, so that the last one
    // stays short; one where two buffers a block would cost resident blocks
    using Z = ZTwo<R0, R1>;
    constexpr size_t buf = (size_t)R0 * R1 * 32 * sizeof(C);
    constexpr bool two = Z::min_blocks * (2 * buf + 1024) <= 227 * 1024;
    const int cg = (g.ncol + 31) / 32;
    const int most = two ? (int)((long long)cg * nb / (3 * 148 * Z::min_blocks)) : 1;
    const int bpb = most < 1 ? 1 : most > 16 ? 16 : most;
    const size_t sm = bpb > 1 ? 2 * buf : buf;
    raise_smem_limit(k_zsticks_inverse2<C, R0, R1>, sm);
    k_zsticks_inverse2<C, R0, R1><<<dim3(cg, (nb + bpb - 1) / bpb), Z::threads, sm, st>>>(psi, ldp, work, nb, bpb, g);
}

template <typename C, int COLS>
void zsticks_inverse_launch(const C* psi, int ldp, C* work, int nb, const HGeom& g, cudaStream_t st) {
    dim3 grid((g.ncol + COLS - 1) / COLS, nb);
    size_t sm = align16<C>(g.nz) + (size_t)COLS * g.lsz * sizeof(C);
    raise_smem_limit(k_zsticks_inverse<C, COLS>, sm);
    k_zsticks_inverse<C, COLS><<<grid, 256, sm, st>>>(psi, ldp, work, g);
}

template <typename C>
void launch_zsticks_inverse(const C* psi, int ldp, C* work, int nb, const HGeom& g,
                            cudaStream_t st) {
    count_launch();
    int key;
    if (two_radix<C>(g.az, key)) {
#define CHFSI_ZI(A, B) case A * 100 + B: zsticks_inverse2_launch<C, A, B>(psi, ldp, work, nb, g, st); return;
        if constexpr (sizeof(C) == 16) {
            switch (key) { CHFSI_ZPLANS64(CHFSI_ZI) }
        } else {
            switch (key) { CHFSI_ZPLANS32(CHFSI_ZI) }
        }
#undef CHFSI_ZI
    }
    switch (g.tune_cols) {
    case 16: zsticks_inverse_launch<C, 16>(psi, ldp, work, nb, g, st); break;
    case 64: zsticks_inverse_launch<C, 64>(psi, ldp, work, nb, g, st); break;
    default: zsticks_inverse_launch<C, 32>(psi, ldp, work, nb, g, st); break;
    }
}

size_t planes_smem_bytes(const HGeom& g, size_t csize) {
    auto a16 = [](size_t b) { return (b + 15) & ~(size_t)15; };
    return a16(g.nx * csize) + a16(g.ny * csize) + (size_t)g.ny * g.lsx * csize +
           (size_t)g.nxact * sizeof(int);
}

template <typename C, int V>
void planes_vloc_variant(C* work, const double* veff, int nb, const HGeom& g, cudaStream_t st) {
    dim3 grid(g.nz, nb);
    size_t sm = planes_smem_bytes(g, sizeof(C));
    raise_smem_limit(k_planes_vloc<C, V>, sm);
    k_planes_vloc<C, V><<<grid, PlanesCfg<C, V>::threads, sm, st>>>(work, veff, g);
}

template <int V, int R0, int R1>
void planes_vloc_x2(float2* work, const double* veff, int nb, const HGeom& g, cudaStream_t st) {
    const size_t sm = 2 * align16<float2>(R0 * R1) + (size_t)R0 * R1 * ((R0 * R1) | 1) * sizeof(float4) +
                      (size_t)g.nxact * sizeof(int);
    raise_smem_limit(k_planes_vloc_p3x2<V, R0, R1>, sm);
    k_planes_vloc_p3x2<V, R0, R1><<<dim3(g.nz, (nb + 1) / 2), PlanesCfg<double2, V>::threads, sm, st>>>(
        work, veff, nb, g);
}

template <typename C, int R0, int R1>
void planes_vloc2_launch(C* work, const double* veff, int nb, const HGeom& g, cudaStream_t st) {
    constexpr int NB = sizeof(C) == 8 ? 2 : 1;
    using P = PlaneTwo<R0, R1>;
    if constexpr (NB == 2 && P::fit >= 2) {
        switch (g.tune_planes) {
        case 1: planes_vloc_x2<1, R0, R1>(work, veff, nb, g, st); return;
        case 2: planes_vloc_x2<2, R0, R1>(work, veff, nb, g, st); return;
        default: planes_vloc_x2<0, R0, R1>(work, veff, nb, g, st); return;
        }
    } else {
        dim3 grid(g.nz, (nb + NB - 1) / NB);
        raise_smem_limit(k_planes_vloc2<C, NB, R0, R1>, P::bytes);
        k_planes_vloc2<C, NB, R0, R1><<<grid, P::threads, P::bytes, st>>>(work, veff, nb, g);
    }
}

// Square planes on a plan that is compiled in
template <typename C>
bool planes_vloc_fixed(C* work, const double* veff, int nb, const HGeom& g, cudaStream_t st) {
    int key, ky;
    if (!g.fixed_planes || !g.colidx_t || g.nx != g.ny || !two_radix<C>(g.ax, key) ||
        !two_radix<C>(g.ay, ky) || key != ky)
        return false;
#define CHFSI_PV(A, B) case A * 100 + B: planes_vloc2_launch<C, A, B>(work, veff, nb, g, st); return true;
    if constexpr (sizeof(C) == 16) {
        switch (key) { CHFSI_PLANES64(CHFSI_PV) }
    } else {
        switch (key) { CHFSI_PLANES32(CHFSI_PV) }
    }
#undef CHFSI_PV
    return false;
}

template <typename C>
void launch_planes_vloc(C* work, const double* veff, int nb, const HGeom& g, cudaStream_t st) {
    count_launch();
    if (planes_vloc_fixed<C>(work, veff, nb, g, st)) return;
    switch (g.tune_planes) {
    case 1: planes_vloc_variant<C, 1>(work, veff, nb, g, st); break;
    case 2: planes_vloc_variant<C, 2>(work, veff, nb, g, st); break;
    default: planes_vloc_variant<C, 0>(work, veff, nb, g, st); break;
    }
}

template <typename C, int MODE, int R0, int R1>
void zsticks_forward2_launch(const C* work, const C* psi, int ldp, C* out, int ldo, int nb,
                             const HGeom& g, const Epilogue& e, cudaStream_t st) {
    dim3 grid((g.ncol + 31) / 32, nb);
    const size_t sm = (size_t)R0 * R1 * 32 * sizeof(C);
    raise_smem_limit(k_zsticks_forward2<C, MODE, R0, R1>, sm);
    k_zsticks_forward2<C, MODE, R0, R1><<<grid, ZTwo<R0, R1>::threads, sm, st>>>(work, psi, ldp, out, ldo,
                                                                              g, e);
}

template <typename C, int MODE, int COLS>
void zsticks_forward_launch(const C* work, const C* psi, int ldp, C* out, int ldo, int nb,
                            const HGeom& g, const Epilogue& e, cudaStream_t st) {
    dim3 grid((g.ncol + COLS - 1) / COLS, nb);
    size_t sm = align16<C>(g.nz) + (size_t)COLS * g.lsz * sizeof(C);
    raise_smem_limit(k_zsticks_forward<C, MODE, COLS>, sm);
    k_zsticks_forward<C, MODE, COLS><<<grid, 256, sm, st>>>(work, psi, ldp, out, ldo, g, e);
}

template <typename C, int MODE>
void zsticks_forward_mode(const C* work, const C* psi, int ldp, C* out, int ldo, int nb,
                          const HGeom& g, const Epilogue& e, cudaStream_t st) {
    int key;
    if (two_radix<C>(g.az, key)) {
#define CHFSI_ZF(A, B) case A * 100 + B: zsticks_forward2_launch<C, MODE, A, B>(work, psi, ldp, out, ldo, nb, g, e, st); return;
        if constexpr (sizeof(C) == 16) {
            switch (key) { CHFSI_ZPLANS64(CHFSI_ZF) }
        } else {
            switch (key) { CHFSI_ZPLANS32(CHFSI_ZF) }
        }
#undef CHFSI_ZF
    }
    switch (g.tune_cols) {
    case 16: zsticks_forward_launch<C, MODE, 16>(work, psi, ldp, out, ldo, nb, g, e, st); break;
    case 64: zsticks_forward_launch<C, MODE, 64>(work, psi, ldp, out, ldo, nb, g, e, st); break;
    default: zsticks_forward_launch<C, MODE, 32>(work, psi, ldp, out, ldo, nb, g, e, st); break;
    }
}

template <typename C>
void launch_zsticks_forward(const C* work, const C* psi, int ldp, C* out, int ldo, int nb,
                            const HGeom& g, const Epilogue& e, cudaStream_t st) {
    count_launch();
    switch (e.mode) {
    case kEpiApply: zsticks_forward_mode<C, kEpiApply>(work, psi, ldp, out, ldo, nb, g, e, st); break;
    case kEpiChebFirst: zsticks_forward_mode<C, kEpiChebFirst>(work, psi, ldp, out, ldo, nb, g, e, st); break;
    case kEpiResid: zsticks_forward_mode<C, kEpiResid>(work, psi, ldp, out, ldo, nb, g, e, st); break;
    default: zsticks_forward_mode<C, kEpiCheb>(work, psi, ldp, out, ldo, nb, g, e, st); break;
    }
}

int density_groups(int nz, int nb) {
    const int groups = std::max(1, std::min(nb, (2 * 148 + nz - 1) / nz));
    const int bpg = (nb + groups - 1) / groups;
    return (nb + bpg - 1) / bpg;
}

template <int R0, int R1>
void planes_density2_launch(const double2* work, const double* occ, int nb, int bpg, int groups,
                            double scale, double* part, const HGeom& g, cudaStream_t st) {
    using P = PlaneTwo<R0, R1>;
    raise_smem_limit(k_planes_density2<R0, R1>, P::bytes);
    k_planes_density2<R0, R1><<<dim3(g.nz, groups), 32 * P::shared_warps, P::bytes, st>>>(work, occ, nb, bpg, scale,
                                                                                 part, g);
}

void launch_planes_density(const double2* work, const double* occ, int nb, double scale, double* rho,
                           double* part, const HGeom& g, cudaStream_t st) {
    count_launch(2);
    const int groups = density_groups(g.nz, nb), bpg = (nb + groups - 1) / groups;
    int key = 0, ky;
    const bool fixed = g.colidx_t && g.nx == g.ny && two_radix<double2>(g.ax, key) &&
                       two_radix<double2>(g.ay, ky) && key == ky;
    switch (fixed ? key : 0) {
#define CHFSI_PD(A, B) \
    case A * 100 + B: planes_density2_launch<A, B>(work, occ, nb, bpg, groups, scale, part, g, st); break;
        CHFSI_PLANES64(CHFSI_PD)
#undef CHFSI_PD
    default: {
        const size_t sm = planes_smem_bytes(g, sizeof(double2));
        raise_smem_limit(k_planes_density<24>, sm);
        k_planes_density<24><<<dim3(g.nz, groups), 512, sm, st>>>(work, occ, nb, bpg, scale, part, g);
    }
    }
    const size_t n = (size_t)g.nx * g.ny * g.nz;
    k_sum_parts<<<grid_for(n, 256), 256, 0, st>>>(part, groups, n, rho);
}

template <typename C>
void launch_axis_fft(C* data, int nx, int ny, int nz, int axis, bool forward, const AxisPlan& P,
                     cudaStream_t st) {
    count_launch();
    const int lb = 16;
    int blocks;
    if (axis == 0) blocks = (ny * nz + lb - 1) / lb;
    else blocks = ((nx + lb - 1) / lb) * (axis == 1 ? nz : ny);
    size_t sm = align16<C>(P.n) + (size_t)lb * (P.n | 1) * sizeof(C);
    raise_smem_limit(k_axis_fft<C, true>, sm);
    raise_smem_limit(k_axis_fft<C, false>, sm);
    if (forward) k_axis_fft<C, true><<<blocks, 256, sm, st>>>(data, nx, ny, nz, axis, P, lb);
    else k_axis_fft<C, false><<<blocks, 256, sm, st>>>(data, nx, ny, nz, axis, P, lb);
}

void launch_real_to_complex(const double* r, double2* c, size_t n, cudaStream_t st) {
    count_launch();
    k_real_to_complex<<<grid_for(n, 256), 256, 0, st>>>(r, c, n);
}
void launch_take_real(const double2* c, double* r, size_t n, cudaStream_t st) {
    count_launch();
    k_take_real<<<grid_for(n, 256), 256, 0, st>>>(c, r, n);
}
void launch_hartree_gspace(double2* c, const GridRecip& gr, double omega, double* eh_acc,
                           cudaStream_t st) {
    count_launch();
    size_t n = (size_t)gr.nx * gr.ny * gr.nz;
    k_hartree_gspace<<<grid_for(n, 256), 256, 0, st>>>(c, gr, omega, eh_acc);
}
void launch_assemble_veff(const double* vloc, const double2* vh, const double* rho, double* veff,
                          size_t n, double dv, double* exc_acc, cudaStream_t st) {
    count_launch();
    k_assemble_veff<<<grid_for(n, 256), 256, 0, st>>>(vloc, vh, rho, veff, n, dv, exc_acc);
}
void launch_energy_terms(const double* rho_out, const double* veff, const double* vloc, size_t n,
                         double dv, double* exc_acc, double* dc_acc, cudaStream_t st) {
    count_launch();
    k_energy_terms<<<grid_for(n, 256), 256, 0, st>>>(rho_out, veff, vloc, n, dv, exc_acc, dc_acc);
}

#define CHFSI_INST(C)                                                                        \
    template void launch_zsticks_inverse<C>(const C*, int, C*, int, const HGeom&, cudaStream_t); \
    template void launch_planes_vloc<C>(C*, const double*, int, const HGeom&, cudaStream_t);     \
    template void launch_zsticks_forward<C>(const C*, const C*, int, C*, int, int, const HGeom&, \
                                            const Epilogue&, cudaStream_t);                      \
    template void launch_axis_fft<C>(C*, int, int, int, int, bool, const AxisPlan&, cudaStream_t);
CHFSI_INST(double2)
CHFSI_INST(float2)
#undef CHFSI_INST

}  // namespace chfsi
