// Dense FP64 eigenproblem of the Rayleigh-Ritz step: Cholesky factor and its
// inverse, and the Hermitian eigensolver (role of cuSOLVER ZHEGVD itype 1,
// src/device/solver.rs:47-95).
//
//   chol_inv   S = L L^H -> L^-1, blocked (32 columns), one cooperative launch
//   heev       A = Q T Q^H (Householder, T real tridiagonal), T = Z W Z^T by
//              divide and conquer, U = Q Z
//
// The parallel Jacobi these replace takes about ten sweeps of n - 1 rotation
// steps, each ending in a barrier over the grid; the reduction to tridiagonal
// form takes one pass of n steps with one barrier each, and what follows has
// no chain longer than the tree's depth.  Measured (us, here / parallel Jacobi
// with its serial Cholesky): 160 rows, nearly diagonal: eigenproblem 715 / 2,670,
// factor and inverse 163 / 826; 576 rows, dense: 3,450 / 132,600 and 620 / 25,900;
// 20 rows: 160 / 206 and 18 / 35.  Of the 3,450: reduction 2,440, back
// transformation 380, merges 505, leaves 80.
//
// Divide and conquer follows Cuppen (Numer. Math. 36 (1981) 177) with the
// eigenvectors of the rank-one updates from recomputed z (Gu, Eisenstat, SIAM
// J. Matrix Anal. Appl. 16 (1995) 172), which keeps them orthogonal to working
// precision, and the two-pole rational iteration for the secular equation (Li,
// LAPACK Working Note 89 (1994)) inside a bracket.
#include "dense.hpp"
#include "launch_count.hpp"
#include "smem_limit.hpp"

#include <algorithm>
#include <cooperative_groups.h>
#include <utility>

namespace cg = cooperative_groups;

namespace chfsi {

namespace {

constexpr double kEps = 1.1102230246251565e-16;  // 2^-53
// what the sweep count says of a solve that did not converge (above any limit
// a caller has)
constexpr int kNoConvergence = 1 << 20;

__device__ __forceinline__ double2 c_mul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// acc += a b,  acc += conj(a) b,  acc -= a conj(b)
__device__ __forceinline__ void c_fma(double2& acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, fma(-a.y, b.y, acc.x));
    acc.y = fma(a.x, b.y, fma(a.y, b.x, acc.y));
}
__device__ __forceinline__ void c_fma_conj(double2& acc, double2 a, double2 b) {
    acc.x = fma(a.x, b.x, fma(a.y, b.y, acc.x));
    acc.y = fma(a.x, b.y, fma(-a.y, b.x, acc.y));
}
__device__ __forceinline__ void c_fms_rconj(double2& acc, double2 a, double2 b) {
    acc.x = fma(-a.x, b.x, fma(-a.y, b.y, acc.x));
    acc.y = fma(-a.y, b.x, fma(a.x, b.y, acc.y));
}
__device__ __forceinline__ double warp_add(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
__device__ __forceinline__ double2 warp_add(double2 v) {
    return make_double2(warp_add(v.x), warp_add(v.y));
}

// ------------------------------------------------- Cholesky and inverse
constexpr int kCB = 32, kCL = kCB + 1;
constexpr int kCTile = kCB * kCL;  // one tile in shared memory

// tile (32 x 32, zero outside n) of a row-major matrix -> shared memory
__device__ __forceinline__ void tile_load(double2* t, const double2* A, int n, int r0, int c0) {
    for (int u = threadIdx.x; u < kCB * kCB; u += blockDim.x) {
        const int r = u >> 5, c = u & 31;
        t[r * kCL + c] = r0 + r < n && c0 + c < n ? __ldcg(A + (size_t)(r0 + r) * n + c0 + c)
                                                  : make_double2(0.0, 0.0);
    }
}
// products of two tiles, 2 x 2 outputs per thread: a b (CONJT false) or a b^H
template <bool CONJT>
__device__ __forceinline__ void tile_mul(const double2* a, const double2* b, double2 (&o)[2][2]) {
    const int r = (threadIdx.x >> 4) * 2, c = (threadIdx.x & 15) * 2;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j) o[i][j] = make_double2(0.0, 0.0);
#pragma unroll 8
    for (int k = 0; k < kCB; ++k) {
        const double2 x0 = a[r * kCL + k], x1 = a[(r + 1) * kCL + k];
        double2 y0, y1;
        if (CONJT) {
            y0 = b[c * kCL + k];
            y1 = b[(c + 1) * kCL + k];
            y0.y = -y0.y;
            y1.y = -y1.y;
        } else {
            y0 = b[k * kCL + c];
            y1 = b[k * kCL + c + 1];
        }
        c_fma(o[0][0], x0, y0);
        c_fma(o[0][1], x0, y1);
        c_fma(o[1][0], x1, y0);
        c_fma(o[1][1], x1, y1);
    }
}

// A: Hermitian, its lower triangle is overwritten by the factor (diagonal
// blocks aside); X <- L^-1 (lower triangular, upper part zero).  info: 0 or the
// failing column + 1.  A pivot fails when it is not above n 2^-52 times its
// column's original diagonal entry (singular to working precision).
// Step J: every block factors the 32 x 32 diagonal tile itself, together with
// the tile's inverse (unit-lower form, one reciprocal and one barrier per
// column); panel tiles A_IJ L_JJ^-H and the rows X_J = L_JJ^-1 X_J are shared
// out; after a grid barrier the trailing tiles A_IC -= L_IJ L_CJ^H and
// X_IC -= L_IJ X_J.  Bound by the diagonal tile's chain of 32 reciprocals and the
// two grid barriers of a step, about 32 us together.
__global__ void __launch_bounds__(256)
k_chol_inv(double2* A, double2* X, int n, int* info) {
    cg::grid_group grid = cg::this_grid();
    extern __shared__ double2 csm[];
    double2* D = csm;                  // diagonal tile
    double2* V = csm + kCTile;         // its inverse
    double2* ta = csm + 2 * kCTile;
    double2* tb = csm + 3 * kCTile;
    double* dia = reinterpret_cast<double*>(csm + 4 * kCTile);  // original diagonal
    __shared__ double2 colk[2][kCB], rowk[2][kCB];
    __shared__ double pivot[2];
    const int nbk = (n + kCB - 1) / kCB, tid = threadIdx.x;
    const double rel = (double)n * 2.220446049250313e-16;
    for (int i = tid; i < n; i += blockDim.x) dia[i] = A[(size_t)i * n + i].x;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + tid; t < (size_t)n * n;
         t += (size_t)gridDim.x * blockDim.x)
        X[t] = make_double2(0.0, 0.0);
    grid.sync();
    const int r2 = (tid >> 4) * 2, c2 = (tid & 15) * 2;
    for (int J = 0; J < nbk; ++J) {
        const int j0 = J * kCB, nj = min(kCB, n - j0);
        tile_load(D, A, n, j0, j0);
        __syncthreads();
        // thread: row fi, columns fm + 8 q of the tile (m > k: factor, m <= k:
        // inverse) in registers; column k of the factor, row k of the inverse and
        // the pivot's reciprocal pass through shared memory, two slots in turn
        const int fi = tid >> 3, fm = tid & 7;
        double2 dv[4], iv[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            dv[q] = D[fi * kCL + fm + 8 * q];
            iv[q] = make_double2(fi == fm + 8 * q ? 1.0 : 0.0, 0.0);
        }
        if (fm == 0) {
            colk[0][fi] = dv[0];
            if (fi == 0) pivot[0] = dv[0].x;
        }
        if (fi == 0)
#pragma unroll
            for (int q = 0; q < 4; ++q) rowk[0][fm + 8 * q] = iv[q];
        __syncthreads();
        int fail = 0;
        double mine = 1.0;  // this row's pivot
        for (int k = 0; k < nj; ++k) {
            const int sl = k & 1;
            const double d = pivot[sl];
            if (!(d > 0.0) || (j0 + k > 0 && !(d > rel * dia[j0 + k]))) { fail = j0 + k + 1; break; }
            if (fi == k) mine = d;
            const double inv = 1.0 / d;
            if (fi > k) {
                double2 l = colk[sl][fi];
                l.x *= inv;
                l.y *= inv;
                const double2 nl = make_double2(-l.x, -l.y);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const int m = fm + 8 * q;
                    if (m > k) {
                        if (m <= fi) c_fms_rconj(dv[q], l, colk[sl][m]);
                    } else {
                        c_fma(iv[q], nl, rowk[sl][m]);
                    }
                    if (m == k + 1) {
                        colk[sl ^ 1][fi] = dv[q];
                        if (fi == k + 1) pivot[sl ^ 1] = dv[q].x;
                    }
                    if (fi == k + 1) rowk[sl ^ 1][m] = iv[q];
                }
            }
            __syncthreads();
        }
        if (fail) {  // the same in every block
            if (blockIdx.x == 0 && tid == 0) *info = fail;
            return;
        }
        {
            const double s = fi < nj ? rsqrt(mine) : 1.0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const int m = fm + 8 * q;
                V[fi * kCL + m] = m <= fi ? make_double2(iv[q].x * s, iv[q].y * s) : make_double2(0.0, 0.0);
            }
        }
        __syncthreads();
        // panel tiles below, row block J of X
        for (int t = blockIdx.x; t < nbk; t += gridDim.x) {
            double2 o[2][2];
            if (t > J) {
                tile_load(ta, A, n, t * kCB, j0);
                __syncthreads();
                tile_mul<true>(ta, V, o);
            } else if (t < J) {
                tile_load(ta, X, n, j0, t * kCB);
                __syncthreads();
                tile_mul<false>(V, ta, o);
            } else {
                __syncthreads();
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int j = 0; j < 2; ++j) o[i][j] = V[(r2 + i) * kCL + c2 + j];
            }
            double2* dst = t > J ? A : X;
            const int r0 = t > J ? t * kCB : j0, c0 = t > J ? j0 : t * kCB;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j)
                    if (r0 + r2 + i < n && c0 + c2 + j < n)
                        dst[(size_t)(r0 + r2 + i) * n + c0 + c2 + j] = o[i][j];
            __syncthreads();
        }
        if (J + 1 == nbk) break;
        grid.sync();
        // trailing tiles: column blocks 0 .. J of X, J + 1 .. I of A
        const int m = nbk - J - 1, items = m * (J + 1) + m * (m + 1) / 2;
        for (int t = blockIdx.x; t < items; t += gridDim.x) {
            int u = t, I = J + 1;
            while (u >= I + 1) { u -= I + 1; ++I; }
            const int C = u;
            double2 o[2][2];
            tile_load(ta, A, n, I * kCB, j0);
            if (C > J) tile_load(tb, A, n, C * kCB, j0);
            else tile_load(tb, X, n, j0, C * kCB);
            __syncthreads();
            if (C > J) tile_mul<true>(ta, tb, o);
            else tile_mul<false>(ta, tb, o);
            double2* dst = C > J ? A : X;
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 2; ++j) {
                    const int r = I * kCB + r2 + i, c = C * kCB + c2 + j;
                    if (r < n && c < n) {
                        double2* e = dst + (size_t)r * n + c;
                        const double2 v = __ldcg(e);
                        *e = make_double2(v.x - o[i][j].x, v.y - o[i][j].y);
                    }
                }
            __syncthreads();
        }
        grid.sync();
    }
    if (blockIdx.x == 0 && tid == 0) *info = 0;
}

// ------------------------------------------------- tridiagonal reduction
// A = Q T Q^H, Q = H_0 H_1 ... H_{n-2}, H_j = I - sigma_j u_j u_j^H with u_j = x -
// beta e_{j+1} for the column x below diagonal j (u_j zero up to j, not
// normalised), sigma_j = -1 / (beta conj(x_{j+1} - beta)).  The matrix lies in
// shared memory, rows dealt out over the blocks.  Step j: each block applies the
// rank-two update of step j - 1 to its rows and multiplies them, in the same
// sweep, by x without its first entry (the norm is not needed for that), and
// publishes for each of its rows the entry of that product q and of column j + 1,
// a.  Behind the barrier's arrival every block reduces |x|^2 and forms beta and
// sigma; past it, with u_{j+1} = x_{j+1} - beta,
//   A u = q + a u_{j+1},   w = sigma A u - (|sigma|^2 / 2) (u^H A u) u,
//   a <- a - u w_{j+1}^* - w u_{j+1}^*
// and the new a is the next x.  What bounds it is that chain, not the 16 n^3 / 3
// flops: 2.5 us a step at 160 rows and 4.2 at 576, of which the barrier takes 0.2
// and 1.2 and the rest is two block-wide sums read back from shared memory and the
// sweep over the rows.  CL: one thread-block cluster (n <= 256): a cheaper barrier
// (390 clocks, the grid's takes 2,300), q and a pushed into every block's shared
// memory instead of the round trip through L2.
// The rows are scaled by a power of two to a largest entry next to 1 (its top word
// in *top, zero before the launch; the eigenvalues are scaled back at the end), and
// columns with |x|^2 < 1e-140 then count as zero: sigma is about 1 / |x|^2, and its
// square and beta |u|^2 leave the range of the exponents for |x| below 1e-77 and
// above 1e77 otherwise.
__device__ __forceinline__ unsigned tri_top(double2 v) {
    const unsigned x = ((unsigned)__double2hiint(v.x) & 0x7fffffffu) | (__double2loint(v.x) != 0);
    const unsigned y = ((unsigned)__double2hiint(v.y) & 0x7fffffffu) | (__double2loint(v.y) != 0);
    return max(x, y);
}
__device__ __forceinline__ double tri_scale(unsigned top) {
    const int f = (int)(top >> 20);
    if (top == 0 || f == 2047) return 1.0;
    return __longlong_as_double((long long)max(1, 2046 - f) << 52);
}
constexpr int kTriPer = 5;  // vector entries per thread (n <= 5 x 256)
constexpr int kTriCluster = 256;  // largest n of the cluster form
template <bool CL> struct TriCfg {
    static constexpr int threads = CL ? 512 : 256;
    static constexpr int per = CL ? 1 : kTriPer;
    static constexpr int vectors = CL ? 7 : 3;  // shared memory beside the rows
};

template <bool CL>
__global__ void __launch_bounds__(TriCfg<CL>::threads)
k_tridiag(const double2* __restrict__ A, int n, int rows, double2* Vh, double2* tau, double* d,
          double* e, double2* P, unsigned* top) {
    constexpr int T = TriCfg<CL>::threads, W = T / 32, KP = TriCfg<CL>::per;
    extern __shared__ double2 tsm[];
    double2* M = tsm;                      // own rows
    double2* xc = M + (size_t)rows * n;    // x of this step, zero up to j + 1
    double2* up = xc + n;                  // u, w of the step before
    double2* wp = up + n;
    double2* pl = wp + n;                  // CL: [2][n][2], q and a
    __shared__ double red[2][W];
    __shared__ double2 psum[64], pcol[16];
    const int G = gridDim.x, rank = blockIdx.x, tid = threadIdx.x;
    const int lane = tid & 31, warp = tid >> 5;
    const int nw = min(W, (n + 31) / 32);  // warps that hold vector entries
    // block-wide sums, in every thread; two buffers, one block barrier per call
    int rb = 0;
    auto sum = [&](double v) {
        v = warp_add(v);
        if (lane == 0) red[rb][warp] = v;
        __syncthreads();
        v = red[rb][0];
        for (int w = 1; w < nw; ++w) v += red[rb][w];
        rb ^= 1;
        return v;
    };
    unsigned big = 0;
    for (int l = 0; l < rows; ++l) {
        const int i = rank + l * G;
        if (i < n)
            for (int k = tid; k < n; k += T) {
                const double2 v = A[(size_t)i * n + k];
                M[(size_t)l * n + k] = v;
                big = max(big, tri_top(v));
            }
    }
    big = __reduce_max_sync(0xffffffffu, big);
    if (lane == 0) atomicMax(top, big);
    __threadfence();
    // also: a block's shared memory may be stored to only once the block runs
    if constexpr (CL) cg::this_cluster().sync();
    else cg::this_grid().sync();
    const double scale = tri_scale(__ldcg(top));
    for (int l = 0; l < rows; ++l)
        if (rank + l * G < n)
            for (int k = tid; k < n; k += T) {
                M[(size_t)l * n + k].x *= scale;
                M[(size_t)l * n + k].y *= scale;
            }
    const int wpr = rows <= W ? W / rows : 1, rpp = W / wpr;  // warps per row, rows at a time
    double2 x[KP];
#pragma unroll
    for (int q = 0; q < KP; ++q) {
        const int k = tid + q * T;
        x[q] = make_double2(0.0, 0.0);
        if (k > 0 && k < n) x[q] = make_double2(A[k].x * scale, -A[k].y * scale);
        if (k < n) xc[k] = k > 1 ? x[q] : make_double2(0.0, 0.0);
    }
    double2 alpha = make_double2(A[1].x * scale, -A[1].y * scale);  // x_{j+1}
    double dj = A[0].x * scale;
    __syncthreads();
    for (int j = 0; j < n - 1; ++j) {
        double2* Pj = (CL ? pl : P) + (size_t)(j & 1) * 2 * n;
        for (int l0 = 0; l0 < rows; l0 += rpp) {
            const int l = l0 + warp / wpr, seg = warp % wpr, i = rank + l * G;
            const bool live = l < rows && i < n && i > j && warp < rpp * wpr;
            double2 acc = make_double2(0.0, 0.0), col = acc;
            if (live) {
                double2* row = M + (size_t)l * n;
                double2 ui = acc, wi = acc;
                if (j > 0) {
                    ui = up[i];
                    wi = wp[i];
                }
                // four entries at a time, all loads before the stores
                const int step = 32 * wpr, k0 = j + 1 + seg * 32 + lane;
                for (int kb = k0; kb - lane < n; kb += 4 * step) {
                    double2 a[4], wk[4], uk[4], xk[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int k = kb + q * step;
                        a[q] = wk[q] = uk[q] = xk[q] = make_double2(0.0, 0.0);
                        if (k < n) {
                            a[q] = row[k];
                            xk[q] = xc[k];
                            if (j > 0) {
                                wk[q] = wp[k];
                                uk[q] = up[k];
                            }
                        }
                    }
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        c_fms_rconj(a[q], ui, wk[q]);
                        c_fms_rconj(a[q], wi, uk[q]);
                        c_fma(acc, a[q], xk[q]);
                    }
                    if (kb == k0) col = a[0];
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        const int k = kb + q * step;
                        if (k < n) row[k] = a[q];
                    }
                }
            }
            acc = warp_add(acc);
            col.x = __shfl_sync(0xffffffffu, col.x, 0);  // segment 0, lane 0: column j + 1
            col.y = __shfl_sync(0xffffffffu, col.y, 0);
            if (wpr > 1) {
                if (lane == 0 && l < rows && warp < rpp * wpr) {
                    psum[l * wpr + seg] = acc;
                    if (seg == 0) pcol[l] = col;
                }
            } else if (live) {
                if constexpr (CL) {
                    if (lane < 2 * G)
                        *cg::this_cluster().map_shared_rank(Pj + 2 * i + (lane & 1), lane >> 1) =
                            lane & 1 ? col : acc;
                } else if (lane < 2) {
                    Pj[2 * i + lane] = lane & 1 ? col : acc;
                }
            }
        }
        if (wpr > 1) {
            __syncthreads();
            const int half = tid & 1, l = CL ? (tid >> 1) / G : tid >> 1, i = rank + l * G;
            if (l < rows && i < n && i > j) {
                double2 s = half ? pcol[l] : make_double2(0.0, 0.0);
                if (!half)
                    for (int g = 0; g < wpr; ++g) {
                        s.x += psum[l * wpr + g].x;
                        s.y += psum[l * wpr + g].y;
                    }
                if constexpr (CL) *cg::this_cluster().map_shared_rank(Pj + 2 * i + half, (tid >> 1) % G) = s;
                else Pj[2 * i + half] = s;
            }
        }
        double beta = alpha.x;
        double2 u0 = make_double2(0.0, 0.0), sg = make_double2(0.0, 0.0);
        auto reflector = [&]() {
            double v = 0.0;
#pragma unroll
            for (int q = 0; q < KP; ++q) {
                const int k = tid + q * T;
                if (k > j + 1 && k < n) v += x[q].x * x[q].x + x[q].y * x[q].y;
            }
            v = sum(v);
            const double s2 = alpha.x * alpha.x + alpha.y * alpha.y + v;
            if ((v != 0.0 || alpha.y != 0.0) && !(s2 < 1e-140)) {
                beta = -copysign(s2 * rsqrt(s2), alpha.x);
                u0 = make_double2(alpha.x - beta, alpha.y);
                const double q = -1.0 / (beta * (u0.x * u0.x + u0.y * u0.y));
                sg = make_double2(u0.x * q, u0.y * q);
            }
            if (rank == j % G)
#pragma unroll
                for (int q = 0; q < KP; ++q) {
                    const int k = tid + q * T;
                    if (k < n)
                        Vh[(size_t)j * n + k] = k <= j ? make_double2(0.0, 0.0) : k == j + 1 ? u0 : x[q];
                }
            if (rank == 0 && tid == 0) {
                tau[j] = sg;
                d[j] = dj;
                e[j] = beta;
            }
        };
        if constexpr (CL) {
            cg::cluster_group cl = cg::this_cluster();
            auto token = cl.barrier_arrive();
            reflector();
            cl.barrier_wait(std::move(token));
        } else {
            cg::grid_group gr = cg::this_grid();
            auto token = gr.barrier_arrive();
            reflector();
            gr.barrier_wait(std::move(token));
        }
        auto get = [](const double2* p) {
            if constexpr (CL) return *p;
            else return __ldcg(p);
        };
        const bool more = j + 2 < n;
        // A u of this thread's entries, column j + 1, u^H A u
        double2 au[KP], ak[KP];
        double v = 0.0;
#pragma unroll
        for (int q = 0; q < KP; ++q) {
            const int k = tid + q * T;
            au[q] = ak[q] = make_double2(0.0, 0.0);
            if (k > j + 1 && k < n) {
                au[q] = get(Pj + 2 * k);
                ak[q] = get(Pj + 2 * k + 1);
            }
        }
        const double2 q1 = get(Pj + 2 * j + 2), a1 = get(Pj + 2 * j + 3);
        double2 q2 = more ? get(Pj + 2 * j + 4) : q1;
        const double2 a2 = more ? get(Pj + 2 * j + 5) : a1;
        const double2 x2 = more ? xc[j + 2] : u0;
#pragma unroll
        for (int q = 0; q < KP; ++q) {
            const int k = tid + q * T;
            if (k > j + 1 && k < n) {
                c_fma(au[q], ak[q], u0);
                v = fma(x[q].x, au[q].x, fma(x[q].y, au[q].y, v));
            }
        }
        const double2 au1 = make_double2(fma(a1.x, u0.x, q1.x), fma(a1.x, u0.y, q1.y));
        v = sum(v) + u0.x * au1.x + u0.y * au1.y;
        const double c = 0.5 * (sg.x * sg.x + sg.y * sg.y) * v;
        auto w_of = [&](double2 z, double2 u) {
            double2 w = c_mul(sg, z);
            w.x -= c * u.x;
            w.y -= c * u.y;
            return w;
        };
        const double2 w1 = w_of(au1, u0);
        dj = a1.x - 2.0 * (u0.x * w1.x + u0.y * w1.y);
        auto next = [&](double2 a, double2 w, double2 u) {  // entry of the next x
            c_fms_rconj(a, u, w1);
            c_fms_rconj(a, w, u0);
            return a;
        };
        if (more) {
            c_fma(q2, a2, u0);
            alpha = next(a2, w_of(q2, x2), x2);
        }
#pragma unroll
        for (int q = 0; q < KP; ++q) {
            const int k = tid + q * T;
            if (k >= n) continue;
            double2 u = make_double2(0.0, 0.0), w = u;
            if (k > j + 1) {
                u = x[q];
                w = w_of(au[q], u);
                x[q] = next(ak[q], w, u);
            } else if (k == j + 1) {
                u = u0;
                w = w1;
            }
            up[k] = u;
            wp[k] = w;
        }
        // every thread has read x_{j+2} out of xc before the barrier in sum()
#pragma unroll
        for (int q = 0; q < KP; ++q) {
            const int k = tid + q * T;
            if (k < n) xc[k] = k > j + 2 ? x[q] : make_double2(0.0, 0.0);
        }
        __syncthreads();
    }
    if (rank == 0 && tid == 0) {
        d[n - 1] = dj;
        e[n - 1] = 0.0;
    }
    if constexpr (CL) cg::this_cluster().sync();
}

// The reflectors in groups of kGrp, H_j H_{j+1} .. H_{j+kGrp-1} = I - V T V^H
// with T upper triangular (compact WY; Schreiber, Van Loan, SIAM J. Sci. Stat.
// Comput. 10 (1989) 53): one warp per group forms V^H V and T.
constexpr int kGrp = 4;
__global__ void __launch_bounds__(128)
k_wy(const double2* __restrict__ Vh, const double2* __restrict__ tau, int n, double2* __restrict__ Tg) {
    const int g = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31, j0 = g * kGrp;
    if (j0 > n - 2) return;
    double2 G[kGrp][kGrp];
#pragma unroll
    for (int a = 0; a < kGrp; ++a)
#pragma unroll
        for (int b = 0; b < kGrp; ++b) G[a][b] = make_double2(0.0, 0.0);
    for (int k = j0 + 1 + lane; k < n; k += 32) {
        double2 v[kGrp];
#pragma unroll
        for (int a = 0; a < kGrp; ++a)
            v[a] = j0 + a <= n - 2 ? Vh[(size_t)(j0 + a) * n + k] : make_double2(0.0, 0.0);
#pragma unroll
        for (int a = 0; a < kGrp; ++a)
#pragma unroll
            for (int b = a + 1; b < kGrp; ++b) c_fma_conj(G[a][b], v[a], v[b]);
    }
    double2 T[kGrp][kGrp];
#pragma unroll
    for (int b = 0; b < kGrp; ++b) {
        const double2 tb = j0 + b <= n - 2 ? tau[j0 + b] : make_double2(0.0, 0.0);
#pragma unroll
        for (int a = 0; a < kGrp; ++a) {
            T[a][b] = make_double2(0.0, 0.0);
            if (a < b) G[a][b] = warp_add(G[a][b]);
        }
        T[b][b] = tb;
        // column b: -tau_b T (V^H v_b)
#pragma unroll
        for (int a = 0; a < b; ++a) {
            double2 s = make_double2(0.0, 0.0);
#pragma unroll
            for (int c = a; c < b; ++c) c_fma(s, T[a][c], G[c][b]);
            s = c_mul(s, tb);
            T[a][b] = make_double2(-s.x, -s.y);
        }
    }
    if (lane == 0)
#pragma unroll
        for (int a = 0; a < kGrp; ++a)
#pragma unroll
            for (int b = 0; b < kGrp; ++b) Tg[(size_t)g * kGrp * kGrp + a * kGrp + b] = T[a][b];
}

// U = Q Z: one warp per column of Z (a row of Zt), the column in registers (NQ
// entries per lane, n <= 32 NQ), groups of reflectors from the last to the
// first, each brought into shared memory while the one before it is applied.
// The four dot products of a group are reduced together; a reflector at a time
// took 4.3 us each at n = 576, this kernel about 0.5.  out[i][c], row-major.
constexpr int kBackWarps = 4;
template <int NQ>
__global__ void __launch_bounds__(32 * kBackWarps)
k_back(const double2* __restrict__ Vh, const double2* __restrict__ Tg, const double* __restrict__ Zt,
       int n, double2* __restrict__ out) {
    extern __shared__ double2 bsm[];  // [2][kGrp][32 NQ]
    constexpr int L = 32 * NQ;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int c = blockIdx.x * kBackWarps + warp;
    double2 z[NQ];
#pragma unroll
    for (int q = 0; q < NQ; ++q) {
        const int k = lane + 32 * q;
        z[q] = make_double2(c < n && k < n ? Zt[(size_t)c * n + k] : 0.0, 0.0);
    }
    const int groups = (n - 1 + kGrp - 1) / kGrp;
    auto load = [&](int g, int slot) {
        double2* dst = bsm + (size_t)slot * kGrp * L;
        for (int a = 0; a < kGrp; ++a) {
            const int j = g * kGrp + a;
            for (int k = tid; k < L; k += 32 * kBackWarps) {
                const bool in = j <= n - 2 && k < n;
                const unsigned sa = (unsigned)__cvta_generic_to_shared(dst + a * L + k);
                const double2* src = Vh + (in ? (size_t)j * n + k : 0);
                asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(sa), "l"(src),
                             "r"(in ? 16 : 0) : "memory");
            }
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    load(groups - 1, 0);
    for (int g = groups - 1, slot = 0; g >= 0; --g, slot ^= 1) {
        if (g > 0) {
            load(g - 1, slot ^ 1);
            asm volatile("cp.async.wait_group 1;" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;" ::: "memory");
        }
        __syncthreads();
        const double2* v = bsm + (size_t)slot * kGrp * L + lane;
        double2 T[kGrp * kGrp];
#pragma unroll
        for (int a = 0; a < kGrp * kGrp; ++a) T[a] = Tg[(size_t)g * kGrp * kGrp + a];
        double2 s[kGrp];
#pragma unroll
        for (int a = 0; a < kGrp; ++a) s[a] = make_double2(0.0, 0.0);
        const int q0 = (g * kGrp + 1) >> 5;  // entries before it are zero in the group
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (q >= q0)
#pragma unroll
                for (int a = 0; a < kGrp; ++a) c_fma_conj(s[a], v[a * L + 32 * q], z[q]);
#pragma unroll
        for (int a = 0; a < kGrp; ++a) s[a] = warp_add(s[a]);
        double2 t[kGrp];
#pragma unroll
        for (int a = 0; a < kGrp; ++a) {
            t[a] = make_double2(0.0, 0.0);
#pragma unroll
            for (int b = a; b < kGrp; ++b) c_fma(t[a], T[a * kGrp + b], s[b]);
            t[a].x = -t[a].x;
            t[a].y = -t[a].y;
        }
#pragma unroll
        for (int q = 0; q < NQ; ++q)
            if (q >= q0)
#pragma unroll
                for (int a = 0; a < kGrp; ++a) c_fma(z[q], t[a], v[a * L + 32 * q]);
        __syncthreads();
    }
    if (c < n)
#pragma unroll
        for (int q = 0; q < NQ; ++q) {
            const int k = lane + 32 * q;
            if (k < n) out[(size_t)k * n + c] = z[q];
        }
}

template <int NQ>
cudaError_t launch_back(const double2* Vh, const double2* Tg, const double* Zt, int n, double2* U,
                        cudaStream_t st) {
    const size_t smem = (size_t)2 * kGrp * 32 * NQ * sizeof(double2);
    if (cudaError_t e = raise_smem_limit(k_back<NQ>, smem)) return e;
    k_back<NQ><<<(n + kBackWarps - 1) / kBackWarps, 32 * kBackWarps, smem, st>>>(Vh, Tg, Zt, n, U);
    return cudaGetLastError();
}

// ------------------------------------------------- divide and conquer
constexpr int kLeaf = 24;

__host__ __device__ __forceinline__ int dc_bound(int n, int level, int b) {
    return (int)(((long long)n * b) >> level);
}
// block of index t at a level
__device__ __forceinline__ int dc_block(int n, int level, int t) {
    int b = (int)(((long long)t << level) / n);
    while (dc_bound(n, level, b) > t) --b;
    while (dc_bound(n, level, b + 1) <= t) ++b;
    return b;
}

struct DcWork {
    int n;
    double *d, *e;             // tridiagonal
    double *D[2], *Zt[2];      // eigenvalues and eigenvectors (rows) per level parity
    double *kd, *kz, *kl, *km; // kept poles, z, eigenvalues, offsets from their poles
    double *zh, *dd, *rho;     // recomputed z, deflated eigenvalues, 1 / (rank-one weight)
    double* S;                 // eigenvectors of the rank-one problems (rows)
    int *ks, *ds, *org, *rank, *K;
    int* sweeps;
};

// Leaf problems (at most kLeaf rows): cyclic Jacobi in shared memory.  The
// splits subtract |e| from the two diagonal entries beside them.  One warp per
// rotated pair, a lane per column.
constexpr int kLeafWarps = kLeaf / 2;
constexpr int kLeafSweeps = 30;
__global__ void __launch_bounds__(32 * kLeafWarps) k_dc_leaf(DcWork w, int level) {
    constexpr int LS = kLeaf + 1;
    __shared__ double a[kLeaf * LS], v[kLeaf * LS];
    __shared__ double cs[kLeaf / 2][2];
    __shared__ int pq[kLeaf / 2][2];
    __shared__ double off[kLeafWarps], tot[kLeafWarps];
    const int n = w.n, o = dc_bound(n, level, blockIdx.x), N = dc_bound(n, level, blockIdx.x + 1) - o;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;  // lane: column (N <= 24)
    for (int i = warp; i < N; i += kLeafWarps) {
        const int k = lane;
        if (k >= N) continue;
        double x = 0.0;
        if (i == k) {
            x = w.d[o + i];
            if (i == 0 && o > 0) x -= fabs(w.e[o - 1]);
            if (i == N - 1 && o + N < n) x -= fabs(w.e[o + N - 1]);
        } else if (i == k + 1) x = w.e[o + k];
        else if (k == i + 1) x = w.e[o + i];
        a[i * LS + k] = x;
        v[i * LS + k] = i == k ? 1.0 : 0.0;
    }
    __syncthreads();
    const int m = N + (N & 1), np = m / 2;
    int sweep = 0;
    bool bad = false;
    for (;; ++sweep) {
        double f = 0.0, t = 0.0;
        for (int i = warp; i < N; i += kLeafWarps) {
            const double x = lane < N ? a[i * LS + lane] * a[i * LS + lane] : 0.0;
            t += x;
            if (i != lane) f += x;
        }
        f = warp_add(f);
        t = warp_add(t);
        if (lane == 0) { off[warp] = f; tot[warp] = t; }
        __syncthreads();
        f = t = 0.0;
#pragma unroll
        for (int g = 0; g < kLeafWarps; ++g) {
            f += off[g];
            t += tot[g];
        }
        // rotated entries are set to zero, so the sum falls quadratically well
        // below rounding; also leaves on NaN
        if (!(f > 1e-34 * t)) break;
        if (sweep == kLeafSweeps) {
            bad = f > 1e-28 * t;  // short of working precision, not just of its last bits
            break;
        }
        for (int s = 0; s < m - 1; ++s) {
            if (tid < np) {  // circle method: pair tid of step s
                int x = tid == 0 ? 0 : tid - 1 + s, y = m - 2 - tid + s;
                if (x >= m - 1) x -= m - 1;
                if (tid > 0) ++x;
                if (y >= m - 1) y -= m - 1;
                ++y;
                const int p = min(x, y), q = max(x, y);
                pq[tid][0] = p;
                pq[tid][1] = q;
                double c = 1.0, sn = 0.0;
                if (q < N) {
                    const double apq = a[p * LS + q], app = a[p * LS + p], aqq = a[q * LS + q];
                    if (apq != 0.0) {
                        // c^2 = (1 + cos 2t) / 2, sin t = sin 2t / (2 c): two rsqrt in
                        // a row instead of two divisions, a square root and a rsqrt
                        const double dl = 0.5 * (aqq - app), h = dl * dl + apq * apq;
                        if (h > 1e-280) {
                            const double ri = rsqrt(h), c2 = fma(0.5 * fabs(dl), ri, 0.5);
                            const double rc = rsqrt(c2);
                            c = c2 * rc;
                            sn = copysign(0.5, dl) * apq * ri * rc;
                        } else {
                            const double th = dl / apq;
                            const double tt = (th >= 0.0 ? 1.0 : -1.0) / (fabs(th) + sqrt(1.0 + th * th));
                            c = rsqrt(1.0 + tt * tt);
                            sn = tt * c;
                        }
                    }
                }
                cs[tid][0] = c;
                cs[tid][1] = sn;
            }
            __syncthreads();
            if (warp < np) {  // rows
                const int i = warp, p = pq[i][0], q = pq[i][1];
                if (q < N && lane < N) {
                    const double c = cs[i][0], sn = cs[i][1], x = a[p * LS + lane], y = a[q * LS + lane];
                    a[p * LS + lane] = c * x - sn * y;
                    a[q * LS + lane] = sn * x + c * y;
                }
            }
            __syncthreads();
            if (warp < np) {  // columns
                const int i = warp, p = pq[i][0], q = pq[i][1];
                if (q < N && lane < N) {
                    const double c = cs[i][0], sn = cs[i][1];
                    double x = a[lane * LS + p], y = a[lane * LS + q];
                    a[lane * LS + p] = lane == q ? 0.0 : c * x - sn * y;
                    a[lane * LS + q] = lane == p ? 0.0 : sn * x + c * y;
                    x = v[lane * LS + p];
                    y = v[lane * LS + q];
                    v[lane * LS + p] = c * x - sn * y;
                    v[lane * LS + q] = sn * x + c * y;
                }
            }
            __syncthreads();
        }
    }
    __syncthreads();
    for (int i = tid; i < N; i += 32 * kLeafWarps) {
        const double x = a[i * LS + i];
        bad |= !isfinite(x);
        int r = 0;
        for (int k = 0; k < N; ++k) {
            const double y = a[k * LS + k];
            r += y < x || (y == x && k < i);
        }
        w.D[0][o + r] = x;
        for (int k = 0; k < N; ++k) w.Zt[0][(size_t)(o + r) * n + o + k] = v[k * LS + i];
    }
    if (bad) atomicMax(w.sweeps, kNoConvergence);
    else if (tid == 0) atomicMax(w.sweeps, sweep);
}

// Deflation of the merges of one level (blocks 2b, 2b + 1 of level + 1): poles
// sorted, entries with a negligible z or closer than the tolerance to their
// neighbour (rotated away) set aside.  One block per merge; the serial scan
// runs only where two neighbours are close.
__global__ void __launch_bounds__(256) k_dc_deflate(DcWork w, int level, int par) {
    extern __shared__ double dsm[];
    __shared__ double wmax[8];
    __shared__ int wcnt[8];
    __shared__ int sh_k, sh_nr;
    const int n = w.n, b = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int o = dc_bound(n, level, b), m = dc_bound(n, level + 1, 2 * b + 1),
              N = dc_bound(n, level, b + 1) - o, n1 = m - o, n2 = N - n1;
    const double* D = w.D[par] + o;
    double* Zt = w.Zt[par];
    double* ds = dsm;            // poles, ascending
    double* zs = ds + N;
    double* rc = zs + N;         // rotations
    double* rs = rc + N;
    int* src = (int*)(rs + N);
    int* rp = src + N;
    int* rq = rp + N;
    int* small = rq + N;
    const double ee = w.e[m - 1], rho = 2.0 * fabs(ee), sg = ee < 0.0 ? -1.0 : 1.0;
    for (int i = tid; i < N; i += 256) {
        src[i] = o + i;
        ds[i] = zs[i] = 0.0;
    }
    __syncthreads();
    double mx = 0.0;
    for (int i = tid; i < N; i += 256) {
        const double x = D[i];
        const double z = 0.7071067811865476 *
                         (i < n1 ? Zt[(size_t)(o + i) * n + m - 1] : sg * Zt[(size_t)(o + i) * n + m]);
        // rank in the merged order: first half before equal ones of the second
        int lo = 0, hi = i < n1 ? n2 : n1;
        const double* other = i < n1 ? D + n1 : D;
        while (lo < hi) {
            const int q = (lo + hi) >> 1;
            const bool before = i < n1 ? other[q] < x : other[q] <= x;
            if (before) lo = q + 1;
            else hi = q;
        }
        const int pos = (i < n1 ? i : i - n1) + lo;
        ds[pos] = x;
        zs[pos] = z;
        src[pos] = o + i;
        mx = fmax(mx, fabs(x));
        mx = fmax(mx, rho * fabs(z));
    }
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, q));
    if (lane == 0) wmax[warp] = mx;
    if (tid == 0) sh_k = sh_nr = 0;
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 8; ++q) mx = fmax(mx, wmax[q]);
    const double tol = 16.0 * kEps * mx;
    // entries with a negligible z, and whether neighbours among the others are close
    for (int i = tid; i < N; i += 256) small[i] = !(rho * fabs(zs[i]) > tol);
    __syncthreads();
    int close = 0;
    for (int i = tid; i < N; i += 256) {
        if (small[i]) continue;
        int p = i - 1;
        while (p >= 0 && small[p]) --p;
        if (p >= 0) {
            const double s = zs[p], c = zs[i];
            close |= fabs((ds[i] - ds[p]) * c * s) <= tol * (c * c + s * s);
        }
    }
    close = __syncthreads_or(close);
    double* kd = w.kd + o;
    double* kz = w.kz + o;
    int* ks = w.ks + o;
    double* dd = w.dd + o;
    int* dsrc = w.ds + o;
    if (!close) {
        for (int i0 = 0; i0 < N; i0 += 256) {  // stable compaction
            const int i = i0 + tid;
            const bool keep = i < N && !small[i];
            const unsigned mask = __ballot_sync(0xffffffffu, keep);
            if (lane == 0) wcnt[warp] = __popc(mask);
            __syncthreads();
            int before = sh_k;
            for (int q = 0; q < warp; ++q) before += wcnt[q];
            before += __popc(mask & ((1u << lane) - 1u));
            if (keep) {
                kd[before] = ds[i];
                kz[before] = zs[i];
                ks[before] = src[i];
            } else if (i < N) {
                dd[i - before] = ds[i];
                dsrc[i - before] = src[i];
            }
            __syncthreads();
            if (tid == 0)
                for (int q = 0; q < 8; ++q) sh_k += wcnt[q];
            __syncthreads();
        }
    } else {
        if (tid == 0) {
            int K = 0, nd = 0, nr = 0, p = -1;
            for (int i = 0; i < N; ++i) {
                if (small[i]) {
                    dd[nd] = ds[i];
                    dsrc[nd++] = src[i];
                    continue;
                }
                if (p >= 0) {
                    double s = zs[p], c = zs[i];
                    const double t2 = c * c + s * s, gap = ds[i] - ds[p];
                    if (fabs(gap * c * s) <= tol * t2) {
                        const double t = sqrt(t2);
                        c /= t;
                        s = -s / t;
                        zs[i] = t;
                        rp[nr] = src[p];
                        rq[nr] = src[i];
                        rc[nr] = c;
                        rs[nr++] = s;
                        const double dp = ds[p] * c * c + ds[i] * s * s;
                        ds[i] = ds[p] * s * s + ds[i] * c * c;
                        dd[nd] = dp;
                        dsrc[nd++] = src[p];
                    } else {
                        kd[K] = ds[p];
                        kz[K] = zs[p];
                        ks[K++] = src[p];
                    }
                }
                p = i;
            }
            if (p >= 0) {
                kd[K] = ds[p];
                kz[K] = zs[p];
                ks[K++] = src[p];
            }
            sh_k = K;
            sh_nr = nr;
        }
        __syncthreads();
        const int nr = sh_nr;
        for (int i = tid; i < N; i += 256)
            for (int q = 0; q < nr; ++q) {
                double* x = Zt + (size_t)rp[q] * n + o + i;
                double* y = Zt + (size_t)rq[q] * n + o + i;
                const double u = *x, v = *y;
                *x = rc[q] * u + rs[q] * v;
                *y = rc[q] * v - rs[q] * u;
            }
    }
    if (tid == 0) {
        w.K[b] = sh_k;
        w.rho[b] = 1.0 / rho;
    }
}

// Root j of 1/rho + sum z_i^2 / (d_i - x): one warp per root, bracketed two-pole
// iteration on the offset from the nearer pole.
constexpr int kSecularSteps = 100;
__global__ void __launch_bounds__(128) k_dc_secular(DcWork w, int level) {
    const int n = w.n, t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= n) return;
    const int b = dc_block(n, level, t), o = dc_bound(n, level, b), j = t - o, K = w.K[b];
    if (j >= K) return;
    const double* d = w.kd + o;
    const double* z = w.kz + o;
    const double ri = w.rho[b];
    const bool last = j == K - 1;
    double z2 = 0.0;
    for (int i = lane; i < K; i += 32) z2 += z[i] * z[i];
    z2 = warp_add(z2);
    if (K == 1) {
        if (lane == 0) {
            w.km[t] = z2 / ri;
            w.org[t] = 0;
            w.kl[t] = d[0] + z2 / ri;
        }
        return;
    }
    // sums and derivatives of the poles up to and past `split`, at offset mu
    // from pole q
    const int split = last ? K - 2 : j;
    auto eval = [&](int q, double mu, double& psi, double& dpsi, double& phi, double& dphi) {
        psi = dpsi = phi = dphi = 0.0;
        const double dq = d[q];
        for (int i = lane; i < K; i += 32) {
            const double r = z[i] / ((d[i] - dq) - mu), u = z[i] * r;
            if (i <= split) { psi += u; dpsi += r * r; }
            else { phi += u; dphi += r * r; }
        }
        psi = warp_add(psi);
        dpsi = warp_add(dpsi);
        phi = warp_add(phi);
        dphi = warp_add(dphi);
    };
    int q = j;
    double lo = 0.0, hi = last ? z2 / ri : d[j + 1] - d[j];  // open ends, f(lo) < 0 < f(hi)
    double psi, dpsi, phi, dphi;
    double mu = 0.5 * hi;
    eval(j, mu, psi, dpsi, phi, dphi);
    double f = ri + psi + phi;
    if (!last && f < 0.0) {  // right half: offsets from pole j + 1, negative
        q = j + 1;
        const double gap = hi;
        lo = -0.5 * gap;
        hi = 0.0;
        mu = lo;
        eval(q, mu, psi, dpsi, phi, dphi);
        f = ri + psi + phi;
    } else if (f < 0.0) {
        lo = mu;
    } else {
        hi = mu;
    }
    // the two poles of the interpolation
    const double pa = d[split] - d[q], pb = d[split + 1] - d[q];
    double width = hi - lo;
    bool bad = false;
    for (int it = 0;; ++it) {
        const double err = 8.0 * (fabs(psi) + fabs(phi)) + ri + fabs(mu) * (dpsi + dphi);
        bad = !isfinite(f);
        if (!(fabs(f) > kEps * err) || bad) break;
        if (it == kSecularSteps) {
            bad = fabs(f) > 0x1p20 * kEps * err;
            break;
        }
        if (f < 0.0) lo = fmax(lo, mu);
        else hi = fmin(hi, mu);
        if (hi - lo <= 2.0 * kEps * fmax(fabs(lo), fabs(hi))) break;
        const double da = pa - mu, db = pb - mu;
        double c = f - da * dpsi - db * dphi;
        const double a = (da + db) * f - da * db * (dpsi + dphi), bb = da * db * f;
        if (last && c < 0.0) c = fabs(c);
        const double disc = sqrt(fabs(a * a - 4.0 * bb * c));
        double eta;
        if (last) eta = a >= 0.0 ? (a + disc) / (2.0 * c) : 2.0 * bb / (a - disc);
        else eta = a <= 0.0 ? (a - disc) / (2.0 * c) : 2.0 * bb / (a + disc);
        if (!(f * eta < 0.0)) eta = -f / (dpsi + dphi);
        double next = mu + eta;
        // outside the bracket, or a bracket that no longer shrinks: halve it (in
        // the exponent next to a pole)
        bool halve = !(next > lo && next < hi);
        if (it >= 8 && it % 4 == 0) {
            halve |= hi - lo > 0.5 * width;
            width = hi - lo;
        }
        if (halve) {
            const double s = fmin(fabs(lo), fabs(hi)), l = fmax(fabs(lo), fabs(hi));
            if (s == 0.0) next = copysign(l * 0x1p-10, lo + hi);
            else if (l > 4.0 * s) next = copysign(sqrt(s) * sqrt(l), lo + hi);
            else next = 0.5 * (lo + hi);
        }
        if (next == mu) break;
        mu = next;
        eval(q, mu, psi, dpsi, phi, dphi);
        f = ri + psi + phi;
    }
    if (lane == 0) {
        w.km[t] = mu;
        w.org[t] = q;
        w.kl[t] = d[q] + mu;
        if (bad) atomicMax(w.sweeps, kNoConvergence);
    }
}

// z recomputed so that the computed roots are exact for it: z_i^2 is the product
// of (x_j - d_i) over that of (d_j - d_i).  One warp per entry.
__global__ void __launch_bounds__(128) k_dc_zhat(DcWork w, int level) {
    const int n = w.n, t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= n) return;
    const int b = dc_block(n, level, t), o = dc_bound(n, level, b), i = t - o, K = w.K[b];
    if (i >= K) return;
    const double* d = w.kd + o;
    const double di = d[i];
    double p = 1.0;
    for (int j = lane; j < K; j += 32) {
        const double x = (d[w.org[o + j]] - di) + w.km[o + j];  // root j minus d_i
        if (j < i) p *= x / (d[j] - di);
        else if (j < K - 1) p *= x / (d[j + 1] - di);
        else p *= x;
    }
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) p *= __shfl_xor_sync(0xffffffffu, p, q);
    if (lane == 0) w.zh[t] = copysign(sqrt(fabs(p)), w.kz[t]);
}

// Normalised eigenvectors of the rank-one problems (rows of S) and the place of
// every eigenvalue, kept or deflated, in ascending order.  One warp per entry.
__global__ void __launch_bounds__(128) k_dc_vectors(DcWork w, int level, int par) {
    const int n = w.n, t = blockIdx.x * 4 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (t >= n) return;
    const int b = dc_block(n, level, t), o = dc_bound(n, level, b), j = t - o, K = w.K[b];
    const int nd = dc_bound(n, level, b + 1) - o - K;
    const double* d = w.kd + o;
    int r = 0;
    double x;
    if (j < K) {
        const double dq = d[w.org[t]], mu = w.km[t];
        double s = 0.0;
        double* S = w.S + (size_t)t * n;
        for (int i = lane; i < K; i += 32) {
            const double u = w.zh[o + i] / ((d[i] - dq) - mu);
            S[i] = u;
            s += u * u;
        }
        s = 1.0 / sqrt(warp_add(s));
        if (lane == 0 && !(s > 0.0 && isfinite(s))) atomicMax(w.sweeps, kNoConvergence);
        for (int i = lane; i < K; i += 32) S[i] *= s;
        x = w.kl[t];
        for (int i = lane; i < nd; i += 32) r += w.dd[o + i] < x;
    } else {
        x = w.dd[o + j - K];
        for (int i = lane; i < nd; i += 32) {
            const double y = w.dd[o + i];
            r += y < x || (y == x && i < j - K);
        }
        for (int i = lane; i < K; i += 32) r += w.kl[o + i] <= x;
    }
#pragma unroll
    for (int q = 16; q > 0; q >>= 1) r += __shfl_xor_sync(0xffffffffu, r, q);
    if (j < K) r += j;
    if (lane == 0) {
        w.rank[t] = o + r;
        w.D[par ^ 1][o + r] = x;
    }
}

// Eigenvectors of the merged problems: rows of S times the kept rows of the
// halves (K x K by K x N), deflated rows copied.  32 x 64 tiles.
__global__ void __launch_bounds__(256) k_dc_update(DcWork w, int level, int par) {
    __shared__ double sa[32][17], sb[16][66];
    const int n = w.n, b = blockIdx.z, o = dc_bound(n, level, b), N = dc_bound(n, level, b + 1) - o;
    const int K = w.K[b], j0 = blockIdx.y * 32, i0 = blockIdx.x * 64, tid = threadIdx.x;
    if (j0 >= N || i0 >= N) return;
    const double* Z = w.Zt[par];
    double* Zn = w.Zt[par ^ 1];
    const int jr = (tid >> 4) * 2, ic = (tid & 15) * 4;
    double acc[2][4] = {};
    if (j0 < K)
        for (int k0 = 0; k0 < K; k0 += 16) {
            for (int u = tid; u < 32 * 16; u += 256) {
                const int r = u >> 4, k = u & 15;
                sa[r][k] = j0 + r < K && k0 + k < K ? w.S[(size_t)(o + j0 + r) * n + k0 + k] : 0.0;
            }
            for (int u = tid; u < 16 * 64; u += 256) {
                const int k = u >> 6, i = u & 63;
                sb[k][i] = k0 + k < K && i0 + i < N ? Z[(size_t)w.ks[o + k0 + k] * n + o + i0 + i] : 0.0;
            }
            __syncthreads();
#pragma unroll
            for (int k = 0; k < 16; ++k) {
                const double x0 = sa[jr][k], x1 = sa[jr + 1][k];
#pragma unroll
                for (int c = 0; c < 4; ++c) {
                    const double y = sb[k][ic + c];
                    acc[0][c] = fma(x0, y, acc[0][c]);
                    acc[1][c] = fma(x1, y, acc[1][c]);
                }
            }
            __syncthreads();
        }
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const int j = j0 + jr + r;
        if (j >= N) continue;
        const double* from = j >= K ? Z + (size_t)w.ds[o + j - K] * n + o : nullptr;
        double* to = Zn + (size_t)w.rank[o + j] * n + o;
#pragma unroll
        for (int c = 0; c < 4; ++c) {
            const int i = i0 + ic + c;
            if (i < N) to[i] = from ? from[i] : acc[r][c];
        }
    }
}

__global__ void k_heev1(const double2* A, double* w, double2* U, int* sweeps) {
    w[0] = A[0].x;
    U[0] = make_double2(1.0, 0.0);
    *sweeps = isfinite(A[0].x) ? 0 : kNoConvergence;
}

__global__ void k_copy_eig(const double* __restrict__ D, int n, const unsigned* __restrict__ top,
                           double* __restrict__ w, int* sweeps) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    w[i] = D[i] / tri_scale(*top);
    if (!isfinite(D[i])) atomicMax(sweeps, kNoConvergence);
}

int dc_levels(int n) {
    int l = 0;
    while ((n + (1 << l) - 1) >> l > kLeaf) ++l;
    return l;
}

struct TriPlan { int blocks, rows; size_t smem; };
TriPlan tri_plan(int n, int blocks, int vectors) {
    TriPlan p;
    p.rows = (n + blocks - 1) / blocks;
    p.blocks = (n + p.rows - 1) / p.rows;
    p.smem = ((size_t)p.rows + vectors) * n * sizeof(double2);
    return p;
}
constexpr size_t kTriSmem = 200 * 1024;

int device_sms() {
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return sms;
}

}  // namespace

cudaError_t chol_inv(double2* A, double2* X, int n, int* info, cudaStream_t st) {
    const size_t smem = 4 * kCTile * sizeof(double2) + (size_t)n * sizeof(double);
    if (cudaError_t e = raise_smem_limit(k_chol_inv, smem)) return e;
    const int nbk = (n + kCB - 1) / kCB;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_chol_inv, 256, smem);
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    // one block per trailing tile of the middle step
    int blocks = std::min(device_sms(), std::max(1, nbk * nbk / 4 + nbk / 2));
    count_launch();
    void* args[] = {&A, &X, &n, &info};
    return cudaLaunchCooperativeKernel((const void*)k_chol_inv, dim3(blocks), dim3(256), args, smem, st);
}

// sizes whose rows fit the shared memory of the grid
bool heev_fits(int n) {
    return n <= kTriPer * 256 && tri_plan(n, 148, TriCfg<false>::vectors).smem <= kTriSmem;
}

size_t heev_scratch_doubles(int n) {
    return 5 * (size_t)n * n + 36 * (size_t)n + 128;
}

cudaError_t heev(const double2* A, int n, double* w, double2* U, double* scratch, int* sweeps_out,
                 cudaStream_t st) {
    const size_t nn = (size_t)n * n;
    if (n == 1) {
        count_launch();
        k_heev1<<<1, 1, 0, st>>>(A, w, U, sweeps_out);
        return cudaGetLastError();
    }
    double* s = (double*)(((uintptr_t)scratch + 15) & ~(uintptr_t)15);
    double2* Vh = (double2*)s;
    double2* tau = Vh + nn;
    double2* P = tau + n;      // q and a of two steps in turn
    DcWork q{};
    q.n = n;
    double2* Tg = P + 4 * n;   // T of each reflector group, 16 entries per 4 columns
    double* at = (double*)(Tg + 4 * n + 16);
    auto take = [&](size_t k) { double* p = at; at += k; return p; };
    q.Zt[0] = take(nn);
    q.Zt[1] = take(nn);
    unsigned* top = (unsigned*)take(1);
    q.S = take(nn);
    double** vecs[] = {&q.d, &q.e, &q.D[0], &q.D[1], &q.kd, &q.kz, &q.kl, &q.km, &q.zh, &q.dd, &q.rho};
    for (double** v : vecs) *v = take(n);
    int** ints[] = {&q.ks, &q.ds, &q.org, &q.rank, &q.K};
    for (int** v : ints) *v = (int*)take(n);
    q.sweeps = sweeps_out;
    cudaError_t e = cudaMemsetAsync(sweeps_out, 0, sizeof(int), st);
    if (e == cudaSuccess) e = cudaMemsetAsync(q.Zt[0], 0, (2 * nn + 1) * sizeof(double), st);
    if (e != cudaSuccess) return e;
    // ---- A = Q T Q^H
    count_launch();
    bool done = false;
    if (n <= kTriCluster) {
        const TriPlan p = tri_plan(n, std::min(16, (n + 3) / 4), TriCfg<true>::vectors);
        raise_smem_limit(k_tridiag<true>, p.smem);
        cudaFuncSetAttribute(k_tridiag<true>, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
        cudaLaunchConfig_t lc = {};
        lc.gridDim = dim3(p.blocks);
        lc.blockDim = dim3(TriCfg<true>::threads);
        lc.dynamicSmemBytes = p.smem;
        lc.stream = st;
        cudaLaunchAttribute attr[1];
        attr[0].id = cudaLaunchAttributeClusterDimension;
        attr[0].val.clusterDim.x = p.blocks;
        attr[0].val.clusterDim.y = 1;
        attr[0].val.clusterDim.z = 1;
        lc.attrs = attr;
        lc.numAttrs = 1;
        int clusters = 0;
        if (p.smem <= kTriSmem &&
            cudaOccupancyMaxActiveClusters(&clusters, k_tridiag<true>, &lc) == cudaSuccess && clusters >= 1)
            done = cudaLaunchKernelEx(&lc, k_tridiag<true>, A, n, p.rows, Vh, tau, q.d, q.e, P, top) == cudaSuccess;
        cudaGetLastError();  // a refused configuration: the grid version
    }
    if (!done) {
        TriPlan p = tri_plan(n, std::min(device_sms(), std::max(1, (n + 3) / 4)), TriCfg<false>::vectors);
        if ((e = raise_smem_limit(k_tridiag<false>, p.smem)) != cudaSuccess) return e;
        void* args[] = {&A, &n, &p.rows, &Vh, &tau, &q.d, &q.e, &P, &top};
        e = cudaLaunchCooperativeKernel((const void*)k_tridiag<false>, dim3(p.blocks),
                                        dim3(TriCfg<false>::threads), args, p.smem, st);
        if (e != cudaSuccess) return e;
    }
    // ---- T = Z W Z^T
    const int levels = dc_levels(n);
    count_launch(4 + 5 * levels);
    k_dc_leaf<<<1 << levels, 32 * kLeafWarps, 0, st>>>(q, levels);
    int par = 0;
    for (int l = levels - 1; l >= 0; --l, par ^= 1) {
        const int most = (n >> l) + 1;
        const size_t smem = (size_t)most * (4 * sizeof(double) + 4 * sizeof(int));
        if ((e = raise_smem_limit(k_dc_deflate, smem)) != cudaSuccess) return e;
        k_dc_deflate<<<1 << l, 256, smem, st>>>(q, l, par);
        k_dc_secular<<<(n + 3) / 4, 128, 0, st>>>(q, l);
        k_dc_zhat<<<(n + 3) / 4, 128, 0, st>>>(q, l);
        k_dc_vectors<<<(n + 3) / 4, 128, 0, st>>>(q, l, par);
        k_dc_update<<<dim3((most + 63) / 64, (most + 31) / 32, 1 << l), 256, 0, st>>>(q, l, par);
    }
    k_copy_eig<<<(n + 255) / 256, 256, 0, st>>>(q.D[par], n, top, w, sweeps_out);
    // ---- U = Q Z.  A size takes the next rung up, with the entries past it idle; 5
    // and 18 are those of the 64- and 216-atom cells' 160 and 576 bands, the others
    // keep the steps between sizes below a factor of two from 96 rows on.
    k_wy<<<((n + kGrp - 1) / kGrp + 3) / 4, 128, 0, st>>>(Vh, tau, n, Tg);
    if (n <= 32) return launch_back<1>(Vh, Tg, q.Zt[par], n, U, st);
    if (n <= 96) return launch_back<3>(Vh, Tg, q.Zt[par], n, U, st);
    if (n <= 160) return launch_back<5>(Vh, Tg, q.Zt[par], n, U, st);
    if (n <= 256) return launch_back<8>(Vh, Tg, q.Zt[par], n, U, st);
    if (n <= 384) return launch_back<12>(Vh, Tg, q.Zt[par], n, U, st);
    if (n <= 576) return launch_back<18>(Vh, Tg, q.Zt[par], n, U, st);
    if (n <= 768) return launch_back<24>(Vh, Tg, q.Zt[par], n, U, st);
    return launch_back<40>(Vh, Tg, q.Zt[par], n, U, st);
}

}  // namespace chfsi
