// Small dense FP64 kernels of the Rayleigh-Ritz step and the scalar
// plumbing of the filter (bounds, norm guard, Lanczos), all on the device so
// the ChFSI iteration needs no host round trip until the eigenvalues return.
//
// Rayleigh-Ritz follows the Cholesky reduction of the reference's CPU
// path (src/eigensolver/subspace_diag.rs:229-391):
//   S = L L^H (info = failing column as ZPOTRF), Li = L^-1,
//   B = Li H Li^H (Hermitian-symmetrised), B U = U diag(w),
//   V = Li^H U; psi <- psi V (caller).
// It replaces cuSOLVER ZHEGVD itype 1 (src/device/solver.rs:47-95).  The factor
// and the eigensolver are in heev.cu; a parallel cyclic Jacobi (round-robin pair
// ordering, one cooperative launch) serves the sizes past those of heev().
#include "dense.hpp"
#include "launch_count.hpp"
#include "smem_limit.hpp"

#include <cooperative_groups.h>

namespace cg = cooperative_groups;

namespace chfsi {

namespace {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
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

__global__ void k_symmetrize(const double2* __restrict__ in, double2* __restrict__ out, int n) {
    const size_t nn = (size_t)n * n;
    for (size_t t = blockIdx.x * (size_t)blockDim.x + threadIdx.x; t < nn;
         t += (size_t)gridDim.x * blockDim.x) {
        const int i = (int)(t / n), j = (int)(t % n);
        const double2 a = in[(size_t)i * n + j], b = in[(size_t)j * n + i];
        out[t] = make_double2(0.5 * (a.x + b.x), 0.5 * (a.y - b.y));
    }
}

// C = op(A) op(B), n x n row-major; op 0 = N, 1 = conjugate transpose.
template <int OPA, int OPB>
__global__ void __launch_bounds__(256)
k_small_gemm(const double2* __restrict__ A, const double2* __restrict__ B, double2* __restrict__ C,
             int n) {
    __shared__ double2 As[16][17], Bs[16][17];
    const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
    const int i = blockIdx.y * 16 + ty, j = blockIdx.x * 16 + tx;
    double2 acc = make_double2(0.0, 0.0);
    for (int k0 = 0; k0 < n; k0 += 16) {
        {
            const int r = blockIdx.y * 16 + ty, k = k0 + tx;
            double2 v = make_double2(0.0, 0.0);
            if (r < n && k < n) {
                if (OPA == 0) v = A[(size_t)r * n + k];
                else { v = A[(size_t)k * n + r]; v.y = -v.y; }
            }
            As[ty][tx] = v;
            const int kb = k0 + ty, cc = blockIdx.x * 16 + tx;
            double2 w = make_double2(0.0, 0.0);
            if (kb < n && cc < n) {
                if (OPB == 0) w = B[(size_t)kb * n + cc];
                else { w = B[(size_t)cc * n + kb]; w.y = -w.y; }
            }
            Bs[ty][tx] = w;
        }
        __syncthreads();
#pragma unroll
        for (int k = 0; k < 16; ++k) {
            const double2 a = As[ty][k], b = Bs[k][tx];
            acc.x = fma(a.x, b.x, acc.x);
            acc.x = fma(-a.y, b.y, acc.x);
            acc.y = fma(a.x, b.y, acc.y);
            acc.y = fma(a.y, b.x, acc.y);
        }
        __syncthreads();
    }
    if (i < n && j < n) C[(size_t)i * n + j] = acc;
}

// Circle-method pairing of step s over m = n + (n & 1) indices: pair i of
// step s is (min(a, b), max(a, b)).
// Every argument reduced below lies in (-(m - 1), 2 (m - 1)), so one
// conditional add or subtract replaces the integer modulo.
__device__ __forceinline__ int jac_wrap(int x, int M) { return x >= M ? x - M : (x < 0 ? x + M : x); }
__device__ __forceinline__ void jac_pair(int m, int s, int i, int& p, int& q) {
    const int M = m - 1;
    const int a = i == 0 ? 0 : 1 + jac_wrap(i - 1 + s, M);
    const int b = 1 + jac_wrap(m - 2 - i + s, M);
    p = min(a, b);
    q = max(a, b);
}
// Pair index and partner of column k at step s.
__device__ __forceinline__ void jac_partner(int m, int s, int k, int& pi, int& partner) {
    const int M = m - 1;
    const int j = k == 0 ? 0 : jac_wrap(k - 1 - s, M) + 1;
    const int jj = m - 1 - j;
    pi = min(j, jj);
    partner = jj == 0 ? 0 : 1 + jac_wrap(jj - 1 + s, M);
}

// Parallel cyclic Jacobi with one grid barrier per rotation step.
//   phase 1 (step s): each warp takes its pairs (p, q), computes the rotation
//     from A, writes rows p, q of X = G^H A and the rotation parameters
//     (double-buffered by step parity)
//   grid barrier
//   phase 2 (step s): each warp builds the rows it owns at step s + 1 as
//     A[r] = X[r] G, mixing the columns of every pair of step s, and updates
//     its share of V rows the same way (through a shared-memory row buffer)
// Rows read in phase 1 of step s + 1 were written by the same warp in phase 2
// of step s, so no second barrier is needed.  All accesses are row-wise.
__global__ void __launch_bounds__(256)
k_jacobi2(double2* A, double2* V, double2* X, int n, int max_sweeps, double tol2, double* scratch,
          double* rot, int* sweeps_out) {
    cg::grid_group grid = cg::this_grid();
    extern __shared__ double2 rowbuf_all[];  // 8 warps x n
    __shared__ double red[32];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int nwarps = (gridDim.x * blockDim.x) >> 5;
    double2* rowbuf = rowbuf_all + (size_t)wib * n;
    const size_t nn = (size_t)n * n;
    const size_t gtid = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    const size_t gstride = (size_t)gridDim.x * blockDim.x;
    for (size_t t = gtid; t < nn; t += gstride)
        V[t] = make_double2((t / n) == (t % n) ? 1.0 : 0.0, 0.0);
    double tot = 0.0;
    for (size_t t = gtid; t < nn; t += gstride) tot += A[t].x * A[t].x + A[t].y * A[t].y;
    tot = block_sum(tot, red);
    if (threadIdx.x == 0) atomicAdd(&scratch[0], tot);
    grid.sync();
    const double total = scratch[0];
    const int m = n + (n & 1);
    const int npairs = m / 2;
    const int nsteps = m - 1;
    int sweep = 0;
    bool converged = false;
    for (; sweep < max_sweeps && !converged; ++sweep) {
        for (int s = 0; s < nsteps; ++s) {
            double* rs = rot + 4 * (size_t)npairs * (s & 1);
            // ---- phase 1
            for (int pi = gw; pi < npairs; pi += nwarps) {
                int p, q;
                jac_pair(m, s, pi, p, q);
                double c = 1.0, sn = 0.0, phr = 1.0, phi = 0.0;
                if (q < n) {
                    const double2 apq = A[(size_t)p * n + q];
                    const double app = A[(size_t)p * n + p].x, aqq = A[(size_t)q * n + q].x;
                    const double bm = hypot(apq.x, apq.y);
                    if (bm > 1e-300 && bm > 1e-18 * sqrt(fabs(app * aqq))) {
                        phr = apq.x / bm;
                        phi = apq.y / bm;
                        const double tau = (aqq - app) / (2.0 * bm);
                        const double t = (tau >= 0.0 ? 1.0 : -1.0) / (fabs(tau) + sqrt(1.0 + tau * tau));
                        c = 1.0 / sqrt(1.0 + t * t);
                        sn = t * c;
                    }
                    for (int k = lane; k < n; k += 32) {
                        const double2 apk = A[(size_t)p * n + k], aqk = A[(size_t)q * n + k];
                        const double2 pa = make_double2(phr * aqk.x - phi * aqk.y, phr * aqk.y + phi * aqk.x);
                        X[(size_t)p * n + k] = make_double2(c * apk.x - sn * pa.x, c * apk.y - sn * pa.y);
                        X[(size_t)q * n + k] = make_double2(sn * apk.x + c * pa.x, sn * apk.y + c * pa.y);
                    }
                } else if (p < n) {
                    for (int k = lane; k < n; k += 32) X[(size_t)p * n + k] = A[(size_t)p * n + k];
                }
                if (lane == 0) {
                    rs[4 * pi + 0] = c; rs[4 * pi + 1] = sn; rs[4 * pi + 2] = phr; rs[4 * pi + 3] = phi;
                }
            }
            grid.sync();
            // ---- phase 2: rows owned at the next step, A[r] = X[r] G(s)
            const int s2 = (s + 1) % nsteps;
            auto mix = [&](const double2* src, int k) -> double2 {
                int pi, partner;
                jac_partner(m, s, k, pi, partner);
                const double2 xk = src[k];
                if (partner >= n) return xk;
                const double c = rs[4 * pi + 0], sn = rs[4 * pi + 1];
                const double phr = rs[4 * pi + 2], phi = rs[4 * pi + 3];
                const double2 xp = src[partner];
                if (k < partner) {  // k is p: X_rp c + X_rq (-s conj(ph))
                    const double2 qc = make_double2(phr * xp.x + phi * xp.y, phr * xp.y - phi * xp.x);
                    return make_double2(c * xk.x - sn * qc.x, c * xk.y - sn * qc.y);
                }
                // k is q: X_rp s + X_rq c conj(ph)
                const double2 qc = make_double2(phr * xk.x + phi * xk.y, phr * xk.y - phi * xk.x);
                return make_double2(sn * xp.x + c * qc.x, sn * xp.y + c * qc.y);
            };
            for (int pi = gw; pi < npairs; pi += nwarps) {
                int p, q;
                jac_pair(m, s2, pi, p, q);
                for (int h = 0; h < 2; ++h) {
                    const int r = h == 0 ? p : q;
                    if (r >= n) continue;
                    const double2* xr = X + (size_t)r * n;
                    for (int k = lane; k < n; k += 32) A[(size_t)r * n + k] = mix(xr, k);
                }
            }
            for (int r = gw; r < n; r += nwarps) {
                double2* vr = V + (size_t)r * n;
                for (int k = lane; k < n; k += 32) rowbuf[k] = mix(vr, k);
                __syncwarp();
                for (int k = lane; k < n; k += 32) vr[k] = rowbuf[k];
                __syncwarp();
            }
            __syncwarp();
        }
        // off-diagonal norm of the rows this warp owns at step 0
        double off = 0.0;
        for (int pi = gw; pi < npairs; pi += nwarps) {
            int p, q;
            jac_pair(m, 0, pi, p, q);
            for (int h = 0; h < 2; ++h) {
                const int r = h == 0 ? p : q;
                if (r >= n) continue;
                for (int k = lane; k < n; k += 32)
                    if (k != r) off += A[(size_t)r * n + k].x * A[(size_t)r * n + k].x +
                                       A[(size_t)r * n + k].y * A[(size_t)r * n + k].y;
            }
        }
        off = block_sum(off, red);
        if (threadIdx.x == 0) atomicAdd(&scratch[1 + sweep], off);
        grid.sync();
        converged = scratch[1 + sweep] <= tol2 * total;
    }
    if (gtid == 0) *sweeps_out = converged ? sweep : max_sweeps;
}

// Sort eigenvalues ascending (stable by index) and permute eigenvector columns.
__global__ void __launch_bounds__(1024)
k_sort_eig(const double2* __restrict__ A, const double2* __restrict__ V, int n,
           double* __restrict__ w_out, double2* __restrict__ U) {
    extern __shared__ int perm_smem[];
    int* dest = perm_smem;  // dest[i] = rank of eigenvalue i
    for (int i = threadIdx.x; i < n; i += blockDim.x) {
        const double wi = A[(size_t)i * n + i].x;
        int r = 0;
        for (int j = 0; j < n; ++j) {
            const double wj = A[(size_t)j * n + j].x;
            r += (wj < wi) || (wj == wi && j < i);
        }
        dest[i] = r;
        w_out[r] = wi;
    }
    __syncthreads();
    for (size_t t = threadIdx.x; t < (size_t)n * n; t += blockDim.x) {
        const int row = (int)(t / n), i = (int)(t % n);
        U[(size_t)row * n + dest[i]] = V[t];
    }
}

// One cluster of kMinmaxBlocks blocks: the range of a 72^3 potential in 13 us (170
// with a single block, which has too few loads in flight), of 40^3 in 7.5 (32).
constexpr int kMinmaxBlocks = 8;
__global__ void __launch_bounds__(1024) k_minmax(const double* __restrict__ v, size_t n, double* out) {
    cg::cluster_group cluster = cg::this_cluster();
    __shared__ double smin[32], smax[32], both[2];
    double lo = 1e300, hi = -1e300;
    const size_t step = (size_t)kMinmaxBlocks * 1024;
    size_t i = cluster.block_rank() * (size_t)1024 + threadIdx.x;
    for (; i + 3 * step < n; i += 4 * step) {
        const double a = v[i], b = v[i + step], c = v[i + 2 * step], d = v[i + 3 * step];
        lo = fmin(lo, fmin(fmin(a, b), fmin(c, d)));
        hi = fmax(hi, fmax(fmax(a, b), fmax(c, d)));
    }
    for (; i < n; i += step) {
        lo = fmin(lo, v[i]);
        hi = fmax(hi, v[i]);
    }
    auto reduce = [&]() {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
        }
    };
    reduce();
    if ((threadIdx.x & 31) == 0) { smin[threadIdx.x >> 5] = lo; smax[threadIdx.x >> 5] = hi; }
    __syncthreads();
    if (threadIdx.x < 32) {
        lo = smin[threadIdx.x];
        hi = smax[threadIdx.x];
        reduce();
        if (threadIdx.x == 0) { both[0] = lo; both[1] = hi; }
    }
    cluster.sync();
    if (cluster.block_rank() == 0 && threadIdx.x == 0) {
        for (int b = 1; b < kMinmaxBlocks; ++b) {
            const double* o = cluster.map_shared_rank(both, b);
            lo = fmin(lo, o[0]);
            hi = fmax(hi, o[1]);
        }
        out[0] = lo;
        out[1] = hi;
    }
    cluster.sync();
}

__global__ void __launch_bounds__(256)
k_sumsq(const double2* __restrict__ x, size_t n, double* acc) {
    __shared__ double red[32];
    double s = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        s += x[i].x * x[i].x + x[i].y * x[i].y;
    s = block_sum(s, red);
    if (threadIdx.x == 0) atomicAdd(acc, s);
}

// Largest eigenvalue of the Lanczos tridiagonal by Sturm bisection.
__device__ double tridiag_max(const double* d, const double* e, int k) {
    double lo = 1e300, hi = -1e300;
    for (int i = 0; i < k; ++i) {
        const double r = (i > 0 ? fabs(e[i - 1]) : 0.0) + (i < k - 1 ? fabs(e[i]) : 0.0);
        lo = fmin(lo, d[i] - r);
        hi = fmax(hi, d[i] + r);
    }
    for (int it = 0; it < 200; ++it) {
        const double mid = 0.5 * (lo + hi);
        if (mid <= lo || mid >= hi) break;
        int c = 0;
        double q = d[0] - mid;
        if (q < 0) ++c;
        for (int i = 1; i < k; ++i) {
            const double qq = q == 0.0 ? 1e-300 : q;
            q = d[i] - mid - e[i - 1] * e[i - 1] / qq;
            if (q < 0) ++c;
        }
        if (c >= k) hi = mid; else lo = mid;
    }
    return hi;
}

// Spectral bounds (src/eigensolver/chebyshev.rs:225-254).  coef[0..5] =
// lambda_max, eps_cut, center c, half-width e, 1/e, -c/e.  lanczos: k alphas
// followed by k squared residual norms |f_j|^2 (null: kinetic + potential-
// range bound); the Lanczos bound is lambda_max(T_k) + |f_k| (Zhou 2010).
__global__ void k_bounds(double kin_max, const double* __restrict__ minmax,
                         const double* __restrict__ eig, int n_eig, const double* lanczos, int k,
                         double lm_scale, double* coef) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    double lm;
    if (lanczos) {
        double e[64];
        for (int i = 0; i < k - 1 && i < 64; ++i) e[i] = sqrt(lanczos[k + i]);
        lm = tridiag_max(lanczos, e, k) + sqrt(lanczos[2 * k - 1]);
    } else {
        lm = kin_max + (minmax[1] - minmax[0]);
    }
    lm *= lm_scale;  // generalised problem: lambda_max(H) / lambda_min(S)
    double cut;
    if (!eig || n_eig == 0) cut = lm / 3.0;
    else {
        const double e0 = eig[0], el = eig[n_eig - 1];
        cut = fmin(el + 0.2 * (el - e0), lm * 0.95);
    }
    const double c = (lm + cut) / 2.0, e = (lm - cut) / 2.0;
    coef[0] = lm; coef[1] = cut; coef[2] = c; coef[3] = e;
    coef[4] = 1.0 / e;
    coef[5] = -c / e;
}

// 10x norm-growth guard over the squared norms of one filter
// (src/eigensolver/chebyshev.rs:552-563), checked for k >= 2 as the
// reference does; status[0] = first failing degree (0 = none).
__global__ void k_norm_guard(const double* __restrict__ nsq, int ndeg, int* status) {
    if (threadIdx.x != 0 || blockIdx.x != 0) return;
    int fail = 0;
    for (int k = 2; k <= ndeg && !fail; ++k) {
        const double prev = sqrt(nsq[k - 1]), cur = sqrt(nsq[k]);
        const double growth = prev > 0.0 ? cur / prev : 1.0;
        if (growth > 10.0 || !(cur == cur)) fail = k;
    }
    status[0] = fail;
}

// ---- Lanczos helpers (vectors of n complex, scalars on device)
__global__ void k_scale_by_rsqrt(double2* v, size_t n, const double* nsq) {
    const double s = 1.0 / sqrt(*nsq);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x)
        v[i] = make_double2(v[i].x * s, v[i].y * s);
}
// f -= beta v0 (if beta_sq); alpha_acc += Re<v, f>
__global__ void __launch_bounds__(256)
k_lanczos_a(double2* f, const double2* v, const double2* v0, const double* beta_sq, size_t n,
            double* alpha_acc) {
    __shared__ double red[32];
    const double bt = beta_sq ? sqrt(*beta_sq) : 0.0;
    double s = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        double2 x = f[i];
        if (beta_sq) { x.x -= bt * v0[i].x; x.y -= bt * v0[i].y; f[i] = x; }
        s += v[i].x * x.x + v[i].y * x.y;
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) atomicAdd(alpha_acc, s);
}
// f -= alpha v; fn_acc += |f|^2
__global__ void __launch_bounds__(256)
k_lanczos_b(double2* f, const double2* v, const double* alpha, size_t n, double* fn_acc) {
    __shared__ double red[32];
    const double a = *alpha;
    double s = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        double2 x = f[i];
        x.x -= a * v[i].x;
        x.y -= a * v[i].y;
        f[i] = x;
        s += x.x * x.x + x.y * x.y;
    }
    s = block_sum(s, red);
    if (threadIdx.x == 0) atomicAdd(fn_acc, s);
}
// v0 = v; v = f / sqrt(fn)
__global__ void k_lanczos_c(const double2* f, double2* v, double2* v0, size_t n, const double* fn) {
    const double s = 1.0 / sqrt(*fn);
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        v0[i] = v[i];
        v[i] = make_double2(f[i].x * s, f[i].y * s);
    }
}
// beta[j] = sqrt(fn)
__global__ void k_lanczos_store_beta(const double* fn, double* beta) {
    if (threadIdx.x == 0) *beta = sqrt(*fn);
}

// ---- Pulay helpers
__global__ void k_pulay_push(const double* rin, const double* rout, double* hr, double* hres,
                             size_t n) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        hr[i] = rin[i];
        hres[i] = rout[i] - rin[i];
    }
}
__global__ void __launch_bounds__(256)
k_dots(const double* __restrict__ x, const double* const* ys, int m, size_t n, double* out) {
    __shared__ double red[32];
    double acc[kPulayMax];
    for (int j = 0; j < kPulayMax; ++j) acc[j] = 0.0;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        const double xi = x[i];
#pragma unroll
        for (int j = 0; j < kPulayMax; ++j)
            if (j < m) acc[j] += xi * ys[j][i];
    }
    for (int j = 0; j < m; ++j) {
        const double s = block_sum(acc[j], red);
        if (threadIdx.x == 0) atomicAdd(&out[j], s);
    }
}
struct PulayCoef { double c[kPulayMax]; };
__global__ void k_pulay_combine(const double* const* hr, const double* const* hres, int m,
                                PulayCoef pc, double alpha, size_t n, double* out) {
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
         i += (size_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int j = 0; j < m; ++j) s += pc.c[j] * (hr[j][i] + alpha * hres[j][i]);
        out[i] = s;
    }
}

int grid_for(size_t n) {
    size_t b = (n + 255) / 256;
    return (int)(b < 148 * 8 ? b : 148 * 8);
}

}  // namespace

void symmetrize(const double2* in, double2* out, int n, cudaStream_t st) {
    count_launch();
    k_symmetrize<<<grid_for((size_t)n * n), 256, 0, st>>>(in, out, n);
}
void small_gemm(int opa, int opb, const double2* A, const double2* B, double2* C, int n,
                cudaStream_t st) {
    count_launch();
    dim3 grid((n + 15) / 16, (n + 15) / 16);
    if (opa == 0 && opb == 0) k_small_gemm<0, 0><<<grid, 256, 0, st>>>(A, B, C, n);
    else if (opa == 0 && opb == 1) k_small_gemm<0, 1><<<grid, 256, 0, st>>>(A, B, C, n);
    else if (opa == 1 && opb == 0) k_small_gemm<1, 0><<<grid, 256, 0, st>>>(A, B, C, n);
    else k_small_gemm<1, 1><<<grid, 256, 0, st>>>(A, B, C, n);
}
size_t jacobi_scratch_doubles(int n, int max_sweeps) {
    // sweep norms, double-buffered rotations, X (n x n complex)
    return 1 + (size_t)max_sweeps + 8 * (size_t)((n + 1) / 2 + 1) + 2 * (size_t)n * n + 2;
}
cudaError_t jacobi(double2* A, double2* V, int n, int max_sweeps, double tol2, double* scratch,
                   int* sweeps_out, cudaStream_t st) {
    count_launch();
    cudaMemsetAsync(scratch, 0, sizeof(double) * (1 + max_sweeps), st);
    const int npairs = (n + 1) / 2;
    double* rot = scratch + 1 + max_sweeps;
    double2* X = (double2*)(rot + 8 * (size_t)(npairs + 1));
    if (((uintptr_t)X) & 15) X = (double2*)(((uintptr_t)X + 15) & ~(uintptr_t)15);
    int dev = 0, sms = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int warps_per_block = 8;
    int blocks = (npairs + warps_per_block - 1) / warps_per_block;
    const size_t smem = (size_t)warps_per_block * n * sizeof(double2);
    if (cudaError_t e = raise_smem_limit(k_jacobi2, smem)) return e;
    int per_sm = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_jacobi2, 256, smem);
    if (per_sm < 1) per_sm = 1;
    if (blocks > sms * per_sm) blocks = sms * per_sm;
    if (blocks < 1) blocks = 1;
    void* args[] = {&A, &V, &X, &n, &max_sweeps, &tol2, &scratch, &rot, &sweeps_out};
    return cudaLaunchCooperativeKernel((const void*)k_jacobi2, dim3(blocks), dim3(256), args, smem, st);
}
void sort_eig(const double2* A, const double2* V, int n, double* w, double2* U, cudaStream_t st) {
    count_launch();
    k_sort_eig<<<1, 1024, sizeof(int) * n, st>>>(A, V, n, w, U);
}
void minmax(const double* v, size_t n, double* out, cudaStream_t st) {
    count_launch();
    cudaLaunchConfig_t lc = {};
    lc.gridDim = dim3(kMinmaxBlocks);
    lc.blockDim = dim3(1024);
    lc.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = kMinmaxBlocks;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    lc.attrs = at;
    lc.numAttrs = 1;
    cudaLaunchKernelEx(&lc, k_minmax, v, n, out);
}
void sumsq(const double2* x, size_t n, double* acc, cudaStream_t st) {
    count_launch();
    k_sumsq<<<grid_for(n), 256, 0, st>>>(x, n, acc);
}
void bounds(double kin_max, const double* minmax_dev, const double* eig_dev, int n_eig,
            const double* lanczos, int k, double lm_scale, double* coef, cudaStream_t st) {
    count_launch();
    k_bounds<<<1, 32, 0, st>>>(kin_max, minmax_dev, eig_dev, n_eig, lanczos, k, lm_scale, coef);
}
void norm_guard(const double* nsq, int ndeg, int* status, cudaStream_t st) {
    count_launch();
    k_norm_guard<<<1, 32, 0, st>>>(nsq, ndeg, status);
}
void scale_by_rsqrt(double2* v, size_t n, const double* nsq, cudaStream_t st) {
    count_launch();
    k_scale_by_rsqrt<<<grid_for(n), 256, 0, st>>>(v, n, nsq);
}
void lanczos_a(double2* f, const double2* v, const double2* v0, const double* beta_sq, size_t n,
               double* alpha_acc, cudaStream_t st) {
    count_launch();
    k_lanczos_a<<<grid_for(n), 256, 0, st>>>(f, v, v0, beta_sq, n, alpha_acc);
}
void lanczos_b(double2* f, const double2* v, const double* alpha, size_t n, double* fn_acc,
               cudaStream_t st) {
    count_launch();
    k_lanczos_b<<<grid_for(n), 256, 0, st>>>(f, v, alpha, n, fn_acc);
}
void lanczos_c(const double2* f, double2* v, double2* v0, size_t n, const double* fn,
               cudaStream_t st) {
    count_launch();
    k_lanczos_c<<<grid_for(n), 256, 0, st>>>(f, v, v0, n, fn);
}
void lanczos_store_beta(const double* fn, double* beta, cudaStream_t st) {
    count_launch();
    k_lanczos_store_beta<<<1, 32, 0, st>>>(fn, beta);
}
void pulay_push(const double* rin, const double* rout, double* hr, double* hres, size_t n,
                cudaStream_t st) {
    count_launch();
    k_pulay_push<<<grid_for(n), 256, 0, st>>>(rin, rout, hr, hres, n);
}
void dots(const double* x, const double* const* ys, int m, size_t n, double* out, cudaStream_t st) {
    count_launch();
    k_dots<<<grid_for(n), 256, 0, st>>>(x, ys, m, n, out);
}
void pulay_combine(const double* const* hr, const double* const* hres, int m, const double* c,
                   double alpha, size_t n, double* out, cudaStream_t st) {
    count_launch();
    PulayCoef pc{};
    for (int j = 0; j < m && j < kPulayMax; ++j) pc.c[j] = c[j];
    k_pulay_combine<<<grid_for(n), 256, 0, st>>>(hr, hres, m, pc, alpha, n, out);
}

}  // namespace chfsi
