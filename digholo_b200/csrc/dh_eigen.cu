// FP64 eigenvalues (and the eigenvectors of the smallest and largest) of a
// Hermitian matrix on the GPU, for the power meter: the squared singular
// values of the batch coefficient matrix that digHolo takes from cgesvd
// (svdSingularValues, digHolo.cpp:3021-3055; digHoloPowerMeter
// digHolo.cpp:11012-11062) are the eigenvalues of its FP64 Gram matrix, and
// MDL = s_min^2 / s_max^2 needs only their extremes -- and for its gradient
// the two extreme eigenvectors.
//
// Three phases:
//   1. Householder tridiagonalisation, A = Q T Q^H, Q = H_0 H_1 ... H_{n-2},
//      H_k = I - tau_k v_k v_k^H with v_k[k+1] = 1 (the reflector convention
//      of LAPACK's zlarfg / zhetd2, lower triangle).  The rank-2 update of
//      step k - 1 is applied in the same pass that forms A v_k for step k.
//      Up to n = 304 the matrix stays in the shared memory of one block or of
//      a cluster of eight (k_heev_cluster); beyond, one block of 1024 threads
//      works on it in global memory, L2-resident (k_heev).
//   2. Eigenvalues of the real symmetric tridiagonal T (the reflectors make
//      every off-diagonal real) by Sturm-count bisection, ascending: all of
//      them, or the two extremes with a warp group's count points per pass.
//   3. On request, inverse iteration on T for the smallest and largest
//      eigenvalue (tridiagonal LU with partial pivoting, one thread each),
//      then u = Q z by applying the reflectors in reverse order (one warp
//      each).
// Bound in both kernels: the latency of the n dependent steps, not bytes or
// FLOPs (n = 110 is 0.2 MB and 7 MFLOP).  One 110 x 110 matrix, extremes
// only: 709 us by k_heev, 364 by the cluster with a quotient per Sturm step
// and 256 threads a block, 262 with sturmCount's minors and 128 threads;
// all eigenvalues and two eigenvectors of n = 110 / 240 / 300: 1084 / 4320 /
// 7355 us by k_heev, 848 / 2415 / 3787 by the cluster.
// No block waits on a memory flag; the cluster's barrier is the hardware's.
#include <cuda_runtime.h>

#include <cfloat>
#include <cmath>
#include <cstdio>

#include "dh_host.h"

namespace {

constexpr int NT = 1024;

__device__ __forceinline__ double2 cmulD(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
// conj(a) * b
__device__ __forceinline__ double2 cmulcD(double2 a, double2 b) {
    return make_double2(a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x);
}

// Sum over the block; every thread gets the result.  red holds 33 entries.
__device__ double2 blockSum(double2 v, double2* red) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        v.x += __shfl_xor_sync(0xffffffffu, v.x, o);
        v.y += __shfl_xor_sync(0xffffffffu, v.y, o);
    }
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        double2 w = lane < (int)(blockDim.x >> 5) ? red[lane] : make_double2(0.0, 0.0);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            w.x += __shfl_xor_sync(0xffffffffu, w.x, o);
            w.y += __shfl_xor_sync(0xffffffffu, w.y, o);
        }
        if (lane == 0) red[32] = w;
    }
    __syncthreads();
    const double2 r = red[32];
    __syncthreads();
    return r;
}

__device__ double blockMinMax(double v, double* red, bool isMax) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        const double u = __shfl_xor_sync(0xffffffffu, v, o);
        v = isMax ? fmax(v, u) : fmin(v, u);
    }
    if (lane == 0) red[warp] = v;
    __syncthreads();
    if (warp == 0) {
        double w = lane < (int)(blockDim.x >> 5) ? red[lane] : (isMax ? -DBL_MAX : DBL_MAX);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const double u = __shfl_xor_sync(0xffffffffu, w, o);
            w = isMax ? fmax(w, u) : fmin(w, u);
        }
        if (lane == 0) red[32] = w;
    }
    __syncthreads();
    const double r = red[32];
    __syncthreads();
    return r;
}

// Number of eigenvalues of the tridiagonal (D, E2 = off-diagonal squared,
// scaled to norm <= 1) below x: the sign changes of the leading minors p_i =
// (d_i - x) p_{i-1} - e_{i-1}^2 p_{i-2}, whose ratios are the pivots of
// LAPACK's dstebz and carry the same backward error, with one FMA instead of
// a quotient in the chain.  Both minors are rescaled by a power of two every
// four steps; a minor that vanishes counts as a change (dstebz's pivot
// -pivmin) and goes on as a negligible multiple of its predecessor.
__device__ int sturmCount(const double* D, const double* E2, int n, double x) {
    int cnt = 0;
    double p0 = 1.0, p1 = D[0] - x;   // p_{i-2}, p_{i-1}
    auto settle = [&]() {
        if (p1 == 0.0) {
            p0 = p0 < 0.0 ? -1.0 : 1.0;
            p1 = -1e-140 * p0;
        }
        cnt += (p1 < 0.0) != (p0 < 0.0);
    };
    settle();
    for (int i = 1; i < n; i++) {
        const double p2 = fma(D[i] - x, p1, -E2[i - 1] * p0);
        p0 = p1;
        p1 = p2;
        settle();
        if ((i & 3) == 3) {
            const int e = (__double2hiint(fmax(fabs(p0), fabs(p1))) >> 20) & 0x7ff;
            const double s = __hiloint2double((2046 - min(max(e, 1), 2045)) << 20, 0);
            p0 *= s;
            p1 *= s;
        }
    }
    return cnt;
}

struct HeevArgs {
    double2* G;         // [count][n][n] column-major (element (i, j) at j n + i); overwritten
    int n;
    double* W;          // [count][n] eigenvalues, ascending
    double2* vecs;      // [count][2][n]: eigenvectors of the smallest and largest eigenvalue, or null
    double2* tau;       // [count][n] work
    double* lu;         // [count][2][6 n] work (inverse iteration)
    int extremes;       // 1: only W[0] and W[n-1] (the other entries untouched)
    double* trace;      // [count] sum of the eigenvalues (the tridiagonal's diagonal sum), or null
};

// Phases 2 and 3 on the tridiagonal (D, E, E2) in shared memory, by one block
// of THREADS threads; the reflectors lie in a.G's columns and a.tau.
template <int THREADS>
__device__ void eigenTail(const HeevArgs& a, double* D, const double* E, double* E2) {
    const int n = a.n, t = threadIdx.x;
    double2* A = a.G + (size_t)blockIdx.y * n * n;
    double2* tau = a.tau + (size_t)blockIdx.y * n;
    // ---- 2. eigenvalues by bisection (Gershgorin interval)
    double lo = DBL_MAX, hi = -DBL_MAX;
    for (int i = t; i < n; i += THREADS) {
        const double r = (i > 0 ? fabs(E[i - 1]) : 0.0) + (i + 1 < n ? fabs(E[i]) : 0.0);
        lo = fmin(lo, D[i] - r);
        hi = fmax(hi, D[i] + r);
    }
    __shared__ double redd[33];
    lo = blockMinMax(lo, redd, false);
    hi = blockMinMax(hi, redd, true);
    const double scale = fmax(fabs(lo), fabs(hi));
    // power of two (exact) that brings the interval to order 1, and back
    int ex = 0;
    if (scale > 0.0 && isfinite(scale)) ex = min(max(ilogb(scale) + 1, -1000), 1000);
    const double down = scalbn(1.0, -ex), up = scalbn(1.0, ex);
    lo *= down;
    hi *= down;
    const double tol = scale > 0.0 ? 4.0 * DBL_EPSILON * (scale * down) + 4.0 * DBL_MIN : 0.0;
    lo -= tol;
    hi += tol;
    double* W = a.W + (size_t)blockIdx.y * n;
    if (a.trace && t == 0) {
        double tr = 0.0;
        for (int i = 0; i < n; i++) tr += D[i];
        a.trace[blockIdx.y] = tr;
    }
    __syncthreads();
    for (int i = t; i < n; i += THREADS) {
        const double e = E[i] * down;
        D[i] *= down;
        E2[i] = e * e;
    }
    __syncthreads();
    if (a.extremes) {
        // the smallest and the largest eigenvalue only (what MDL and its
        // gradient use): a group of up to four warps each, one count point a
        // thread but the last, so six or seven bits of the interval per Sturm
        // count; every thread of a group holds the same interval
        constexpr int GW = THREADS >= 256 ? 4 : THREADS / 64;   // warps of a group
        constexpr int GP = 32 * GW;
        static_assert(GW >= 1, "two groups");
        __shared__ int first[2 * GW];
        const int warp = t >> 5, lane = t & 31, grp = warp / GW & 1, p = t % GP;
        const bool active = t < 2 * GP;
        const int m = grp == 0 ? 0 : n - 1;
        double l = lo, h = hi;
        for (int it = 0; it < 100; it++) {
            if (__syncthreads_and(!active || !(h - l > tol))) break;
            const double step = (h - l) * (1.0 / GP);
            const bool above = active && p < GP - 1 && sturmCount(D, E2, n, l + step * (double)(p + 1)) > m;
            const unsigned bits = __ballot_sync(0xffffffffu, above);
            if (active && lane == 0) first[warp] = bits ? 32 * (warp % GW) + __ffs(bits) - 1 : GP - 1;
            __syncthreads();
            if (active) {   // first count point above eigenvalue m
                int f = GP - 1;
                for (int g = 0; g < GW; g++) f = min(f, first[GW * grp + g]);
                const double nh = f < GP - 1 ? l + step * (double)(f + 1) : h;
                const double nl = f > 0 ? l + step * (double)f : l;
                l = nl;
                h = nh;
            }
        }
        if (active && p == 0) W[m] = 0.5 * (l + h) * up;
    } else {
        // quadrisection, four lanes per eigenvalue: lanes 0-2 of a group
        // count at the interval's quarter points, the group keeps the
        // quarter holding eigenvalue m (two bits per Sturm count instead of
        // one).  Every lane of a group holds the same interval, so the
        // group's trip count is uniform.
        const int lane = t & 31, q4 = t & 3;
        const unsigned gmask = 0xFu << (lane & ~3);
        for (int m = t >> 2; m < n; m += THREADS / 4) {
            double l = lo, h = hi;
            for (int it = 0; it < 200 && h - l > tol; it++) {
                const double step = 0.25 * (h - l);
                const double x = l + step * (double)(q4 + 1);
                const bool above = q4 < 3 && sturmCount(D, E2, n, x) > m;
                const unsigned bits = (__ballot_sync(gmask, above) >> (lane & ~3)) & 7u;
                const int f = bits ? __ffs(bits) - 1 : 3;   // first quarter point above eigenvalue m
                const double nh = f < 3 ? l + step * (double)(f + 1) : h;
                const double nl = f > 0 ? l + step * (double)f : l;
                l = nl;
                h = nh;
            }
            if (q4 == 0) W[m] = 0.5 * (l + h) * up;
        }
    }
    if (!a.vecs) return;
    __syncthreads();

    // ---- 3. eigenvectors of the smallest and largest eigenvalue
    const int warp = t >> 5, lane = t & 31;
    if (warp >= 2) return;
    const double sigma = W[warp == 0 ? 0 : n - 1];
    double2* u = a.vecs + ((size_t)blockIdx.y * 2 + warp) * n;
    double* lu = a.lu + ((size_t)blockIdx.y * 2 + warp) * 6 * n;
    double* dl = lu;
    double* dd = lu + n;
    double* du = lu + 2 * n;
    double* du2 = lu + 3 * n;
    double* z = lu + 4 * n;
    int* piv = reinterpret_cast<int*>(lu + 5 * n);
    if (lane == 0) {
        const double tiny = DBL_EPSILON * fmax(scale, DBL_MIN);
        for (int i = 0; i < n; i++) {
            dd[i] = D[i] * up - sigma;
            if (i + 1 < n) { dl[i] = E[i]; du[i] = E[i]; }
            du2[i] = 0.0;
        }
        // LU with partial pivoting (the elimination of LAPACK's dgttrf)
        for (int i = 0; i + 1 < n; i++) {
            if (fabs(dd[i]) >= fabs(dl[i])) {
                piv[i] = i;
                if (dd[i] == 0.0) dd[i] = tiny;
                const double f = dl[i] / dd[i];
                dl[i] = f;
                dd[i + 1] -= f * du[i];
            } else {
                piv[i] = i + 1;
                const double f = dd[i] / dl[i];
                dd[i] = dl[i];
                dl[i] = f;
                const double tmp = du[i];
                du[i] = dd[i + 1];
                dd[i + 1] = tmp - f * dd[i + 1];
                if (i + 2 < n) {
                    du2[i] = du[i + 1];
                    du[i + 1] = -f * du[i + 1];
                }
            }
        }
        if (dd[n - 1] == 0.0) dd[n - 1] = tiny;
        for (int i = 0; i < n; i++) z[i] = 1.0 + 0.5 * (double)((i * 7919) % 97) / 97.0;
        for (int rep = 0; rep < 3; rep++) {
            for (int i = 0; i + 1 < n; i++) {
                if (piv[i] == i) {
                    z[i + 1] -= dl[i] * z[i];
                } else {
                    const double tmp = z[i];
                    z[i] = z[i + 1];
                    z[i + 1] = tmp - dl[i] * z[i];
                }
            }
            z[n - 1] /= dd[n - 1];
            if (n > 1) z[n - 2] = (z[n - 2] - du[n - 2] * z[n - 1]) / dd[n - 2];
            for (int i = n - 3; i >= 0; i--) z[i] = (z[i] - du[i] * z[i + 1] - du2[i] * z[i + 2]) / dd[i];
            double nrm = 0.0;
            for (int i = 0; i < n; i++) nrm = fmax(nrm, fabs(z[i]));
            if (!(nrm > 0.0) || !isfinite(nrm)) {
                for (int i = 0; i < n; i++) z[i] = (i == (warp == 0 ? 0 : n - 1)) ? 1.0 : 0.0;
                break;
            }
            for (int i = 0; i < n; i++) z[i] /= nrm;
        }
    }
    __syncwarp();
    // u = H_0 H_1 ... H_{n-2} z, normalised
    for (int i = lane; i < n; i += 32) u[i] = make_double2(z[i], 0.0);
    __syncwarp();
    for (int k = n - 2; k >= 0; k--) {
        const double2* col = A + (size_t)k * n;
        double2 d = make_double2(0.0, 0.0);
        for (int i = k + 1 + lane; i < n; i += 32) {
            const double2 v = i == k + 1 ? make_double2(1.0, 0.0) : col[i];
            const double2 p = cmulcD(v, u[i]);
            d.x += p.x;
            d.y += p.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            d.x += __shfl_xor_sync(0xffffffffu, d.x, o);
            d.y += __shfl_xor_sync(0xffffffffu, d.y, o);
        }
        const double2 td = cmulD(tau[k], d);
        __syncwarp();
        for (int i = k + 1 + lane; i < n; i += 32) {
            const double2 v = i == k + 1 ? make_double2(1.0, 0.0) : col[i];
            const double2 p = cmulD(v, td);
            u[i].x -= p.x;
            u[i].y -= p.y;
        }
        __syncwarp();
    }
    double nn = 0.0;
    for (int i = lane; i < n; i += 32) nn += u[i].x * u[i].x + u[i].y * u[i].y;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nn += __shfl_xor_sync(0xffffffffu, nn, o);
    const double inv = nn > 0.0 ? 1.0 / sqrt(nn) : 0.0;
    for (int i = lane; i < n; i += 32) u[i] = make_double2(u[i].x * inv, u[i].y * inv);
}

__global__ void __launch_bounds__(NT, 1) k_heev(HeevArgs a) {
    extern __shared__ double2 smem[];
    const int n = a.n, t = threadIdx.x;
    double2* A = a.G + (size_t)blockIdx.y * n * n;
    double2* tau = a.tau + (size_t)blockIdx.y * n;
    double2* vk = smem;             // reflector of this step, by row index
    double2* vp = vk + n;           // reflector of the previous step
    double2* xp = vp + n;           // w of the previous step (A22 -= v w^H + w v^H)
    double2* y = xp + n;            // A22 v
    double2* part = y + n;          // NT partial sums
    double* D = reinterpret_cast<double*>(part + NT);
    double* E = D + n;
    double* E2 = E + n;
    __shared__ double2 red[33];
    __shared__ double2 scal[2];

    // ---- 1. tridiagonalisation
    bool havePrev = false;
    for (int k = 0; k + 1 < n; k++) {
        const int L = n - k - 1;
        double2* col = A + (size_t)k * n;
        // (a) the previous update on column k, rows k..n-1
        if (havePrev) {
            for (int i = k + t; i < n; i += NT) {
                const double2 u1 = cmulD(vp[i], make_double2(xp[k].x, -xp[k].y));
                const double2 u2 = cmulD(xp[i], make_double2(vp[k].x, -vp[k].y));
                double2 c = col[i];
                c.x -= u1.x + u2.x;
                c.y -= u1.y + u2.y;
                col[i] = c;
            }
        }
        __syncthreads();
        // (b) reflector for col[k+1 .. n-1]: alpha = col[k+1], x = col[k+2 ..]
        double2 s = make_double2(0.0, 0.0);
        for (int i = k + 2 + t; i < n; i += NT) s.x += col[i].x * col[i].x + col[i].y * col[i].y;
        s = blockSum(s, red);
        if (t == 0) {
            D[k] = col[k].x;
            const double2 alpha = col[k + 1];
            const double xnorm2 = s.x;
            double beta, tr, ti;
            double2 sc;
            if (xnorm2 == 0.0 && alpha.y == 0.0) {
                beta = alpha.x;
                tr = 0.0; ti = 0.0;
                sc = make_double2(0.0, 0.0);
            } else {
                const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2);
                beta = alpha.x >= 0.0 ? -nrm : nrm;
                tr = (beta - alpha.x) / beta;
                ti = -alpha.y / beta;
                // 1 / (alpha - beta)
                const double dr = alpha.x - beta, di = alpha.y;
                const double den = dr * dr + di * di;
                sc = make_double2(dr / den, -di / den);
            }
            E[k] = beta;
            E2[k] = beta * beta;
            tau[k] = make_double2(tr, ti);
            scal[0] = make_double2(tr, ti);
            scal[1] = sc;
        }
        __syncthreads();
        const double2 tk = scal[0], sc = scal[1];
        for (int i = k + 1 + t; i < n; i += NT) {
            double2 v;
            if (i == k + 1) {
                v = make_double2(1.0, 0.0);
            } else {
                v = cmulD(col[i], sc);
                col[i] = v;   // kept for the back-transformation
            }
            vk[i] = v;
        }
        __syncthreads();
        // (c) the previous update on the trailing block (rows, columns >= k+1)
        // fused with y = A22 v_k
        const int Lr = min(((L + 31) / 32) * 32, NT);
        const int groups = NT / Lr;
        for (int r0 = 0; r0 < L; r0 += Lr) {
            const int ri = r0 + (t % Lr), g = t / Lr;
            double2 acc = make_double2(0.0, 0.0);
            if (ri < L && g < groups) {
                const int i = k + 1 + ri;
                const double2 vpi = havePrev ? vp[i] : make_double2(0.0, 0.0);
                const double2 xpi = havePrev ? xp[i] : make_double2(0.0, 0.0);
                // CB columns per pass, their loads issued before any store:
                // the trailing block lives in L2, and one load in flight per
                // thread would leave each pass waiting on L2 latency CB times
                constexpr int CB = 4;
                for (int j0 = k + 1 + g; j0 < n; j0 += CB * groups) {
                    double2 e[CB];
#pragma unroll
                    for (int q = 0; q < CB; q++) {
                        const int j = j0 + q * groups;
                        e[q] = j < n ? A[(size_t)j * n + i] : make_double2(0.0, 0.0);
                    }
#pragma unroll
                    for (int q = 0; q < CB; q++) {
                        const int j = j0 + q * groups;
                        if (j >= n) break;
                        if (havePrev) {
                            const double2 u1 = cmulD(vpi, make_double2(xp[j].x, -xp[j].y));
                            const double2 u2 = cmulD(xpi, make_double2(vp[j].x, -vp[j].y));
                            e[q].x -= u1.x + u2.x;
                            e[q].y -= u1.y + u2.y;
                            A[(size_t)j * n + i] = e[q];
                        }
                        const double2 p = cmulD(e[q], vk[j]);
                        acc.x += p.x;
                        acc.y += p.y;
                    }
                }
            }
            part[t] = acc;
            __syncthreads();
            if (t < Lr && r0 + t < L) {
                double2 sum = make_double2(0.0, 0.0);
                for (int gg = 0; gg < groups; gg++) {
                    sum.x += part[gg * Lr + t].x;
                    sum.y += part[gg * Lr + t].y;
                }
                y[k + 1 + r0 + t] = sum;
            }
            __syncthreads();
        }
        // (d) x = tau y, alpha = -tau (x^H v) / 2, w = x + alpha v
        double2 d = make_double2(0.0, 0.0);
        for (int i = k + 1 + t; i < n; i += NT) {
            const double2 x = cmulD(tk, y[i]);
            y[i] = x;
            const double2 p = cmulcD(x, vk[i]);
            d.x += p.x;
            d.y += p.y;
        }
        d = blockSum(d, red);
        const double2 al = cmulD(make_double2(-0.5 * tk.x, -0.5 * tk.y), d);
        for (int i = k + 1 + t; i < n; i += NT) {
            const double2 w = cmulD(al, vk[i]);
            xp[i] = make_double2(y[i].x + w.x, y[i].y + w.y);
            vp[i] = vk[i];
        }
        havePrev = true;
        __syncthreads();
    }
    if (t == 0) {
        const int k = n - 1;
        double2 c = A[(size_t)k * n + k];
        if (havePrev) {
            const double2 u1 = cmulD(vp[k], make_double2(xp[k].x, -xp[k].y));
            const double2 u2 = cmulD(xp[k], make_double2(vp[k].x, -vp[k].y));
            c.x -= u1.x + u2.x;
        }
        D[k] = c.x;
        E[k] = 0.0;
        E2[k] = 0.0;
    }
    __syncthreads();

    eigenTail<NT>(a, D, E, E2);
}

// ---------------------------------------------------------------- in shared memory, by a cluster
// The same solver for matrices whose rows fit the shared memory of a cluster
// of CC blocks (CC = 1 or 8; n up to 304).  Row i lives on block i mod CC, both
// triangles, and stays there; a lane holds columns lane + 32 q of the vectors
// in registers.  Per step, two phases and one cluster barrier:
//   M  every warp updates its rows i > k with the previous reflector's
//      (v, w), forms y_i = (A v_k)_i and sends it to every block; the owner
//      of row k + 1 sends that row too (the next column, conjugated);
//   S  every warp, redundantly and in registers, forms w_k, applies the
//      update to the received row and builds reflector k + 1 from it, so that
//      nothing is exchanged between S and the next M.
// y and the row are double-buffered by the step's parity.  Bound: the latency
// of S (two warp sums, a square root and two quotients in FP64) and of the
// cluster barrier.

struct HeevClSmem {
    size_t y, row, vw, d, rows, total;
};
__host__ __device__ inline HeevClSmem heevClSmem(int n, int cc) {
    HeevClSmem s;
    s.y = 0;                                         // [2][n]
    s.row = s.y + sizeof(double2) * 2 * n;           // [2][n]
    s.vw = s.row + sizeof(double2) * 2 * n;          // v, w of the last applied reflector [2][n]
    s.d = s.vw + sizeof(double2) * 2 * n;            // D, E, E2
    s.rows = s.d + (sizeof(double) * 3 * n + 15) / 16 * 16;
    s.total = s.rows + sizeof(double2) * (size_t)((n + cc - 1) / cc) * n;
    return s;
}

__device__ __forceinline__ unsigned clusterRank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
// `p` of this block's shared memory at the same place in block `rank`'s.
__device__ __forceinline__ unsigned remoteShared(const void* p, unsigned rank) {
    unsigned a = (unsigned)__cvta_generic_to_shared(p), r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
    return r;
}
__device__ __forceinline__ void storeRemote(unsigned addr, double v) {
    asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(addr), "d"(v) : "memory");
}
__device__ __forceinline__ void storeRemote(unsigned addr, double2 v) {
    asm volatile("st.shared::cluster.v2.f64 [%0], {%1, %2};" ::"r"(addr), "d"(v.x), "d"(v.y) : "memory");
}
__device__ __forceinline__ void clusterBarrier() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ double warpSum(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

template <int Q, int CC, int CNT>
__global__ void __launch_bounds__(CNT, 1) k_heev_cluster(HeevArgs a) {
    extern __shared__ double2 smem[];
    const int n = a.n, t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int rank = CC > 1 ? (int)clusterRank() : 0;
    double2* G = a.G + (size_t)blockIdx.y * n * n;
    double2* tau = a.tau + (size_t)blockIdx.y * n;
    const HeevClSmem L = heevClSmem(n, CC);
    unsigned char* sm = reinterpret_cast<unsigned char*>(smem);
    double2* ybuf = reinterpret_cast<double2*>(sm + L.y);
    double2* rbuf = reinterpret_cast<double2*>(sm + L.row);
    double2* sv = reinterpret_cast<double2*>(sm + L.vw);
    double2* sw = sv + n;
    double* D = reinterpret_cast<double*>(sm + L.d);
    double* E = D + n;
    double* E2 = E + n;
    double2* rows = reinterpret_cast<double2*>(sm + L.rows);
    const int nl = (n - rank + CC - 1) / CC;   // rows of this block
    auto barrier = [&]() {
        if (CC > 1) clusterBarrier();
        else __syncthreads();
    };
    // row i = conj(column i)
    for (int li = warp; li < nl; li += CNT / 32) {
        const int i = rank + CC * li;
        for (int j = lane; j < n; j += 32) {
            const double2 g = G[(size_t)i * n + j];
            rows[(size_t)li * n + j] = make_double2(g.x, -g.y);
        }
    }
    for (int i = t; i < 2 * n; i += CNT) sv[i] = make_double2(0.0, 0.0);
    double2 v[Q], vp[Q], wp[Q], c[Q];   // this reflector; the applied one and its w; the next column
#pragma unroll
    for (int q = 0; q < Q; q++) {
        const int j = lane + 32 * q;
        vp[q] = wp[q] = v[q] = make_double2(0.0, 0.0);
        c[q] = j < n ? G[j] : make_double2(0.0, 0.0);
    }
    barrier();   // the matrix is read before the reflectors overwrite it
    double2 tk = make_double2(0.0, 0.0);
    // reflector k of the column c (rows k ..): v, tau, D, E
    auto reflect = [&](int k) {
        double2 alpha = make_double2(0.0, 0.0);
        double x2 = 0.0, diag = 0.0;
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int i = lane + 32 * q;
            if (i == k + 1) alpha = c[q];
            if (i == k) diag = c[q].x;
            if (i > k + 1) x2 += c[q].x * c[q].x + c[q].y * c[q].y;
        }
        const double xnorm2 = warpSum(x2);
        alpha.x = __shfl_sync(0xffffffffu, alpha.x, (k + 1) & 31);
        alpha.y = __shfl_sync(0xffffffffu, alpha.y, (k + 1) & 31);
        diag = __shfl_sync(0xffffffffu, diag, k & 31);
        double beta = alpha.x;
        double2 sc = make_double2(0.0, 0.0);
        tk = make_double2(0.0, 0.0);
        if (xnorm2 != 0.0 || alpha.y != 0.0) {
            const double nrm = sqrt(alpha.x * alpha.x + alpha.y * alpha.y + xnorm2);
            beta = alpha.x >= 0.0 ? -nrm : nrm;
            // 1 / (alpha - beta)
            const double dr = alpha.x - beta, di = alpha.y;
            const double rb = 1.0 / beta, rden = 1.0 / (dr * dr + di * di);
            tk = make_double2(-dr * rb, -di * rb);
            sc = make_double2(dr * rden, -di * rden);
        }
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int i = lane + 32 * q;
            v[q] = i == k + 1 ? make_double2(1.0, 0.0) : (i > k + 1 && i < n ? cmulD(c[q], sc) : make_double2(0.0, 0.0));
            if (a.vecs && rank == 0 && warp == 0 && i > k + 1 && i < n) G[(size_t)k * n + i] = v[q];
        }
        if (rank == 0 && t == 0) {
            D[k] = diag;
            E[k] = beta;
            E2[k] = beta * beta;
            tau[k] = tk;
        }
    };
    reflect(0);
    for (int k = 0; k + 1 < n; k++) {
        double2* y = ybuf + (k & 1) * n;
        double2* rk = rbuf + (k & 1) * n;
        // ---- M: two rows at a time
        const int li0 = k + 1 > rank ? (k + 1 - rank + CC - 1) / CC : 0;
        for (int li = li0 + 2 * warp; li < nl; li += 2 * (CNT / 32)) {
            const bool two = li + 1 < nl;
            const int i0 = rank + CC * li, i1 = two ? i0 + CC : i0;
            double2* r0 = rows + (size_t)li * n;
            double2* r1 = rows + (size_t)(two ? li + 1 : li) * n;
            const double2 v0 = sv[i0], w0 = sw[i0], v1 = sv[i1], w1 = sw[i1];
            double2 s0 = make_double2(0.0, 0.0), s1 = s0;
#pragma unroll
            for (int q = 0; q < Q; q++) {
                if (32 * q + 31 <= k || 32 * q >= n) continue;   // warp-uniform
                const int j = lane + 32 * q;
                if (j < n) {
                    double2 e = r0[j], f = r1[j];
                    const double2 a1 = vp[q], b1 = wp[q];
                    e.x -= v0.x * b1.x + v0.y * b1.y + w0.x * a1.x + w0.y * a1.y;
                    e.y -= v0.y * b1.x - v0.x * b1.y + w0.y * a1.x - w0.x * a1.y;
                    f.x -= v1.x * b1.x + v1.y * b1.y + w1.x * a1.x + w1.y * a1.y;
                    f.y -= v1.y * b1.x - v1.x * b1.y + w1.y * a1.x - w1.x * a1.y;
                    r0[j] = e;
                    if (two) r1[j] = f;
                    s0.x += e.x * v[q].x - e.y * v[q].y;
                    s0.y += e.x * v[q].y + e.y * v[q].x;
                    s1.x += f.x * v[q].x - f.y * v[q].y;
                    s1.y += f.x * v[q].y + f.y * v[q].x;
                    if (i0 == k + 1 || i1 == k + 1) {   // the next column's row, to every block (i1 only as i0's copy)
                        const double2 o = i0 == k + 1 ? e : f;
                        if (CC == 1) {
                            rk[j] = o;
                        } else {
#pragma unroll
                            for (int r = 0; r < CC; r++) storeRemote(remoteShared(rk + j, r), o);
                        }
                    }
                }
            }
            // four sums over the warp: lane group l / 8 ends with (row l / 16, part (l / 8) % 2)
            const bool up = lane & 16, im = lane & 8;
            const double2 keep = up ? s1 : s0, send = up ? s0 : s1;
            const double kx = keep.x + __shfl_xor_sync(0xffffffffu, send.x, 16);
            const double ky = keep.y + __shfl_xor_sync(0xffffffffu, send.y, 16);
            double z = (im ? ky : kx) + __shfl_xor_sync(0xffffffffu, im ? kx : ky, 8);
#pragma unroll
            for (int o = 4; o > 0; o >>= 1) z += __shfl_xor_sync(0xffffffffu, z, o);
            if (!up || two) {
                double* at = reinterpret_cast<double*>(y + (up ? i1 : i0)) + (im ? 1 : 0);
                if (CC == 1) {
                    if ((lane & 7) == 0) *at = z;
                } else {
                    storeRemote(remoteShared(at, lane & 7), z);   // one lane per block
                }
            }
        }
        barrier();
        // ---- S: x = tau y, w = x - tau (x^H v) v / 2, the next column and its reflector
        double2 x[Q];
        double dx = 0.0, dy = 0.0;
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int i = lane + 32 * q;
            x[q] = i > k && i < n ? cmulD(tk, y[i]) : make_double2(0.0, 0.0);
            const double2 p = cmulcD(x[q], v[q]);
            dx += p.x;
            dy += p.y;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            dx += __shfl_xor_sync(0xffffffffu, dx, o);
            dy += __shfl_xor_sync(0xffffffffu, dy, o);
        }
        const double2 al = cmulD(make_double2(-0.5 * tk.x, -0.5 * tk.y), make_double2(dx, dy));
        double2 w1 = make_double2(0.0, 0.0);
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int i = lane + 32 * q;
            const double2 s = cmulD(al, v[q]);
            vp[q] = v[q];
            wp[q] = make_double2(x[q].x + s.x, x[q].y + s.y);
            if (i == k + 1) w1 = wp[q];
            if (i < n) {   // every warp writes the same values; read in the next M, rewritten after its barrier
                sv[i] = vp[q];
                sw[i] = wp[q];
            }
        }
        w1.x = __shfl_sync(0xffffffffu, w1.x, (k + 1) & 31);
        w1.y = __shfl_sync(0xffffffffu, w1.y, (k + 1) & 31);
#pragma unroll
        for (int q = 0; q < Q; q++) {
            const int i = lane + 32 * q;
            c[q] = make_double2(0.0, 0.0);
            if (i > k && i < n) {
                const double2 r = rk[i];   // row k + 1: the column's conjugate; v_{k+1} = 1
                c[q].x = r.x - (vp[q].x * w1.x + vp[q].y * w1.y + wp[q].x);
                c[q].y = -r.y - (vp[q].y * w1.x - vp[q].x * w1.y + wp[q].y);
            }
        }
        __syncwarp();
        if (k + 2 < n) {
            reflect(k + 1);
        } else if (rank == 0 && warp == 0) {
#pragma unroll
            for (int q = 0; q < Q; q++)
                if (lane + 32 * q == n - 1) D[n - 1] = c[q].x;
            if (lane == 0) {
                E[n - 1] = 0.0;
                E2[n - 1] = 0.0;
            }
        }
    }
    if (rank != 0) return;   // nothing is sent after the last barrier
    __syncthreads();
    eigenTail<CNT>(a, D, E, E2);
}

template <int Q, int CC, int CNT>
cudaError_t launchHeevCluster(const HeevArgs& a, int count, cudaStream_t s) {
    const size_t smem = heevClSmem(a.n, CC).total;
    cudaError_t e = dh::setSmemOnce(reinterpret_cast<const void*>(k_heev_cluster<Q, CC, CNT>), (int)smem);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(CC, count);
    cfg.blockDim = dim3(CNT);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = CC;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_heev_cluster<Q, CC, CNT>, a);
}

// Shared memory holds the rows: of one block up to n = 115, of eight up to 304
// (216 KB each).  One block up to 64; beyond, eight are faster also where one
// would do (metrics of 200 and 256 frames, n = 72 / 90 / 110: 237 / 279 / 354
// us against 287 / 358 / 491 by one block).  128 threads a block up to n = 128,
// where the phase every warp repeats is the longer one (metrics of 256 frames,
// n = 110: 480 us against 493 with 256 threads, when the host's part still
// followed the solver's); 256 beyond, where the rows are (n = 240: 2415 us
// against 3148 with 128 and 2860 with 512).
cudaError_t launchHeevFits(const HeevArgs& a, int count, cudaStream_t s) {
    const int n = a.n;
    if (n < 2 || n > 304 || count > 65535) return cudaErrorNotSupported;
    if (n <= 64) return launchHeevCluster<2, 1, 256>(a, count, s);
    if (n <= 128) return launchHeevCluster<4, 8, 128>(a, count, s);
    if (n <= 256) return launchHeevCluster<8, 8, 256>(a, count, s);
    return launchHeevCluster<10, 8, 256>(a, count, s);
}

size_t heevSmem(int n) { return sizeof(double2) * (4 * (size_t)n + NT) + sizeof(double) * 3 * (size_t)n; }

}  // namespace

// Work buffers of the eigen solver, grown on demand and owned by the caller.
struct DhEigen {
    void* work = nullptr;
    size_t bytes = 0;
};

static int ensureWork(DhEigen& e, size_t need) {
    if (need <= e.bytes && e.work) return 0;
    if (e.work) cudaFree(e.work);
    e.work = nullptr;
    e.bytes = 0;
    if (cudaMalloc(&e.work, need) != cudaSuccess) return 1;
    e.bytes = need;
    return 0;
}

// Largest matrix the solvers take (k_heev's shared memory).
int dh_eigen_max_n() { return 2048; }

// `count` Hermitian n x n matrices G (column-major, consecutive, overwritten):
// eigenvalues ascending into W[count][n]; with vecs non-null the unit
// eigenvectors of the smallest and the largest eigenvalue into
// vecs[count][2][n] (complex double).
int dh_eigen_solve(DhEigen& e, void* G, int n, int count, double* W, void* vecs, cudaStream_t s, int extremes = 0,
                   double* trace = nullptr) {
    if (n < 1 || n > dh_eigen_max_n() || count < 1) return 2;
    const size_t need = (size_t)count * n * sizeof(double2) + (size_t)count * 2 * 6 * n * sizeof(double);
    if (ensureWork(e, need)) return 3;
    HeevArgs a;
    a.G = static_cast<double2*>(G);
    a.n = n;
    a.W = W;
    a.vecs = static_cast<double2*>(vecs);
    a.tau = static_cast<double2*>(e.work);
    a.lu = reinterpret_cast<double*>(static_cast<char*>(e.work) + (size_t)count * n * sizeof(double2));
    a.extremes = extremes;
    a.trace = trace;
    {
        const cudaError_t fe = launchHeevFits(a, count, s);
        if (fe == cudaSuccess) return 0;
        if (fe != cudaErrorNotSupported) return 5;
    }
    const size_t smem = heevSmem(n);
    static size_t smemSet = 0;
    if (smem > 48 * 1024 && smem > smemSet) {
        if (cudaFuncSetAttribute(k_heev, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return 4;
        smemSet = smem;
    }
    k_heev<<<dim3(1, count), NT, smem, s>>>(a);
    return cudaGetLastError() == cudaSuccess ? 0 : 5;
}

int dh_eigen_values(DhEigen& e, void* G, int n, double* W, cudaStream_t s) {
    return dh_eigen_solve(e, G, n, 1, W, nullptr, s);
}

// The smallest and largest eigenvalue (W[0], W[n-1]; the other entries of W
// untouched), with vecs non-null their eigenvectors, and the eigenvalue sum.
int dh_eigen_extremes(DhEigen& e, void* G, int n, int count, double* W, void* vecs, double* trace, cudaStream_t s) {
    return dh_eigen_solve(e, G, n, count, W, vecs, s, 1, trace);
}

DhEigen* dh_eigen_create() { return new DhEigen(); }
void dh_eigen_destroy(DhEigen* e) {
    if (e) {
        if (e->work) cudaFree(e->work);
        delete e;
    }
}

extern "C" {

// Eigenvalues of one Hermitian n x n matrix given in host memory
// (column-major complex double, interleaved re/im), ascending into W (host);
// with vecs non-null the unit eigenvectors of the smallest and largest
// eigenvalue into vecs[2][n] complex (host).  A utility around the power
// meter's solver; runs on the current device and waits for it.
// No counterpart in the reference (its power meter calls LAPACK cgesvd).
int digHoloB200EigenHermitian(int n, const double* G, double* W, double* vecs) {
    if (n < 1 || n > dh_eigen_max_n()) return 5;   // DIGHOLO_ERROR_INVALIDDIMENSION
    if (!G || !W) return 3;                         // DIGHOLO_ERROR_NULLPOINTER
    DhEigen e;
    void* dG = nullptr;
    double* dW = nullptr;
    void* dV = nullptr;
    const size_t gb = (size_t)n * n * sizeof(double2);
    int rc = 0;
    if (cudaMalloc(&dG, gb) != cudaSuccess || cudaMalloc(&dW, n * sizeof(double)) != cudaSuccess ||
        (vecs && cudaMalloc(&dV, 2 * (size_t)n * sizeof(double2)) != cudaSuccess)) {
        rc = 9;                                     // DIGHOLO_ERROR_MEMORYALLOCATION
    } else if (cudaMemcpy(dG, G, gb, cudaMemcpyHostToDevice) != cudaSuccess ||
               dh_eigen_solve(e, dG, n, 1, dW, dV, 0) != 0 || cudaDeviceSynchronize() != cudaSuccess ||
               cudaMemcpy(W, dW, n * sizeof(double), cudaMemcpyDeviceToHost) != cudaSuccess ||
               (vecs && cudaMemcpy(vecs, dV, 2 * (size_t)n * sizeof(double2), cudaMemcpyDeviceToHost) != cudaSuccess)) {
        rc = 1;
    }
    if (dG) cudaFree(dG);
    if (dW) cudaFree(dW);
    if (dV) cudaFree(dV);
    if (e.work) cudaFree(e.work);
    return rc;
}

}  // extern "C"
