// Adjoint of the batch path for gradient-driven AutoAlign: the gradient of
// the captured power S = sum |c_mn|^2 (IL = 10 log10 S + const, the power
// meter's insertion loss, digHolo.cpp:3105-3143 and 11012-11062) with
// respect to each polarisation's beam centre, tilt, defocus and basis waist,
// with the Fourier-window selection held fixed.
//
// With V = -conj(A R) the tilt-removed field (A the reconstructed field, R
// the reference wave of digHolo.cpp:10386-10504, phase
//   phi(x, y) = (-k0 tx + offx) x + bcx (-k0 tx) + focal x^2 + (same in y),
//   focal = -pi D / lambda),
// and c_mn = sum_xy Hx_m(x) Hy_n(y) V(x, y) (the separable overlap,
// digHolo.cpp:2149-2341, in float), dS = 2 Re sum_mn conj(c_mn) dc_mn
//   = 2 Re sum_xy Abar dV + 2 Re sum_xy Abar_w dw V,
// Abar = sum_mn conj(c_mn) Hx_m Hy_n (the adjoint field) and
// Abar_w = sum_mn conj(c_mn) d(Hx_m Hy_n)/dw.  The tangents of V are
//   dV/dtx = V i k0 u (x + bcx),   dV/dty = V i k0 u (y + bcy)   (u = pi/180),
//   dV/dD  = V i (pi / lambda) (x^2 + y^2),
//   dV/dbcx = -conj(A_x R) + V i k0 u tx,  A_x the field of the window times
//             i kx (the beam-centre phase of digHoloCopyWindow, digHolo.cpp:1955-2035),
// and for the waist the Hermite-Gaussian ladder relation
//   dpsi_m/dw = -(1 / 2w) (sqrt(m (m-1)) psi_{m-2} - sqrt((m+1)(m+2)) psi_{m+2}).
// Per-field partial sums of Re sum conj(c) dc for the six parameters and the
// field's sum |c|^2, from the Fourier windows where the inverse stage is
// separable (k_align_grad_window), else from the pixels of V, Vx and Vy, one
// block per (frame, polarisation) field.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "dh_common.cuh"
#include "dh_f32x2.cuh"
#include "dh_grad.h"
#include "dh_host.h"

using namespace dh;


// Window of the beam-centre derivatives: Wx = i kx W, Wy = i ky W.
__global__ void k_window_deriv(const float2* __restrict__ W, const float* __restrict__ kxw, const float* __restrict__ kyw,
                               int w, int h, int polCount, int units, float2* __restrict__ Wx, float2* __restrict__ Wy) {
    const size_t total = (size_t)units * w * h;
    for (size_t e = blockIdx.x * (size_t)blockDim.x + threadIdx.x; e < total; e += (size_t)gridDim.x * blockDim.x) {
        const size_t unit = e / ((size_t)w * h);
        const int rem = (int)(e - unit * w * h);
        const int j = rem / w, c = rem - j * w;
        const int pol = (int)(unit % polCount);
        const float2 v = W[e];
        const float kx = kxw[pol * w + c], ky = kyw[pol * h + j];
        Wx[e] = make_float2(-kx * v.y, kx * v.x);
        Wy[e] = make_float2(-ky * v.y, ky * v.x);
    }
}

// blockDim.x = 256; shared: U, Uw [G][ny] complex, hx/hy derivative rows.
__global__ void __launch_bounds__(256) k_align_grad(DhGradParams p) {
    extern __shared__ float2 sg[];
    const int unit = blockIdx.x;
    const int P = p.polCount, G = p.G, M = p.M, nx = p.nx, ny = p.ny;
    const int pol = unit % P, frame = unit / P;
    const int GE = G + 2;
    float2* cc = sg;                                   // [M] conj(c)
    float2* U = cc + M;                                // [G][ny]  sum_n conj(c_mn) Hy_n(y)
    float2* Uw = U + (size_t)G * ny;                   // [G][ny]  sum_n conj(c_mn) Hy'_n(y)
    float* dhx = reinterpret_cast<float*>(Uw + (size_t)G * ny);   // [G][nx] Hx'_m
    float* dhy = dhx + (size_t)G * nx;                              // [G][ny] Hy'_n
    float* red = dhy + (size_t)G * ny;                              // [8 warps][7]
    const float* hxp = p.hx + (size_t)pol * GE * nx;
    const float* hyp = p.hy + (size_t)pol * GE * ny;
    const float w0 = p.waist[pol];
    const int tid = threadIdx.x;

    float spow = 0.f;   // captured power of this field
    for (int mode = tid; mode < M; mode += blockDim.x) {
        const size_t ci = (size_t)frame * P * M + (size_t)pol * M + mode;
        const float2 c = p.coefs[ci];
        cc[mode] = p.weights ? p.weights[ci] : make_float2(c.x, -c.y);
        spow = fmaf(c.x, c.x, fmaf(c.y, c.y, spow));
    }
    // ladder derivatives of the modes with respect to the waist
    for (int e = tid; e < G * nx; e += blockDim.x) {
        const int m = e / nx, x = e - m * nx;
        float v = 0.f;
        if (m >= 2) v += sqrtf((float)(m * (m - 1))) * hxp[(m - 2) * nx + x];
        v -= sqrtf((float)((m + 1) * (m + 2))) * hxp[(m + 2) * nx + x];
        dhx[e] = -v / (2.0f * w0);
    }
    for (int e = tid; e < G * ny; e += blockDim.x) {
        const int n = e / ny, y = e - n * ny;
        float v = 0.f;
        if (n >= 2) v += sqrtf((float)(n * (n - 1))) * hyp[(n - 2) * ny + y];
        v -= sqrtf((float)((n + 1) * (n + 2))) * hyp[(n + 2) * ny + y];
        dhy[e] = -v / (2.0f * w0);
    }
    __syncthreads();
    // U[m][y] = sum_n conj(c_mn) Hy_n(y) over the modes m + n < G (digHolo.cpp:1245-1265 order)
    for (int e = tid; e < G * ny; e += blockDim.x) {
        const int m = e / ny, y = e - m * ny;
        float2 u = make_float2(0.f, 0.f), uw = make_float2(0.f, 0.f);
        for (int n = 0; m + n < G; n++) {
            const int g = m + n;
            const float2 c = cc[g * (g + 1) / 2 + n];
            const float hv = hyp[n * ny + y], dv = dhy[n * ny + y];
            u.x = fmaf(c.x, hv, u.x); u.y = fmaf(c.y, hv, u.y);
            uw.x = fmaf(c.x, dv, uw.x); uw.y = fmaf(c.y, dv, uw.y);
        }
        U[e] = u;
        Uw[e] = uw;
    }
    __syncthreads();

    const float2* Vp = p.V + (size_t)unit * nx * ny;
    const float2* Vxp = p.Vx + (size_t)unit * nx * ny;
    const float2* Vyp = p.Vy + (size_t)unit * nx * ny;
    const float k0u = p.k0u[pol];
    const float txr = p.tiltX[pol], tyr = p.tiltY[pol];
    const float bx = p.bcx[pol], by = p.bcy[pol];
    float s[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, spow};
    for (int e = tid; e < nx * ny; e += blockDim.x) {
        const int y = e / nx, x = e - y * nx;
        float2 a = make_float2(0.f, 0.f), aw = make_float2(0.f, 0.f);
        for (int m = 0; m < G; m++) {
            const float hv = hxp[m * nx + x], dv = dhx[m * nx + x];
            const float2 u = U[m * ny + y], uw = Uw[m * ny + y];
            a.x = fmaf(hv, u.x, a.x); a.y = fmaf(hv, u.y, a.y);
            aw.x = fmaf(dv, u.x, fmaf(hv, uw.x, aw.x));
            aw.y = fmaf(dv, u.y, fmaf(hv, uw.y, aw.y));
        }
        const float2 v = Vp[e], vx = Vxp[e], vy = Vyp[e];
        // Re(Abar V i) = -Im(Abar V)
        const float imAV = a.x * v.y + a.y * v.x;
        const float xv = p.xAxis[x], yv = p.yAxis[y];
        s[0] += -imAV * k0u * (xv + bx);
        s[1] += -imAV * k0u * (yv + by);
        s[2] += -imAV * p.piOverLambda * (xv * xv + yv * yv);
        s[3] += (a.x * vx.x - a.y * vx.y) - imAV * k0u * txr;
        s[4] += (a.x * vy.x - a.y * vy.y) - imAV * k0u * tyr;
        s[5] += aw.x * v.x - aw.y * v.y;
    }
#pragma unroll
    for (int k = 0; k < 7; k++)
        for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
    if ((tid & 31) == 0)
        for (int k = 0; k < 7; k++) red[(tid >> 5) * 7 + k] = s[k];
    __syncthreads();
    if (tid < 7) {
        float t = 0.f;
        for (int wv = 0; wv < (int)(blockDim.x >> 5); wv++) t += red[wv * 7 + tid];
        p.out[(size_t)unit * 7 + tid] = t;
    }
}

// The same contraction for G <= GM, register-tiled: each thread owns one
// column x of the field, with Hx_m(x) and dHx_m/dw(x) for m < GM in
// registers, and walks the rows y = ty, ty + YS, ...; the row sums U[m][y]
// and Uw[m][y] sit in shared memory as one float4 per (m, y), which a warp
// (32 columns of one row) reads as a broadcast.  Rows G <= m < GM of the
// table are zero, so the unrolled mode loop needs no bound check.  Per pixel
// and mode: one shared load and six FMAs (the generic kernel above reads
// four values per pixel and mode).
template <int GM>
__global__ void __launch_bounds__(256) k_align_grad_reg(DhGradParams p) {
    extern __shared__ float4 sg4[];
    const int unit = blockIdx.x;
    const int P = p.polCount, G = p.G, M = p.M, nx = p.nx, ny = p.ny;
    const int pol = unit % P, frame = unit / P;
    const int GE = G + 2;
    float4* UU = sg4;                                                 // [GM][ny] {U, Uw}
    float2* cc = reinterpret_cast<float2*>(UU + (size_t)GM * ny);     // [M] conj(c)
    float* dhy = reinterpret_cast<float*>(cc + M);                    // [G][ny] Hy'_n
    float* red = dhy + (size_t)G * ny;                                // [8 warps][7]
    const float* hxp = p.hx + (size_t)pol * GE * nx;
    const float* hyp = p.hy + (size_t)pol * GE * ny;
    const float w0 = p.waist[pol];
    const float ladder = -1.0f / (2.0f * w0);
    const int tid = threadIdx.x;

    float spow = 0.f;
    for (int mode = tid; mode < M; mode += blockDim.x) {
        const size_t ci = (size_t)frame * P * M + (size_t)pol * M + mode;
        const float2 c = p.coefs[ci];
        cc[mode] = p.weights ? p.weights[ci] : make_float2(c.x, -c.y);
        spow = fmaf(c.x, c.x, fmaf(c.y, c.y, spow));
    }
    for (int e = tid; e < G * ny; e += blockDim.x) {
        const int n = e / ny, y = e - n * ny;
        float v = 0.f;
        if (n >= 2) v += sqrtf((float)(n * (n - 1))) * hyp[(n - 2) * ny + y];
        v -= sqrtf((float)((n + 1) * (n + 2))) * hyp[(n + 2) * ny + y];
        dhy[e] = v * ladder;
    }
    __syncthreads();
    for (int e = tid; e < GM * ny; e += blockDim.x) {
        const int m = e / ny, y = e - m * ny;
        float4 u = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int n = 0; m + n < G; n++) {
            const int g = m + n;
            const float2 c = cc[g * (g + 1) / 2 + n];
            const float hv = hyp[n * ny + y], dv = dhy[n * ny + y];
            u.x = fmaf(c.x, hv, u.x); u.y = fmaf(c.y, hv, u.y);
            u.z = fmaf(c.x, dv, u.z); u.w = fmaf(c.y, dv, u.w);
        }
        UU[e] = u;
    }
    __syncthreads();

    const size_t base = (size_t)unit * nx * ny;
    const float2* Vp = p.V + base;
    const float2* Vxp = p.Vx + base;
    const float2* Vyp = p.Vy + base;
    const int XT = nx < 256 ? nx : 256;   // nx is a power of two
    const int YS = 256 / XT;
    const int tx = tid % XT, ty = tid / XT;
    const float bx = p.bcx[pol], by = p.bcy[pol];
    // sums: Im(Abar V) (x + bcx), Im(Abar V) (y + bcy), Im(Abar V) (x^2 + y^2),
    // Re(Abar Vx), Re(Abar Vy), Re(Abar_w V), Im(Abar V)
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f, s4 = 0.f, s5 = 0.f, si = 0.f;
    for (int x0 = 0; x0 < nx; x0 += XT) {
        const int x = x0 + tx;
        float hr[GM], dr[GM];
#pragma unroll
        for (int m = 0; m < GM; m++) {
            hr[m] = 0.f;
            dr[m] = 0.f;
            if (m < G) {
                hr[m] = hxp[m * nx + x];
                float v = 0.f;
                if (m >= 2) v += sqrtf((float)(m * (m - 1))) * hxp[(m - 2) * nx + x];
                v -= sqrtf((float)((m + 1) * (m + 2))) * hxp[(m + 2) * nx + x];
                dr[m] = v * ladder;
            }
        }
        const float xv = p.xAxis[x];
        for (int y = ty; y < ny; y += YS) {
            const size_t e = (size_t)y * nx + x;
            const float2 v = Vp[e], vx = Vxp[e], vy = Vyp[e];
            float2 a = make_float2(0.f, 0.f), aw = make_float2(0.f, 0.f);
            const float4* Uy = UU + y;
#pragma unroll
            for (int m = 0; m < GM; m++) {
                const float4 u = Uy[m * ny];
                a.x = fmaf(hr[m], u.x, a.x);
                a.y = fmaf(hr[m], u.y, a.y);
                aw.x = fmaf(dr[m], u.x, fmaf(hr[m], u.z, aw.x));
                aw.y = fmaf(dr[m], u.y, fmaf(hr[m], u.w, aw.y));
            }
            const float imAV = a.x * v.y + a.y * v.x;
            const float yv = p.yAxis[y];
            s0 = fmaf(imAV, xv + bx, s0);
            s1 = fmaf(imAV, yv + by, s1);
            s2 = fmaf(imAV, xv * xv + yv * yv, s2);
            s3 += a.x * vx.x - a.y * vx.y;
            s4 += a.x * vy.x - a.y * vy.y;
            s5 += aw.x * v.x - aw.y * v.y;
            si += imAV;
        }
    }
    const float k0u = p.k0u[pol];
    // Re(Abar V i) = -Im(Abar V); the beam-centre tangents carry -Im(Abar V) k0 u t
    float s[7] = {-k0u * s0, -k0u * s1, -p.piOverLambda * s2, s3 - k0u * p.tiltX[pol] * si,
                  s4 - k0u * p.tiltY[pol] * si, s5, spow};
#pragma unroll
    for (int k = 0; k < 7; k++)
        for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
    if ((tid & 31) == 0)
        for (int k = 0; k < 7; k++) red[(tid >> 5) * 7 + k] = s[k];
    __syncthreads();
    if (tid < 7) {
        float t = 0.f;
        for (int wv = 0; wv < (int)(blockDim.x >> 5); wv++) t += red[wv * 7 + tid];
        p.out[(size_t)unit * 7 + tid] = t;
    }
}

// The same contraction with four columns per thread in packed pairs (f32x2),
// G <= GM - 2: lanes along the columns, four each, so that one shared load
// serves four pixels and one instruction two.  The waist derivative's adjoint
// field is written in the modes themselves, the ladder relation applied to
// the coefficients instead of the modes:
//   Abar_w = sum_mn D_mn Hx_m Hy_n,  D_mn = -(1 / 2w) (
//       sqrt((m+1)(m+2)) conj(c_{m+2,n}) - sqrt((m-1) m) conj(c_{m-2,n}) + (same in n)),
// m + n < G + 2, which leaves four FMAs per pixel and mode where the
// derivative modes need six.  Bound: latency (32 % of the issue slots at 16
// warps per SM; 2.9 TB/s of V, Vx, Vy).  1024 fields of 128 x 128, 15 groups:
// 141 us; k_align_grad_reg 195.
template <int GM, int CP>
__global__ void __launch_bounds__(256) k_align_grad_tile(DhGradParams p) {
    extern __shared__ float4 sg4[];
    const int unit = blockIdx.x;
    const int P = p.polCount, G = p.G, M = p.M, nx = p.nx, ny = p.ny;
    const int pol = unit % P, frame = unit / P;
    const int GE = G + 2;
    float4* UD = sg4;                                                 // [ny][GM][2] {ux, ux, uy, uy}, {dx, dx, dy, dy}
    float4* CD = UD + (size_t)2 * GM * ny;                            // [n][m] {conj(c), D}
    float* red = reinterpret_cast<float*>(CD + GM * GM);              // [8 warps][7]
    const float* hxp = p.hx + (size_t)pol * GE * nx;
    const float* hyp = p.hy + (size_t)pol * GE * ny;
    const float ladder = -1.0f / (2.0f * p.waist[pol]);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;

    float spow = 0.f;
    for (int mode = tid; mode < M; mode += blockDim.x) {
        const float2 c = p.coefs[(size_t)frame * P * M + (size_t)pol * M + mode];
        spow = fmaf(c.x, c.x, fmaf(c.y, c.y, spow));
    }
    const float2* src = (p.weights ? p.weights : p.coefs) + (size_t)frame * P * M + (size_t)pol * M;
    const float sgn = p.weights ? 1.0f : -1.0f;
    auto coef = [&](int m, int n) {
        if (m < 0 || n < 0 || m + n >= G) return make_float2(0.f, 0.f);
        const int g = m + n;
        const float2 c = src[g * (g + 1) / 2 + n];
        return make_float2(c.x, sgn * c.y);
    };
    for (int e = tid; e < GM * GM; e += 256) {
        const int n = e / GM, m = e - n * GM;
        const float2 c = coef(m, n), a = coef(m + 2, n), b = coef(m - 2, n), d = coef(m, n + 2), f = coef(m, n - 2);
        const float wa = sqrtf((float)((m + 1) * (m + 2))), wb = sqrtf((float)((m - 1) * m));
        const float wd = sqrtf((float)((n + 1) * (n + 2))), wf = sqrtf((float)((n - 1) * n));
        CD[e] = make_float4(c.x, c.y, ladder * (wa * a.x - wb * b.x + wd * d.x - wf * f.x),
                            ladder * (wa * a.y - wb * b.y + wd * d.y - wf * f.y));
    }
    __syncthreads();
    // row sums: each thread one y, every second m
    for (int y = tid >> 1; y < ny; y += 128) {
        constexpr int HM = GM / 2;
        const int par = tid & 1;
        f2x us[HM], ds[HM];
#pragma unroll
        for (int i = 0; i < HM; i++) us[i] = ds[i] = pk(0.f, 0.f);
        for (int n = 0; n < GE; n++) {
            const f2x h = pk1(__ldg(hyp + (size_t)n * ny + y));
            const ulonglong2* c = reinterpret_cast<const ulonglong2*>(CD + n * GM + par);
#pragma unroll
            for (int i = 0; i < HM; i++) {
                const ulonglong2 v = c[2 * i];
                us[i] = fma2(v.x, h, us[i]);
                ds[i] = fma2(v.y, h, ds[i]);
            }
        }
        float4* o = UD + ((size_t)y * GM + par) * 2;
#pragma unroll
        for (int i = 0; i < HM; i++) {
            const float2 u = upk(us[i]), d = upk(ds[i]);
            o[4 * i] = make_float4(u.x, u.x, u.y, u.y);
            o[4 * i + 1] = make_float4(d.x, d.x, d.y, d.y);
        }
    }
    __syncthreads();

    const size_t base = (size_t)unit * nx * ny;
    constexpr int CT = 2 * CP;                       // columns per thread
    const int LX = nx / CT < 32 ? nx / CT : 32;      // lanes per row (nx is a power of two, at least CT)
    const int rows = 8 * (32 / LX);                  // rows in flight per block
    const int y0 = warp * (32 / LX) + lane / LX;
    const float bx = p.bcx[pol], by = p.bcy[pol];
    // sums: Im(Abar V) (x + bcx), Im(Abar V) (y + bcy), Im(Abar V) (x^2 + y^2),
    // Re(Abar Vx), Re(Abar Vy), Re(Abar_w V), Im(Abar V)
    float s0 = 0.f, s1 = 0.f, s2 = 0.f, s3 = 0.f, s4 = 0.f, s5 = 0.f, si = 0.f;
    for (int x0 = (lane % LX) * CT; x0 < nx; x0 += LX * CT) {
        f2x hr[CP][GM];
#pragma unroll
        for (int q = 0; q < CP; q++)
#pragma unroll
            for (int m = 0; m < GM; m++) {
                const float2 v = m < GE ? __ldg(reinterpret_cast<const float2*>(hxp + (size_t)m * nx + x0 + 2 * q)) : make_float2(0.f, 0.f);
                hr[q][m] = pk(v.x, v.y);
            }
        float col[CT];
#pragma unroll
        for (int q = 0; q < CT; q++) col[q] = 0.f;
        for (int y = y0; y < ny; y += rows) {
            const size_t e = base + (size_t)y * nx + x0;
            float4 v[CP], vx[CP], vy[CP];
#pragma unroll
            for (int q = 0; q < CP; q++) {
                v[q] = __ldg(reinterpret_cast<const float4*>(p.V + e) + q);
                vx[q] = __ldg(reinterpret_cast<const float4*>(p.Vx + e) + q);
                vy[q] = __ldg(reinterpret_cast<const float4*>(p.Vy + e) + q);
            }
            f2x ar[CP], ai[CP], wr[CP], wi[CP];
#pragma unroll
            for (int q = 0; q < CP; q++) ar[q] = ai[q] = wr[q] = wi[q] = pk(0.f, 0.f);
            const ulonglong2* u = reinterpret_cast<const ulonglong2*>(UD + (size_t)y * GM * 2);
#pragma unroll
            for (int m = 0; m < GM; m++) {
                const ulonglong2 uc = u[2 * m], dc = u[2 * m + 1];
#pragma unroll
                for (int q = 0; q < CP; q++) {
                    if (m < GM - 2) {
                        ar[q] = fma2(hr[q][m], uc.x, ar[q]);
                        ai[q] = fma2(hr[q][m], uc.y, ai[q]);
                    }
                    wr[q] = fma2(hr[q][m], dc.x, wr[q]);
                    wi[q] = fma2(hr[q][m], dc.y, wi[q]);
                }
            }
            float row = 0.f;
#pragma unroll
            for (int q = 0; q < CP; q++) {
                const float2 axr = upk(ar[q]), axi = upk(ai[q]), awr = upk(wr[q]), awi = upk(wi[q]);
                const float im0 = axr.x * v[q].y + axi.x * v[q].x, im1 = axr.y * v[q].w + axi.y * v[q].z;
                col[2 * q] += im0;
                col[2 * q + 1] += im1;
                row += im0 + im1;
                s3 += (axr.x * vx[q].x - axi.x * vx[q].y) + (axr.y * vx[q].z - axi.y * vx[q].w);
                s4 += (axr.x * vy[q].x - axi.x * vy[q].y) + (axr.y * vy[q].z - axi.y * vy[q].w);
                s5 += (awr.x * v[q].x - awi.x * v[q].y) + (awr.y * v[q].z - awi.y * v[q].w);
            }
            const float yv = p.yAxis[y];
            s1 = fmaf(row, yv + by, s1);
            s2 = fmaf(row, yv * yv, s2);
        }
#pragma unroll
        for (int q = 0; q < CT; q++) {
            const float xv = p.xAxis[x0 + q];
            s0 = fmaf(col[q], xv + bx, s0);
            s2 = fmaf(col[q], xv * xv, s2);
            si += col[q];
        }
    }
    const float k0u = p.k0u[pol];
    // Re(Abar V i) = -Im(Abar V); the beam-centre tangents carry -Im(Abar V) k0 u t
    float s[7] = {-k0u * s0, -k0u * s1, -p.piOverLambda * s2, s3 - k0u * p.tiltX[pol] * si,
                  s4 - k0u * p.tiltY[pol] * si, s5, spow};
#pragma unroll
    for (int k = 0; k < 7; k++)
        for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
    if (lane == 0)
        for (int k = 0; k < 7; k++) red[warp * 7 + k] = s[k];
    __syncthreads();
    if (tid < 7) {
        float t = 0.f;
        for (int wv = 0; wv < 8; wv++) t += red[wv * 7 + tid];
        p.out[(size_t)unit * 7 + tid] = t;
    }
}

// ---------------------------------------------------------------- in the Fourier window
// The same sums from the Fourier window W alone.  A is the inverse transform
// of W, and the modes, the reference wave and the weights x, x^2, kx of the
// tangents are all separable, so every sum over pixels is a sum over the
// window:
//   sum_xy conj(Abar) f(x) g(y) A R = sum_jc W[j][c] sum_mn c_mn F_m[c] K_n[j],
//   F_m[c] = sum_x f(x) Hx_m(x) Rx(x) exp(2 pi i col_c x / nx),   K_n[j] alike,
// with Abar V = -conj(conj(Abar) A R).  One small kernel makes the tables F
// and K (five each: 1, x + bcx, x^2, kx, the waist derivative of the modes)
// for the configuration; a field then costs about (2 w h G + 5 (w + h) G^2 / 2)
// complex products on w h values, where the pixels cost 4 nx ny G on three
// fields of nx ny that had to be made and stored first.

// F (axis 0) or K (axis 1) of one mode and polarisation per block, summed in
// FP64: out[axis][pol][5][G][side].  The samples' factors (mode and waist
// derivative times wave, position) are formed once, in shared memory.
__global__ void __launch_bounds__(256) k_grad_tables(DhGradWindowParams p) {
    extern __shared__ double sd[];
    const int m = blockIdx.x, axis = blockIdx.y, pol = blockIdx.z, tid = threadIdx.x;
    const int side = axis ? p.h : p.w, logn = axis ? p.logny : p.lognx, n = 1 << logn;
    const int GE = p.G + 2;
    const float* H = (axis ? p.hy : p.hx) + (size_t)pol * GE * n;
    const float* R = p.refWaveF + (size_t)pol * 2 * (p.nx + p.ny) + (axis ? 2 * p.nx : 0);
    const float* ax = axis ? p.yAxis : p.xAxis;
    const double bc = axis ? p.bcy[pol] : p.bcx[pol];
    const float* kt = (axis ? p.ky : p.kx) + pol * side;
    float2* out = (axis ? p.tabY : p.tabX) + (size_t)pol * 5 * p.G * side;
    double* part = sd;                                     // [8][256]
    double2* tw = reinterpret_cast<double2*>(sd + 8 * 256);   // [n] exp(+2 pi i x / n)
    float4* smp = reinterpret_cast<float4*>(tw + n);       // [n] {mode, derivative, Rr, Ri}
    float* pos = reinterpret_cast<float*>(smp + n);        // [n]
    {
        const double ladder = -1.0 / (2.0 * (double)p.waist[pol]);
        const double la = m > 1 ? ladder * sqrt((double)(m * (m - 1))) : 0.0, lb = -ladder * sqrt((double)((m + 1) * (m + 2)));
        for (int x = tid; x < n; x += 256) {
            const float2 e = __ldg(&p.twiddle[x << (TW_LOG - logn)]);
            tw[x] = make_double2(e.x, -e.y);
            const double hw = (m > 1 ? la * H[(size_t)(m - 2) * n + x] : 0.0) + lb * H[(size_t)(m + 2) * n + x];
            smp[x] = make_float4(H[(size_t)m * n + x], (float)hw, R[x], R[n + x]);
            pos[x] = ax[x];
        }
    }
    __syncthreads();
    const int nf = side < 256 ? side : 256, S = 256 / nf;   // side is a power of two
    const int q = tid / nf;
    for (int f = tid % nf; f < side; f += nf) {
        int col = f;
        if (!p.lowres) col = axis ? f + p.sy[pol] + n / 2 : p.sx0[pol] + f;
        double a[8];
        for (int v = 0; v < 8; v++) a[v] = 0.0;
#pragma unroll 4
        for (int x = q; x < n; x += S) {
            const double2 e = tw[(unsigned)(col * x) & (unsigned)(n - 1)];
            const float4 s = smp[x];
            const double rr = s.z, ri = s.w;
            const double tr = rr * e.x - ri * e.y, ti = ri * e.x + rr * e.y;   // Rx exp(+)
            const double xv = pos[x], gr = s.x * tr, gi = s.x * ti;
            a[0] += gr;
            a[1] += gi;
            a[2] += (xv + bc) * gr;
            a[3] += (xv + bc) * gi;
            a[4] += xv * xv * gr;
            a[5] += xv * xv * gi;
            a[6] += s.y * tr;
            a[7] += s.y * ti;
        }
        for (int v = 0; v < 8; v++) part[(size_t)v * 256 + tid] = a[v];
        __syncthreads();
        if (q == 0) {
            for (int u = 1; u < S; u++)
                for (int v = 0; v < 8; v++) a[v] += part[(size_t)v * 256 + u * nf + tid];
            const double k = kt[f];
            const size_t o = (size_t)m * side + f, st = (size_t)p.G * side;
            out[o] = make_float2((float)a[0], (float)a[1]);
            out[st + o] = make_float2((float)a[2], (float)a[3]);
            out[2 * st + o] = make_float2((float)a[4], (float)a[5]);
            out[3 * st + o] = make_float2((float)(k * a[0]), (float)(k * a[1]));
            out[4 * st + o] = make_float2((float)a[6], (float)a[7]);
        }
        __syncthreads();
    }
}

constexpr int GB = 3;   // blocks per SM of the window kernel (2 and 4: the same time)

// Half of a field's sums, by 128 threads.  An item is one window column (row)
// u and four modes n of the other axis, 2 i, 2 i + 1 and their mirrors
// G - 1 - n, whose lengths G - n add up to the same for every i:
//   Y_n = sum_v B_n[v] W(u, v)   (B the other axis's base table)
//   s[k] += (sum_m c_mn T^k_m[u]) Y_n,   k = 1, lin, quad, k, waist.
// XS: u = column, n the modes of y; else u = row, n those of x.  c[m][n], zero
// for m + n >= G.
template <bool XS>
__device__ __forceinline__ void gradHalf(const float2* __restrict__ W, int ld, const float2* __restrict__ c, int G,
                                         const float2* __restrict__ T, const float2* __restrict__ B, int logu, int nv,
                                         int t, float (&s)[5]) {
    const int nu = 1 << logu, half = (G + 1) >> 1, quads = (half + 1) >> 1;
    const int st = G << logu;
    for (int item = t; item < quads << logu; item += 128) {
        const int i = item >> logu, u = item & (nu - 1);
        const int n0 = 2 * i, n1 = min(2 * i + 1, half - 1);
        const int n[4] = {n0, n1, G - 1 - n0, G - 1 - n1};
        const bool use[4] = {true, n1 != n0, n[2] != n0, n1 != n0 && n[3] != n1};
        float2 y[4];
        const float4* b[4];
#pragma unroll
        for (int k = 0; k < 4; k++) {
            y[k] = make_float2(0.f, 0.f);
            b[k] = reinterpret_cast<const float4*>(B + (size_t)n[k] * nv);
        }
#pragma unroll 4
        for (int v = 0; v < nv; v += 2) {
            const float2 w0 = XS ? W[(size_t)v * ld + u] : W[(size_t)u * ld + v];
            const float2 w1 = XS ? W[(size_t)(v + 1) * ld + u] : W[(size_t)u * ld + v + 1];
#pragma unroll
            for (int k = 0; k < 4; k++) {
                const float4 q = b[k][v >> 1];
                y[k].x = fmaf(q.x, w0.x, fmaf(-q.y, w0.y, y[k].x));
                y[k].y = fmaf(q.x, w0.y, fmaf(q.y, w0.x, y[k].y));
                y[k].x = fmaf(q.z, w1.x, fmaf(-q.w, w1.y, y[k].x));
                y[k].y = fmaf(q.z, w1.y, fmaf(q.w, w1.x, y[k].y));
            }
        }
#pragma unroll
        for (int k = 0; k < 4; k++)
            if (!use[k]) y[k] = make_float2(0.f, 0.f);   // a mode counts once
        // z_m = sum of c_mn Y_n over the four n serves the five tables
        const float2* tu = T + u;
#pragma unroll 2
        for (int m = 0; m < G - n0; m++) {
            const float2* cm = c + m * G;
            float zr = 0.f, zi = 0.f;
#pragma unroll
            for (int k = 0; k < 4; k++) {
                if (k >= 2 && m > n1) break;   // the mirrors end at m = n
                const float2 a = cm[n[k]];
                zr = fmaf(a.x, y[k].x, fmaf(-a.y, y[k].y, zr));
                zi = fmaf(a.x, y[k].y, fmaf(a.y, y[k].x, zi));
            }
            const float2* tm = tu + (m << logu);
            const float2 t1 = tm[st], t2 = tm[2 * st], t3 = tm[3 * st], t4 = tm[4 * st];
            if (XS) {
                const float2 t0 = tm[0];
                s[0] = fmaf(t0.x, zi, fmaf(t0.y, zr, s[0]));
            }
            s[1] = fmaf(t1.x, zi, fmaf(t1.y, zr, s[1]));
            s[2] = fmaf(t2.x, zi, fmaf(t2.y, zr, s[2]));
            s[3] = fmaf(t3.x, zi, fmaf(t3.y, zr, s[3]));
            s[4] = fmaf(t4.x, zr, fmaf(-t4.y, zi, s[4]));
        }
    }
}

// One (frame, polarisation) at a time per block of a fixed polarisation, the x
// tables' sums by its first four warps, the y tables' by the others; SM: the
// tables and the window in shared memory (this build's kernels keep the L1
// small, so the tables would come from the L2 each time).
// Bound: the shared-memory reads of the products (14.7 M instructions at 62 %
// of the issue slots, 5 % of the DRAM).  1024 fields of 128 x 128 (32 x 32
// windows), 15 groups: 28 us, and 7 for the tables (47 with one unit per block
// and the tables in global memory, 11 with each table's samples fetched in its
// loop); the pixel path took 10 + 108 us for the
// derivative fields, 30 more in the batch for V and 141 for its contraction.
template <bool SM>
__global__ void __launch_bounds__(256, GB) k_align_grad_window(DhGradWindowParams p) {
    extern __shared__ float4 sg4[];
    __shared__ float red[8 * 7];
    const int P = p.polCount, G = p.G, M = p.M, w = p.w, h = p.h;
    const int pol = blockIdx.x % P;   // the grid is a multiple of P
    const int tid = threadIdx.x;
    const int nt = SM ? 5 * G * (w + h) : 0;
    float2* st = reinterpret_cast<float2*>(sg4);   // the polarisation's tables, x then y
    float2* c = st + nt;                           // [m][n] and [n][m]: conj of Abar's coefficients, zero for m + n >= G
    float2* sw = c + 2 * G * G;                    // [h][w + 1]
    const float2* tx = p.tabX + (size_t)pol * 5 * G * w;
    const float2* ty = p.tabY + (size_t)pol * 5 * G * h;
    if (SM) {
        const int nx4 = 5 * G * w / 2;
        for (int e = tid; e < nt / 2; e += 256)
            sg4[e] = e < nx4 ? __ldg(reinterpret_cast<const float4*>(tx) + e) : __ldg(reinterpret_cast<const float4*>(ty) + e - nx4);
    }
    const float k0u = p.k0u[pol];
    for (int unit = blockIdx.x; unit < p.frameCount * P; unit += gridDim.x) {
        const int frame = unit / P;
        const float2* win = p.window + (size_t)unit * h * w;
        // in the order of the other gradient kernels
        float spow = 0.f;
        for (int mode = tid; mode < M; mode += 256) {
            const float2 v = p.coefs[(size_t)frame * P * M + (size_t)pol * M + mode];
            spow = fmaf(v.x, v.x, fmaf(v.y, v.y, spow));
        }
        const float2* src = (p.weights ? p.weights : p.coefs) + (size_t)frame * P * M + (size_t)pol * M;
        const float sgn = p.weights ? -1.0f : 1.0f;   // conj(Abar's coefficients)
        for (int e = tid; e < G * G; e += 256) {
            const int n = e / G, m = e - n * G, g = m + n;
            float2 v = make_float2(0.f, 0.f);
            if (g < G) {
                v = src[g * (g + 1) / 2 + n];
                v.y *= sgn;
            }
            c[m * G + n] = v;
            c[G * G + e] = v;
        }
        if (SM)
            for (int e = tid; e < h * w; e += 256) sw[(e >> p.logw) * (w + 1) + (e & (w - 1))] = win[e];
        __syncthreads();
        float sx[5] = {0.f, 0.f, 0.f, 0.f, 0.f}, sy[5] = {0.f, 0.f, 0.f, 0.f, 0.f};
        if (SM) {
            if (tid < 128) gradHalf<true>(sw, w + 1, c, G, st, st + 5 * G * w, p.logw, h, tid, sx);
            else gradHalf<false>(sw, w + 1, c + G * G, G, st + 5 * G * w, st, p.logh, w, tid - 128, sy);
        } else {
            if (tid < 128) gradHalf<true>(win, w, c, G, tx, ty, p.logw, h, tid, sx);
            else gradHalf<false>(win, w, c + G * G, G, ty, tx, p.logh, w, tid - 128, sy);
        }
        // Im(Abar V) = Im, Re(Abar V) = -Re of the sums (Abar V = -conj of them)
        float s[7] = {-k0u * sx[1], -k0u * sy[1], -p.piOverLambda * (sx[2] + sy[2]), sx[3] - k0u * p.tiltX[pol] * sx[0],
                      sy[3] - k0u * p.tiltY[pol] * sx[0], -(sx[4] + sy[4]), spow};
#pragma unroll
        for (int k = 0; k < 7; k++)
            for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
        if ((tid & 31) == 0)
            for (int k = 0; k < 7; k++) red[(tid >> 5) * 7 + k] = s[k];
        __syncthreads();   // also: c and the window are free for the next unit
        if (tid < 7) {
            float t = 0.f;
            for (int wv = 0; wv < 8; wv++) t += red[wv * 7 + tid];
            p.out[(size_t)unit * 7 + tid] = t;
        }
        // red is rewritten only after the next unit's first barrier
    }
}

// The power term of the gradient kernels alone (their first loop and their
// block reduction, in the same order).
__global__ void __launch_bounds__(256) k_align_power(DhGradParams p) {
    __shared__ float red[8 * 7];
    const int unit = blockIdx.x;
    const int P = p.polCount, M = p.M;
    const int pol = unit % P, frame = unit / P;
    const int tid = threadIdx.x;
    float spow = 0.f;
    for (int mode = tid; mode < M; mode += blockDim.x) {
        const float2 c = p.coefs[(size_t)frame * P * M + (size_t)pol * M + mode];
        spow = fmaf(c.x, c.x, fmaf(c.y, c.y, spow));
    }
    float s[7] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, spow};
#pragma unroll
    for (int k = 0; k < 7; k++)
        for (int off = 16; off > 0; off >>= 1) s[k] += __shfl_xor_sync(0xffffffffu, s[k], off);
    if ((tid & 31) == 0)
        for (int k = 0; k < 7; k++) red[(tid >> 5) * 7 + k] = s[k];
    __syncthreads();
    if (tid < 7) {
        float t = 0.f;
        for (int wv = 0; wv < (int)(blockDim.x >> 5); wv++) t += red[wv * 7 + tid];
        p.out[(size_t)unit * 7 + tid] = t;
    }
}

cudaError_t dh_launch_align_power(const DhGradParams& p, cudaStream_t s) {
    k_align_power<<<(unsigned)(p.frameCount * p.polCount), 256, 0, s>>>(p);
    return cudaGetLastError();
}

// Weights of an eigenvalue's derivative.  For an eigenpair (lambda, u) of
// the Gram matrix of the block A (rows = modes of pol0 [and pol1], columns
// = frames; column-major A[b rows + j]), d lambda = 2 Re sum_jb w_jb dA_jb
// with w_jb = conj(p_j) q_b and (p, q) = (u, A^H u) for the mode-space Gram
// A A^H, (A u, u) for the frame-space Gram A^H A.  W[b][pol M + m] +=
// alpha w_jb, row j < M of pol0, j >= M of pol1.  One thread per (j, b).
__global__ void k_mdl_weights(const float2* __restrict__ A, int rows, int batch, int rowsGram,
                              const double2* __restrict__ u, double alpha, int pol0, int pol1, int polCount, int M,
                              float2* __restrict__ W) {
    const int total = rows * batch;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int b = e / rows, j = e - b * rows;
        double2 pj, qb;
        if (rowsGram) {
            pj = u[j];
            double re = 0.0, im = 0.0;   // (A^H u)_b = sum_i conj(A_ib) u_i
            for (int i = 0; i < rows; i++) {
                const float2 a = A[(size_t)b * rows + i];
                re += (double)a.x * u[i].x + (double)a.y * u[i].y;
                im += (double)a.x * u[i].y - (double)a.y * u[i].x;
            }
            qb = make_double2(re, im);
        } else {
            double re = 0.0, im = 0.0;   // (A u)_j = sum_c A_jc u_c
            for (int c = 0; c < batch; c++) {
                const float2 a = A[(size_t)c * rows + j];
                re += (double)a.x * u[c].x - (double)a.y * u[c].y;
                im += (double)a.x * u[c].y + (double)a.y * u[c].x;
            }
            pj = make_double2(re, im);
            qb = u[b];
        }
        // conj(p_j) q_b
        const double wr = pj.x * qb.x + pj.y * qb.y, wi = pj.x * qb.y - pj.y * qb.x;
        const int pol = j < M ? pol0 : pol1, m = j < M ? j : j - M;
        float2* wp = W + (size_t)b * polCount * M + (size_t)pol * M + m;
        wp->x += (float)(alpha * wr);
        wp->y += (float)(alpha * wi);
    }
}

cudaError_t dh_launch_mdl_weights(const float2* A, int rows, int batch, int rowsGram, const double2* u, double alpha,
                                  int pol0, int pol1, int polCount, int M, float2* W, cudaStream_t s) {
    const int total = rows * batch;
    int blocks = (total + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    if (blocks < 1) blocks = 1;
    k_mdl_weights<<<blocks, 256, 0, s>>>(A, rows, batch, rowsGram, u, alpha, pol0, pol1, polCount, M, W);
    return cudaGetLastError();
}

cudaError_t dh_launch_window_deriv(const float2* W, const float* kxw, const float* kyw, int w, int h, int polCount, int units,
                                   float2* Wx, float2* Wy, cudaStream_t s) {
    const size_t total = (size_t)units * w * h;
    int blocks = (int)((total + 255) / 256);
    if (blocks > 4096) blocks = 4096;
    if (blocks < 1) blocks = 1;
    k_window_deriv<<<blocks, 256, 0, s>>>(W, kxw, kyw, w, h, polCount, units, Wx, Wy);
    return cudaGetLastError();
}

template <int GM>
static cudaError_t launchAlignGradReg(const DhGradParams& p, size_t smem, cudaStream_t s) {
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(k_align_grad_reg<GM>), (int)smem);
    if (e != cudaSuccess) return e;
    k_align_grad_reg<GM><<<(unsigned)(p.frameCount * p.polCount), 256, smem, s>>>(p);
    return cudaGetLastError();
}

template <int GM, int CP>
static cudaError_t launchAlignGradTile(const DhGradParams& p, cudaStream_t s) {
    const size_t smem = sizeof(float4) * ((size_t)2 * GM * p.ny + GM * GM) + sizeof(float) * 8 * 7;
    if (smem > 200 * 1024) return cudaErrorNotSupported;
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(k_align_grad_tile<GM, CP>), (int)smem);
    if (e != cudaSuccess) return e;
    k_align_grad_tile<GM, CP><<<(unsigned)(p.frameCount * p.polCount), 256, smem, s>>>(p);
    return cudaGetLastError();
}

cudaError_t dh_launch_align_grad(const DhGradParams& p, cudaStream_t s) {
    const bool pow2 = p.nx > 0 && (p.nx & (p.nx - 1)) == 0;
    // four (G <= 16) or two columns per thread where the row sums fit shared
    // memory (18 or 34 modes x 32 bytes x ny: up to 256 and 128 rows), else
    // one column per thread
    if (pow2 && p.nx >= 16 && p.G <= 32 &&
        ((reinterpret_cast<uintptr_t>(p.V) | reinterpret_cast<uintptr_t>(p.Vx) | reinterpret_cast<uintptr_t>(p.Vy)) & 15) == 0 &&
        (reinterpret_cast<uintptr_t>(p.hx) & 7) == 0) {
        const cudaError_t e = p.G <= 16 ? launchAlignGradTile<18, 2>(p, s) : launchAlignGradTile<34, 1>(p, s);
        if (e != cudaErrorNotSupported) return e;
        cudaGetLastError();
    }
    if (pow2 && p.G <= 32) {
        const int GM = p.G <= 16 ? 16 : 32;
        const size_t smemReg = sizeof(float4) * (size_t)GM * p.ny + sizeof(float2) * (size_t)p.M +
                               sizeof(float) * ((size_t)p.G * p.ny + 8 * 7);
        if (smemReg <= 200 * 1024) return GM == 16 ? launchAlignGradReg<16>(p, smemReg, s) : launchAlignGradReg<32>(p, smemReg, s);
    }
    const size_t smem = sizeof(float2) * ((size_t)p.M + 2 * (size_t)p.G * p.ny) + sizeof(float) * ((size_t)p.G * (p.nx + p.ny) + 8 * 7);
    if (smem > 200 * 1024) return cudaErrorNotSupported;
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(k_align_grad), (int)smem);
    if (e != cudaSuccess) return e;
    k_align_grad<<<(unsigned)(p.frameCount * p.polCount), 256, smem, s>>>(p);
    return cudaGetLastError();
}

size_t dh_grad_tables_elems(int P, int G, int w, int h) { return (size_t)P * 5 * G * (w + h); }

// The two coefficient tables [m][n] and [n][m]; 1 KB is left for the kernel's
// own arrays.  Up to 120 groups.
static size_t gradCoefBytes(int G) { return sizeof(float2) * 2 * (size_t)G * G; }
bool dh_grad_window_fits(int G) { return gradCoefBytes(G) <= 226 * 1024; }

// The refusal of the pixel kernels (fields whose row sums exceed shared
// memory) holds here too: what can be aligned does not depend on a calibration.
cudaError_t dh_launch_align_grad_window(const DhGradWindowParams& p, cudaStream_t s) {
    const size_t reg = sizeof(float4) * (size_t)(p.G <= 16 ? 16 : 32) * p.ny + sizeof(float2) * (size_t)p.M +
                       sizeof(float) * ((size_t)p.G * p.ny + 8 * 7);
    const size_t any = sizeof(float2) * ((size_t)p.M + 2 * (size_t)p.G * p.ny) +
                       sizeof(float) * ((size_t)p.G * (p.nx + p.ny) + 8 * 7);
    if ((p.G > 32 || reg > 200 * 1024) && any > 200 * 1024) return cudaErrorNotSupported;
    if (p.lognx > TW_LOG || p.logny > TW_LOG || !dh_grad_window_fits(p.G)) return cudaErrorNotSupported;
    const size_t ts = 256 * 8 * sizeof(double) + (sizeof(double2) + sizeof(float4) + sizeof(float)) * (size_t)(p.nx > p.ny ? p.nx : p.ny);
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(k_grad_tables), (int)ts);
    if (e != cudaSuccess) return e;
    k_grad_tables<<<dim3(p.G, 2, p.polCount), 256, ts, s>>>(p);
    e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    const unsigned units = (unsigned)(p.frameCount * p.polCount);
    // the base tables are read in pairs
    if ((reinterpret_cast<uintptr_t>(p.tabX) | reinterpret_cast<uintptr_t>(p.tabY)) & 15) return cudaErrorInvalidValue;
    const size_t cs = gradCoefBytes(p.G);
    const size_t ws = cs + sizeof(float2) * ((size_t)p.h * (p.w + 1) + 5 * (size_t)p.G * (p.w + p.h));
    const bool sm = ws <= 200 * 1024;
    unsigned grid = (unsigned)smCountCached() * GB / p.polCount * p.polCount;
    if (grid > units) grid = units;
    if (sm) {
        e = setSmemOnce(reinterpret_cast<const void*>(k_align_grad_window<true>), (int)ws);
        if (e != cudaSuccess) return e;
        k_align_grad_window<true><<<grid, 256, ws, s>>>(p);
    } else {
        e = setSmemOnce(reinterpret_cast<const void*>(k_align_grad_window<false>), (int)cs);
        if (e != cudaSuccess) return e;
        k_align_grad_window<false><<<grid, 256, cs, s>>>(p);
    }
    return cudaGetLastError();
}
