// Inverse stage for full-resolution fields of 32 and 64 pixels
// (IFFTResolutionMode 0; 128-pixel fields: dh_field128.cu): the Fourier
// window placed in the H x W plane -> IFFT -> field statistics -> reference
// wave, -conj, int16 rounding (k_field_full); and the separable HG overlap of
// int16 fields on the CUDA cores (k_overlap_f32).  Same results as k_inverse
// in full-resolution mode and as the reference's FFTW c2c backward
// digHolo.cpp:8734, digHoloFieldAnalysis digHolo.cpp:2354, applyTilt16
// digHolo.cpp:2701-2837 and overlapFieldSeparable16 digHolo.cpp:2149-2341.
//
// Pruned IFFT: only the h x w window is non-zero.  Along y, the window rows
// sit at row_j = (r0 + j) mod H; with y = (H/h) t + u the column transform
// of column c splits into H/h independent h-point inverse FFTs
//   A[(H/h) t + u][c] = IFFT_h( b_u )[t],  b_u[row_j mod h] = win[j][c] e^{2 pi i row_j u / H},
// and along x in the same way with W/w w-point inverse FFTs per row.  Each
// thread owns 32 pixels of the field in registers (two w = 16 tasks or one
// w = 32 task) until the block has the field maximum.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "dh_common.cuh"
#include "dh_host.h"
#include "dh_params.h"
#include "dh_fft.cuh"

using namespace dh;


// W, H: FFT window (= field) size; WW: IFFT window size (h = w = WW).
// blockDim.x = H * W / 32; one block per (frame, polarisation).
template <int W, int H, int WW>
__global__ void __launch_bounds__(H * W / 32, 1) k_field_full(DhInvParams p) {
    constexpr int LOG = ilog2F(WW);
    constexpr int TX = W / WW, TY = H / WW;
    constexpr int TPT = 32 / WW;                    // stage-2 tasks per thread
    constexpr int NT = H * W / 32;
    constexpr int ALD = WW + 1;                     // stage-1 buffer row stride (complex)
    constexpr int SLD = W + 8;                      // int16 staging row stride (elements)
    extern __shared__ float4 smf4[];
    float2* A = reinterpret_cast<float2*>(smf4);                      // [H][ALD]
    short* sR = reinterpret_cast<short*>(A + H * ALD);                // [H][SLD]
    short* sI = sR + H * SLD;
    constexpr int TWLD = WW + 1;                    // padded: lanes with different u hit different banks
    float2* tw1 = reinterpret_cast<float2*>(sI + H * SLD);           // [TY][TWLD] e^{2 pi i row_k u / H}
    float2* tw2 = tw1 + TY * TWLD;                                     // [TX][TWLD] e^{2 pi i col_k u / W}
    float* xax = reinterpret_cast<float*>(tw2 + TX * TWLD);          // [W]
    int* refX = reinterpret_cast<int*>(xax + W);                      // [W] packed (xr, xi)
    StatF* red = reinterpret_cast<StatF*>(refX + W);                  // [NT / 32]

    const int unit = blockIdx.x;
    const int P = p.polCount;
    const int pol = unit % P, frame = unit / P;
    const int tid = threadIdx.x;
    const short* ref = p.refWave + (size_t)pol * 2 * (W + H);
    const int r0 = ((p.sy[pol] + H / 2) % H + H) % H;
    const int sx0 = p.sx0[pol];
    for (int x = tid; x < W; x += NT) {
        xax[x] = p.xAxis[x];
        refX[x] = ((int)(unsigned short)ref[x]) | ((int)ref[W + x] << 16);
    }
    // twiddles of the decimated sub-transforms: input k of sub-problem u
    for (int e = tid; e < TY * WW; e += NT) {
        const int u = e / WW, k = e % WW;
        const int row = (r0 + ((k - r0) & (WW - 1))) & (H - 1);
        tw1[u * TWLD + k] = expPos(p.twiddle, row * u, H);
    }
    for (int e = tid; e < TX * WW; e += NT) {
        const int u = e / WW, k = e % WW;
        const int col = (sx0 + ((k - sx0) & (WW - 1))) & (W - 1);
        tw2[u * TWLD + k] = expPos(p.twiddle, col * u, W);
    }
    __syncthreads();

    // stage 1: columns c < WW, u < TY
    const float2* win = p.window + (size_t)unit * WW * WW;
    for (int task = tid; task < WW * TY; task += NT) {
        const int c = task % WW, u = task / WW;
        float2 b[WW];
#pragma unroll
        for (int k = 0; k < WW; k++) {
            const int j = (k - r0) & (WW - 1);
            b[k] = cmul(__ldg(&win[j * WW + c]), tw1[u * TWLD + k]);
        }
        ifftDIFf<WW>(b);
#pragma unroll
        for (int i = 0; i < WW; i++) A[(TY * brevF<LOG>(i) + u) * ALD + c] = b[i];
    }
    __syncthreads();

    // stage 2: rows y < H, u < TX; the field stays in registers
    float2 f[TPT][WW];
    int ty[TPT], tu[TPT];
#pragma unroll
    for (int q = 0; q < TPT; q++) {
        const int task = tid + NT * q;
        const int y = task / TX, u = task % TX;
        ty[q] = y;
        tu[q] = u;
#pragma unroll
        for (int k = 0; k < WW; k++) {
            const int c = (k - sx0) & (WW - 1);
            f[q][k] = cmul(A[y * ALD + c], tw2[u * TWLD + k]);
        }
        ifftDIFf<WW>(f[q]);
    }

    // statistics over the untilted field (digHolo.cpp:8866-8870)
    const float yShift = fabsf((p.yAxis[1] - p.yAxis[0]) * (float)H);
    const float inv = (float)(1.0 / ((double)W * (double)H));
    StatF st = {0.f, -1, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
    for (int q = 0; q < TPT; q++) {
        const int y = ty[q];
        const float yv = p.yAxis[y];
        const float yw = yv + (yv < 0.f ? yShift : 0.f);
        float Prow = 0.f, cxrow = 0.f, e4 = 0.f;
#pragma unroll
        for (int i = 0; i < WW; i++) {
            const int x = TX * brevF<LOG>(i) + tu[q];
            const float2 a = f[q][i];
            const float I0 = fmaf(a.x, a.x, a.y * a.y);
            const float I = I0 * inv;
            const int idx = 2 * y * W + x;
            if (I0 > st.maxI || (I0 == st.maxI && idx > st.maxIdx)) { st.maxI = I0; st.maxIdx = idx; }
            Prow += I;
            cxrow = fmaf(xax[x], I, cxrow);
            e4 = fmaf(I, I, e4);
        }
        st.P += Prow;
        st.cx += cxrow;
        st.cy = fmaf(yv, Prow, st.cy);
        st.cyw = fmaf(yw, Prow, st.cyw);
        st.e4 += e4;
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) {
        const float mI = __shfl_xor_sync(0xffffffffu, st.maxI, off);
        const int mIdx = __shfl_xor_sync(0xffffffffu, st.maxIdx, off);
        statMerge(st, mI, mIdx, __shfl_xor_sync(0xffffffffu, st.P, off), __shfl_xor_sync(0xffffffffu, st.cx, off),
                  __shfl_xor_sync(0xffffffffu, st.cy, off), __shfl_xor_sync(0xffffffffu, st.cyw, off),
                  __shfl_xor_sync(0xffffffffu, st.e4, off));
    }
    if ((tid & 31) == 0) red[tid >> 5] = st;
    __syncthreads();
    StatF tot = red[0];
    for (int i = 1; i < NT / 32; i++) {
        const StatF o = red[i];
        statMerge(tot, o.maxI, o.maxIdx, o.P, o.cx, o.cy, o.cyw, o.e4);
    }
    const float scale = (float)(32767.0 / (double)sqrtf(tot.maxI));
    if (tid == 0) {
        const int S = p.statsStride;
        float* s = p.stats;
        const int col = pol * S + frame;
        const int per = P * S;
        s[0 * per + col] = tot.P;
        s[1 * per + col] = tot.cx / tot.P;
        s[2 * per + col] = tot.cy / tot.P;
        s[3 * per + col] = scale;
        s[4 * per + col] = __int_as_float(tot.maxIdx);
        s[5 * per + col] = p.dA * (tot.P * tot.P / tot.e4);
        s[6 * per + col] = tot.cyw / tot.P;
    }

    // reference wave, -conj(A . ref), int16 rounding (digHolo.cpp:2741-2833)
    const float K = (float)(1.0 / (16383.0 * 16383.0));
    const size_t fieldOff = (size_t)unit * W * H;
#pragma unroll
    for (int q = 0; q < TPT; q++) {
        const int y = ty[q];
        const int yr = ref[2 * W + y], yi = ref[2 * W + H + y];
#pragma unroll
        for (int i = 0; i < WW; i++) {
            const int x = TX * brevF<LOG>(i) + tu[q];
            const int rx = refX[x];
            const int xr = (short)(rx & 0xFFFF), xi = rx >> 16;
            const float adjR = (float)(yr * xr - yi * xi) * K;
            const float adjI = (float)(yr * xi + yi * xr) * K;
            const float2 a = f[q][i];
            const float vr = __fsub_rn(__fmul_rn(a.y, adjI), __fmul_rn(a.x, adjR));
            const float vi = __fadd_rn(__fmul_rn(a.x, adjI), __fmul_rn(a.y, adjR));
            if (p.field32) {
                const float* rf = p.refWaveF + (size_t)pol * 2 * (W + H);
                const float2 rxf = make_float2(rf[x], rf[W + x]);
                const float2 ryf = make_float2(rf[2 * W + y], rf[2 * W + H + y]);
                const float2 w = cmul(a, cmul(ryf, rxf));
                p.field32[fieldOff + (size_t)y * W + x] = make_float2(-w.x, w.y);
            }
            sR[y * SLD + x] = roundSat16(scale * vr);
            sI[y * SLD + x] = roundSat16(scale * vi);
        }
    }
    if (p.fieldsOnly) return;   // block-uniform
    __syncthreads();
    // coalesced copy of the int16 planes
    constexpr int CH = W / 8;   // 16-byte chunks per row
    uint4* gR = reinterpret_cast<uint4*>(p.fieldR + fieldOff);
    uint4* gI = reinterpret_cast<uint4*>(p.fieldI + fieldOff);
    for (int e = tid; e < H * CH; e += NT) {
        const int y = e / CH, q = e % CH;
        gR[e] = *reinterpret_cast<const uint4*>(sR + y * SLD + 8 * q);
        gI[e] = *reinterpret_cast<const uint4*>(sI + y * SLD + 8 * q);
    }
}

// Separable overlap of int16 fields on the CUDA cores (FP32 accumulation):
// T[y][m] = sum_x F[y][x] Hx[m][x] with one thread per (row, plane) and the
// modes in registers, then c_mn = sum_y Hy[n][y] T[y][m] per mode.
// One block per (frame, polarisation); blockDim.x = 2 * ny.
template <int GMAX>
__global__ void __launch_bounds__(256) k_overlap_f32(DhInvParams p, int nx, int ny) {
    extern __shared__ float smo[];
    const int G = p.maxMG, M = p.modeCount;
    const int unit = blockIdx.x;
    const int P = p.polCount;
    const int pol = unit % P, frame = unit / P;
    const int tid = threadIdx.x;
    float* hx = smo;                                   // [nx][GMAX] (x-major: one float4 row per x)
    float* hy = hx + nx * GMAX;                        // [G][ny]
    float* T = hy + G * ny;                            // [2][ny][G + 1]
    const short* gx = p.hgX + (size_t)pol * G * nx;
    const short* gy = p.hgY + (size_t)pol * G * ny;
    for (int e = tid; e < nx * GMAX; e += blockDim.x) {
        const int x = e / GMAX, m = e % GMAX;
        hx[e] = m < G ? (float)gx[m * nx + x] : 0.f;
    }
    for (int e = tid; e < G * ny; e += blockDim.x) hy[e] = (float)gy[e];
    __syncthreads();
    const size_t npix = (size_t)nx * ny;
    {
        const int plane = tid / ny, y = tid % ny;
        const short* row = (plane ? p.fieldI : p.fieldR) + (size_t)unit * npix + (size_t)y * nx;
        float acc[GMAX];
#pragma unroll
        for (int m = 0; m < GMAX; m++) acc[m] = 0.f;
        for (int x0 = 0; x0 < nx; x0 += 8) {
            const uint4 raw = __ldg(reinterpret_cast<const uint4*>(row + x0));
            const unsigned wv[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
            for (int t = 0; t < 8; t++) {
                const float v = (float)(short)((wv[t >> 1] >> (16 * (t & 1))) & 0xFFFF);
                const float4* hv = reinterpret_cast<const float4*>(hx + (x0 + t) * GMAX);
#pragma unroll
                for (int m4 = 0; m4 < GMAX / 4; m4++) {
                    const float4 h = hv[m4];
                    acc[4 * m4 + 0] = fmaf(v, h.x, acc[4 * m4 + 0]);
                    acc[4 * m4 + 1] = fmaf(v, h.y, acc[4 * m4 + 1]);
                    acc[4 * m4 + 2] = fmaf(v, h.z, acc[4 * m4 + 2]);
                    acc[4 * m4 + 3] = fmaf(v, h.w, acc[4 * m4 + 3]);
                }
            }
        }
        float* Tp = T + ((size_t)plane * ny + y) * (G + 1);
#pragma unroll
        for (int m = 0; m < GMAX; m++)
            if (m < G) Tp[m] = acc[m];   // unrolled: acc stays in registers
    }
    __syncthreads();
    const int S = p.statsStride;
    const float scale = p.stats[3 * P * S + pol * S + frame];
    const float fieldScale = 1.0f / scale;
    const float* sxp = p.hgScaleX + pol * G;
    const float* syp = p.hgScaleY + pol * G;
    for (int mode = tid; mode < M; mode += blockDim.x) {
        int g = (int)((sqrtf(8.0f * mode + 1.0f) - 1.0f) * 0.5f);
        while ((g + 1) * (g + 2) / 2 <= mode) g++;
        while (g * (g + 1) / 2 > mode) g--;
        const int n = mode - g * (g + 1) / 2;
        const int m = g - n;
        const float* hn = hy + n * ny;
        float cr = 0.f, ci = 0.f;
        for (int y = 0; y < ny; y++) {
            cr = fmaf(hn[y], T[(size_t)y * (G + 1) + m], cr);
            ci = fmaf(hn[y], T[((size_t)ny + y) * (G + 1) + m], ci);
        }
        const float ms = (float)((double)sxp[m] * (double)syp[n] * (double)fieldScale);
        p.coefs[(size_t)frame * P * M + (size_t)pol * M + mode] = make_float2(cr * ms, ci * ms);
    }
}

// The same overlap for any number of mode groups: the x-modes in chunks of
// OVC (T[y][m] of one chunk in shared memory, the int16 field re-read per
// chunk), then c_mn for the modes whose m falls in the chunk, with Hy read
// from global memory.  Per chunk the sums run in k_overlap_f32's order, so
// the coefficients equal its bit for bit.  The fallback beyond the
// register-tiled overlaps (more than 64 mode groups, or more than 32 on
// fields taller than 128 rows).  One block of 256 threads per (frame,
// polarisation).
constexpr int OVC = 16;
__global__ void __launch_bounds__(256) k_overlap_f32_chunked(DhInvParams p, int nx, int ny) {
    extern __shared__ float smo[];
    const int G = p.maxMG, M = p.modeCount;
    const int unit = blockIdx.x;
    const int P = p.polCount;
    const int pol = unit % P, frame = unit / P;
    const int tid = threadIdx.x;
    float* hx = smo;                                   // [nx][OVC]
    float* T = hx + (size_t)nx * OVC;                  // [2][ny][OVC + 1]
    const short* gx = p.hgX + (size_t)pol * G * nx;
    const short* gy = p.hgY + (size_t)pol * G * ny;
    const size_t npix = (size_t)nx * ny;
    const int S = p.statsStride;
    const float fieldScale = 1.0f / p.stats[3 * P * S + pol * S + frame];
    const float* sxp = p.hgScaleX + pol * G;
    const float* syp = p.hgScaleY + pol * G;
    for (int m0 = 0; m0 < G; m0 += OVC) {
        __syncthreads();   // the previous chunk's tables are consumed
        for (int e = tid; e < nx * OVC; e += blockDim.x) {
            const int x = e / OVC, m = m0 + e % OVC;
            hx[e] = m < G ? (float)gx[(size_t)m * nx + x] : 0.f;
        }
        __syncthreads();
        for (int r = tid; r < 2 * ny; r += blockDim.x) {
            const int plane = r / ny, y = r - plane * ny;
            const short* row = (plane ? p.fieldI : p.fieldR) + (size_t)unit * npix + (size_t)y * nx;
            float acc[OVC];
#pragma unroll
            for (int m = 0; m < OVC; m++) acc[m] = 0.f;
            for (int x0 = 0; x0 < nx; x0 += 8) {
                const uint4 raw = __ldg(reinterpret_cast<const uint4*>(row + x0));
                const unsigned wv[4] = {raw.x, raw.y, raw.z, raw.w};
#pragma unroll
                for (int t = 0; t < 8; t++) {
                    const float v = (float)(short)((wv[t >> 1] >> (16 * (t & 1))) & 0xFFFF);
                    const float4* hv = reinterpret_cast<const float4*>(hx + (x0 + t) * OVC);
#pragma unroll
                    for (int m4 = 0; m4 < OVC / 4; m4++) {
                        const float4 h = hv[m4];
                        acc[4 * m4 + 0] = fmaf(v, h.x, acc[4 * m4 + 0]);
                        acc[4 * m4 + 1] = fmaf(v, h.y, acc[4 * m4 + 1]);
                        acc[4 * m4 + 2] = fmaf(v, h.z, acc[4 * m4 + 2]);
                        acc[4 * m4 + 3] = fmaf(v, h.w, acc[4 * m4 + 3]);
                    }
                }
            }
            float* Tp = T + (size_t)r * (OVC + 1);
#pragma unroll
            for (int m = 0; m < OVC; m++) Tp[m] = acc[m];
        }
        __syncthreads();
        for (int mode = tid; mode < M; mode += blockDim.x) {
            int g = (int)((sqrtf(8.0f * mode + 1.0f) - 1.0f) * 0.5f);
            while ((g + 1) * (g + 2) / 2 <= mode) g++;
            while (g * (g + 1) / 2 > mode) g--;
            const int n = mode - g * (g + 1) / 2;
            const int m = g - n;
            if (m < m0 || m >= m0 + OVC) continue;
            const short* hn = gy + (size_t)n * ny;
            const float* t0 = T + (m - m0);
            const float* t1 = T + (size_t)ny * (OVC + 1) + (m - m0);
            float cr = 0.f, ci = 0.f;
            for (int y = 0; y < ny; y++) {
                const float hv = (float)hn[y];
                cr = fmaf(hv, t0[(size_t)y * (OVC + 1)], cr);
                ci = fmaf(hv, t1[(size_t)y * (OVC + 1)], ci);
            }
            const float ms = (float)((double)sxp[m] * (double)syp[n] * (double)fieldScale);
            p.coefs[(size_t)frame * P * M + (size_t)pol * M + mode] = make_float2(cr * ms, ci * ms);
        }
    }
}

cudaError_t dh_launch_field128(const DhInvParams& p, int withOverlap, cudaStream_t s);

namespace {

template <int W, int H, int WW>
cudaError_t launchField(const DhInvParams& p, cudaStream_t s) {
    constexpr int NT = H * W / 32;
    const size_t smem = sizeof(float2) * (size_t)H * (WW + 1) + sizeof(short) * 2 * (size_t)H * (W + 8) +
                        sizeof(float2) * (size_t)(H / WW + W / WW) * (WW + 1) + sizeof(float) * W + sizeof(int) * W +
                        sizeof(StatF) * (NT / 32);
    auto kern = k_field_full<W, H, WW>;
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(kern), (int)smem);
    if (e != cudaSuccess) return e;
    kern<<<(unsigned)(p.frameCount * p.polCount), NT, smem, s>>>(p);
    return cudaGetLastError();
}

template <int GMAX>
cudaError_t launchOverlapF32(const DhInvParams& p, int nx, int ny, cudaStream_t s) {
    const size_t smem = sizeof(float) * ((size_t)nx * GMAX + (size_t)p.maxMG * ny + 2 * (size_t)ny * (p.maxMG + 1));
    if (smem > 200 * 1024) return cudaErrorNotSupported;
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(k_overlap_f32<GMAX>), (int)smem);
    if (e != cudaSuccess) return e;
    k_overlap_f32<GMAX><<<(unsigned)(p.frameCount * p.polCount), 2 * ny, smem, s>>>(p, nx, ny);
    return cudaGetLastError();
}

}  // namespace

// Full-resolution field kernels up to 128 x 128; cudaErrorNotSupported
// outside their shapes.  withOverlap: fuse the tensor-core overlap (128 x 128
// fields, maxMG <= 32); *fused reports whether it did, or, beside
// cudaErrorNotSupported, that the fields alone are supported.
cudaError_t dh_launch_field_full(const DhInvParams& p, int withOverlap, int* fused, cudaStream_t s) {
    *fused = 0;
    if (p.lowres || p.logW != p.logH) return cudaErrorNotSupported;
    const bool pow2 = p.logw == p.logh && p.w == (1 << p.logw) && p.h == (1 << p.logh);
    if (p.logW == 7) {
        const int ovl = withOverlap && p.maxMG > 0 && p.coefs && p.maxMG <= 32;
        const cudaError_t e = dh_launch_field128(p, ovl, s);
        *fused = ovl && (e != cudaErrorNotSupported || pow2);
        return e;
    }
    if (!pow2) return cudaErrorNotSupported;
    if (p.frameCount * p.polCount <= 0) return cudaSuccess;
    const int W = 1 << p.logW, w = 1 << p.logw;
    if (w == 16) {
        if (W == 64) return launchField<64, 64, 16>(p, s);
        if (W == 32) return launchField<32, 32, 16>(p, s);
    } else if (w == 32) {
        if (W == 64) return launchField<64, 64, 32>(p, s);
    }
    return cudaErrorNotSupported;
}

// FP32 overlap of the int16 fields [unit][ny][nx]; cudaErrorNotSupported
// outside its shapes (2 ny <= 256 threads, nx a multiple of 8, G <= 64).
cudaError_t dh_launch_overlap_f32(const DhInvParams& p, int nx, int ny, cudaStream_t s) {
    if (p.maxMG <= 0 || !p.coefs) return cudaSuccess;
    if (2 * ny > 256 || nx % 8 != 0 || ny < 16) return cudaErrorNotSupported;
    if (p.maxMG <= 16) return launchOverlapF32<16>(p, nx, ny, s);
    if (p.maxMG <= 32) return launchOverlapF32<32>(p, nx, ny, s);
    if (p.maxMG <= 64) return launchOverlapF32<64>(p, nx, ny, s);
    return cudaErrorNotSupported;
}

// The chunked FP32 overlap (any maxMG); cudaErrorNotSupported when nx is not
// a multiple of 8 or the chunk tables exceed shared memory.
cudaError_t dh_launch_overlap_f32_chunked(const DhInvParams& p, int nx, int ny, cudaStream_t s) {
    if (p.maxMG <= 0 || !p.coefs) return cudaSuccess;
    if (nx % 8 != 0 || nx < 8 || ny < 1) return cudaErrorNotSupported;
    const size_t smem = sizeof(float) * ((size_t)nx * OVC + 2 * (size_t)ny * (OVC + 1));
    if (smem > 227 * 1024) return cudaErrorNotSupported;
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(k_overlap_f32_chunked), (int)smem);
    if (e != cudaSuccess) return e;
    k_overlap_f32_chunked<<<(unsigned)(p.frameCount * p.polCount), 256, smem, s>>>(p, nx, ny);
    return cudaGetLastError();
}
