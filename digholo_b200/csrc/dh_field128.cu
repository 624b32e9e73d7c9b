// Inverse stage of 128 x 128 full-resolution fields (IFFTResolutionMode 0)
// with square IFFT windows of 16, 32 or 48 pixels: the Fourier window placed
// in the H x W plane -> IFFT -> field statistics -> reference wave, -conj,
// int16 rounding, then the separable HG overlap on the tensor cores
// (digHolo.cpp:8734, 2354, 2701-2837 and 2149-2341).
//
// Transform.  Along each axis, output 8 t + u (u < 8) is a 16-point inverse
// DFT over t of the window's samples folded modulo 16 (F = w / 16 samples per
// point) with the phase e^{2 pi i k u / 128}.  32-pixel windows run the first
// stage of a 32-point radix-2 transform instead of the fold: u < 4 takes the
// sums, u >= 4 the twiddled differences.
//
// One persistent block of 512 threads per SM.  Each thread holds 32 pixels of
// the field in registers (one row, two adjacent u, 16 t), as packed pairs
// that go through the transform, the statistics and the quantisation two at
// a time (f32x2: half the instructions of scalar code, the same bits), and
// end as one 32-bit store of two int16 pixels.  Tables, the modes' operand
// and the row constants are laid out once per block.  Per unit (frame,
// polarisation) three barriers separate
//   1. row transform and statistics of unit n; the window of unit n + 1 is
//      on its way (cp.async);
//   2. overlap sums of unit n - 1 out of tensor memory; int16 rounding of
//      unit n into the staging planes;
//   3. the tensor-core products of unit n are issued; some warps run the
//      column transform of unit n + 1, the others copy unit n's planes out
//      and contract unit n - 1's sums with Hy.
//
// Overlap.  T[y][m] = sum_x F[y][x] Hx[m][x] exactly in integers: the staged
// int16 rows are the A operand as they lie (bytes 2 x: low, 2 x + 1: high).
// As u8 with the modes' digits at the even bytes of B (zeros between) they
// contribute the low bytes, as s8 with the digits at the odd bytes the high
// ones.  The digits are the two bytes of Hx + 32768 (both u8, so one product
// of N = 2 GN takes both), and the last mode row is the constant 1, whose sums
// S undo the offset: T = sum F (Hx + 32768) - 32768 S.
//
// Bound: the phases' latency with four warps per scheduler (46 % of the issue
// slots, 54 instructions per pixel).  2048 units, 16-pixel windows, 15 groups:
// 110 us; 304 us with one block per unit, scalar arithmetic (116 instructions
// per pixel) and bf16 products.
#include <cuda_runtime.h>
#include <math.h>
#include <stdint.h>

#include "dh_common.cuh"
#include "dh_f32x2.cuh"
#include "dh_fft.cuh"
#include "dh_host.h"
#include "dh_params.h"
#include "dh_tc.cuh"

using namespace dh;

namespace {

constexpr int N = 128;        // field side
constexpr int NT = 512;       // threads per block
constexpr int TS = N;         // row stride (floats) of the overlap sums and of Hy
constexpr int STG = 2 * N * N * 2;   // staging bytes: R and I planes

__host__ __device__ constexpr int brev4c(int i) {
    return ((i & 1) << 3) | ((i & 2) << 1) | ((i & 4) >> 1) | ((i & 8) >> 3);
}

// Shared-memory plan (byte offsets from a 1024-byte aligned base); the host
// computes the same numbers.
struct F128Smem {
    int bop, win, a, t, hy, sc, tw1, tw2, rot1, rot2, refX, modes, red, misc, total;
};
// Whether the column-stage output holds each part twice (where it fits).
__host__ __device__ constexpr bool f128Dup(int F, int GN) { return F == 1 ? GN < 48 : F == 2 && GN == 16; }

__host__ __device__ constexpr F128Smem f128Smem(int F, bool ovl, int GN, int G, int M) {
    F128Smem s{};
    const int w = 16 * F;
    int o = STG;
    s.bop = o;
    o += ovl ? 8 * GN * 128 : 0;                 // [even, odd][2 atoms][2 GN][128 B]
    s.win = o;
    o += w * w * 8;
    s.a = o;                                     // [128][w + 1] (re, re, im, im), or (re, im)
    o += N * (w + 1) * (f128Dup(F, GN) ? 16 : 8);
    s.t = o;
    o += ovl ? 2 * GN * TS * 4 : 0;
    s.hy = o;
    o += ovl ? (G + 3) / 4 * 4 * TS * 4 : 0;
    s.sc = o;                                    // [2][GN] mode scales along x and y
    o += ovl ? 2 * GN * 4 : 0;
    s.tw1 = o;                                   // [8 or 4 u][w or 16] float2
    o += (F == 2 ? 4 * 32 : 8 * 16) * 8;
    s.rot1 = o;                                  // F >= 3: [8 u][F] float2
    o += F >= 3 ? (8 * F * 8 + 15) / 16 * 16 : 0;
    s.tw2 = o;                                   // [k][pairs] {tr, ti}, then [k][pairs] {-ti}
    o += 64 * 24;
    s.rot2 = o;
    o += F >= 3 ? 4 * F * 24 : 0;
    s.refX = o;                                  // [64] (xr, xi, xr', xi') of pixels 2 q, 2 q + 1
    o += 64 * 16;
    s.red = o;                                   // [5][512] statistics of the threads
    o += 5 * NT * 4;
    s.modes = o;
    o += ovl ? (M * 4 + 15) / 16 * 16 : 0;
    s.misc = o;
    o += 112;
    s.total = o + 1024;
    return s;
}

__device__ __forceinline__ void cpAsync16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(tc::sAddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsyncWait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One 64-pixel x 128-row tile of the swizzled staging planes to the field.
__device__ __forceinline__ void storeTile(const CUtensorMap* map, const void* src, int x, int y) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.tile.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(tc::sAddr(src))
                 : "memory");
}
__device__ __forceinline__ void storeCommit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// the staging planes have been read / the field has been written
__device__ __forceinline__ void storeWaitRead() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void storeWait() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// Two int32 to one word of two saturated int16 (lo in the low half).
__device__ __forceinline__ uint32_t packSat(int lo, int hi) {
    uint32_t r;
    asm("cvt.pack.sat.s16.s32 %0, %1, %2;" : "=r"(r) : "r"(hi), "r"(lo));
    return r;
}

// Round half to even of |v| < 2^22.
__device__ __forceinline__ int roundMagic(float v) { return __float_as_int(__fadd_rn(v, 12582912.0f)) - 0x4B400000; }

// Within int16, -32768 for NaN.
__device__ __forceinline__ float clamp16(float v) { return fminf(fmaxf(v, -32768.0f), 32767.0f); }

__device__ __forceinline__ float2 cfmaS(float2 a, float2 b, float2 c) {
    return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

// Twiddle pairs for the packed complex product: table[n] of (re, im), then of -im.
__device__ __forceinline__ void putTwiddle(f2x* table, int n, int at, float2 a, float2 b) {
    table[2 * at] = pk(a.x, b.x);
    table[2 * at + 1] = pk(a.y, b.y);
    table[2 * n + at] = pk(-a.y, -b.y);
}

// The 16 folded and phased inputs of one column sub-problem u of window column c.
template <int F>
__device__ __forceinline__ void columnInputs(const float2* win, int c, int u, int r0, const float2* tw1, const float2* rot1,
                                             float2 (&b)[16]) {
    constexpr int W = 16 * F;
    if (F == 2) {
        const bool diff = u >= 4;
        const float2* tw = tw1 + (u & 3) * 32;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const float2 a0 = cmul(win[((k - r0) & 31) * W + c], tw[k]);
            const float2 a1 = cmul(win[((k + 16 - r0) & 31) * W + c], tw[k + 16]);
            if (!diff) {
                b[k] = cadd(a0, a1);
            } else {
                const float2 d = csub(a0, a1);
                const float2 t = tw128(4 * k);
                b[k] = k == 0 ? d : (k == 8 ? make_float2(-d.y, d.x) : cmul(d, make_float2(t.x, -t.y)));
            }
        }
    } else {
        const float2* tw = tw1 + u * 16;
#pragma unroll
        for (int k = 0; k < 16; k++) {
            const int j = (k - r0) & 15;
            float2 v = win[j * W + c];
#pragma unroll
            for (int f = 1; f < F; f++) v = cfmaS(win[(j + 16 * f) * W + c], rot1[u * F + f], v);
            b[k] = cmul(v, tw[k]);
        }
    }
}

template <int F, bool OVL, int GN>
__global__ void __launch_bounds__(NT, 1)
    k_field128(const __grid_constant__ CUtensorMap mapR, const __grid_constant__ CUtensorMap mapI, DhInvParams p, int units) {
    constexpr int W = 16 * F;
    constexpr int ALD = W + 1;
    constexpr bool DUP = f128Dup(F, GN);  // rows of A hold each part twice: the packed operands as loaded
    constexpr int S1W = F == 1 ? 4 : 8;   // warps of the column transform
    constexpr int TMCOLS = GN == 16 ? 128 : (GN == 32 ? 256 : 512);
    extern __shared__ float4 smf4[];
    unsigned char* base = tc::alignShared1024(reinterpret_cast<unsigned char*>(smf4));
    const F128Smem L = f128Smem(F, OVL, GN, OVL ? p.maxMG : 0, OVL ? p.modeCount : 0);
    unsigned char* stg = base;                                        // [plane][atom][128][128 B], swizzled
    unsigned char* bop = base + L.bop;
    float2* win = reinterpret_cast<float2*>(base + L.win);
    float4* A = reinterpret_cast<float4*>(base + L.a);
    float* T = reinterpret_cast<float*>(base + L.t);                  // [plane * GN + m][TS]
    float* hy = reinterpret_cast<float*>(base + L.hy);                // [n][TS]
    float* sc = reinterpret_cast<float*>(base + L.sc);                // [x, y][GN]
    float2* tw1 = reinterpret_cast<float2*>(base + L.tw1);
    float2* rot1 = reinterpret_cast<float2*>(base + L.rot1);
    f2x* tw2 = reinterpret_cast<f2x*>(base + L.tw2);
    f2x* rot2 = reinterpret_cast<f2x*>(base + L.rot2);
    int4* refX = reinterpret_cast<int4*>(base + L.refX);
    float* red = reinterpret_cast<float*>(base + L.red);
    int* modeMN = reinterpret_cast<int*>(base + L.modes);
    uint64_t* bar = reinterpret_cast<uint64_t*>(base + L.misc);
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(bar + 1);
    int* maxBits = reinterpret_cast<int*>(tmemSlot + 1);              // [2] by unit parity
    int* maxIdx = maxBits + 2;                                        // [2]
    float* sums = reinterpret_cast<float*>(maxIdx + 2);               // [2][5]

    const int P = p.polCount;
    const int pol = blockIdx.x % P;           // the grid is a multiple of P
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const short* ref = p.refWave + (size_t)pol * 4 * N;
    const int r0 = ((p.sy[pol] + N / 2) % N + N) % N;
    const int sx0 = p.sx0[pol];
    const int G = p.maxMG, M = p.modeCount;

    // ---- tables, once per block
    if (F == 2) {
        for (int e = tid; e < 4 * 32; e += NT) {
            const int u = e >> 5, k = e & 31;
            tw1[e] = expPos(p.twiddle, ((r0 + ((k - r0) & 31)) & (N - 1)) * u, N);
        }
        for (int e = tid; e < 2 * 32; e += NT) {
            const int u = 2 * (e >> 5), k = e & 31;
            const int col = (sx0 + ((k - sx0) & 31)) & (N - 1);
            const float2 a = expPos(p.twiddle, col * u, N), b = expPos(p.twiddle, col * (u + 1), N);
            putTwiddle(tw2, 64, 2 * k + (e >> 5), a, b);
        }
    } else {
        for (int e = tid; e < 8 * 16; e += NT) {
            const int u = e >> 4, k = e & 15;
            tw1[e] = expPos(p.twiddle, (r0 + ((k - r0) & 15)) * u, N);
        }
        for (int e = tid; e < 4 * 16; e += NT) {
            const int u = 2 * (e >> 4), k = e & 15;
            const int col = sx0 + ((k - sx0) & 15);
            const float2 a = expPos(p.twiddle, col * u, N), b = expPos(p.twiddle, col * (u + 1), N);
            putTwiddle(tw2, 64, 4 * k + (e >> 4), a, b);
        }
        if (F >= 3) {
            for (int e = tid; e < 8 * F; e += NT) rot1[e] = expPos(p.twiddle, 16 * (e % F) * (e / F), N);
            for (int e = tid; e < 4 * F; e += NT) {
                const int u = 2 * (e / F), f = e % F;
                const float2 a = expPos(p.twiddle, 16 * f * u, N), b = expPos(p.twiddle, 16 * f * (u + 1), N);
                putTwiddle(rot2, 4 * F, 4 * f + (e / F), a, b);
            }
        }
    }
    for (int q = tid; q < N / 2; q += NT)
        refX[q] = make_int4(ref[2 * q], ref[N + 2 * q], ref[2 * q + 1], ref[N + 2 * q + 1]);
    if (tid < 2) { maxBits[tid] = 0; maxIdx[tid] = -1; }
    if (OVL) {
        for (int e = tid; e < GN * 16; e += NT) {
            // bytes of Hx + 32768: row m the low digit, row GN + m the high one
            const int m = e >> 4, q = e & 15;
            uint4 raw = make_uint4(0, 0, 0, 0);
            if (m < G) {
                raw = __ldg(reinterpret_cast<const uint4*>(p.hgX + ((size_t)pol * G + m) * N) + q);
                raw = make_uint4(raw.x ^ 0x80008000u, raw.y ^ 0x80008000u, raw.z ^ 0x80008000u, raw.w ^ 0x80008000u);
            } else if (m == GN - 1) {
                raw = make_uint4(0x00010001u, 0x00010001u, 0x00010001u, 0x00010001u);
            }
            unsigned char* d = bop + (q >> 3) * 2 * GN * 128 + m * 128 + (((q & 7) ^ (m & 7)) << 4);
            const uint32_t E = 0x00FF00FFu;
            const uint4 lo = make_uint4(raw.x & E, raw.y & E, raw.z & E, raw.w & E);
            const uint4 hi = make_uint4((raw.x >> 8) & E, (raw.y >> 8) & E, (raw.z >> 8) & E, (raw.w >> 8) & E);
            *reinterpret_cast<uint4*>(d) = lo;
            *reinterpret_cast<uint4*>(d + GN * 128) = hi;
            *reinterpret_cast<uint4*>(d + 4 * GN * 128) = make_uint4(lo.x << 8, lo.y << 8, lo.z << 8, lo.w << 8);
            *reinterpret_cast<uint4*>(d + 5 * GN * 128) = make_uint4(hi.x << 8, hi.y << 8, hi.z << 8, hi.w << 8);
        }
        for (int e = tid; e < (G + 3) / 4 * 4 * N; e += NT) hy[e] = e < G * N ? (float)p.hgY[(size_t)pol * G * N + e] : 0.f;
        for (int e = tid; e < G; e += NT) {
            sc[e] = p.hgScaleX[pol * G + e];
            sc[GN + e] = p.hgScaleY[pol * G + e];
        }
        for (int mode = tid; mode < M; mode += NT) {
            int g = (int)((sqrtf(8.0f * mode + 1.0f) - 1.0f) * 0.5f);
            while ((g + 1) * (g + 2) / 2 <= mode) g++;
            while (g * (g + 1) / 2 > mode) g--;
            const int n = mode - g * (g + 1) / 2;
            modeMN[mode] = ((g - n) << 16) | n;
        }
        if (tid == 0) tc::mbarInitTc(bar);
        if (warp == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::sAddr(tmemSlot)),
                         "n"(TMCOLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        tc::fenceProxyAsync();
        tc::fenceBeforeSync();
    }
    // the first unit's window
    auto fetchWindow = [&](int unit) {
        const float2* src = p.window + (size_t)unit * W * W;
        for (int e = tid; e < W * W / 2; e += NT) cpAsync16(win + 2 * e, src + 2 * e);
    };
    // column transform: column c lands at position (c + sx0) mod 16 (32 for F = 2) of A's rows
    auto columns = [&](int first, int step) {
        for (int task = first; task < 8 * W; task += step) {
            const int c = task % W, u = task / W;
            float2 b[16];
            columnInputs<F>(win, c, u, r0, tw1, rot1, b);
            ifftDIFf<16>(b);
            const int pos = F == 2 ? ((c + sx0) & 31) : (((c + sx0) & 15) + (c & ~15));
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int at = (8 * brev4c(i) + u) * ALD + pos;
                if (DUP)
                    A[at] = make_float4(b[i].x, b[i].x, b[i].y, b[i].y);
                else
                    reinterpret_cast<float2*>(A)[at] = b[i];
            }
        }
    };
    int unit = blockIdx.x;
    dependentWait();
    if (unit < units) fetchWindow(unit);
    cpAsyncWait();
    __syncthreads();
    uint32_t tmem = 0;
    if (OVL) {
        tc::fenceAfterSync();
        tmem = *tmemSlot;
    }
    columns(tid, NT);

    // this thread's pixels: row y, x = 8 t + u and 8 t + u + 1
    const int y = F == 2 ? 16 * (warp >> 1) + (lane >> 1) : 8 * warp + (lane >> 2);
    const int u = F == 2 ? 4 * (warp & 1) + 2 * (lane & 1) : 2 * (lane & 3);
    const int yr = ref[2 * N + y], yi = ref[3 * N + y];
    const float yv = p.yAxis[y];
    const float yw = yv + (yv < 0.f ? fabsf((p.yAxis[1] - p.yAxis[0]) * (float)N) : 0.f);
    const float dx = p.xAxis[1] - p.xAxis[0], xc = p.xAxis[N / 2];
    const float inv = 1.0f / (float)(N * N);
    unsigned char* myStg = stg + y * 128 + 2 * u;
    const int sw = (y & 7) << 4;
    const float* refF = p.refWaveF + (size_t)pol * 4 * N;

    // overlap coefficients of the unit whose sums lie in T, four y-modes by
    // four x-modes of both planes per warp (each lane four rows y); lane l
    // ends with output (n, m, plane) = (l / 8, (l / 2) % 4, l % 2)
    auto contract = [&](int doneUnit, float scale, int first, int step) {
        const float fieldScale = 1.0f / scale;
        const int g4 = (G + 3) / 4;
        float* out = reinterpret_cast<float*>(p.coefs + (size_t)doneUnit * M);
        for (int tile = first; tile < g4 * (g4 + 1) / 2; tile += step) {
            const int mn = modeMN[tile];
            const int m0 = 4 * (mn >> 16), n0 = 4 * (mn & 0xFFFF);
            float4 t[8];
#pragma unroll
            for (int j = 0; j < 8; j++) t[j] = reinterpret_cast<const float4*>(T + ((j & 1) * GN + m0 + (j >> 1)) * TS)[lane];
            float v[32];
#pragma unroll
            for (int n = 0; n < 4; n++) {
                const float4 h = reinterpret_cast<const float4*>(hy + (n0 + n) * TS)[lane];
                const f2x h0 = pk(h.x, h.y), h1 = pk(h.z, h.w);
#pragma unroll
                for (int j = 0; j < 8; j++) {
                    const float2 c = upk(fma2(h1, pk(t[j].z, t[j].w), mul2(h0, pk(t[j].x, t[j].y))));
                    v[8 * n + j] = c.x + c.y;
                }
            }
#pragma unroll
            for (int off = 16; off >= 1; off >>= 1) {
                const bool up = lane & off;
#pragma unroll
                for (int i = 0; i < off; i++) {
                    const float keep = up ? v[i + off] : v[i], send = up ? v[i] : v[i + off];
                    v[i] = keep + __shfl_xor_sync(0xffffffffu, send, off);
                }
            }
            const int n = n0 + (lane >> 3), m = m0 + ((lane >> 1) & 3);
            if (m + n < G) {
                const float ms = (float)((double)sc[m] * (double)sc[GN + n] * (double)fieldScale);
                out[2 * ((m + n) * (m + n + 1) / 2 + n) + (lane & 1)] = v[0] * ms;
            }
        }
    };
    // the sums of the last issued products: tensor memory -> T
    auto readSums = [&]() {
        tc::fenceAfterSync();
        constexpr int MC = GN / 2;                       // x-modes per warp
        const int pl = warp >> 3, m0 = ((warp >> 2) & 1) * MC;
        const uint32_t row = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(pl * 4 * GN);
        const int yy = (warp & 3) * 32 + lane;
        uint32_t e1[8], o1[8];                           // the last eight x-modes: the constant mode among them
        tc::tmemLoad8(row + GN - 8, e1);
        tc::tmemLoad8(row + 3 * GN - 8, o1);
        tc::tmemWaitLoad8(e1);
        tc::tmemWaitLoad8(o1);
        const int S0 = 128 * (int)e1[7], S1 = 128 * (int)o1[7];
#pragma unroll
        for (int c0 = 0; c0 < MC; c0 += 8) {
            uint32_t e0[8], o0[8];
            tc::tmemLoad8(row + m0 + c0, e0);
            tc::tmemLoad8(row + GN + m0 + c0, e1);
            tc::tmemLoad8(row + 2 * GN + m0 + c0, o0);
            tc::tmemLoad8(row + 3 * GN + m0 + c0, o1);
            tc::tmemWaitLoad8(e0);
            tc::tmemWaitLoad8(e1);
            tc::tmemWaitLoad8(o0);
            tc::tmemWaitLoad8(o1);
#pragma unroll
            for (int i = 0; i < 8; i++)
                T[(pl * GN + m0 + c0 + i) * TS + yy] =
                    fmaf((float)((int)o1[i] - S1), 65536.0f,
                         fmaf((float)((int)e1[i] + (int)o0[i] - S0), 256.0f, (float)(int)e0[i]));
        }
        tc::fenceBeforeSync();
    };

    int it = 0, prev = -1;
    float prevScale = 1.f;
    bool ok = true;
    __syncthreads();
    for (; unit < units; unit += gridDim.x, it++) {
        const int par = it & 1;
        const int nextUnit = unit + gridDim.x;
        if (nextUnit < units) fetchWindow(nextUnit);
        // ---- row transform of this thread's pixel pairs
        f2x fr[16], fi[16];
        auto rowSample = [&](int k) {   // (re, re), (im, im)
            if (DUP) return reinterpret_cast<const ulonglong2*>(A)[y * ALD + k];
            const float2 v = reinterpret_cast<const float2*>(A)[y * ALD + k];
            return make_ulonglong2(pk1(v.x), pk1(v.y));
        };
        if (F == 2) {
            const ulonglong2* tw = reinterpret_cast<const ulonglong2*>(tw2) + (u & 2) / 2;   // 2 pairs
            const f2x* ntw = tw2 + 128 + (u & 2) / 2;
            auto twiddle = [&](int k, f2x& re, f2x& im) {
                const ulonglong2 t = tw[2 * k];
                cmul2(re, im, t.x, t.y, ntw[2 * k]);
            };
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const ulonglong2 a = rowSample(k), b = rowSample(k + 16);
                f2x ar = a.x, ai = a.y, br = b.x, bi = b.y;
                twiddle(k, ar, ai);
                twiddle(k + 16, br, bi);
                if (u < 4) {   // warp-uniform
                    fr[k] = add2(ar, br);
                    fi[k] = add2(ai, bi);
                } else if (k == 8) {
                    fr[k] = sub2(bi, ai);
                    fi[k] = sub2(ar, br);
                } else {
                    fr[k] = sub2(ar, br);
                    fi[k] = sub2(ai, bi);
                    if (k != 0) {
                        const float2 t = tw128(4 * k);
                        cmul2(fr[k], fi[k], pk1(t.x), pk1(-t.y), pk1(t.y));
                    }
                }
            }
        } else {
            const ulonglong2* tw = reinterpret_cast<const ulonglong2*>(tw2) + u / 2;   // 4 pairs
            const f2x* ntw = tw2 + 128 + u / 2;
            const ulonglong2* rot = reinterpret_cast<const ulonglong2*>(rot2) + u / 2;
            const f2x* nrot = rot2 + 8 * F + u / 2;
#pragma unroll
            for (int k = 0; k < 16; k++) {
                const ulonglong2 a = rowSample(k);
                fr[k] = a.x;
                fi[k] = a.y;
#pragma unroll
                for (int f = 1; f < F; f++) {
                    const ulonglong2 b = rowSample(k + 16 * f);
                    const f2x br = b.x, bi = b.y;
                    const ulonglong2 r = rot[4 * f];
                    fr[k] = fma2(br, r.x, fma2(bi, nrot[4 * f], fr[k]));
                    fi[k] = fma2(br, r.y, fma2(bi, r.x, fi[k]));
                }
                const ulonglong2 t = tw[4 * k];
                cmul2(fr[k], fi[k], t.x, t.y, ntw[4 * k]);
            }
        }
        ifftDIF2<16>(fr, fi);

        const size_t fieldOff = (size_t)unit * N * N;
        if (p.field32) {
            // -conj(A R) with the unquantised wave
            const float2 ryf = make_float2(refF[2 * N + y], refF[3 * N + y]);
            float4* out = reinterpret_cast<float4*>(p.field32 + fieldOff + (size_t)y * N + u);
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const int x = 8 * brev4c(i) + u;
                const float2 a = upk(fr[i]), b = upk(fi[i]);
                const float2 rx = __ldg(reinterpret_cast<const float2*>(refF + x));
                const float2 ry = __ldg(reinterpret_cast<const float2*>(refF + N + x));
                const float2 w0 = cmul(make_float2(a.x, b.x), cmul(ryf, make_float2(rx.x, ry.x)));
                const float2 w1 = cmul(make_float2(a.y, b.y), cmul(ryf, make_float2(rx.y, ry.y)));
                out[4 * brev4c(i)] = make_float4(-w0.x, w0.y, -w1.x, w1.y);
            }
        }
        if (!OVL && p.fieldsOnly) {   // block-uniform
            cpAsyncWait();
            __syncthreads();
            if (nextUnit < units) columns(tid, NT);
            __syncthreads();
            continue;
        }

        // ---- statistics over the untilted field (digHolo.cpp:8866-8870)
        f2x sP = pk(0.f, 0.f), sX = sP, sE = sP;
        float mx = 0.f;
        const f2x inv2 = pk1(inv);
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const f2x I0 = fma2(fr[i], fr[i], mul2(fi[i], fi[i]));
            const float2 v = upk(I0);
            mx = fmaxf(fmaxf(mx, v.x), v.y);
            const f2x I = mul2(I0, inv2);
            sP = add2(sP, I);
            sX = fma2(I, pk1((float)(8 * brev4c(i) - N / 2)), sX);
            sE = fma2(I, I, sE);
        }
        {
            const float2 v = upk(sP), t = upk(sX), e = upk(sE);
            const float Prow = v.x + v.y;
            const float xs = fmaf((float)u, Prow, v.y) + (t.x + t.y);   // x = dx (index - N / 2) + xc
            red[tid] = Prow;
            red[NT + tid] = fmaf(dx, xs, xc * Prow);
            red[2 * NT + tid] = yv * Prow;
            red[3 * NT + tid] = yw * Prow;
            red[4 * NT + tid] = e.x + e.y;
        }
        const unsigned wm = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
        if (lane == 0) atomicMax(&maxBits[par], (int)wm);
        cpAsyncWait();
        // the planes of the previous unit have left the staging buffer
        if (tid == NT - 64) storeWaitRead();
        if (OVL && it > 0) {
            // ... and its products have read it
            const bool done = tc::mbarWaitTc(bar, (unsigned)((it - 1) & 1));
            if (done) readSums();
            ok = !__syncthreads_or(!done);
            if (!ok) break;
        } else {
            __syncthreads();
        }
        const float maxI = __int_as_float(maxBits[par]);
        const float scale = __fdiv_rn(32767.0f, sqrtf(maxI));
        if (mx == maxI) {
            // the pixel that holds the maximum: the largest index on ties
            int best = -1;
#pragma unroll
            for (int i = 0; i < 16; i++) {
                const float2 v = upk(fma2(fr[i], fr[i], mul2(fi[i], fi[i])));
                const int idx = 2 * y * N + 8 * brev4c(i) + u;
                if (v.x == maxI) best = max(best, idx);
                if (v.y == maxI) best = max(best, idx + 1);
            }
            atomicMax(&maxIdx[par], best);
        }
        // ---- reference wave, -conj(A . ref), int16 rounding (digHolo.cpp:2741-2833).
        // Within a finite, nonzero field |scale v| stays below 2^22 and the
        // packing saturates; otherwise (scale infinite or zero) the value is
        // clamped first, NaN to -32768.
        const f2x K2 = pk1((float)(1.0 / (16383.0 * 16383.0)));
        const f2x scale2 = pk1(scale);
        const bool plain = maxI > 0.f && maxI < 1e37f;
#pragma unroll
        for (int i = 0; i < 16; i++) {
            const int t = brev4c(i);
            const int4 rx = refX[4 * t + (u >> 1)];
            const f2x adjR = mul2(pk((float)(yr * rx.x - yi * rx.y), (float)(yr * rx.z - yi * rx.w)), K2);
            const f2x adjI = mul2(pk((float)(yr * rx.y + yi * rx.x), (float)(yr * rx.w + yi * rx.z)), K2);
            // scalar sums: the packed forms of a product and a sum may be fused into one rounding
            const float2 p0 = upk(mul2(fi[i], adjI)), p1 = upk(mul2(fr[i], adjR));
            const float2 p2 = upk(mul2(fr[i], adjI)), p3 = upk(mul2(fi[i], adjR));
            const f2x vr = mul2(scale2, pk(__fsub_rn(p0.x, p1.x), __fsub_rn(p0.y, p1.y)));
            const f2x vi = mul2(scale2, pk(__fadd_rn(p2.x, p3.x), __fadd_rn(p2.y, p3.y)));
            float2 a = upk(vr), b = upk(vi);
            if (!plain) {   // block-uniform
                a = make_float2(clamp16(a.x), clamp16(a.y));
                b = make_float2(clamp16(b.x), clamp16(b.y));
            }
            const uint32_t wr = packSat(roundMagic(a.x), roundMagic(a.y));
            const uint32_t wi = packSat(roundMagic(b.x), roundMagic(b.y));
            unsigned char* d = myStg + (t >> 3) * (N * 128) + (((t & 7) << 4) ^ sw);
            *reinterpret_cast<uint32_t*>(d) = wr;
            *reinterpret_cast<uint32_t*>(d + 2 * N * 128) = wi;
        }
        tc::fenceProxyAsync();
        __syncthreads();

        // ---- products of this unit; columns of the next; planes out; the previous unit's coefficients
        if (OVL && warp == NT / 32 - 1) {
            if (lane == 0) {
                tc::fenceAfterSync();
                const uint32_t a0 = tc::sAddr(stg), b0 = tc::sAddr(bop);
#pragma unroll
                for (int pl = 0; pl < 2; pl++) {
                    const uint32_t d = tmem + (uint32_t)(pl * 4 * GN);
#pragma unroll
                    for (int k = 0; k < 8; k++) {
                        const uint64_t ad = tc::smemDesc(a0 + (uint32_t)(pl * 2 + (k >> 2)) * (N * 128) + (uint32_t)(k & 3) * 32);
                        const uint32_t kb = b0 + (uint32_t)(k >> 2) * (2 * GN * 128) + (uint32_t)(k & 3) * 32;
                        tc::mmaI8(d, ad, tc::smemDesc(kb), tc::instrDescI8s(128, 2 * GN, false, false), k > 0);
                        tc::mmaI8(d + 2 * GN, ad, tc::smemDesc(kb + 4 * GN * 128), tc::instrDescI8s(128, 2 * GN, true, false), k > 0);
                    }
                }
                tc::mmaCommit(bar);
            }
            __syncwarp();
        }
        if (warp < S1W) {
            if (nextUnit < units) columns(tid, 32 * S1W);
        } else {
            if (tid == NT - 64) {
#pragma unroll
                for (int a = 0; a < 2; a++) {
                    storeTile(&mapR, stg + a * N * 128, 64 * a, unit * N);
                    storeTile(&mapI, stg + (2 + a) * N * 128, 64 * a, unit * N);
                }
                storeCommit();
            }
            if (OVL && prev >= 0 && warp < NT / 32 - 2) contract(prev, prevScale, warp - S1W, NT / 32 - 2 - S1W);
            // the statistics: one warp per sum
            const int j = warp - S1W;
            if (j < 5) {
                const float4* r4 = reinterpret_cast<const float4*>(red + j * NT);
                float s = 0.f;
#pragma unroll
                for (int q = 0; q < NT / 128; q++) {
                    const float4 v = r4[q * 32 + lane];
                    s += (v.x + v.y) + (v.z + v.w);
                }
#pragma unroll
                for (int off = 16; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
                if (lane == 0) sums[par * 5 + j] = s;
            }
        }
        if (tid == 0) { maxBits[par ^ 1] = 0; }
        __syncthreads();
        if (tid == NT - 32) {
            const int S = p.statsStride, frame = unit / P;
            float* s = p.stats + pol * S + frame;
            const int per = P * S;
            const float* v = sums + par * 5;
            s[0] = v[0];
            s[1 * per] = v[1] / v[0];
            s[2 * per] = v[2] / v[0];
            s[3 * per] = scale;
            s[4 * per] = __int_as_float(maxIdx[par]);
            s[5 * per] = p.dA * (v[0] * v[0] / v[4]);
            s[6 * per] = v[3] / v[0];
            maxIdx[par] = -1;
        }
        prev = unit;
        prevScale = scale;
    }
    if (tid == NT - 64) storeWait();
    if (OVL) {
        if (ok && it > 0) {
            ok = !__syncthreads_or(!tc::mbarWaitTc(bar, (unsigned)((it - 1) & 1)));
            if (ok) {
                readSums();
                __syncthreads();
                contract(prev, prevScale, warp, NT / 32);
            }
        }
        if (!ok && tid == 0 && p.status) {
            *(volatile int*)p.status = 2;
            __threadfence_system();
        }
        tc::fenceBeforeSync();
        __syncthreads();
        if (warp == 0) {
            tc::fenceAfterSync();
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMCOLS)
                         : "memory");
        }
    }
}

template <int F, bool OVL, int GN>
cudaError_t launchF(const DhInvParams& p, cudaStream_t s) {
    const F128Smem L = f128Smem(F, OVL, GN, OVL ? p.maxMG : 0, OVL ? p.modeCount : 0);
    if (L.total > 227 * 1024) return cudaErrorNotSupported;
    auto kern = k_field128<F, OVL, GN>;
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(kern), L.total);
    if (e != cudaSuccess) return e;
    const int units = p.frameCount * p.polCount;
    CUtensorMap mapR, mapI;
    memset(&mapR, 0, sizeof(mapR));
    memset(&mapI, 0, sizeof(mapI));
    if (OVL || !p.fieldsOnly) {
        const unsigned long long rows = (unsigned long long)units * N;
        if (!frameTensorMap(mapR, p.fieldR, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, N, rows, 64, N) ||
            !frameTensorMap(mapI, p.fieldI, CU_TENSOR_MAP_DATA_TYPE_UINT16, 2, N, rows, 64, N))
            return cudaErrorNotSupported;
    }
    int grid = smCountCached();
    grid -= grid % p.polCount;   // a block keeps its polarisation
    if (grid > units) grid = units;
    return launchDependent(kern, (unsigned)grid, NT, L.total, s, p.afterForward != 0, mapR, mapI, p, units);
}

template <int F>
cudaError_t launchG(const DhInvParams& p, int withOverlap, cudaStream_t s) {
    if (!withOverlap) return launchF<F, false, 16>(p, s);
    // one mode row of the operand is the constant
    if (p.maxMG < 16) return launchF<F, true, 16>(p, s);
    if (p.maxMG < 32) return launchF<F, true, 32>(p, s);
    return launchF<F, true, 48>(p, s);
}

}  // namespace

// 128 x 128 full-resolution fields with square IFFT windows of 16, 32 or 48
// pixels; cudaErrorNotSupported outside its shapes.  withOverlap: fuse the
// tensor-core overlap (up to 32 mode groups).
cudaError_t dh_launch_field128(const DhInvParams& p, int withOverlap, cudaStream_t s) {
    if (p.lowres || p.refCal || p.logW != 7 || p.logH != 7 || p.w != p.h || p.w % 16 || p.w > 48) return cudaErrorNotSupported;
    if (withOverlap && (p.maxMG <= 0 || p.maxMG > 32 || !p.coefs)) return cudaErrorNotSupported;
    // 16-byte accesses to the caller's buffers
    const uintptr_t al = reinterpret_cast<uintptr_t>(p.fieldR) | reinterpret_cast<uintptr_t>(p.fieldI) |
                         reinterpret_cast<uintptr_t>(p.field32) | reinterpret_cast<uintptr_t>(p.window);
    if (al % 16) return cudaErrorNotSupported;
    if (p.frameCount * p.polCount <= 0) return cudaSuccess;
    const int F = p.w / 16;
    return F == 1 ? launchG<1>(p, withOverlap, s) : F == 2 ? launchG<2>(p, withOverlap, s) : launchG<3>(p, withOverlap, s);
}
