// Inverse stage of full-resolution 512-pixel-wide fields (IFFTResolutionMode
// 0 with a 512-wide FFT window and an IFFT window of at most 64 x 64: the
// large-field workload, 2048 x 2048 frames with 512 x 512 FFT windows): the
// Fourier window placed in the H x W plane -> IFFT -> field statistics ->
// reference wave, -conj, int16 rounding -> separable HG overlap, i.e. the
// reference's FFTW c2c backward (digHolo.cpp:8734), digHoloFieldAnalysis
// (digHolo.cpp:2354), applyTilt16 (digHolo.cpp:2701-2837) and
// overlapFieldSeparable16 (digHolo.cpp:2149-2341).
//
// Transform.  E[y][x] = sum_j sum_c win[j][c] e^{2 pi i (r0 + j) y / H}
// e^{2 pi i (sx0 + c) x / W}.  With y = Ry s + u (Ry = H / 64) the column
// transform of window column c is, for every u, one 64-point inverse DFT over
// m = (r0 + j) mod 64 of win[j][c] e^{2 pi i (r0 + j) u / H}; with
// x = 8 t + v the row transform is, for every v, one 64-point inverse DFT over
// m = (sx0 + c) mod 64 of A[c] e^{2 pi i (sx0 + c) v / W}.  A 64-point
// transform runs on four lanes, 16 points each: a 16-point DFT in registers,
// the twiddle e^{2 pi i lane s1 / 64}, and a 4-point DFT across the lanes.
//
// k_cols512 writes the column stage's output A[unit][y][c] once (32 rows of
// it are 16 KB; a chunk of 256 units stays in L2).  k_field512 then takes 32
// rows at a time, twice: a statistics pass (the int16 scale depends on the
// maximum over the whole field) and a quantising pass.  Blocks are persistent,
// 512 threads, the next rows arriving by cp.async.  A thread holds two
// adjacent v of one row as packed pairs (f32x2): 32 pixels; the lanes' values
// are exchanged through a warp-private buffer, four s1 at a time, so that the
// 4-point DFT is again in registers, and every store carries two pixels.
//
// Overlap.  T[row][m] = sum_x F[row][x] Hx[m][x] of int16 F (R and I rows) and
// int16 Hx is exact in integers: with F = 256 Fh + Fl (Fh signed, Fl
// unsigned bytes) and likewise Hx, four tcgen05.mma.kind::i8 products
// (int32 accumulators in tensor memory, |partial| < 2^25 for 256 pixels) give
// T = 65536 hh + 256 (hl + lh) + ll.  The 128 operand rows are the 32 field
// rows x (R, I) x the two halves of x, so one buffer of 64 KB serves a pass
// and its products run under the next pass's row transform.  Two passes' sums
// are contracted with Hy in FP32; a last kernel sums the 64-row bands.
//
// Bound: the transforms' latency (44 % of the issue slots in both passes with
// four warps per scheduler).  192 units of 512 x 512, 30 groups: columns 25 us,
// statistics 89, quantising and overlap 201 (its global stores 11, the
// contraction 24, the products' issue 7); the band kernels before, which
// repeated the column stage in each pass and used scalar arithmetic, 190 and
// 340.
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

constexpr int WF = 512;       // field width
constexpr int NT = 512;       // threads per block of k_field512
constexpr int RP = 32;        // rows per pass
constexpr int BR = 64;        // rows per band (two passes)
// strides (floats) of the overlap sums [pass][half][plane, m][32 rows] and of
// Hy [n][pass][32 rows]: the 16-byte accesses of a contraction's lanes
// (consecutive m, both passes) fall into distinct banks
constexpr int TS = RP + 4;
constexpr int HP = RP + 4, HS = 2 * HP;
__host__ __device__ constexpr int tPass(int GN) { return 4 * GN * TS + 16; }
constexpr int APITCH = 64;    // buffered row of A (complex): column c at (c + sx0) mod 64, the others zero
constexpr int GNMAX = 32;
constexpr int ITEMS = 256;    // contraction items, at most 144 (32 mode groups), then end marks
// Units whose column stage is held at a time: at most 64 MiB, half of the L2,
// since windows of up to 64 rows have w H <= 512 x 64.
constexpr int CHUNK = 256;

enum { P_STATS = 0, P_QUANT = 1, P_I8 = 2 };

// cos and sin of 2 pi m / 16, m = 0..9
__device__ __constant__ float kC[10] = {1.0f, 0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f, 0.0f,
                                        -0.38268343236508977f, -0.70710678118654752f, -0.92387953251128674f, -1.0f,
                                        -0.92387953251128674f};
__device__ __constant__ float kS[10] = {0.0f, 0.38268343236508977f, 0.70710678118654752f, 0.92387953251128674f, 1.0f,
                                        0.92387953251128674f, 0.70710678118654752f, 0.38268343236508977f, 0.0f,
                                        -0.38268343236508977f};

// 4-point inverse DFT in place (exp(+2 pi i / 4)), natural order.
__device__ __forceinline__ void idft4(float2& a0, float2& a1, float2& a2, float2& a3) {
    const float2 s02 = cadd(a0, a2), d02 = csub(a0, a2);
    const float2 s13 = cadd(a1, a3), d13 = csub(a1, a3);
    const float2 r = make_float2(-d13.y, d13.x);   // +i d13
    a0 = cadd(s02, s13);
    a1 = cadd(d02, r);
    a2 = csub(s02, s13);
    a3 = csub(d02, r);
}

// 16-point inverse DFT in registers, natural order in and out.
__device__ __forceinline__ void idft16(float2 (&v)[16]) {
#pragma unroll
    for (int n2 = 0; n2 < 4; n2++) idft4(v[n2], v[4 + n2], v[8 + n2], v[12 + n2]);
#pragma unroll
    for (int k1 = 1; k1 < 4; k1++) {
#pragma unroll
        for (int n2 = 1; n2 < 4; n2++) {
            const int m = n2 * k1;
            v[4 * k1 + n2] = cmul(v[4 * k1 + n2], make_float2(kC[m], kS[m]));
        }
    }
#pragma unroll
    for (int k1 = 0; k1 < 4; k1++) idft4(v[4 * k1], v[4 * k1 + 1], v[4 * k1 + 2], v[4 * k1 + 3]);
    // X[k1 + 4 k2] sits at v[4 k1 + k2]: transpose the 4 x 4 index grid
    float2 t[16];
#pragma unroll
    for (int k = 0; k < 16; k++) t[k] = v[4 * (k & 3) + (k >> 2)];
#pragma unroll
    for (int k = 0; k < 16; k++) v[k] = t[k];
}

// 64-point inverse DFT on the four lanes l = lane & 3 of a lane quad:
// in v[m1] = x[4 m1 + l], out v[s1] = X[s1 + 16 brev2(l)].  tw64p[k] =
// e^{2 pi i k / 64}.  All 32 lanes of the warp take part.
__device__ __forceinline__ void ifft64q(float2 (&v)[16], int l, const float2* tw64p) {
    idft16(v);
#pragma unroll
    for (int s1 = 1; s1 < 16; s1++) v[s1] = cmul(v[s1], tw64p[(l * s1) & 63]);
    // X[s2] = sum_l y_l i^{l s2}: butterflies across lane bit 1, then bit 0
    const float sA = (l & 2) ? -1.0f : 1.0f;
    const float sB = (l & 1) ? -1.0f : 1.0f;
    const bool rot = (l & 3) == 3;   // bit 0 and bit 1: times i before the second butterfly
#pragma unroll
    for (int s1 = 0; s1 < 16; s1++) {
        float2 a = v[s1];
        const float ox = __shfl_xor_sync(0xffffffffu, a.x, 2);
        const float oy = __shfl_xor_sync(0xffffffffu, a.y, 2);
        a = make_float2(fmaf(sA, a.x, ox), fmaf(sA, a.y, oy));
        if (rot) a = make_float2(-a.y, a.x);
        const float px = __shfl_xor_sync(0xffffffffu, a.x, 1);
        const float py = __shfl_xor_sync(0xffffffffu, a.y, 1);
        v[s1] = make_float2(fmaf(sB, a.x, px), fmaf(sB, a.y, py));
    }
}

__host__ __device__ constexpr int brev2(int l) { return ((l & 1) << 1) | ((l >> 1) & 1); }

// The same transforms on packed pairs, operation for operation.
__device__ __forceinline__ void idft4p(f2x& r0, f2x& i0, f2x& r1, f2x& i1, f2x& r2, f2x& i2, f2x& r3, f2x& i3) {
    const f2x sr = add2(r0, r2), si = add2(i0, i2), dr = sub2(r0, r2), di = sub2(i0, i2);
    const f2x tr = add2(r1, r3), ti = add2(i1, i3), er = sub2(r1, r3), ei = sub2(i1, i3);
    r0 = add2(sr, tr);
    i0 = add2(si, ti);
    r1 = sub2(dr, ei);
    i1 = add2(di, er);
    r2 = sub2(sr, tr);
    i2 = sub2(si, ti);
    r3 = add2(dr, ei);
    i3 = sub2(di, er);
}
// X[k] ends at index 4 (k mod 4) + k / 4.
__device__ __forceinline__ void idft16p(f2x (&re)[16], f2x (&im)[16]) {
    constexpr float c1 = 0.92387953251128674f, s1 = 0.38268343236508977f, r = 0.70710678118654752f;
    constexpr float tc[10] = {1.0f, c1, r, s1, 0.0f, -s1, -r, -c1, -1.0f, -c1};
    constexpr float ts[10] = {0.0f, s1, r, c1, 1.0f, c1, r, s1, 0.0f, -s1};
#pragma unroll
    for (int n = 0; n < 4; n++) idft4p(re[n], im[n], re[4 + n], im[4 + n], re[8 + n], im[8 + n], re[12 + n], im[12 + n]);
#pragma unroll
    for (int k = 1; k < 4; k++) {
#pragma unroll
        for (int n = 1; n < 4; n++) cmul2(re[4 * k + n], im[4 * k + n], pk1(tc[n * k]), pk1(ts[n * k]), pk1(-ts[n * k]));
    }
#pragma unroll
    for (int k = 0; k < 4; k++)
        idft4p(re[4 * k], im[4 * k], re[4 * k + 1], im[4 * k + 1], re[4 * k + 2], im[4 * k + 2], re[4 * k + 3], im[4 * k + 3]);
}

// Column stage of one (unit, u): A[unit][Ry s + u][c].
__global__ void __launch_bounds__(256) k_cols512(DhInvParams p, int unit0, float2* A) {
    __shared__ float2 colTw[64], tw64p[64];
    const int H = 1 << p.logH, Ry = H / 64, w = p.w, h = p.h;
    const int local = blockIdx.x / Ry, u = blockIdx.x % Ry, unit = unit0 + local;
    const int pol = unit % p.polCount;
    const int tid = threadIdx.x, l = tid & 3, c = tid >> 2;
    const int r0 = ((p.sy[pol] + H / 2) % H + H) % H;
    if (tid < 64) {
        tw64p[tid] = expPos(p.twiddle, tid, 64);
        colTw[tid] = tid < h ? expPos(p.twiddle, ((r0 + tid) % H) * u, H) : make_float2(0.f, 0.f);
    }
    __syncthreads();
    if (c >= w) return;   // whole warps: w is a multiple of 8
    const float2* win = p.window + (size_t)unit * w * h;
    float2 v[16];
#pragma unroll
    for (int m1 = 0; m1 < 16; m1++) {
        const int j = (4 * m1 + l - r0) & 63;
        v[m1] = j < h ? cmul(__ldg(&win[(size_t)j * w + c]), colTw[j]) : make_float2(0.f, 0.f);
    }
    ifft64q(v, l, tw64p);
    float2* out = A + ((size_t)local * H + u) * w + c;
#pragma unroll
    for (int s1 = 0; s1 < 16; s1++) out[(size_t)Ry * (s1 + 16 * brev2(l)) * w] = v[s1];
}

// Shared-memory plan; the host computes the same numbers.
struct F512Smem {
    int op, b, t, hy, a, ex, rowTw, tw, refX, red, items, misc, total;
};
__host__ __device__ constexpr F512Smem f512Smem(int pass, int GN, int G) {
    F512Smem s{};
    int o = 0;
    s.op = o;
    o += pass == P_I8 ? 2 * 2 * 128 * 128 : 0;        // low, high bytes: [2 atoms][128 rows][128 B]
    s.b = o;
    o += pass == P_I8 ? 2 * 4 * GN * 128 : 0;         // [2 atoms][digit, half, m][128 B]
    s.t = o;
    o += pass == P_I8 ? 2 * tPass(GN) * 4 : 0;  // [pass][half][plane, m][32 rows]
    s.hy = o;
    o += pass == P_I8 ? (G + 3) / 4 * 4 * HS * 4 : 0; // [n][pass][32 rows]
    s.a = o;
    o += 2 * RP * APITCH * 8;
    s.ex = o;
    o += NT / 32 * 2048 * (pass == P_STATS ? 4 : 1);  // one, or all, of the four rounds
    s.rowTw = o;
    o += 64 * 4 * 24;                                 // [(c + sx0) mod 64][v pair] (tr, ti), then -ti
    s.tw = o;
    o += 16 * 4 * 24;                                 // [s1][l] (tr, tr), (ti, ti), then -ti
    s.refX = o;
    o += pass != P_STATS ? WF / 2 * 16 : 0;
    s.red = o;
    o += pass == P_STATS ? 5 * 16 * 4 : 0;            // [sum][warp]
    s.items = o;
    o += pass == P_I8 ? ITEMS * 4 : 0;                // the contraction's (m, n0) items, then -1
    s.misc = o;
    o += 96;
    s.total = o + 1024;
    return s;
}

struct F512Args {
    const float2* A;             // [unit - unit0][y][c]
    StatF* part;                 // [unit][H / 64] partial statistics
    float* passMax;              // [unit][H / 32] maximum intensity of each pass's rows
    float* unitMax;              // [unit] maximum intensity
    float2* partCoefs;           // [unit][H / 64][modeCount]
    const unsigned char* hx;     // [pol][2 atoms][4 GN][128 B]: the operand's rows
    int unit0, units;            // this chunk
};

__device__ __forceinline__ void cpAsync8(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;" ::"r"(tc::sAddr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cpAsyncWait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// Round half to even of |v| < 2^22: the integer in the low half's two's complement.
__device__ __forceinline__ uint32_t roundMagic(float v) { return (uint32_t)__float_as_int(__fadd_rn(v, 12582912.0f)); }
// Within int16, -32768 for NaN.
__device__ __forceinline__ float clamp16(float v) { return fminf(fmaxf(v, -32768.0f), 32767.0f); }

template <int PASS, int GN>
__global__ void __launch_bounds__(NT, 1) k_field512(DhInvParams p, F512Args a) {
    constexpr bool QUANT = PASS != P_STATS;
    constexpr bool I8 = PASS == P_I8;
    constexpr int TMCOLS = 8 * GN;
    const int W = WF, H = 1 << p.logH, w = p.w;
    extern __shared__ float4 smf4[];
    unsigned char* base = tc::alignShared1024(reinterpret_cast<unsigned char*>(smf4));
    const F512Smem L = f512Smem(PASS, GN, I8 ? p.maxMG : 0);
    unsigned char* op = base + L.op;
    unsigned char* bop = base + L.b;
    float* T = reinterpret_cast<float*>(base + L.t);
    float* hy = reinterpret_cast<float*>(base + L.hy);
    float2* Abuf = reinterpret_cast<float2*>(base + L.a);
    const ulonglong2* rowTw = reinterpret_cast<const ulonglong2*>(base + L.rowTw);
    const f2x* nrowTw = reinterpret_cast<const f2x*>(base + L.rowTw) + 512;
    const ulonglong2* tw = reinterpret_cast<const ulonglong2*>(base + L.tw);
    const f2x* ntw = reinterpret_cast<const f2x*>(base + L.tw) + 128;
    int4* refX = reinterpret_cast<int4*>(base + L.refX);
    float* red = reinterpret_cast<float*>(base + L.red);
    int* itemMN = reinterpret_cast<int*>(base + L.items);
    uint64_t* bar = reinterpret_cast<uint64_t*>(base + L.misc);   // the products
    uint32_t* tmemSlot = reinterpret_cast<uint32_t*>(bar + 1);
    unsigned* passMax = reinterpret_cast<unsigned*>(bar + 2);     // [2] maxima of a band's passes (float bits)
    unsigned long long& bandMax = *reinterpret_cast<unsigned long long*>(bar + 3);   // (maximum, index + 1)

    const int P = p.polCount, pol = blockIdx.x % P;   // the grid is a multiple of P
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int pr = lane & 3, l = (lane >> 2) & 3, v0 = 2 * pr;
    const int row = 4 * (warp >> 1) + (warp & 1) + 2 * (lane >> 4);   // two rows per warp, swizzles apart
    const int sx0 = p.sx0[pol];
    const short* ref = p.refWave + (size_t)pol * 2 * (W + H);
    const float* refF = p.refWaveF + (size_t)pol * 2 * (W + H);
    const int G = I8 ? p.maxMG : 0, M = p.modeCount;

    // ---- tables
    {
        f2x* t = reinterpret_cast<f2x*>(base + L.rowTw);
        for (int e = tid; e < 256; e += NT) {
            const int c = ((e >> 2) - sx0) & 63, v = 2 * (e & 3);
            const float2 x = expPos(p.twiddle, ((sx0 + c) % W) * v, W), y = expPos(p.twiddle, ((sx0 + c) % W) * (v + 1), W);
            t[2 * e] = pk(x.x, y.x);
            t[2 * e + 1] = pk(x.y, y.y);
            t[512 + e] = pk(-x.y, -y.y);
        }
        t = reinterpret_cast<f2x*>(base + L.tw);
        for (int e = tid; e < 64; e += NT) {
            const float2 x = expPos(p.twiddle, ((e & 3) * (e >> 2)) & 63, 64);
            t[2 * e] = pk1(x.x);
            t[2 * e + 1] = pk1(x.y);
            t[128 + e] = pk1(-x.y);
        }
    }
    for (int e = tid; e < 2 * RP * APITCH; e += NT) Abuf[e] = make_float2(0.f, 0.f);
    if (QUANT) {
        for (int q = tid; q < W / 2; q += NT) refX[q] = make_int4(ref[2 * q], ref[W + 2 * q], ref[2 * q + 1], ref[W + 2 * q + 1]);
    }
    if (tid < 2) passMax[tid] = 0;
    if (tid == 0) bandMax = 0;
    if (I8) {
        // items of the contraction: x-mode m with y-modes n0 .. n0 + 3, m + n0 < G
        for (int e = tid; e < ITEMS; e += NT) {
            int n0 = 0, k = e;
            while (n0 < G && k >= G - n0) {
                k -= G - n0;
                n0 += 4;
            }
            itemMN[e] = n0 < G ? (k << 16) | n0 : -1;
        }
        for (int e = tid; e < (G + 3) / 4 * 4 * HS; e += NT) hy[e] = 0.f;
        const uint4* src = reinterpret_cast<const uint4*>(a.hx + (size_t)pol * 8 * GN * 128);
        for (int e = tid; e < 8 * GN * 8; e += NT) reinterpret_cast<uint4*>(bop)[e] = __ldg(src + e);
        if (tid == 0) tc::mbarInitTc(bar);
        if (warp == 0) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(tc::sAddr(tmemSlot)), "n"(TMCOLS)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
        }
        tc::fenceProxyAsync();
        tc::fenceBeforeSync();
    }
    __syncthreads();
    uint32_t tmem = 0;
    if (I8) {
        tc::fenceAfterSync();
        tmem = *tmemSlot;
    }

    // ---- this block's passes: item = (frame of its polarisation, rows), a band being two passes in a row
    constexpr int PPI = BR / RP;                            // passes per item
    const int perUnit = H / BR;
    const int lanes = gridDim.x / P;
    const int items = a.units / P * perUnit;
    const int first = blockIdx.x / P;
    const int mine = first < items ? (items - first + lanes - 1) / lanes * PPI : 0;
    auto locate = [&](int n, int& unit, int& y0) {          // pass n of this block
        const int item = first + n / PPI * lanes;
        unit = item / perUnit * P + pol;
        y0 = (item % perUnit) * RP * PPI + n % PPI * RP;
    };
    // a warp fetches its own two rows of pass n
    auto fetch = [&](int n) {
        int unit, y0;
        locate(n, unit, y0);
        const float2* src = a.A + ((size_t)unit * H + y0) * w;
        float2* dst = Abuf + (n & 1) * RP * APITCH;
        const int r = 4 * (warp >> 1) + (warp & 1);
        for (int c = lane; c < w; c += 32) {
            const int at = (c + sx0) & 63;
            cpAsync8(dst + r * APITCH + at, src + r * w + c);
            cpAsync8(dst + (r + 2) * APITCH + at, src + (r + 2) * w + c);
        }
    };
    ulonglong2* ex = reinterpret_cast<ulonglong2*>(base + L.ex) + warp * (QUANT ? 128 : 512);
    // the sums of the last issued products: tensor memory -> T[pass]
    auto readSums = [&](int par) {
        tc::fenceAfterSync();
        const int half = (warp >> 1) & 1, plane = warp & 1, m0 = (warp >> 2) * (GN / 4);
        const uint32_t at = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(half * GN + m0);
        float* t = T + par * tPass(GN) + (half * 2 * GN + plane * GN + m0) * TS + lane;
#pragma unroll
        for (int c0 = 0; c0 < GN / 4; c0 += 4) {
            uint32_t e0[4], e1[4], o0[4], o1[4];
            tc::tmemLoad4(at + c0, e0);
            tc::tmemLoad4(at + 2 * GN + c0, e1);
            tc::tmemLoad4(at + 4 * GN + c0, o0);
            tc::tmemLoad4(at + 6 * GN + c0, o1);
            tc::tmemWaitLoad4(e0);
            tc::tmemWaitLoad4(e1);
            tc::tmemWaitLoad4(o0);
            tc::tmemWaitLoad4(o1);
#pragma unroll
            for (int i = 0; i < 4; i++)
                t[(c0 + i) * TS] =
                    fmaf((float)(int)o1[i], 65536.0f, fmaf((float)((int)e1[i] + (int)o0[i]), 256.0f, (float)(int)e0[i]));
        }
        tc::fenceBeforeSync();
    };
    // Hy of a band's rows
    auto loadHy = [&](int y0) {
        for (int e = tid; e < G * BR; e += NT) {
            const int nn = e >> 6, r = e & 63;
            hy[nn * HS + (r >> 5) * HP + (r & 31)] = (float)__ldg(p.hgY + ((size_t)pol * G + nn) * H + y0 + r);
        }
    };
    // a band's partial coefficients: four lanes per item, one for 16 of the 64 rows each
    // (by the first `warps` warps)
    auto contract = [&](int unit, int y0, int warps) {
        const int ps = tid & 1, q0 = (tid & 2) * (RP / 16);
        float2* out = a.partCoefs + ((size_t)(a.unit0 + unit) * (H / BR) + y0 / BR) * M;
        for (int item = tid >> 2; item < ITEMS && itemMN[item & ~7] >= 0; item += 8 * warps) {   // whole warps
            const int mn = itemMN[item], m = mn < 0 ? 0 : mn >> 16, n0 = mn < 0 ? 0 : mn & 0xFFFF;
            const ulonglong2* r0 = reinterpret_cast<const ulonglong2*>(T + ps * tPass(GN) + m * TS) + q0;
            const ulonglong2* r1 = r0 + 2 * GN * TS / 4;
            const ulonglong2* i0 = r0 + GN * TS / 4;
            const ulonglong2* i1 = i0 + 2 * GN * TS / 4;
            const ulonglong2* hn = reinterpret_cast<const ulonglong2*>(hy + n0 * HS + ps * HP) + q0;
            f2x cr[4], ci[4];
#pragma unroll
            for (int i = 0; i < 4; i++) cr[i] = ci[i] = pk(0.f, 0.f);
#pragma unroll 2
            for (int q = 0; q < RP / 8; q++) {
                const ulonglong2 u = r0[q], v = r1[q], s = i0[q], t = i1[q];
                const f2x ra = add2(u.x, v.x), rb = add2(u.y, v.y), ia = add2(s.x, t.x), ib = add2(s.y, t.y);
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    const ulonglong2 h = hn[i * HS / 4 + q];
                    cr[i] = fma2(h.y, rb, fma2(h.x, ra, cr[i]));
                    ci[i] = fma2(h.y, ib, fma2(h.x, ia, ci[i]));
                }
            }
            float2 mine = make_float2(0.f, 0.f);
#pragma unroll
            for (int i = 0; i < 4; i++) {
                const float2 c = upk(cr[i]), d = upk(ci[i]);
                float x = c.x + c.y, y = d.x + d.y;
                x += __shfl_xor_sync(0xffffffffu, x, 1);
                y += __shfl_xor_sync(0xffffffffu, y, 1);
                x += __shfl_xor_sync(0xffffffffu, x, 2);
                y += __shfl_xor_sync(0xffffffffu, y, 2);
                if ((tid & 3) == i) mine = make_float2(x, y);
            }
            const int nn = n0 + (tid & 3);
            if (mn >= 0 && m + nn < G) out[(m + nn) * (m + nn + 1) / 2 + nn] = mine;
        }
    };

    const float inv = (float)(1.0 / ((double)W * (double)H));
    const float dx = p.xAxis[1] - p.xAxis[0], xc = p.xAxis[WF / 2];
    const float yShift = fabsf((p.yAxis[1] - p.yAxis[0]) * (float)H);
    bool ok = true;
    if (mine > 0) fetch(0);
    StatF st = {0.f, -1, 0.f, 0.f, 0.f, 0.f, 0.f};
    int n = 0;
    for (; n < mine; n++) {
        int unit, y0;
        locate(n, unit, y0);
        const int gu = a.unit0 + unit, frame = gu / P, y = y0 + row, par = n & 1;
        cpAsyncWait();   // this pass's rows; the other buffer's readers are past their last barrier or this warp
        __syncwarp();
        if (n + 1 < mine) fetch(n + 1);
        float scale = 0.f, unitMax = 0.f, rowsMax = 0.f;
        int yr = 0, yi = 0;
        if (QUANT) {
            unitMax = __ldg(a.unitMax + gu);
            rowsMax = __ldg(a.passMax + (size_t)gu * (H / RP) + y0 / RP);
            scale = __ldg(p.stats + (size_t)(3 * P + pol) * p.statsStride + frame);
            yr = ref[2 * W + y];
            yi = ref[2 * W + H + y];
        }
        // ---- row transform
        f2x re[16], im[16];
        {
            const float2* arow = Abuf + (par * RP + row) * APITCH + l;
#pragma unroll
            for (int m1 = 0; m1 < 16; m1++) {
                const float2 s = arow[4 * m1];
                re[m1] = pk1(s.x);
                im[m1] = pk1(s.y);
                const ulonglong2 t = rowTw[16 * m1 + 4 * l + pr];
                cmul2(re[m1], im[m1], t.x, t.y, nrowTw[16 * m1 + 4 * l + pr]);
            }
        }
        idft16p(re, im);
        // four s1 at a time: twiddle, exchange, 4-point DFT over the lanes;
        // (j, s2) ends at 4 j + s2 with t = 4 j + l + 16 s2
        f2x fr[16], fi[16];
        constexpr int BATCH = QUANT ? 1 : 4;   // rounds between two barriers
#pragma unroll
        for (int j = 0; j < 4; j++) {
            if (j % BATCH == 0) {
                if (j) __syncwarp();
#pragma unroll
                for (int i = 0; i < 4 * BATCH; i++) {
                    const int s1 = 4 * j + i, k = 4 * (s1 & 3) + (s1 >> 2);
                    if (s1) {
                        const ulonglong2 t = tw[4 * s1 + l];
                        cmul2(re[k], im[k], t.x, t.y, ntw[4 * s1 + l]);
                    }
                    ex[i * 32 + (lane ^ ((i & 3) << 2))] = make_ulonglong2(re[k], im[k]);
                }
                __syncwarp();
            }
            f2x yr_[4], yi_[4];
#pragma unroll
            for (int s = 0; s < 4; s++) {
                // s1 = 4 j + l from source lane s
                const ulonglong2 t = ex[(j % BATCH * 4 + l) * 32 + ((lane & 16) | ((s ^ l) << 2) | pr)];
                yr_[s] = t.x;
                yi_[s] = t.y;
            }
            const f2x b0r = add2(yr_[0], yr_[2]), b0i = add2(yi_[0], yi_[2]), b2r = sub2(yr_[0], yr_[2]), b2i = sub2(yi_[0], yi_[2]);
            const f2x b1r = add2(yr_[1], yr_[3]), b1i = add2(yi_[1], yi_[3]), b3r = sub2(yr_[1], yr_[3]), b3i = sub2(yi_[1], yi_[3]);
            fr[4 * j] = add2(b0r, b1r);
            fi[4 * j] = add2(b0i, b1i);
            fr[4 * j + 2] = sub2(b0r, b1r);
            fi[4 * j + 2] = sub2(b0i, b1i);
            fr[4 * j + 1] = sub2(b2r, b3i);   // b2 + i b3
            fi[4 * j + 1] = add2(b2i, b3r);
            fr[4 * j + 3] = add2(b2r, b3i);
            fi[4 * j + 3] = sub2(b2i, b3r);
        }
        const int x0 = 8 * l + v0;   // pixel pair (j, s2): x = 128 s2 + 32 j + x0

        if (!QUANT) {
            // statistics over the untilted field (digHolo.cpp:8866-8870)
            f2x sP = pk(0.f, 0.f), sX = sP, sE = sP;
            float mx = 0.f;
            const f2x inv2 = pk1(inv);
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const f2x I0 = fma2(fr[q], fr[q], mul2(fi[q], fi[q]));
                const float2 v = upk(I0);
                mx = fmaxf(fmaxf(mx, v.x), v.y);
                const f2x I = mul2(I0, inv2);
                sP = add2(sP, I);
                sX = fma2(I, pk1((float)(128 * (q & 3) + 32 * (q >> 2) - WF / 2)), sX);
                sE = fma2(I, I, sE);
            }
            {
                const float2 v = upk(sP), t = upk(sX), e = upk(sE);
                const float Prow = v.x + v.y;
                const float xs = fmaf((float)x0, Prow, v.y) + (t.x + t.y);
                const float yv = p.yAxis[y];
                st.P += Prow;
                st.cx += fmaf(dx, xs, xc * Prow);   // x = dx (index - W / 2) + xc
                st.cy = fmaf(yv, Prow, st.cy);
                st.cyw = fmaf(yv + (yv < 0.f ? yShift : 0.f), Prow, st.cyw);
                st.e4 += e.x + e.y;
            }
            // the band's maximum and its index (the larger on ties): the lanes
            // that hold a warp's maximum look it up when it may be the band's
            const unsigned wm = __reduce_max_sync(0xffffffffu, __float_as_uint(mx));
            if (lane == 0) atomicMax(&passMax[par], wm);
            if (__float_as_uint(mx) == wm && wm >= (unsigned)(*(volatile unsigned long long*)&bandMax >> 32)) {
                int best = -1;
#pragma unroll
                for (int q = 0; q < 16; q++) {
                    const float2 v = upk(fma2(fr[q], fr[q], mul2(fi[q], fi[q])));
                    const int idx = 2 * y * W + 128 * (q & 3) + 32 * (q >> 2) + x0;
                    if (v.x == mx) best = max(best, idx);
                    if (v.y == mx) best = max(best, idx + 1);
                }
                // index + 1 in the low word: 0 for none (no pixel is a number)
                atomicMax(&bandMax, ((unsigned long long)wm << 32) | (unsigned)(best + 1));
            }
            if (par == 0) continue;
            // the band's record
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) {
                st.P += __shfl_xor_sync(0xffffffffu, st.P, off);
                st.cx += __shfl_xor_sync(0xffffffffu, st.cx, off);
                st.cy += __shfl_xor_sync(0xffffffffu, st.cy, off);
                st.cyw += __shfl_xor_sync(0xffffffffu, st.cyw, off);
                st.e4 += __shfl_xor_sync(0xffffffffu, st.e4, off);
            }
            if (lane < 5) red[lane * 16 + warp] = lane == 0 ? st.P : lane == 1 ? st.cx : lane == 2 ? st.cy : lane == 3 ? st.cyw : st.e4;
            st = {0.f, -1, 0.f, 0.f, 0.f, 0.f, 0.f};
            __syncthreads();
            if (warp < 5) {
                float s = lane < 16 ? red[warp * 16 + lane] : 0.f;
#pragma unroll
                for (int off = 8; off > 0; off >>= 1) s += __shfl_xor_sync(0xffffffffu, s, off);
                StatF* out = a.part + (size_t)gu * (H / BR) + y0 / BR;
                if (lane == 0) (&out->P)[warp] = s;
                if (warp == 0 && lane == 0) {
                    out->maxI = __uint_as_float((unsigned)(bandMax >> 32));
                    out->maxIdx = (int)(unsigned)bandMax - 1;
                    bandMax = 0;
                }
                if (warp == 0 && lane < 2) {
                    a.passMax[(size_t)gu * (H / RP) + y0 / RP - 1 + lane] = __uint_as_float(passMax[lane]);
                    passMax[lane] = 0;
                }
            }
            __syncthreads();
            continue;
        }

        const size_t fieldOff = ((size_t)gu * H + y) * W + x0;
        if (p.field32) {
            // -conj(A R) with the unquantised wave
            const float2 ryf = make_float2(refF[2 * W + y], refF[2 * W + H + y]);
#pragma unroll
            for (int q = 0; q < 16; q++) {
                const int x = 128 * (q & 3) + 32 * (q >> 2);
                const float2 c = upk(fr[q]), d = upk(fi[q]);
                const float2 rx = __ldg(reinterpret_cast<const float2*>(refF + x0 + x));
                const float2 ri = __ldg(reinterpret_cast<const float2*>(refF + W + x0 + x));
                const float2 w0 = cmul(make_float2(c.x, d.x), cmul(ryf, make_float2(rx.x, ri.x)));
                const float2 w1 = cmul(make_float2(c.y, d.y), cmul(ryf, make_float2(rx.y, ri.y)));
                *reinterpret_cast<float4*>(p.field32 + fieldOff + x) = make_float4(-w0.x, w0.y, -w1.x, w1.y);
            }
        }
        if (I8 && n > 0) {
            // the products of the previous pass have read the operand
            ok = !__syncthreads_or(!tc::mbarWaitTc(bar, (unsigned)((n - 1) & 1)));
            if (!ok) break;
            readSums(par ^ 1);   // T of the band before has been contracted: its readers are past this barrier
        } else {
            __syncthreads();
        }
        // ---- reference wave, -conj(A . ref), int16 rounding (digHolo.cpp:2741-2833).
        const f2x K2 = pk1((float)(1.0 / (16383.0 * 16383.0))), scale2 = pk1(scale);
        // Rows whose own maximum is clearly below the field's cannot saturate
        // (|ref| <= 1 + 9e-5): their integers are the sums' low halves.
        const bool fast = scale < 1e30f && scale > 0.f && rowsMax < 0.9995f * unitMax;
        const int rho = row & 7;
        // lane pairs exchange halves: the even lane stores four R pixels, the odd lane four I pixels
        unsigned char* opRow = op + row * 128 + 8 * (l & 1) + 2 * pr;
#pragma unroll
        for (int q = 0; q < 16; q++) {
            const int s2 = q & 3, j = q >> 2, x = 128 * s2 + 32 * j;
            const int4 rx = refX[(x + x0) >> 1];
            const f2x adjR = mul2(pk((float)(yr * rx.x - yi * rx.y), (float)(yr * rx.z - yi * rx.w)), K2);
            const f2x adjI = mul2(pk((float)(yr * rx.y + yi * rx.x), (float)(yr * rx.w + yi * rx.z)), K2);
            // scalar sums: the packed forms of a product and a sum may be fused into one rounding
            const float2 p0 = upk(mul2(fi[q], adjI)), p1 = upk(mul2(fr[q], adjR));
            const float2 p2 = upk(mul2(fr[q], adjI)), p3 = upk(mul2(fi[q], adjR));
            float2 c = upk(mul2(scale2, pk(__fsub_rn(p0.x, p1.x), __fsub_rn(p0.y, p1.y))));
            float2 d = upk(mul2(scale2, pk(__fadd_rn(p2.x, p3.x), __fadd_rn(p2.y, p3.y))));
            if (!fast) {   // block-uniform
                c = make_float2(clamp16(c.x), clamp16(c.y));
                d = make_float2(clamp16(d.x), clamp16(d.y));
            }
            const uint32_t c0 = roundMagic(c.x), c1 = roundMagic(c.y), d0 = roundMagic(d.x), d1 = roundMagic(d.y);
            const uint32_t wr = __byte_perm(c0, c1, 0x5410), wi = __byte_perm(d0, d1, 0x5410);
            *reinterpret_cast<uint32_t*>(p.fieldR + fieldOff + x) = wr;
            *reinterpret_cast<uint32_t*>(p.fieldI + fieldOff + x) = wi;
            if (I8) {
                unsigned char* o = opRow + (s2 & 1) * 16384 + (s2 >> 1) * 8192 + (((2 * j + (l >> 1)) ^ rho) << 4);
                *reinterpret_cast<unsigned short*>(o) = (unsigned short)__byte_perm(c0, c1, 0x4040);
                *reinterpret_cast<unsigned short*>(o + 4096) = (unsigned short)__byte_perm(d0, d1, 0x4040);
                *reinterpret_cast<unsigned short*>(o + 32768) = (unsigned short)__byte_perm(c0, c1, 0x5151);
                *reinterpret_cast<unsigned short*>(o + 32768 + 4096) = (unsigned short)__byte_perm(d0, d1, 0x5151);
            }
        }
        if (!I8) continue;
        tc::fenceProxyAsync();
        __syncthreads();
        // ---- products of this pass; after a band's second pass has been read, its coefficients
        if (warp == NT / 32 - 1) {
            if (lane == 0) {
                tc::fenceAfterSync();
                const uint32_t a0 = tc::sAddr(op), b0 = tc::sAddr(bop);
#pragma unroll
                for (int k = 0; k < 8; k++) {
                    const uint32_t ao = a0 + (uint32_t)(k >> 2) * 16384 + (uint32_t)(k & 3) * 32;
                    const uint64_t al = tc::smemDesc(ao), ah = tc::smemDesc(ao + 32768);
                    const uint32_t bo = b0 + (uint32_t)(k >> 2) * (4 * GN * 128) + (uint32_t)(k & 3) * 32;
                    const uint64_t bl = tc::smemDesc(bo), bh = tc::smemDesc(bo + 2 * GN * 128);
                    tc::mmaI8(tmem, al, bl, tc::instrDescI8s(128, 2 * GN, false, false), k > 0);
                    tc::mmaI8(tmem + 2 * GN, al, bh, tc::instrDescI8s(128, 2 * GN, false, true), k > 0);
                    tc::mmaI8(tmem + 4 * GN, ah, bl, tc::instrDescI8s(128, 2 * GN, true, false), k > 0);
                    tc::mmaI8(tmem + 6 * GN, ah, bh, tc::instrDescI8s(128, 2 * GN, true, true), k > 0);
                }
                tc::mmaCommit(bar);
            }
            __syncwarp();
        } else if (par == 0 && n > 0) {
            int pu, py;
            locate(n - 2, pu, py);
            contract(pu, py, NT / 32 - 1);
        }
        if (par == 1) loadHy(y0 - RP);   // this band's, for the contraction after its sums are read
    }
    if (I8) {
        if (ok && n > 0) {
            ok = !__syncthreads_or(!tc::mbarWaitTc(bar, (unsigned)((n - 1) & 1)));
            if (ok) {
                readSums((n - 1) & 1);
                __syncthreads();
                int pu, py;
                locate(n - 2, pu, py);
                contract(pu, py, NT / 32);
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
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(TMCOLS) : "memory");
        }
    }
}

// The statistics of each unit from its bands' partial records.
__global__ void k_field512_stats(DhInvParams p, const StatF* __restrict__ part, int np, float* unitMax) {
    const int P = p.polCount, S = p.statsStride, per = P * S;
    const int units = p.frameCount * P;
    for (int unit = blockIdx.x * blockDim.x + threadIdx.x; unit < units; unit += gridDim.x * blockDim.x) {
        const StatF* q = part + (size_t)unit * np;
        StatF t = q[0];
        for (int b = 1; b < np; b++) {
            const StatF o = q[b];
            statMerge(t, o.maxI, o.maxIdx, o.P, o.cx, o.cy, o.cyw, o.e4);
        }
        unitMax[unit] = t.maxI;
        float* s = p.stats + (unit % P) * S + unit / P;
        s[0] = t.P;
        s[1 * per] = t.cx / t.P;
        s[2 * per] = t.cy / t.P;
        s[3 * per] = (float)(32767.0 / (double)sqrtf(t.maxI));
        s[4 * per] = __int_as_float(t.maxIdx);
        s[5 * per] = p.dA * (t.P * t.P / t.e4);
        s[6 * per] = t.cyw / t.P;
    }
}

// Hx of every polarisation as the operand's rows (digit, half of x, m): the
// low (unsigned) then the high (signed) bytes of the int16 modes, rows from
// maxMG up zero; 128-byte-swizzled.
__global__ void k_field512_prep_hx(DhInvParams p, int GN, unsigned char* out) {
    const int G = p.maxMG;
    const int total = p.polCount * GN * WF;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int pol = e / (GN * WF), rem = e - pol * GN * WF;
        const int m = rem / WF, x = rem - m * WF;
        const int val = m < G ? (int)p.hgX[((size_t)pol * G + m) * WF + x] : 0;
        const int half = x >> 8, atom = (x >> 7) & 1, chunk = (x & 127) >> 4;
        unsigned char* b = out + (size_t)pol * 8 * GN * 128 + (size_t)atom * 4 * GN * 128;
        const int r = half * GN + m;   // GN is a multiple of 8: the swizzle is the same for both digits
        const int off = ((chunk ^ (r & 7)) << 4) + (x & 15);
        b[r * 128 + off] = (unsigned char)(val & 0xFF);
        b[(2 * GN + r) * 128 + off] = (unsigned char)((val >> 8) & 0xFF);
    }
}

// Sum of the bands' partial coefficients, times sx[m] sy[n] / scale.
__global__ void k_field512_coefs(DhInvParams p, const float2* __restrict__ part, int nb) {
    const int P = p.polCount, M = p.modeCount, G = p.maxMG, S = p.statsStride;
    const int total = p.frameCount * P * M;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int unit = e / M, mode = e % M;
        const int pol = unit % P, frame = unit / P;
        float cr = 0.f, ci = 0.f;
        for (int b = 0; b < nb; b++) {
            const float2 v = part[((size_t)unit * nb + b) * M + mode];
            cr += v.x;
            ci += v.y;
        }
        int g = (int)((sqrtf(8.0f * mode + 1.0f) - 1.0f) * 0.5f);
        while ((g + 1) * (g + 2) / 2 <= mode) g++;
        while (g * (g + 1) / 2 > mode) g--;
        const int n = mode - g * (g + 1) / 2, m = g - n;
        const float scale = p.stats[3 * P * S + pol * S + frame];
        const float fieldScale = 1.0f / scale;
        const float ms = (float)((double)p.hgScaleX[pol * G + m] * (double)p.hgScaleY[pol * G + n] * (double)fieldScale);
        p.coefs[(size_t)frame * P * M + (size_t)pol * M + mode] = make_float2(cr * ms, ci * ms);
    }
}

struct F512Plan {
    int pass, GN, chunk;
    size_t offMax, offPass, offCoefs, offHx, offA, scratch;
};

// cudaErrorNotSupported outside the kernel's shapes: full-resolution fields
// 512 wide and 64 to 4096 high, IFFT windows of at most 64 x 64 (sides
// multiples of 16), no overlap or the tensor-core overlap with maxMG <= 32.
cudaError_t plan512(const DhInvParams& p, int overlapKind, F512Plan& pl) {
    // a reference-wave calibration is applied by k_field_big, not here
    if (p.lowres || p.refCal) return cudaErrorNotSupported;
    const int W = 1 << p.logW, H = 1 << p.logH;
    if (W != WF || H < 64 || H > TW_N) return cudaErrorNotSupported;
    if (p.w < 16 || p.h < 16 || p.w > 64 || p.h > 64 || p.w % 16 || p.h % 16) return cudaErrorNotSupported;
    for (int q = 0; q < p.polCount; q++)
        if (p.sx0[q] < 0) return cudaErrorNotSupported;
    const bool ov = p.maxMG > 0 && p.coefs;
    if (ov && (overlapKind != 0 || p.maxMG > GNMAX)) return cudaErrorNotSupported;
    pl.pass = ov ? P_I8 : P_QUANT;
    pl.GN = ov && p.maxMG > 16 ? 32 : 16;
    const size_t units = (size_t)p.frameCount * p.polCount;
    pl.chunk = units < CHUNK ? (int)units : CHUNK;   // a multiple of polCount (1 or 2)
    pl.offMax = (units * (H / BR) * sizeof(StatF) + 255) / 256 * 256;
    pl.offPass = pl.offMax + (units * sizeof(float) + 255) / 256 * 256;
    pl.offCoefs = pl.offPass + (units * (H / RP) * sizeof(float) + 255) / 256 * 256;
    pl.offHx = pl.offCoefs + (ov ? (units * (H / BR) * p.modeCount * sizeof(float2) + 255) / 256 * 256 : 0);
    pl.offA = pl.offHx + (ov ? (size_t)p.polCount * 8 * pl.GN * 128 : 0);
    pl.scratch = pl.offA + (size_t)pl.chunk * H * p.w * sizeof(float2);
    return cudaSuccess;
}

template <int PASS, int GN>
cudaError_t launch512(const DhInvParams& p, const F512Args& a, cudaStream_t s) {
    const F512Smem L = f512Smem(PASS, GN, PASS == P_I8 ? p.maxMG : 0);
    auto kern = k_field512<PASS, GN>;
    cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(kern), L.total);
    if (e != cudaSuccess) return e;
    const int items = a.units * ((1 << p.logH) / BR);
    int grid = smCountCached();
    grid -= grid % p.polCount;   // a block keeps its polarisation
    if (grid > items) grid = items;
    kern<<<(unsigned)grid, NT, L.total, s>>>(p, a);
    return cudaGetLastError();
}

}  // namespace

// Scratch the kernels need for this launch (0 where they do not apply).
size_t dh_field512_scratch_bytes(const DhInvParams& p, int overlapKind) {
    F512Plan pl;
    if (plan512(p, overlapKind, pl) != cudaSuccess) return 0;
    return pl.scratch;
}

// Full-resolution 512-wide fields: column stage, statistics pass, quantising
// pass (with the exact integer overlap on the tensor cores when maxMG > 0),
// then the coefficient sum.  *overlapUsed: 0 none, 3 integer tensor cores.
cudaError_t dh_launch_field512(const DhInvParams& p, int overlapKind, void* scratch, size_t scratchBytes, int* overlapUsed,
                               cudaStream_t s) {
    *overlapUsed = 0;
    F512Plan pl;
    cudaError_t e = plan512(p, overlapKind, pl);
    if (e != cudaSuccess) return e;
    const int units = p.frameCount * p.polCount, H = 1 << p.logH;
    if (units <= 0) return cudaSuccess;
    if (!scratch || scratchBytes < pl.scratch || (reinterpret_cast<uintptr_t>(scratch) & 255)) return cudaErrorInvalidValue;
    if (((reinterpret_cast<uintptr_t>(p.fieldR) | reinterpret_cast<uintptr_t>(p.fieldI)) & 7) ||
        (reinterpret_cast<uintptr_t>(p.field32) & 15))
        return cudaErrorNotSupported;
    unsigned char* sc = static_cast<unsigned char*>(scratch);
    F512Args a;
    a.part = reinterpret_cast<StatF*>(sc);
    a.unitMax = reinterpret_cast<float*>(sc + pl.offMax);
    a.passMax = reinterpret_cast<float*>(sc + pl.offPass);
    a.partCoefs = reinterpret_cast<float2*>(sc + pl.offCoefs);
    a.hx = sc + pl.offHx;
    a.A = reinterpret_cast<float2*>(sc + pl.offA);
    if (pl.pass == P_I8) {
        const int total = p.polCount * pl.GN * WF;
        k_field512_prep_hx<<<(total + 255) / 256, 256, 0, s>>>(p, pl.GN, sc + pl.offHx);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    // a chunk's column stage and statistics, then its quantising pass (the
    // statistics kernel covers the units whose records are complete)
    for (int u0 = 0; u0 < units; u0 += pl.chunk) {
        a.unit0 = u0;
        a.units = units - u0 < pl.chunk ? units - u0 : pl.chunk;
        k_cols512<<<(unsigned)(a.units * (H / 64)), 256, 0, s>>>(p, u0, reinterpret_cast<float2*>(sc + pl.offA));
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        if ((e = launch512<P_STATS, 16>(p, a, s)) != cudaSuccess) return e;
        DhInvParams pc = p;   // the chunk's frames
        pc.frameCount = a.units / p.polCount;
        pc.stats = p.stats + u0 / p.polCount;
        k_field512_stats<<<(unsigned)(a.units + 63) / 64, 64, 0, s>>>(pc, a.part + (size_t)u0 * (H / BR), H / BR, a.unitMax + u0);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        e = pl.pass == P_QUANT ? launch512<P_QUANT, 16>(p, a, s)
            : pl.GN == 16      ? launch512<P_I8, 16>(p, a, s)
                               : launch512<P_I8, 32>(p, a, s);
        if (e != cudaSuccess) return e;
    }
    if (pl.pass == P_I8) {
        const int total = p.frameCount * p.polCount * p.modeCount;
        int g = (total + 255) / 256;
        if (g > 148 * 16) g = 148 * 16;
        k_field512_coefs<<<g, 256, 0, s>>>(p, a.partCoefs, H / BR);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
        *overlapUsed = 3;
    }
    return cudaSuccess;
}
