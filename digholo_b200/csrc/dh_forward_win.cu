// Forward stage of 128- and 256-pixel-wide FFT windows (up to 256 rows) with
// any IFFT window, in one launch and without the full Fourier plane: row
// transforms, R2C split of the kept kx columns, column transforms and the
// window factors (the reference's FFTW r2c of the window,
// digHolo.cpp:7184-7260, and digHoloCopyWindow, digHolo.cpp:1808-2122).
//
// One block of 256 threads per (frame, polarisation).  A row of W real pixels
// is the complex sequence z[n] = f[2 n] + i f[2 n + 1] of N = W / 2 points,
// transformed by the butterflies of the radix-2 decimation in time that
// k_fourier_rows runs in shared memory, two rows per instruction (f32x2):
// thread g of a row pair loads the 16 samples of bit-reversed positions
// 16 g .. 16 g + 15 straight into registers (four stages), one exchange
// through a warp-private buffer, then the remaining stages for the positions
// s + 16 g of two (N = 128) or four (N = 64) s.  Each thread holds s and
// 16 - s, so the split F[k] of Z[k] and Z[N - k] needs no further exchange,
// and only the kept columns are stored, to shared memory.  The columns go the
// same way, two per instruction, in place; the last stage writes the kept
// rows of the window.
//
// Bound: latency (28 % of the issue slots with 16 warps of 128 registers per
// SM; two rows per thread halve the arithmetic).  1000 windows of 256 x 256
// float pixels, 32 columns kept: 114 us, 2.3 TB/s of frame rows; the plane
// kernels, which moved every stage through shared memory and the kept columns
// through global memory, took 596 us.
#include <cuda_runtime.h>
#include <stdint.h>

#include "dh_common.cuh"
#include "dh_f32x2.cuh"
#include "dh_host.h"
#include "dh_params.h"

using namespace dh;

namespace {

constexpr int NT = 256;

__host__ __device__ constexpr int brevc(int i, int bits) {
    int r = 0;
    for (int b = 0; b < bits; b++) r |= ((i >> b) & 1) << (bits - 1 - b);
    return r;
}

// One stage (butterflies 2^LH apart) of a radix-2 DIT over 16 bit-reversed
// positions, forward.
template <int LH>
__device__ __forceinline__ void ditStage(f2x (&re)[16], f2x (&im)[16]) {
    constexpr int HALF = 1 << LH;
#pragma unroll
    for (int i = 0; i < 8; i++) {
        const int j = i & (HALF - 1), a = 2 * (i - j) + j, b = a + HALF;
        const f2x ar = re[a], ai = im[a];
        if (2 * j == HALF) {   // times -i
            const f2x br = re[b], bi = im[b];
            re[a] = add2(ar, bi);
            im[a] = sub2(ai, br);
            re[b] = sub2(ar, bi);
            im[b] = add2(ai, br);
        } else {
            if (j != 0) {
                const float2 t = tw128(j * (64 >> LH));
                cmul2(re[b], im[b], pk1(t.x), pk1(t.y), pk1(-t.y));
            }
            const f2x br = re[b], bi = im[b];
            re[a] = add2(ar, br);
            im[a] = add2(ai, bi);
            re[b] = sub2(ar, br);
            im[b] = sub2(ai, bi);
        }
    }
}

// One stage (butterflies 16 HALF apart) of a transform of 16 G positions on
// the positions s + 16 g of one s; tw(HALF - 1 + j): exp(-2 pi i (s + 16 j) / (32 HALF)).
template <int G, int HALF, typename Tw>
__device__ __forceinline__ void tailStage(f2x (&re)[G], f2x (&im)[G], const Tw& tw) {
#pragma unroll
    for (int j = 0; j < HALF; j++) {
        f2x tr, ti, nti;
        tw(HALF - 1 + j, tr, ti, nti);
#pragma unroll
        for (int i = 0; i < G / 2 / HALF; i++) {
            const int a = 2 * HALF * i + j, b = a + HALF;
            cmul2(re[b], im[b], tr, ti, nti);
            const f2x ar = re[a], ai = im[a], br = re[b], bi = im[b];
            re[a] = add2(ar, br);
            im[a] = add2(ai, bi);
            re[b] = sub2(ar, br);
            im[b] = sub2(ai, bi);
        }
    }
}
template <int G, typename Tw>
__device__ __forceinline__ void ditTail(f2x (&re)[G], f2x (&im)[G], const Tw& tw) {
    tailStage<G, 1>(re, im, tw);
    tailStage<G, 2>(re, im, tw);
    if constexpr (G >= 8) tailStage<G, 4>(re, im, tw);
    if constexpr (G >= 16) tailStage<G, 8>(re, im, tw);
}

// Two pixels.  Float pairs skip L1 (a row's 64-byte pieces fill whole sectors
// by themselves: 127 us against 130 at 1000 windows of 256 x 256); uint16
// pairs share sectors' lines with the next piece and keep it (111 against 119
// at 800 windows of 128 x 128, 48 kept columns and the inverse included).
__device__ __forceinline__ unsigned loadPair(const unsigned short* p) {
    return __ldg(reinterpret_cast<const unsigned*>(p));
}
__device__ __forceinline__ float2 loadPair(const float* p) {
    float2 v;
    asm volatile("ld.global.nc.L1::no_allocate.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "l"(p));
    return v;
}

struct WinSmem {
    int col, pitch, ex, exRow, twN, twH, twW, total;
};
__host__ __device__ inline WinSmem winSmem(int logN, int H, int w) {
    const int N = 1 << logN;
    WinSmem s;
    s.pitch = w / 2 + 1;                              // float4 per buffered row
    s.col = 0;                                        // [H][pitch] (re, re', im, im') of columns 2 q, 2 q + 1
    int o = H * s.pitch * 16;
    s.exRow = N * 8 + 64;                             // bytes per row pair: the pad spreads the pairs over the banks
    s.ex = o;                                         // per row pair: half of the positions (s < 8, then s >= 8)
    o += NT / (N / 16) * s.exRow;
    s.twN = o;                                        // [G - 1 (stage, j)][16 s] (tr, tr), (ti, ti), then (-ti, -ti)
    o += (N - 16) * 24;
    s.twH = o;                                        // the same for the columns, float2
    o += (H - 16) * 8;
    s.twW = o;                                        // [w] float2, the split's twiddles of the kept columns
    o += w * 8;
    s.total = o;
    return s;
}

template <int LOGN, int LOGH, bool U16>
__global__ void __launch_bounds__(NT, 2) k_forward_win(DhFwdParams f) {
    constexpr int N = 1 << LOGN, H = 1 << LOGH;
    constexpr int G = N / 16;            // positions 16 apart = threads per row pair
    constexpr int SPT = 16 / G;          // s values per thread
    constexpr int GH = H / 16;
    extern __shared__ float4 smf4[];
    unsigned char* sm = reinterpret_cast<unsigned char*>(smf4);
    const int w = f.w, h = f.h;
    const WinSmem L = winSmem(LOGN, H, w);
    float4* col = smf4;
    float* colF = reinterpret_cast<float*>(smf4);
    ulonglong2* twN = reinterpret_cast<ulonglong2*>(sm + L.twN);
    f2x* ntwN = reinterpret_cast<f2x*>(sm + L.twN) + 2 * (N - 16);
    float2* twH = reinterpret_cast<float2*>(sm + L.twH);
    float2* twW = reinterpret_cast<float2*>(sm + L.twW);
    const int unit = blockIdx.x, P = f.polCount, pol = unit % P, frame = unit / P;
    const int tid = threadIdx.x;
    const int sx0 = f.sx0[pol];
    // entry e = 16 (half - 1 + j) + s: exp(-2 pi i (s + 16 j) / (32 half))
    auto tailTwiddle = [&](int e) {
        const int hj = (e >> 4) + 1, lg = 31 - __clz(hj);
        return __ldg(&f.twiddle[((e & 15) + 16 * (hj - (1 << lg))) << (TW_LOG - 5 - lg)]);
    };
    for (int e = tid; e < N - 16; e += NT) {
        const float2 t = tailTwiddle(e);
        twN[e] = make_ulonglong2(pk1(t.x), pk1(t.y));
        ntwN[e] = pk1(-t.y);
    }
    for (int e = tid; e < H - 16; e += NT) twH[e] = tailTwiddle(e);
    for (int c = tid; c < w; c += NT) twW[c] = __ldg(&f.twiddle[(sx0 + c) << (TW_LOG - LOGN - 1)]);
    __syncthreads();

    // ---- rows: thread g of row pair rp
    const int g = tid % G, rp = tid / G;
    ulonglong2* ex = reinterpret_cast<ulonglong2*>(sm + L.ex + rp * L.exRow);
    const int gr = (int)(__brev((unsigned)g) >> (32 - (LOGN - 4)));   // bit-reversed block index
    const long long base = (long long)frame * f.frameStride + (long long)f.cy[pol] * f.frameWidth + f.cx[pol];
    // the s of this thread's outputs: [0] and [1] (and [2] and [3]) are negatives modulo 16
    int sOf[SPT];
    sOf[0] = g;
    sOf[1] = g ? 16 - g : 8;
    if (SPT == 4) {
        sOf[2] = g + 4;
        sOf[3] = 12 - g;
    }
    for (int r0 = 2 * rp; r0 < H; r0 += 2 * NT / G) {
        f2x re[16], im[16];
        {
            const long long o = base + (long long)r0 * f.frameWidth + 2 * gr;
            float2 z0[16], z1[16];
#pragma unroll
            for (int c = 0; c < 16; c++) {   // in address order: both halves of a line together
                const int s = brevc(c, 4);
                const long long e = o + 2 * (c << (LOGN - 4));
                if (U16) {
                    const unsigned u0 = loadPair(static_cast<const unsigned short*>(f.frames) + e);
                    const unsigned u1 = loadPair(static_cast<const unsigned short*>(f.frames) + e + f.frameWidth);
                    z0[s] = make_float2((float)(u0 & 0xFFFFu), (float)(u0 >> 16));
                    z1[s] = make_float2((float)(u1 & 0xFFFFu), (float)(u1 >> 16));
                } else {
                    z0[s] = loadPair(static_cast<const float*>(f.frames) + e);
                    z1[s] = loadPair(static_cast<const float*>(f.frames) + e + f.frameWidth);
                }
            }
            // the first stage pairs the two rows on its way
#pragma unroll
            for (int s = 0; s < 16; s += 2) {
                re[s] = pk(z0[s].x + z0[s + 1].x, z1[s].x + z1[s + 1].x);
                im[s] = pk(z0[s].y + z0[s + 1].y, z1[s].y + z1[s + 1].y);
                re[s + 1] = pk(z0[s].x - z0[s + 1].x, z1[s].x - z1[s + 1].x);
                im[s + 1] = pk(z0[s].y - z0[s + 1].y, z1[s].y - z1[s + 1].y);
            }
        }
        ditStage<1>(re, im);
        ditStage<2>(re, im);
        ditStage<3>(re, im);
        // exchange: position (s, g) at (s mod 8) G + (g ^ (s mod G)), the lower eight s, then the upper
        f2x zr[SPT][G], zi[SPT][G];
#pragma unroll
        for (int up = 0; up < 2; up++) {
            if (up) __syncwarp();
#pragma unroll
            for (int s = 0; s < 8; s++) ex[s * G + (g ^ (s % G))] = make_ulonglong2(re[8 * up + s], im[8 * up + s]);
            __syncwarp();
#pragma unroll
            for (int a = up; a < SPT; a += 2)   // the even entries of sOf are below 8, the odd ones not
#pragma unroll
                for (int b = 0; b < G; b++) {
                    const ulonglong2 v = ex[(sOf[a] & 7) * G + (b ^ (sOf[a] % G))];
                    zr[a][b] = v.x;
                    zi[a][b] = v.y;
                }
        }
        __syncwarp();
#pragma unroll
        for (int a = 0; a < SPT; a++) {
            ditTail<G>(zr[a], zi[a], [&](int hj, f2x& tr, f2x& ti, f2x& nti) {
                const ulonglong2 t = twN[16 * hj + sOf[a]];
                tr = t.x;
                ti = t.y;
                nti = ntwN[16 * hj + sOf[a]];
            });
        }
        // R2C split of the kept columns: F[k] = (Z[k] + conj Z[N-k]) / 2 - i e^{-2 pi i k / W} (Z[k] - conj Z[N-k]) / 2
        float* c0 = colF + r0 * L.pitch * 4;
        float* c1 = c0 + L.pitch * 4;
        auto split = [&](int k, f2x kr, f2x ki, f2x pr, f2x pi) {
            const float2 t = twW[k - sx0];
            const f2x half = pk1(0.5f);
            const f2x er = mul2(add2(kr, pr), half), ei = mul2(sub2(ki, pi), half);
            const f2x orr = mul2(add2(ki, pi), half), oi = mul2(sub2(kr, pr), pk1(-0.5f));
            const float2 vr = upk(add2(er, fma2(pk1(t.x), orr, mul2(pk1(-t.y), oi))));
            const float2 vi = upk(add2(ei, fma2(pk1(t.x), oi, mul2(pk1(t.y), orr))));
            const int q = (k - sx0) >> 1, odd = (k - sx0) & 1;
            c0[4 * q + odd] = vr.x;
            c0[4 * q + 2 + odd] = vi.x;
            c1[4 * q + odd] = vr.y;
            c1[4 * q + 2 + odd] = vi.y;
        };
#pragma unroll
        for (int a = 0; a < SPT; a++) {
#pragma unroll
            for (int b = 0; b < G; b++) {
                const int k = sOf[a] + 16 * b;
                if ((unsigned)(k - sx0) >= (unsigned)w) continue;
                // Z[N - k]: the partner's position G - 1 - b; s = 0 and s = 8 are their own partners
                const int o = a ^ 1, m = G - 1 - b;
                f2x pr = zr[o][m], pi = zi[o][m];
                if (a < 2 && g == 0) {
                    const int ms = a == 0 ? (G - b) % G : m;
                    pr = zr[a][ms];
                    pi = zi[a][ms];
                }
                split(k, zr[a][b], zi[a][b], pr, pi);
            }
        }
        if (g == 0 && N - sx0 < w) split(N, zr[0][0], zi[0][0], zr[0][0], zi[0][0]);
    }
    __syncthreads();

    // ---- columns, in place: position p lies at row bitrev(p)
    const int pairs = w / 2;
    for (int task = tid; task < pairs * GH; task += NT) {
        const int q = task % pairs, b = task / pairs;
        float4* c = col + (int)(__brev((unsigned)b) >> (32 - (LOGH - 4))) * L.pitch + q;
        f2x re[16], im[16];
#pragma unroll
        for (int s = 0; s < 16; s++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(c + (brevc(s, 4) << (LOGH - 4)) * L.pitch);
            re[s] = v.x;
            im[s] = v.y;
        }
        ditStage<0>(re, im);
        ditStage<1>(re, im);
        ditStage<2>(re, im);
        ditStage<3>(re, im);
#pragma unroll
        for (int s = 0; s < 16; s++)
            *reinterpret_cast<ulonglong2*>(c + (brevc(s, 4) << (LOGH - 4)) * L.pitch) = make_ulonglong2(re[s], im[s]);
    }
    __syncthreads();
    const int row0 = ((f.sy[pol] + H / 2) % H + H) % H;
    float2 bc = make_float2(1.0f, 0.0f);
    const bool cal = f.batchCal && f.batchCalCount > 0;
    if (cal) bc = f.batchCal[pol * f.batchCalCount + ((f.frameOffset + frame) % f.batchCalCount)];
    for (int task = tid; task < pairs * 16; task += NT) {
        const int q = task % pairs, s = task / pairs;
        const float4* c = col + (int)(__brev((unsigned)s) >> 28 << (LOGH - 4)) * L.pitch + q;
        f2x re[GH], im[GH];
#pragma unroll
        for (int b = 0; b < GH; b++) {
            const ulonglong2 v = *reinterpret_cast<const ulonglong2*>(c + brevc(b, LOGH - 4) * L.pitch);
            re[b] = v.x;
            im[b] = v.y;
        }
        ditTail<GH>(re, im, [&](int hj, f2x& tr, f2x& ti, f2x& nti) {
            const float2 t = twH[16 * hj + s];
            tr = pk1(t.x);
            ti = pk1(t.y);
            nti = pk1(-t.y);
        });
#pragma unroll
        for (int b = 0; b < GH; b++) {
            const int j = (s + 16 * b - row0) & (H - 1);
            if (j >= h) continue;
            const float2 vr = upk(re[b]), vi = upk(im[b]);
            float2 y0 = make_float2(vr.x, vi.x), y1 = make_float2(vr.y, vi.y);
            if (cal) {
                y0 = cmul(y0, bc);
                y1 = cmul(y1, bc);
            }
            const float4 a = __ldg(reinterpret_cast<const float4*>(f.tabAdj + ((size_t)pol * h + j) * w) + q);
            y0 = cmul(y0, make_float2(a.x, a.y));
            y1 = cmul(y1, make_float2(a.z, a.w));
            reinterpret_cast<float4*>(f.window + ((size_t)unit * h + j) * w)[q] = make_float4(y0.x, y0.y, y1.x, y1.y);
        }
    }
}

template <int LOGN, int LOGH>
cudaError_t launchWin(const DhFwdParams& f, cudaStream_t s) {
    const WinSmem L = winSmem(LOGN, 1 << LOGH, f.w);
    if (L.total > 227 * 1024) return cudaErrorNotSupported;
    const unsigned units = (unsigned)(f.frameCount * f.polCount);
    if (f.inputU16) {
        cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(k_forward_win<LOGN, LOGH, true>), L.total);
        if (e != cudaSuccess) return e;
        k_forward_win<LOGN, LOGH, true><<<units, NT, L.total, s>>>(f);
    } else {
        cudaError_t e = setSmemOnce(reinterpret_cast<const void*>(k_forward_win<LOGN, LOGH, false>), L.total);
        if (e != cudaSuccess) return e;
        k_forward_win<LOGN, LOGH, false><<<units, NT, L.total, s>>>(f);
    }
    return cudaGetLastError();
}

}  // namespace

// cudaErrorNotSupported outside the kernel's shapes: FFT windows 128 or 256
// wide and 64, 128 or 256 high, the window's columns within the R2C half
// plane, its buffered columns within shared memory (up to 80 at 256 rows).
cudaError_t dh_launch_forward_win(const DhFwdParams& f, cudaStream_t s) {
    const int N = 1 << (f.logW - 1);
    if (f.logW < 7 || f.logW > 8 || f.logH < 6 || f.logH > 8 || !f.tabAdj || !f.twiddle || !f.window) return cudaErrorNotSupported;
    if (f.w % 16 || f.h % 16 || f.w <= 0 || f.h <= 0 || f.h > (1 << f.logH)) return cudaErrorNotSupported;
    // pixel pairs in one load
    const size_t es = f.inputU16 ? 2 : 4;
    if (reinterpret_cast<uintptr_t>(f.frames) % (2 * es) || f.frameWidth % 2 || f.frameStride % 2) return cudaErrorNotSupported;
    // window rows and factors as 16-byte pairs
    if ((reinterpret_cast<uintptr_t>(f.window) | reinterpret_cast<uintptr_t>(f.tabAdj)) % 16) return cudaErrorNotSupported;
    for (int p = 0; p < f.polCount; p++)
        if (f.sx0[p] < 0 || f.sx0[p] + f.w > N + 1 || f.cx[p] % 2) return cudaErrorNotSupported;
    if (f.frameCount * f.polCount <= 0) return cudaSuccess;
    if (f.logW == 7)
        return f.logH == 6 ? launchWin<6, 6>(f, s) : f.logH == 7 ? launchWin<6, 7>(f, s) : launchWin<6, 8>(f, s);
    return f.logH == 6 ? launchWin<7, 6>(f, s) : f.logH == 7 ? launchWin<7, 7>(f, s) : launchWin<7, 8>(f, s);
}
