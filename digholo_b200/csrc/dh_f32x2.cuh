// Packed pairs of floats (Blackwell's f32x2 instructions): one instruction
// works on two independent values, each rounded exactly as the scalar
// instruction rounds it, so a pair of transforms runs in lock step with the
// bits of two scalar ones.  A pair is held in one 64-bit register.
#pragma once
#include <cuda_runtime.h>

#include "dh_fft.cuh"

namespace dh {

typedef unsigned long long f2x;

__device__ __forceinline__ f2x pk(float lo, float hi) {
    f2x r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ f2x pk1(float v) { return pk(v, v); }
__device__ __forceinline__ float2 upk(f2x v) {
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
    return r;
}
__device__ __forceinline__ f2x add2(f2x a, f2x b) {
    f2x r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2x sub2(f2x a, f2x b) {
    f2x r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2x mul2(f2x a, f2x b) {
    f2x r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f2x fma2(f2x a, f2x b, f2x c) {
    f2x r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}

// (re, im) *= (tr, ti), ti and its negative given: the rounding of cmul().
__device__ __forceinline__ void cmul2(f2x& re, f2x& im, f2x tr, f2x ti, f2x nti) {
    const f2x r = fma2(re, tr, mul2(im, nti));
    im = fma2(re, ti, mul2(im, tr));
    re = r;
}

// Two radix-2 DIF inverse FFTs of N points in lock step, the operations of
// ifftDIFf<N> one for one: natural-order input, bit-reversed output.
template <int N>
__device__ __forceinline__ void ifftDIF2(f2x (&re)[N], f2x (&im)[N]) {
#pragma unroll
    for (int m = N / 2; m >= 1; m >>= 1) {
#pragma unroll
        for (int blk = 0; blk < N; blk += 2 * m) {
#pragma unroll
            for (int j = 0; j < m; j++) {
                const int p = blk + j, q = blk + j + m;
                const f2x ar = re[p], ai = im[p], br = re[q], bi = im[q];
                re[p] = add2(ar, br);
                im[p] = add2(ai, bi);
                if (2 * j == m) {
                    re[q] = sub2(bi, ai);   // times i
                    im[q] = sub2(ar, br);
                } else {
                    re[q] = sub2(ar, br);
                    im[q] = sub2(ai, bi);
                    if (j != 0) {
                        const float2 t = tw128(j * (128 / (2 * m)));
                        cmul2(re[q], im[q], pk1(t.x), pk1(-t.y), pk1(t.y));
                    }
                }
            }
        }
    }
}

}  // namespace dh
