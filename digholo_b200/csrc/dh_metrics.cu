// Power-meter support on the GPU: gather of one coefficient matrix block and
// its FP64 Gram matrix, whose eigenvalues (dh_eigen.cu, FP64) are the squared
// singular values digHolo takes from cgesvd (digHolo.cpp:3021-3055, used by
// digHoloPowerMeter digHolo.cpp:10980-11011).
#include <cuda_runtime.h>
#include <cuComplex.h>

#include <cstdio>

// Dense column-major block A (rows = svdM modes, cols = batch) from the
// coefficient array coefs[batch][polCount * M]:
//   row j < M      : src0[b][pol0 * M + j]
//   row j >= M     : src1[b][pol1 * M + (j - M)]   (only when rows == 2M)
__global__ void k_gather_block(const float2* __restrict__ src0, const float2* __restrict__ src1, int pol0, int pol1,
                               int polCount, int M, int rows, int batch, float2* __restrict__ A) {
    const int total = rows * batch;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < total; e += gridDim.x * blockDim.x) {
        const int b = e / rows, j = e - b * rows;
        const float2* s = j < M ? src0 + (size_t)b * polCount * M + pol0 * M + j
                                : src1 + (size_t)b * polCount * M + pol1 * M + (j - M);
        A[(size_t)b * rows + j] = *s;
    }
}

// Gram matrix in FP64, column-major n x n:
//   rowsGram (n == rows):  G[i][k] = sum_b A[i][b] conj(A[k][b])
//   batch Gram (n == batch): G[i][k] = sum_j conj(A[j][i]) A[j][k]   (A^H A)
// A block has an 8 x 8 tile of G and four threads per element, each with a
// quarter of every 64 terms; the quarters are added in a fixed order.  Bound:
// the FP64 chain of a thread (K / 4 terms) and, at the sizes of a metrics
// call, the number of blocks: 110 modes x 256 frames 24.3 us with one thread
// per element in 16 x 16 tiles (49 blocks, 256 terms in a row), 8.4 us so; 6 x
// 40 5.9 and 3.4 us, 300 x 700 98 and 74, 600 x 700 293 and 259.
constexpr int GT = 8, GK = 64;
__global__ void __launch_bounds__(256) k_gram(const float2* __restrict__ A, int rows, int batch, int rowsGram,
                                              cuDoubleComplex* __restrict__ G) {
    __shared__ float2 ta[GT][GK + 1];
    __shared__ float2 tb[GT][GK + 1];
    __shared__ double2 part[3][GT * GT];
    const int n = rowsGram ? rows : batch;
    const int K = rowsGram ? batch : rows;
    const int t = threadIdx.x, e = t & 63, q = t >> 6;
    const int x = e & 7, y = e >> 3;
    const int i0 = blockIdx.y * GT, k0 = blockIdx.x * GT;
    double re = 0.0, im = 0.0;
    for (int t0 = 0; t0 < K; t0 += GK) {
        // ta[r][c] = element (i0 + r, t0 + c), tb[r][c] = element (k0 + r, t0 + c)
#pragma unroll
        for (int l = 0; l < 4; l++) {
            const int u = t + 256 * (l & 1);   // element of the 8 x 64 tile
            const int r = rowsGram ? u & 7 : u >> 6, c = rowsGram ? u >> 3 : u & 63;
            const int row = (l < 2 ? i0 : k0) + r, tt = t0 + c;
            float2 v = make_float2(0.f, 0.f);
            if (tt < K && row < n) v = rowsGram ? A[(size_t)tt * rows + row] : A[(size_t)row * rows + tt];
            (l < 2 ? ta : tb)[r][c] = v;
        }
        __syncthreads();
#pragma unroll
        for (int c = 0; c < GK / 4; c++) {
            const float2 a = ta[y][q * (GK / 4) + c];
            const float2 b = tb[x][q * (GK / 4) + c];
            const double ar = a.x, ai = a.y, br = b.x, bi = b.y;
            re += ar * br + ai * bi;
            im += ai * br - ar * bi;   // a * conj(b)
        }
        __syncthreads();
    }
    if (q > 0) part[q - 1][e] = make_double2(re, im);
    __syncthreads();
    if (q > 0) return;
    for (int p = 0; p < 3; p++) {
        re += part[p][e].x;
        im += part[p][e].y;
    }
    const int i = i0 + y, k = k0 + x;
    if (i < n && k < n) G[(size_t)k * n + i] = make_cuDoubleComplex(re, rowsGram ? im : -im);   // else conj(a) * b
}

cudaError_t dh_launch_gather_block(const float2* src0, const float2* src1, int pol0, int pol1, int polCount, int M,
                                   int rows, int batch, float2* A, cudaStream_t s) {
    const int total = rows * batch;
    int blocks = (total + 255) / 256;
    if (blocks > 4096) blocks = 4096;
    k_gather_block<<<blocks, 256, 0, s>>>(src0, src1, pol0, pol1, polCount, M, rows, batch, A);
    return cudaGetLastError();
}

cudaError_t dh_launch_gram(const float2* A, int rows, int batch, int rowsGram, void* G, cudaStream_t s) {
    const int n = rowsGram ? rows : batch;
    dim3 grid((n + GT - 1) / GT, (n + GT - 1) / GT);
    k_gram<<<grid, 256, 0, s>>>(A, rows, batch, rowsGram, static_cast<cuDoubleComplex*>(G));
    return cudaGetLastError();
}
