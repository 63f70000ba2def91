// FP64 SIMT GEMMs (real and complex, row-major, batched by blockIdx.z).
//
// These serve the plain FP64 GPU path and the small complex products of the
// G builder and E_c; on GB300 the FP64 pipe (1.06 TFLOP/s) is the limit, so a
// register-blocked 64x64 tile already sits on the FP64 roofline where its tiles fill the device.
#include "kernels.h"
#include "common.h"

#include <algorithm>

namespace gb {

namespace {

constexpr int BM = 64, BN = 64, BK = 16;

template <typename T>
__global__ void __launch_bounds__(256) k_gemm_real(int M, int N, int K, const T *__restrict__ A, long long lda,
                                                   long long sA, const T *__restrict__ B, long long ldb,
                                                   long long sB, T *__restrict__ C, long long ldc, long long sC,
                                                   T alpha, T beta)
{
    __shared__ T As[BK][BM + 1];
    __shared__ T Bs[BK][BN];
    const int bz = blockIdx.z;
    A += bz * sA;
    B += bz * sB;
    C += bz * sC;
    const int m0 = blockIdx.y * BM, n0 = blockIdx.x * BN;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    T acc[4][4] = {};
    for (int k0 = 0; k0 < K; k0 += BK)
    {
        for (int t = threadIdx.x; t < BM * BK; t += 256)
        {
            const int r = t / BK, kk = t % BK;
            const int gm = m0 + r, gk = k0 + kk;
            As[kk][r] = (gm < M && gk < K) ? A[gm * lda + gk] : T(0);
        }
        for (int t = threadIdx.x; t < BK * BN; t += 256)
        {
            const int kk = t / BN, c = t % BN;
            const int gk = k0 + kk, gn = n0 + c;
            Bs[kk][c] = (gk < K && gn < N) ? B[gk * ldb + gn] : T(0);
        }
        __syncthreads();
#pragma unroll
        for (int kk = 0; kk < BK; ++kk)
        {
            T a[4], b[4];
#pragma unroll
            for (int i = 0; i < 4; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
            for (int j = 0; j < 4; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
            for (int i = 0; i < 4; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) acc[i][j] = fma(a[i], b[j], acc[i][j]);
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
        {
            const int gm = m0 + ty + 16 * i, gn = n0 + tx + 16 * j;
            if (gm < M && gn < N)
            {
                T v = alpha * acc[i][j];
                if (beta != T(0)) v += beta * C[gm * ldc + gn];
                C[gm * ldc + gn] = v;
            }
        }
}

// The same product in 32 x 32 tiles of 128 threads, 4 x 2 outputs each, for shapes whose 64 x 64 tiles leave
// SMs idle: the FP64 pipe of an SM does 1.68 FMAs a clock whatever it holds, so the number of SMs at work and
// the padding of the tiles set the time.  A thread's rows and columns beyond the matrix are left out, and
// the next 16 of K are in flight during a block's FMAs.  Each element's sum runs over k in the same order
// as in the larger tiles.  One GB300, 16 products of 102 x 102 x 102: 134 us in 64 x 64 tiles, now 56.
constexpr int SM_TILE = 32, SM_THREADS = 128, SM_K = 16;

template <typename T>
__global__ void __launch_bounds__(SM_THREADS) k_gemm_small(int M, int N, int K, const T *__restrict__ A, long long lda,
                                                          long long sA, const T *__restrict__ B, long long ldb,
                                                          long long sB, T *__restrict__ C, long long ldc, long long sC,
                                                          T alpha, T beta)
{
    constexpr int NLD = SM_TILE * SM_K / SM_THREADS;
    __shared__ T As[SM_K][SM_TILE + 1];
    __shared__ T Bs[SM_K][SM_TILE];
    A += blockIdx.z * sA;
    B += blockIdx.z * sB;
    C += blockIdx.z * sC;
    const int m0 = blockIdx.y * SM_TILE, n0 = blockIdx.x * SM_TILE;
    // rows ty + 8 i, columns tx + 16 j
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int mi = min(4, (M - m0 + 7) / 8), nj = min(2, (N - n0 + 15) / 16);  // uniform over the CTA
    T ra[NLD], rb[NLD];
    auto fetch = [&](int k0) {
#pragma unroll
        for (int u = 0; u < NLD; ++u)
        {
            const int t = threadIdx.x + u * SM_THREADS;
            const int gm = m0 + t / SM_K, ka = k0 + t % SM_K, kb = k0 + t / SM_TILE, gn = n0 + t % SM_TILE;
            ra[u] = gm < M && ka < K ? A[gm * lda + ka] : T(0);
            rb[u] = kb < K && gn < N ? B[kb * ldb + gn] : T(0);
        }
    };
    T acc[4][2] = {};
    fetch(0);
    for (int k0 = 0; k0 < K; k0 += SM_K)
    {
#pragma unroll
        for (int u = 0; u < NLD; ++u)
        {
            const int t = threadIdx.x + u * SM_THREADS;
            As[t % SM_K][t / SM_K] = ra[u];
            Bs[t / SM_TILE][t % SM_TILE] = rb[u];
        }
        __syncthreads();
        if (k0 + SM_K < K) fetch(k0 + SM_K);
        const int kn = min(SM_K, K - k0);
#pragma unroll 4
        for (int kk = 0; kk < kn; ++kk)
        {
            const T b0 = Bs[kk][tx], b1 = Bs[kk][tx + 16];
#pragma unroll
            for (int i = 0; i < 4; ++i)
                if (i < mi)
                {
                    const T a = As[kk][ty + 8 * i];
                    acc[i][0] = fma(a, b0, acc[i][0]);
                    if (nj == 2) acc[i][1] = fma(a, b1, acc[i][1]);
                }
        }
        __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < 4; ++i)
#pragma unroll
        for (int j = 0; j < 2; ++j)
        {
            const int gm = m0 + ty + 8 * i, gn = n0 + tx + 16 * j;
            if (gm < M && gn < N)
            {
                T v = alpha * acc[i][j];
                if (beta != T(0)) v += beta * C[gm * ldc + gn];
                C[gm * ldc + gn] = v;
            }
        }
}

// 32 x 32 tiles below two CTAs of 64 x 64 an SM; above, the larger tile reads A and B half as often and the
// pipe is busy either way.  2 x 1600 x 102 x 800: 244 us in 104 large tiles, 159 in 350 small ones; FP64 X of
// 1040 x 208 x 208 (two signs): 247 us in 136, 212 in 462.  The grid's y and z limits hold for both.
template <typename T>
void gemm_real(int M, int N, int K, const T *A, long long lda, long long sA, const T *B, long long ldb, long long sB, T *C,
               long long ldc, long long sC, int batch, T alpha, T beta, cudaStream_t st)
{
    const dim3 grid((N + BN - 1) / BN, (M + BM - 1) / BM, batch);
    const dim3 small((N + SM_TILE - 1) / SM_TILE, (M + SM_TILE - 1) / SM_TILE, batch);
    if (static_cast<long long>(grid.x) * grid.y * grid.z < 2 * 152 && small.y <= 65535)
        k_gemm_small<T><<<small, SM_THREADS, 0, st>>>(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, alpha, beta);
    else
        k_gemm_real<T><<<grid, 256, 0, st>>>(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, alpha, beta);
    GB_LAUNCH_CHECK();
}

constexpr int ZB = 32, ZK = 16;

__global__ void __launch_bounds__(256) k_zgemm(int M, int N, int K, const cuDoubleComplex *__restrict__ A,
                                               long long lda, long long sA, const cuDoubleComplex *__restrict__ B,
                                               long long ldb, long long sB, cuDoubleComplex *__restrict__ C,
                                               long long ldc, long long sC)
{
    __shared__ cuDoubleComplex As[ZK][ZB + 1];
    __shared__ cuDoubleComplex Bs[ZK][ZB];
    const int bz = blockIdx.z;
    A += bz * sA;
    B += bz * sB;
    C += bz * sC;
    const int m0 = blockIdx.y * ZB, n0 = blockIdx.x * ZB;
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    cuDoubleComplex acc[2][2];
    for (int i = 0; i < 2; ++i)
        for (int j = 0; j < 2; ++j) acc[i][j] = make_cuDoubleComplex(0, 0);
    for (int k0 = 0; k0 < K; k0 += ZK)
    {
        for (int t = threadIdx.x; t < ZB * ZK; t += 256)
        {
            const int r = t / ZK, kk = t % ZK;
            const int gm = m0 + r, gk = k0 + kk;
            As[kk][r] = (gm < M && gk < K) ? A[gm * lda + gk] : make_cuDoubleComplex(0, 0);
        }
        for (int t = threadIdx.x; t < ZK * ZB; t += 256)
        {
            const int kk = t / ZB, c = t % ZB;
            const int gk = k0 + kk, gn = n0 + c;
            Bs[kk][c] = (gk < K && gn < N) ? B[gk * ldb + gn] : make_cuDoubleComplex(0, 0);
        }
        __syncthreads();
#pragma unroll 4
        for (int kk = 0; kk < ZK; ++kk)
        {
            const cuDoubleComplex a0 = As[kk][ty], a1 = As[kk][ty + 16];
            const cuDoubleComplex b0 = Bs[kk][tx], b1 = Bs[kk][tx + 16];
            acc[0][0] = cuCfma(a0, b0, acc[0][0]);
            acc[0][1] = cuCfma(a0, b1, acc[0][1]);
            acc[1][0] = cuCfma(a1, b0, acc[1][0]);
            acc[1][1] = cuCfma(a1, b1, acc[1][1]);
        }
        __syncthreads();
    }
    for (int i = 0; i < 2; ++i)
        for (int j = 0; j < 2; ++j)
        {
            const int gm = m0 + ty + 16 * i, gn = n0 + tx + 16 * j;
            if (gm < M && gn < N) C[gm * ldc + gn] = acc[i][j];
        }
}

} // namespace

void launch_dgemm(int M, int N, int K, const double *A, long long lda, long long sA, const double *B,
                  long long ldb, long long sB, double *C, long long ldc, long long sC, int batch,
                  double alpha, double beta, cudaStream_t st)
{
    if (M <= 0 || N <= 0 || batch <= 0) return;
    gemm_real(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, batch, alpha, beta, st);
}

void launch_sgemm(int M, int N, int K, const float *A, long long lda, long long sA, const float *B,
                  long long ldb, long long sB, float *C, long long ldc, long long sC, int batch,
                  cudaStream_t st)
{
    if (M <= 0 || N <= 0 || batch <= 0) return;
    gemm_real(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC, batch, 1.0f, 0.0f, st);
}

namespace {
__global__ void k_d2f(const double *__restrict__ in, float *__restrict__ out, long long n)
{
    for (long long i = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; i < n;
         i += static_cast<long long>(gridDim.x) * blockDim.x)
        out[i] = static_cast<float>(in[i]);
}
} // namespace

void launch_d2f(const double *in, float *out, long long n, cudaStream_t st)
{
    if (n <= 0) return;
    const long long blocks = std::min<long long>((n + 255) / 256, 152LL * 16);
    k_d2f<<<static_cast<unsigned>(blocks), 256, 0, st>>>(in, out, n);
    GB_LAUNCH_CHECK();
}

void launch_zgemm(int M, int N, int K, const cuDoubleComplex *A, long long lda, long long sA,
                  const cuDoubleComplex *B, long long ldb, long long sB, cuDoubleComplex *C, long long ldc,
                  long long sC, int batch, cudaStream_t st)
{
    if (M <= 0 || N <= 0 || batch <= 0) return;
    dim3 grid((N + ZB - 1) / ZB, (M + ZB - 1) / ZB, batch);
    k_zgemm<<<grid, 256, 0, st>>>(M, N, K, A, lda, sA, B, ldb, sB, C, ldc, sC);
    GB_LAUNCH_CHECK();
}

} // namespace gb
