// Batched blocked Cholesky factorisation in FP64 (real symmetric or complex Hermitian).
//
// Right-looking, panel width NB = 32, three launches per panel step for the whole batch:
//   k_chol_diag  : one CTA per matrix factors the NB x NB diagonal block in shared memory;
//   k_chol_panel : each CTA solves a 32-row slab of the panel below it, X L11^H = A21;
//   k_chol_update: lower-triangle trailing update A22 -= L21 L21^H in 32 x 32 tiles.
// The real variant chol_batched_r_ozaki uses panels of 64 and does the trailing update on the
// tensor cores with exact integer slices (k_chol_ozaki.cu).
// The diagonal of L is written to diag[b][i]; ln det A = 2 sum_i log L_ii (k_chol_logdet).
// On GB300 the FP64 pipe (~1 TFLOP/s) bounds these kernels; the blocking keeps them off
// the HBM roofline (each trailing element is read and written once per 32 columns).
#include <cuComplex.h>

#include "chol.h"
#include "common.h"

namespace gb {

namespace {

constexpr int NB = 32;

__device__ inline double cre(double x) { return x; }
__device__ inline double cre(cuDoubleComplex x) { return x.x; }
__device__ inline double cconjmul_acc(double acc, double a, double b) { return fma(a, b, acc); }
__device__ inline cuDoubleComplex cconjmul_acc(cuDoubleComplex acc, cuDoubleComplex a, cuDoubleComplex b)
{
    // acc + a * conj(b)
    return make_cuDoubleComplex(acc.x + a.x * b.x + a.y * b.y, acc.y + a.y * b.x - a.x * b.y);
}
__device__ inline double csub(double a, double b) { return a - b; }
__device__ inline cuDoubleComplex csub(cuDoubleComplex a, cuDoubleComplex b) { return cuCsub(a, b); }
__device__ inline double cscale(double a, double s) { return a * s; }
__device__ inline cuDoubleComplex cscale(cuDoubleComplex a, double s) { return make_cuDoubleComplex(a.x * s, a.y * s); }
template <typename T>
__device__ inline T czero();
template <>
__device__ inline double czero<double>() { return 0.0; }
template <>
__device__ inline cuDoubleComplex czero<cuDoubleComplex>() { return make_cuDoubleComplex(0.0, 0.0); }
__device__ inline double cfromreal(double x, double) { return x; }
__device__ inline cuDoubleComplex cfromreal(double x, cuDoubleComplex) { return make_cuDoubleComplex(x, 0.0); }

// Factor the nb x nb diagonal block at k0 into shared memory D (lower triangle).
template <typename T, int NBT>
__device__ void factor_diag(const T *A, int N, int k0, int nb, T (*D)[NBT + 1], int *bad)
{
    for (int t = threadIdx.x; t < nb * nb; t += blockDim.x)
    {
        const int i = t / nb, j = t % nb;
        D[i][j] = j <= i ? A[static_cast<long long>(k0 + i) * N + k0 + j] : czero<T>();
    }
    __syncthreads();
    __shared__ double sinv;  // reciprocal of the current pivot, formed once per step
    for (int p = 0; p < nb; ++p)
    {
        if (threadIdx.x == 0)
        {
            const double d2 = cre(D[p][p]);
            if (!(d2 > 0.0)) *bad = 1;
            const double l = sqrt(fmax(d2, 1e-300));
            D[p][p] = cfromreal(l, D[p][p]);
            sinv = 1.0 / l;
        }
        __syncthreads();
        const double inv = sinv;
        for (int i = p + 1 + threadIdx.x; i < nb; i += blockDim.x) D[i][p] = cscale(D[i][p], inv);
        __syncthreads();
        const int m = nb - p - 1;
        for (int t = threadIdx.x; t < m * m; t += blockDim.x)
        {
            const int i = p + 1 + t / m, j = p + 1 + t % m;
            if (j <= i) D[i][j] = csub(D[i][j], cconjmul_acc(czero<T>(), D[i][p], D[j][p]));
        }
        __syncthreads();
    }
}

// Factor the diagonal block in place (one CTA per matrix) and record the diagonal of L.
template <typename T, int NBT>
__global__ void __launch_bounds__(256) k_chol_diag(T *__restrict__ Aall, int N, int k0, double *__restrict__ diag,
                                                  int *__restrict__ bad)
{
    __shared__ T D[NBT][NBT + 1];
    const int b = blockIdx.x;
    T *A = Aall + static_cast<long long>(b) * N * N;
    const int nb = min(NBT, N - k0);
    factor_diag<T, NBT>(A, N, k0, nb, D, bad + b);
    for (int t = threadIdx.x; t < nb * nb; t += blockDim.x)
    {
        const int i = t / nb, j = t % nb;
        if (j <= i) A[static_cast<long long>(k0 + i) * N + k0 + j] = D[i][j];
    }
    for (int i = threadIdx.x; i < nb; i += blockDim.x) diag[static_cast<long long>(b) * N + k0 + i] = cre(D[i][i]);
}

// Real diagonal block of the tensor-core Cholesky: factor the nb x nb block at k0 in place, record the
// diagonal of L, and with INV form W = L11^-1 (lower triangular, FP64) into Wb[b][64][64], so that the
// panel becomes the product L21 = A21 W^T.
//
// Right-looking, the block in registers: thread (row i, s) holds the columns 8 k + s of row i.  With raw
// column a_i of step p, pivot d and the inverse's unscaled row V_p (1 at p), the rows below take off
// (a_i / d) times a_j to the right of p and (a_i / d) times V_pj up to p; a row's columns up to p belong
// to the inverse and the later ones to A, so one array of 8 holds both.  Square roots wait until the end
// (L_ip = a_i d_p^-1/2, W_p = d_p^-1/2 V_p): a step's chain is one barrier, a product, the update of the
// next column and the next pivot's reciprocal.  Only whole warps skip work: the elements above the
// diagonal are updated with whatever U holds and never read, so loads and FMAs stand without branches
// between them.  A warp FMA occupies its scheduler's FP64 pipe for about 80 clocks and a warp of 4 rows
// costs in proportion to the square of their index, so diag_rows deals the 16 warps' rows to the 4
// schedulers evenly.  One GB300, a 64 x 64 block with its inverse: 216 us with the block in shared memory,
// 128 with the roots in the chain and two barriers a step, 111 with a branch per element, now 80 (and 61 without the
// inverse: the pivots' chain).
constexpr int DIAG_THREADS = 512;

// first of the 4 rows of a warp: warps w, w + 4, w + 8 and w + 12 share a scheduler
__device__ inline int diag_rows(int warp) { return 4 * static_cast<int>(0x621075438BA9CDEFull >> (4 * warp) & 15); }

template <bool INV>
__global__ void __launch_bounds__(DIAG_THREADS) k_chol_diag64(double *__restrict__ Aall, int N, int k0,
                                                             double *__restrict__ diag, int *__restrict__ bad,
                                                             double *__restrict__ Wb)
{
    constexpr int NBT = OZAKI_NB, KC = NBT / 8;
    static_assert(NBT == 64, "eight threads a row, 8 columns each");
    __shared__ double U[2][NBT], rinv[2], piv[NBT], raw[NBT][NBT + 1];
    const int b = blockIdx.x, nb = min(NBT, N - k0);
    const int r0 = diag_rows(threadIdx.x / 32), lane = threadIdx.x % 32;
    const int i = r0 + lane / 8, s = lane % 8;
    double *A = Aall + static_cast<long long>(b) * N * N + static_cast<long long>(k0) * N + k0;
    double v[KC];
#pragma unroll
    for (int k = 0; k < KC; ++k) v[k] = i < nb && 8 * k + s <= i ? A[static_cast<long long>(i) * N + 8 * k + s] : 0.0;
    for (int t = threadIdx.x; t < 2 * NBT; t += DIAG_THREADS) U[t / NBT][t % NBT] = 0.0;
    __syncthreads();
    // column n and the pivot of step n; x is this thread's element of column n (s == n % 8)
    auto hand_column = [&](int n, double &x) {
        if (s != n % 8) return;
        if (i > n && i < nb)
        {
            U[n & 1][i] = x;
            raw[i][n] = x;
            x = 0.0;
        }
        if (i == n)
        {
            if (!(x > 0.0)) bad[b] = 1;
            const double d = fmax(x, 1e-300);
            piv[n] = d;
            rinv[n & 1] = 1.0 / d;
            U[n & 1][n] = 1.0;
            x = 1.0;
        }
    };
    hand_column(0, v[0]);
#pragma unroll
    for (int kp = 0; kp < KC; ++kp)
#pragma unroll 1
        for (int sp = 0; sp < 8; ++sp)
        {
            const int p = 8 * kp + sp;
            if (p >= nb) break;
            __syncthreads();
            if (r0 + 3 <= p) continue;  // the warp's rows are done
            const double *u = U[p & 1] + s;
            const double c = i > p ? u[i - s] * rinv[p & 1] : 0.0;
            const int n = p + 1;
            v[kp] = fma(-c, u[8 * kp], v[kp]);
            if (kp + 1 < KC && 8 * (kp + 1) <= r0 + 3) v[kp + 1] = fma(-c, u[8 * (kp + 1)], v[kp + 1]);
            if (n < nb)
            {
                if (sp < 7)
                    hand_column(n, v[kp]);
                else if (kp + 1 < KC)
                    hand_column(n, v[kp + 1]);
            }
            if (INV)
#pragma unroll
                for (int k = 0; k < kp; ++k) v[k] = fma(-c, u[8 * k], v[k]);
#pragma unroll
            for (int k = kp + 2; k < KC; k += 2)
                if (8 * k <= r0 + 3)
                {
                    v[k] = fma(-c, u[8 * k], v[k]);
                    if (k + 1 < KC) v[k + 1] = fma(-c, u[8 * (k + 1)], v[k + 1]);
                }
            if (INV && i == n && n < nb)
            {
#pragma unroll
                for (int k = 0; k <= kp; ++k)
                    if (8 * k + s < n) U[n & 1][8 * k + s] = v[k];
            }
        }
    __syncthreads();
    if (threadIdx.x < nb)
    {
        const double d = piv[threadIdx.x], l = sqrt(d);
        raw[threadIdx.x][threadIdx.x] = d;
        diag[static_cast<long long>(b) * N + k0 + threadIdx.x] = l;
        piv[threadIdx.x] = 1.0 / l;
    }
    __syncthreads();
    for (int t = threadIdx.x; t < nb * NBT; t += DIAG_THREADS)
    {
        const int r = t / NBT, j = t % NBT;
        if (j <= r) A[static_cast<long long>(r) * N + j] = raw[r][j] * piv[j];
    }
    if constexpr (INV)
    {
        double *w = Wb + (static_cast<long long>(b) * NBT + i) * NBT;
#pragma unroll
        for (int k = 0; k < KC; ++k) w[8 * k + s] = i < nb && 8 * k + s <= i ? v[k] * piv[i] : 0.0;
    }
}

__device__ inline double cfms_conj(double c, double a, double b) { return fma(-a, b, c); }
__device__ inline cuDoubleComplex cfms_conj(cuDoubleComplex c, cuDoubleComplex a, cuDoubleComplex b)
{
    // c - a * conj(b)
    return make_cuDoubleComplex(fma(-a.y, b.y, fma(-a.x, b.x, c.x)), fma(a.x, b.y, fma(-a.y, b.x, c.y)));
}
__device__ inline double cshfl(double v, int src) { return __shfl_sync(0xffffffffu, v, src); }
__device__ inline cuDoubleComplex cshfl(cuDoubleComplex v, int src)
{
    return make_cuDoubleComplex(__shfl_sync(0xffffffffu, v.x, src), __shfl_sync(0xffffffffu, v.y, src));
}

// Panel solve X L11^H = A21 below a full diagonal block (L11 already factored in A), 32 rows a CTA.
// Right-looking, x[p] /= L_pp, then x[q] -= x[p] conj L_qp for every q > p.  Four threads hold a row,
// columns 4 k + s, and pass x[p] on by a shuffle, so that a few rows already give all four schedulers'
// FP64 pipes a warp; that pipe is the bound (a warp FMA takes about 80 clocks of it, 640 of them a warp
// with complex entries).  The staged L11 has a zero diagonal, so the update takes whole quads of columns.
// One GB300, the panels of eight complex 80 x 80 matrices: 122 us a launch with a thread per row, now 31.
constexpr int PANEL_THREADS = 128, PANEL_ROWS = PANEL_THREADS / 4;

template <typename T, int NBT>
__global__ void __launch_bounds__(PANEL_THREADS) k_chol_panel(T *__restrict__ Aall, int N, int k0)
{
    static_assert(NBT % 4 == 0, "four threads share a row's columns");
    constexpr int KC = NBT / 4;
    __shared__ T D[NBT][NBT + 1];
    __shared__ double invd[NBT];
    T *A = Aall + static_cast<long long>(blockIdx.y) * N * N;
    for (int t = threadIdx.x; t < NBT * NBT; t += PANEL_THREADS)
    {
        const int i = t / NBT, j = t % NBT;
        const T v = A[static_cast<long long>(k0 + i) * N + k0 + j];
        D[i][j] = j < i ? v : czero<T>();
        if (j == i) invd[i] = 1.0 / cre(v);
    }
    __syncthreads();
    const int lane = threadIdx.x % 32, s = lane % 4;
    const int r = k0 + NBT + static_cast<int>(blockIdx.x) * PANEL_ROWS + static_cast<int>(threadIdx.x) / 4;
    if (r - lane / 4 >= N) return;  // the whole warp: its rows lie below the matrix
    T *row = A + static_cast<long long>(min(r, N - 1)) * N + k0;
    T x[KC];
#pragma unroll
    for (int k = 0; k < KC; ++k) x[k] = row[4 * k + s];
#pragma unroll
    for (int kp = 0; kp < KC; ++kp)
#pragma unroll
        for (int sp = 0; sp < 4; ++sp)
        {
            const int p = 4 * kp + sp;
            if (s == sp) x[kp] = cscale(x[kp], invd[p]);
            const T xp = cshfl(x[kp], (lane & ~3) | sp);
#pragma unroll
            for (int k = kp; k < KC; ++k) x[k] = cfms_conj(x[k], xp, D[4 * k + s][p]);
        }
    if (r >= N) return;
#pragma unroll
    for (int k = 0; k < KC; ++k) row[4 * k + s] = x[k];
}


// Trailing update of the lower triangle, 32 x 32 tiles (ti >= tj), K = panel width.
template <typename T>
__global__ void __launch_bounds__(256) k_chol_update(T *__restrict__ Aall, int N, int k0, int ntile)
{
    __shared__ T Pi[32][NB + 1];
    __shared__ T Pj[32][NB + 1];
    const int b = blockIdx.y;
    T *A = Aall + static_cast<long long>(b) * N * N;
    const int nb = min(NB, N - k0);
    const int s0 = k0 + nb;
    // blockIdx.x enumerates lower-triangular tile pairs (ti >= tj)
    int t = blockIdx.x, ti = 0;
    while (t > ti)
    {
        t -= ti + 1;
        ++ti;
    }
    const int tj = t;
    if (ti >= ntile) return;
    const int i0 = s0 + ti * 32, j0 = s0 + tj * 32;
    for (int e = threadIdx.x; e < 32 * nb; e += blockDim.x)
    {
        const int r = e / nb, p = e % nb;
        Pi[r][p] = (i0 + r < N) ? A[static_cast<long long>(i0 + r) * N + k0 + p] : czero<T>();
        Pj[r][p] = (j0 + r < N) ? A[static_cast<long long>(j0 + r) * N + k0 + p] : czero<T>();
    }
    __syncthreads();
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;  // 2 x 2 outputs per thread
    T acc[2][2];
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v) acc[u][v] = czero<T>();
    for (int p = 0; p < nb; ++p)
        for (int u = 0; u < 2; ++u)
            for (int v = 0; v < 2; ++v) acc[u][v] = cconjmul_acc(acc[u][v], Pi[ty + 16 * u][p], Pj[tx + 16 * v][p]);
    for (int u = 0; u < 2; ++u)
        for (int v = 0; v < 2; ++v)
        {
            const int i = i0 + ty + 16 * u, j = j0 + tx + 16 * v;
            if (i < N && j < N && j <= i)
            {
                T &a = A[static_cast<long long>(i) * N + j];
                a = csub(a, acc[u][v]);
            }
        }
}

__global__ void k_chol_logdet(const double *__restrict__ diag, int N, double *__restrict__ logdet)
{
    __shared__ double red[256];
    const double *d = diag + static_cast<long long>(blockIdx.x) * N;
    double acc = 0.0;
    for (int i = threadIdx.x; i < N; i += blockDim.x) acc += log(d[i]);
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1)
    {
        if (threadIdx.x < s) red[threadIdx.x] += red[threadIdx.x + s];
        __syncthreads();
    }
    if (threadIdx.x == 0) logdet[blockIdx.x] = 2.0 * red[0];
}

// zero the strict upper triangle (L as a full matrix)
template <typename T>
__global__ void k_zero_upper(T *__restrict__ Aall, int N)
{
    T *A = Aall + static_cast<long long>(blockIdx.y) * N * N;
    const long long nn = static_cast<long long>(N) * N;
    for (long long e = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; e < nn;
         e += static_cast<long long>(gridDim.x) * blockDim.x)
        if (e % N > e / N) A[e] = czero<T>();
}

template <typename T>
int chol_impl(T *A, int N, int batch, double *diag, int *bad, cudaStream_t st)
{
    int launches = 0;
    for (int k0 = 0; k0 < N; k0 += NB)
    {
        const int nb = std::min(NB, N - k0);
        const int rows_below = N - k0 - nb;
        k_chol_diag<T, NB><<<batch, 256, 0, st>>>(A, N, k0, diag, bad);
        GB_LAUNCH_CHECK();
        ++launches;
        if (rows_below > 0)
        {
            // with rows below it the panel is a full one
            dim3 gp((rows_below + PANEL_ROWS - 1) / PANEL_ROWS, batch);
            k_chol_panel<T, NB><<<gp, PANEL_THREADS, 0, st>>>(A, N, k0);
            GB_LAUNCH_CHECK();
            const int ntile = (rows_below + 31) / 32;
            dim3 gu(ntile * (ntile + 1) / 2, batch);
            k_chol_update<T><<<gu, 256, 0, st>>>(A, N, k0, ntile);
            GB_LAUNCH_CHECK();
            launches += 2;
        }
    }
    return launches;
}

} // namespace

int chol_batched_c(cuDoubleComplex *A, int N, int batch, double *diag, int *bad, cudaStream_t st)
{
    return chol_impl(A, N, batch, diag, bad, st);
}

int chol_batched_r(double *A, int N, int batch, double *diag, int *bad, cudaStream_t st)
{
    return chol_impl(A, N, batch, diag, bad, st);
}

int chol_batched_r_ozaki(double *A, int N, int batch, double *diag, int *bad, OzakiWork &w, cudaStream_t st)
{
    constexpr int NBO = OZAKI_NB;
    int launches = 0;
    for (int k0 = 0; k0 < N; k0 += NBO)
    {
        const int nb = std::min(NBO, N - k0);
        const int rows_below = N - k0 - nb;
        if (rows_below == 0)
        {
            k_chol_diag64<false><<<batch, DIAG_THREADS, 0, st>>>(A, N, k0, diag, bad, nullptr);
            GB_LAUNCH_CHECK();
            ++launches;
            continue;
        }
        // every panel with rows below it is a full 64-wide one (panels step by 64)
        k_chol_diag64<true><<<batch, DIAG_THREADS, 0, st>>>(A, N, k0, diag, bad, w.winv);
        GB_LAUNCH_CHECK();
        launches += 1 + ozaki_panel_solve(A, N, batch, k0, w, st);
        launches += ozaki_trailing_update(A, N, batch, k0 + nb, k0, nb, w, st);
    }
    return launches;
}

void chol_logdet(const double *diag, int N, int batch, double *logdet, cudaStream_t st)
{
    k_chol_logdet<<<batch, 256, 0, st>>>(diag, N, logdet);
    GB_LAUNCH_CHECK();
}

void zero_upper_c(cuDoubleComplex *A, int N, int batch, cudaStream_t st)
{
    dim3 g(std::min(1024, (N * N + 255) / 256), batch);
    k_zero_upper<cuDoubleComplex><<<g, 256, 0, st>>>(A, N);
    GB_LAUNCH_CHECK();
}

void zero_upper_r(double *A, int N, int batch, cudaStream_t st)
{
    dim3 g(std::min(1024, (N * N + 255) / 256), batch);
    k_zero_upper<double><<<g, 256, 0, st>>>(A, N);
    GB_LAUNCH_CHECK();
}

} // namespace gb
