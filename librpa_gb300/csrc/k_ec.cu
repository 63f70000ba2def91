// E_c stage kernels: full-matrix assembly from upper atom blocks, trace and
// I - Pi, and an FP64 LU with partial pivoting returning sum log(+-u_ii).
//
// Follows LibRPA's E_c (src/core/epsilon.cpp:270-558 for k points, :43-268 for
// Gamma only): lower blocks are conj-transposes of the upper ones
// (utils_matrix_m_mpi.h:393-455), Pi = V chi0, tr Pi, M = I - Pi, LU, and
// ln det = sum_i log(u_ii) if Re u_ii > 0 else log(-u_ii) (epsilon.cpp:578-592, :640-671).
// Pivot choice follows LAPACK's i*amax: largest |Re|+|Im| (|x| for real), first index on ties.
#include <algorithm>
#include <cmath>
#include <cstdint>
#include <vector>

#include <cooperative_groups.h>

#include "kernels.h"
#include "common.h"

namespace gb {

namespace {

__device__ inline double mag1(double x) { return fabs(x); }
__device__ inline double mag1(cuDoubleComplex x) { return fabs(x.x) + fabs(x.y); }

// out[s][r][c]; row r in atom A (local a), col c in atom B (local b)
__global__ void k_assemble_chi0(const cuDoubleComplex *__restrict__ src, long long slab_stride, int N,
                                const int *__restrict__ atom_of, const int *__restrict__ abf_off,
                                const int *__restrict__ nabf, const int *__restrict__ pair_of, int n_at,
                                const long long *__restrict__ e_off, bool real_only,
                                cuDoubleComplex *__restrict__ outc, double *__restrict__ outr,
                                long long out_stride)
{
    const long long nn = static_cast<long long>(N) * N;
    const int s = blockIdx.y;
    for (long long idx = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; idx < nn;
         idx += static_cast<long long>(gridDim.x) * blockDim.x)
    {
        const int r = static_cast<int>(idx / N), c = static_cast<int>(idx % N);
        const int A = atom_of[r], B = atom_of[c];
        const int a = r - abf_off[A], b = c - abf_off[B];
        const cuDoubleComplex *sl = src + s * slab_stride;
        cuDoubleComplex v;
        if (A <= B)
        {
            const int p = pair_of[A * n_at + B];
            v = sl[e_off[p] + static_cast<long long>(a) * nabf[B] + b];
        }
        else
        {
            const int p = pair_of[B * n_at + A];
            v = sl[e_off[p] + static_cast<long long>(b) * nabf[A] + a];
            v.y = -v.y;
        }
        if (real_only)
            outr[s * out_stride + idx] = v.x;
        else
            outc[s * out_stride + idx] = v;
    }
}

// blk_IJ[2b] = (I, J) with I <= J; block b is nabf[I] x nabf[J] at blob[blk_off[b]]
__global__ void k_assemble_v(const cuDoubleComplex *__restrict__ blob, const long long *__restrict__ blk_off,
                             const int *__restrict__ blk_IJ, const int *__restrict__ abf_off,
                             const int *__restrict__ nabf, int N, bool real_only,
                             cuDoubleComplex *__restrict__ outc, double *__restrict__ outr)
{
    const int b = blockIdx.x;
    const int I = blk_IJ[2 * b], J = blk_IJ[2 * b + 1];
    const int nI = nabf[I], nJ = nabf[J];
    const cuDoubleComplex *src = blob + blk_off[b];
    for (int t = threadIdx.x; t < nI * nJ; t += blockDim.x)
    {
        const int mu = t / nJ, nu = t % nJ;
        const long long r = abf_off[I] + mu, c = abf_off[J] + nu;
        const cuDoubleComplex v = src[t];
        if (real_only)
        {
            outr[r * N + c] = v.x;
            if (I != J) outr[c * N + r] = v.x;
        }
        else
        {
            outc[r * N + c] = v;
            if (I != J) outc[c * N + r] = make_cuDoubleComplex(v.x, -v.y);
        }
    }
}

template <typename T>
__device__ inline T tzero();
template <>
__device__ inline double tzero<double>() { return 0.0; }
template <>
__device__ inline cuDoubleComplex tzero<cuDoubleComplex>() { return make_cuDoubleComplex(0, 0); }

__device__ inline double tadd(double a, double b) { return a + b; }
__device__ inline cuDoubleComplex tadd(cuDoubleComplex a, cuDoubleComplex b) { return cuCadd(a, b); }
__device__ inline double tneg_one_plus(double a, bool diag) { return (diag ? 1.0 : 0.0) - a; }
__device__ inline cuDoubleComplex tneg_one_plus(cuDoubleComplex a, bool diag)
{
    return make_cuDoubleComplex((diag ? 1.0 : 0.0) - a.x, -a.y);
}

template <typename T>
__global__ void k_trace_negate(T *__restrict__ P, int N, T *__restrict__ trace)
{
    T *M = P + static_cast<long long>(blockIdx.x) * N * N;
    __shared__ T red[256];
    T acc = tzero<T>();
    for (int i = threadIdx.x; i < N; i += blockDim.x) acc = tadd(acc, M[static_cast<long long>(i) * N + i]);
    red[threadIdx.x] = acc;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1)
    {
        if (threadIdx.x < s) red[threadIdx.x] = tadd(red[threadIdx.x], red[threadIdx.x + s]);
        __syncthreads();
    }
    if (threadIdx.x == 0) trace[blockIdx.x] = red[0];
    const long long nn = static_cast<long long>(N) * N;
    for (long long idx = threadIdx.x; idx < nn; idx += blockDim.x)
    {
        const bool d = (idx / N) == (idx % N);
        M[idx] = tneg_one_plus(M[idx], d);
    }
}

__device__ inline double tdiv(double a, double b) { return a / b; }
__device__ inline cuDoubleComplex tdiv(cuDoubleComplex a, cuDoubleComplex b) { return cuCdiv(a, b); }
__device__ inline double tfms(double c, double a, double b) { return fma(-a, b, c); }
__device__ inline cuDoubleComplex tfms(cuDoubleComplex c, cuDoubleComplex a, cuDoubleComplex b)
{
    return cuCsub(c, cuCmul(a, b));
}
__device__ inline double tlogpm(double u) { return log(u > 0 ? u : -u); }
__device__ inline cuDoubleComplex tlogpm(cuDoubleComplex u)
{
    if (!(u.x > 0)) u = make_cuDoubleComplex(-u.x, -u.y);
    return make_cuDoubleComplex(log(cuCabs(u)), atan2(u.y, u.x));
}

// LU with partial pivoting of M (N x N, destroyed), logdet = sum of log(+-u_kk).  A cluster of CTAs per
// matrix shares the columns, 4 adjacent ones at a time in turn.  The owner of column k searches it for the
// pivot and hands the column, swapped and with the multipliers in place, to the others through distributed
// shared memory; each CTA then swaps and eliminates in its columns right of k.  STAGED: a CTA's columns stay
// in its shared memory, else in M; per element the operations are the same either way, in the same order.
// The bound is the FP64 pipe, 1.68 FMAs per clock per SM, and below N ~ 100 the latency of a step (pivot
// search, division, hand-over, a thin update).  With one CTA of 1024 threads a matrix, in global memory and
// one q at a time, 16 of 152 SMs worked: 8 x 0.96 ms for 8 q of 16 complex 80 x 80 matrices; now 0.48 ms
// for the 128 together, on two CTAs each.
constexpr int LU_THREADS = 256, LU_CL_MAX = 8, LU_SMEM_MAX = 200 * 1024;

template <typename T, bool STAGED>
__global__ void __launch_bounds__(LU_THREADS) k_lu_logdet(T *__restrict__ Mall, int N, T *__restrict__ logdet)
{
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    const int CL = static_cast<int>(cl.num_blocks()), r = static_cast<int>(cl.block_rank());
    const int m = static_cast<int>(blockIdx.x) / CL;
    T *M = Mall + static_cast<long long>(m) * N * N;
    extern __shared__ __align__(16) unsigned char lu_sm[];
    T *col = reinterpret_cast<T *>(lu_sm);  // [2][N]: row k of column k, and the multipliers below it
    T *diag = col + 2 * N;                  // [N]: the pivots
    T *rowk = diag + N;                     // row k of this CTA's columns
    // local column jl is column j of M, in ascending order
    const int groups = (N + 3) / 4, mine = groups > r ? (groups - r + CL - 1) / CL : 0;
    int nl = 4 * mine;
    if (mine > 0 && (groups - 1) % CL == r) nl -= 4 * groups - N;
    const int width = 4 * ((groups + CL - 1) / CL);
    T *own = rowk + width;  // [N][width]
    auto column = [&](int jl) { return ((jl / 4) * CL + r) * 4 + jl % 4; };
    auto at = [&](int i, int jl) -> T * {
        return STAGED ? own + i * width + jl : M + static_cast<long long>(i) * N + column(jl);
    };
    if (STAGED)
        for (int t = threadIdx.x; t < N * nl; t += LU_THREADS)
        {
            const int i = t / nl, jl = t % nl;
            own[i * width + jl] = M[static_cast<long long>(i) * N + column(jl)];
        }
    cl.sync();  // every CTA runs (its shared memory may be written) and has its columns
    __shared__ unsigned long long bval[LU_THREADS / 32];
    __shared__ int bidx[LU_THREADS / 32], piv_of[2];
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    for (int k = 0; k < N; ++k)
    {
        const int buf = k & 1, gk = k / 4;
        if (gk % CL == r)
        {
            const int kl = gk / CL * 4 + k % 4;
            // pivot (largest magnitude, first index on ties; row k if no element compares)
            unsigned long long best = 0;  // magnitude_key: comparisons of doubles queue on the FP64 pipe
            int bi = N;
            for (int i = k + threadIdx.x; i < N; i += LU_THREADS)
            {
                const unsigned long long v = magnitude_key(mag1(*at(i, kl)));
                if (v > best) { best = v; bi = i; }
            }
            for (int o = 16; o > 0; o >>= 1)
            {
                const unsigned long long v = __shfl_xor_sync(0xffffffffu, best, o);
                const int vi = __shfl_xor_sync(0xffffffffu, bi, o);
                if (v > best || (v == best && vi < bi)) { best = v; bi = vi; }
            }
            if (lane == 0) { bval[warp] = best; bidx[warp] = bi; }
            __syncthreads();
            best = bval[0];
            bi = bidx[0];
            for (int q = 1; q < LU_THREADS / 32; ++q)
                if (bval[q] > best || (bval[q] == best && bidx[q] < bi)) { best = bval[q]; bi = bidx[q]; }
            if (bi >= N) bi = k;
            const T piv = *at(bi, kl);
            for (int i = k + threadIdx.x; i < N; i += LU_THREADS)
            {
                const T v = i == k ? piv : tdiv(*at(i == bi ? k : i, kl), piv);
                for (int q = 0; q < CL; ++q) cl.map_shared_rank(col, q)[buf * N + i] = v;
            }
            if (threadIdx.x < CL) cl.map_shared_rank(piv_of, threadIdx.x)[buf] = bi;
        }
        // one barrier a step: column k + 2 comes into the same buffer, after the barrier of step k + 1
        cl.sync();
        const T *ck = col + buf * N;
        const int p = piv_of[buf];
        if (threadIdx.x == 0) diag[k] = ck[k];
        const int jl0 = (gk > r ? (gk - r + CL - 1) / CL * 4 : 0) + (gk % CL == r ? k % 4 + 1 : 0);
        for (int jl = jl0 + threadIdx.x; jl < nl; jl += LU_THREADS)
        {
            T x = *at(k, jl);
            if (p != k)
            {
                const T y = *at(p, jl);
                *at(p, jl) = x;
                x = y;
            }
            rowk[jl] = x;
        }
        __syncthreads();
        const int na = nl - jl0, nrow = N - k - 1;
        if (na > 0)
            for (int t = threadIdx.x; t < nrow * na; t += LU_THREADS)
            {
                const int i = k + 1 + t / na, jl = jl0 + t % na;
                T *e = at(i, jl);
                *e = tfms(*e, ck[i], rowk[jl]);
            }
        __syncthreads();
    }
    if (r == 0)
    {
        for (int i = threadIdx.x; i < N; i += LU_THREADS) diag[i] = tlogpm(diag[i]);
        __syncthreads();
        if (threadIdx.x == 0)
        {
            T ld = tzero<T>();
            for (int i = 0; i < N; ++i) ld = tadd(ld, diag[i]);
            logdet[m] = ld;
        }
    }
    cl.sync();  // no CTA leaves while another may still write into it
}

// The hand-over buffers no longer fit the shared memory: one CTA a matrix, in global memory throughout.
constexpr int LU_WIDE_THREADS = 1024;

template <typename T>
__global__ void __launch_bounds__(LU_WIDE_THREADS) k_lu_logdet_wide(T *__restrict__ Mall, int N, T *__restrict__ logdet)
{
    T *M = Mall + static_cast<long long>(blockIdx.x) * N * N;
    __shared__ double bval[LU_WIDE_THREADS / 32];
    __shared__ int bidx[LU_WIDE_THREADS / 32];
    __shared__ int piv_s;
    T ld = tzero<T>();
    const int lane = threadIdx.x % 32, warp = threadIdx.x / 32;
    for (int k = 0; k < N; ++k)
    {
        // pivot search (largest magnitude, first index on ties)
        double best = -1.0;
        int bi = N;
        for (int r = k + threadIdx.x; r < N; r += blockDim.x)
        {
            const double m = mag1(M[static_cast<long long>(r) * N + k]);
            if (m > best) { best = m; bi = r; }
        }
        for (int off = 16; off > 0; off >>= 1)
        {
            const double ob = __shfl_down_sync(0xffffffffu, best, off);
            const int oi = __shfl_down_sync(0xffffffffu, bi, off);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if (lane == 0) { bval[warp] = best; bidx[warp] = bi; }
        __syncthreads();
        if (warp == 0)
        {
            best = lane < LU_WIDE_THREADS / 32 ? bval[lane] : -1.0;
            bi = lane < LU_WIDE_THREADS / 32 ? bidx[lane] : N;
            for (int off = 16; off > 0; off >>= 1)
            {
                const double ob = __shfl_down_sync(0xffffffffu, best, off);
                const int oi = __shfl_down_sync(0xffffffffu, bi, off);
                if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
            }
            if (lane == 0) piv_s = bi;
        }
        __syncthreads();
        const int p = piv_s;
        if (p != k && p < N)
            for (int c = k + threadIdx.x; c < N; c += blockDim.x)
            {
                const T t = M[static_cast<long long>(k) * N + c];
                M[static_cast<long long>(k) * N + c] = M[static_cast<long long>(p) * N + c];
                M[static_cast<long long>(p) * N + c] = t;
            }
        __syncthreads();
        const T piv = M[static_cast<long long>(k) * N + k];
        if (threadIdx.x == 0) ld = tadd(ld, tlogpm(piv));
        for (int r = k + 1 + threadIdx.x; r < N; r += blockDim.x)
            M[static_cast<long long>(r) * N + k] = tdiv(M[static_cast<long long>(r) * N + k], piv);
        __syncthreads();
        const int m = N - k - 1;
        const long long nupd = static_cast<long long>(m) * m;
        for (long long t = threadIdx.x; t < nupd; t += blockDim.x)
        {
            const int r = k + 1 + static_cast<int>(t / m), c = k + 1 + static_cast<int>(t % m);
            M[static_cast<long long>(r) * N + c] =
                tfms(M[static_cast<long long>(r) * N + c], M[static_cast<long long>(r) * N + k],
                     M[static_cast<long long>(k) * N + c]);
        }
        __syncthreads();
    }
    if (threadIdx.x == 0) logdet[blockIdx.x] = ld;
}

template <typename T>
void lu_logdet_wide(T *M, int N, int batch, T *logdet, cudaStream_t st)
{
    k_lu_logdet_wide<T><<<batch, LU_WIDE_THREADS, 0, st>>>(M, N, logdet);
    GB_LAUNCH_CHECK();
}

template <typename T>
void lu_logdet(T *M, int N, int batch, T *logdet, cudaStream_t st)
{
    // as many CTAs a matrix as keep all matrices resident together (two CTAs an SM), 8 for a few
    int cl = LU_CL_MAX;
    while (cl > 1 && batch * cl > 2 * 152) cl /= 2;
    const auto bytes = [&](bool staged) {
        const size_t width = 4 * static_cast<size_t>(((N + 3) / 4 + cl - 1) / cl);
        return sizeof(T) * (3 * static_cast<size_t>(N) + width + (staged ? N * width : 0));
    };
    if (bytes(false) > LU_SMEM_MAX)
    {
        lu_logdet_wide(M, N, batch, logdet, st);
        return;
    }
    static PerDeviceOnce attr;
    attr.run([] {
        GB_CUDA(cudaFuncSetAttribute(k_lu_logdet<T, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, LU_SMEM_MAX));
        GB_CUDA(cudaFuncSetAttribute(k_lu_logdet<T, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, LU_SMEM_MAX));
    });
    const bool staged = bytes(true) <= LU_SMEM_MAX;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(batch) * cl);
    cfg.blockDim = dim3(LU_THREADS);
    cfg.dynamicSmemBytes = bytes(staged);
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cl;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    GB_CUDA(cudaLaunchKernelEx(&cfg, staged ? k_lu_logdet<T, true> : k_lu_logdet<T, false>, M, N, logdet));
}

template <typename T>
double lu_compare(const std::vector<double> &h, int N, int batch, cudaStream_t st)
{
    constexpr int comp = sizeof(T) / sizeof(double);
    DevBuf<double> a(h.size()), b(h.size()), la(comp * batch), lb(comp * batch);
    a.upload(h.data(), h.size(), st);
    b.upload(h.data(), h.size(), st);
    lu_logdet(reinterpret_cast<T *>(a.get()), N, batch, reinterpret_cast<T *>(la.get()), st);
    lu_logdet_wide(reinterpret_cast<T *>(b.get()), N, batch, reinterpret_cast<T *>(lb.get()), st);
    std::vector<double> ha(comp * batch), hb(comp * batch);
    la.download(ha.data(), ha.size(), st);
    lb.download(hb.data(), hb.size(), st);
    GB_CUDA(cudaStreamSynchronize(st));
    double worst = 0.0;
    for (size_t i = 0; i < ha.size(); ++i)
    {
        if (ha[i] == hb[i] || (std::isnan(ha[i]) && std::isnan(hb[i]))) continue;
        const double d = std::fabs(ha[i] - hb[i]);
        worst = std::isnan(d) ? INFINITY : std::max(worst, d);
    }
    return worst;
}

} // namespace

double lu_selftest(int N, int batch, bool is_complex, int kind, int seed)
{
    cudaStream_t st;
    GB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    uint64_t x = 0x9E3779B97F4A7C15ull * (static_cast<uint64_t>(seed) + 1);
    std::vector<double> h(static_cast<size_t>(N) * N * batch * (is_complex ? 2 : 1));
    for (double &v : h)
    {
        x ^= x << 13;
        x ^= x >> 7;
        x ^= x << 17;
        v = static_cast<double>(x >> 11) / 9007199254740992.0 * 2.0 - 1.0;
        if (kind == 1) v = std::nearbyint(v * 1.4);
    }
    if (kind == 2) h[h.size() / 2] = std::nan("");
    const double d = is_complex ? lu_compare<cuDoubleComplex>(h, N, batch, st) : lu_compare<double>(h, N, batch, st);
    GB_CUDA(cudaStreamDestroy(st));
    return d;
}

void launch_assemble_chi0(const cuDoubleComplex *src, long long slab_stride, int n_slabs, int N,
                          const int *atom_of, const int *abf_off, const int *nabf, const int *pair_of,
                          int n_at, const long long *e_off, bool real_only, cuDoubleComplex *outc,
                          double *outr, long long out_stride, cudaStream_t st)
{
    const long long nn = static_cast<long long>(N) * N;
    dim3 grid(static_cast<unsigned>(std::min<long long>((nn + 255) / 256, 65535)), n_slabs);
    k_assemble_chi0<<<grid, 256, 0, st>>>(src, slab_stride, N, atom_of, abf_off, nabf, pair_of, n_at, e_off,
                                          real_only, outc, outr, out_stride);
    GB_LAUNCH_CHECK();
}

// The inverse of k_assemble_chi0 on the upper atom pairs: out[s][e_off[p] + a nabf[J] + b] =
// dense[s][(abf_off[I] + a) N + abf_off[J] + b] for pair p = (I, J), a < nabf[I], b < nabf[J].
__global__ void k_scatter_pairs(const cuDoubleComplex *__restrict__ dense, long long dense_stride, int N,
                                const int *__restrict__ pI, const int *__restrict__ pJ, int n_pairs,
                                const int *__restrict__ abf_off, const int *__restrict__ nabf,
                                const long long *__restrict__ e_off, cuDoubleComplex *__restrict__ out,
                                long long slab_stride)
{
    const int s = blockIdx.z;
    for (int p = blockIdx.y; p < n_pairs; p += gridDim.y)
    {
        const int I = pI[p], J = pJ[p], nJ = nabf[J];
        const long long nel = static_cast<long long>(nabf[I]) * nJ;
        const cuDoubleComplex *src = dense + s * dense_stride;
        cuDoubleComplex *dst = out + s * slab_stride + e_off[p];
        for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < nel;
             t += static_cast<long long>(gridDim.x) * blockDim.x)
        {
            const int a = static_cast<int>(t / nJ), b = static_cast<int>(t % nJ);
            dst[t] = src[static_cast<long long>(abf_off[I] + a) * N + abf_off[J] + b];
        }
    }
}

void launch_scatter_pairs(const cuDoubleComplex *dense, long long dense_stride, int n_slabs, int N, const int *pI,
                          const int *pJ, int n_pairs, const int *abf_off, const int *nabf, const long long *e_off,
                          cuDoubleComplex *out, long long slab_stride, cudaStream_t st)
{
    if (n_pairs == 0 || n_slabs == 0) return;
    GB_REQUIRE(n_slabs <= 65535, "too many slabs for one scatter launch");
    const dim3 grid(8, std::min(n_pairs, 65535), n_slabs);
    k_scatter_pairs<<<grid, 256, 0, st>>>(dense, dense_stride, N, pI, pJ, n_pairs, abf_off, nabf, e_off, out,
                                          slab_stride);
    GB_LAUNCH_CHECK();
}

void launch_assemble_v(const cuDoubleComplex *blob, const long long *blk_off, const int *blk_IJ,
                       int n_blocks, const int *abf_off, const int *nabf, int N, bool real_only,
                       cuDoubleComplex *outc, double *outr, cudaStream_t st)
{
    if (n_blocks == 0) return;
    k_assemble_v<<<n_blocks, 256, 0, st>>>(blob, blk_off, blk_IJ, abf_off, nabf, N, real_only, outc, outr);
    GB_LAUNCH_CHECK();
}

void launch_trace_and_negate_c(cuDoubleComplex *P, int N, int batch, cuDoubleComplex *trace, cudaStream_t st)
{
    k_trace_negate<cuDoubleComplex><<<batch, 256, 0, st>>>(P, N, trace);
    GB_LAUNCH_CHECK();
}

void launch_trace_and_negate_r(double *P, int N, int batch, double *trace, cudaStream_t st)
{
    k_trace_negate<double><<<batch, 256, 0, st>>>(P, N, trace);
    GB_LAUNCH_CHECK();
}

void launch_lu_logdet_c(cuDoubleComplex *M, int N, int batch, cuDoubleComplex *logdet, cudaStream_t st)
{
    lu_logdet(M, N, batch, logdet, st);
}

void launch_lu_logdet_r(double *M, int N, int batch, double *logdet, cudaStream_t st)
{
    lu_logdet(M, N, batch, logdet, st);
}

} // namespace gb
