// chi0(R, tau) atom-pair blocks on CUDA cores (FP64 plain path, FP32 variant).
//
// LibRI computes chi0s as two cal_loop3 passes (RPA.hpp:104-137) with labels
// a1b1_a2b2 and a1b2_a2b1 (LRI-cal_loop3.hpp:902-1032).  With the
// supercell products  X_b^I[mu i; (cL,L) l] = sum_{(cK,K) k} C^I[mu i; (cK,K) k] G_b[K;L,RL-RK]_{kl}
// (computed by a GEMM before this kernel) the two labels of one pass (Ga, Gb) are
//   T1[mu,nu] = sum_{i,j} Ga[I;J,RJ]_{ij} sum_{(cL,L) l} X_b^I[mu i;(cL,L) l] C^J[nu j;(L, RL-RJ) l]
//   T2[mu,nu] = sum_{i,j} X_b^I[mu i;(cJ,J) j] X_a^J[nu j;(c(-RJ),I) i]
// T2 uses Re G[I;L,R]_{il} = Re G[L;I,-R]_{li}, which the G builder satisfies exactly up to rounding.
// The passes are (Ga,Gb) = (G+,G-) and (G-,G+).  Only upper pairs I<=J are formed:
// they are the only blocks the R->q transform reads (chi0.cpp:521-534).
//
// Both passes share C^J, so E = sum_pass Ga^T X_b is summed first and contracted once.  One CTA owns a
// 48 x 16 RN (mu, nu) tile of one (pair, cell) block and a part of the supercell orbital axis, which it
// walks LC columns at a time, forming E on the fly; the parts of a tile are a thread-block cluster, whose
// first CTA sums their tiles in order through distributed shared memory (the result does not depend on
// the schedule).  Without the parts a 2-atom cell on 2x2x2 k ran on 24 of 152 SMs.
//
// Bound: FP64, its pipe (1.68 FMAs per clock per SM); FP32, the steps' latency in small cells and
// shared-memory loads in large ones, which is why every operand is read as 4 columns at once.  One GB300,
// per (tau, spin): FP64, 2 atoms of 13/40 on 2x2x2 k 4.67 -> 0.91 ms; FP32, 6 atoms of 36/140 and 13/60
// 4.76 -> 0.75 ms.
#include <cooperative_groups.h>

#include <algorithm>

#include "kernels.h"
#include "common.h"

namespace gb {

namespace {

namespace cg = cooperative_groups;

constexpr int TT = 48;   // mu tile
constexpr int LC = 4;    // supercell columns per K step

__device__ __forceinline__ void load4(const float *p, float (&v)[4])
{
    const float4 x = *reinterpret_cast<const float4 *>(p);
    v[0] = x.x, v[1] = x.y, v[2] = x.z, v[3] = x.w;
}
__device__ __forceinline__ void load4(const double *p, double (&v)[4])
{
    const double2 x = reinterpret_cast<const double2 *>(p)[0], y = reinterpret_cast<const double2 *>(p)[1];
    v[0] = x.x, v[1] = x.y, v[2] = y.x, v[3] = y.y;
}

__device__ __forceinline__ void store4(float *p, const float (&v)[4]) { *reinterpret_cast<float4 *>(p) = make_float4(v[0], v[1], v[2], v[3]); }
__device__ __forceinline__ void store4(double *p, const double (&v)[4])
{
    reinterpret_cast<double2 *>(p)[0] = make_double2(v[0], v[1]);
    reinterpret_cast<double2 *>(p)[1] = make_double2(v[2], v[3]);
}

// Shared memory in elements: [Xs | Es | Cs] of [rows][mp][LC] (mp odd: rows of a warp on different banks;
// rows past the tile's hold nothing, and reach only outputs that are not written),
// then both passes' G as [2][max_nao][mq] where it fits, else G is read from global memory.
struct SimtShape
{
    int mp, mq, tn;
    size_t tiles, gs;  // elements of the three operand tiles, of G
};

template <typename T>
SimtShape simt_shape(const Geom &g, int rn)
{
    SimtShape s;
    s.mp = g.max_nao | 1;
    s.mq = (g.max_nao + 3) / 4 * 4;
    s.tn = 16 * rn;
    // the cluster's sum reuses the operand tiles for [TT][tn]
    s.tiles = std::max<size_t>((2ull * TT + s.tn) * s.mp * LC, static_cast<size_t>(TT) * s.tn);
    s.gs = 2ull * g.max_nao * s.mq;
    return s;
}

template <typename T, int RN>
__global__ void __launch_bounds__(256) k_chi0_simt(const T *__restrict__ Xp, const T *__restrict__ Xm,
                                                   const T *__restrict__ Cm, const T *__restrict__ Gp,
                                                   const T *__restrict__ Gm, Geom g, Pairs pr, SimtShape sh,
                                                   int nsplit, int g_smem, double *__restrict__ out)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T *sm = reinterpret_cast<T *>(smem_raw);
    const int MP = sh.mp, MQ = sh.mq;
    constexpr int TN = 16 * RN;
    T *Xs = sm;                        // [TT][MP][LC]
    T *Es = Xs + TT * MP * LC;         // [TT][MP][LC]
    T *Cs = Es + TT * MP * LC;         // [TN][MP][LC]
    T *gs = sm + sh.tiles;             // [2][max_nao][MQ]

    const int p = blockIdx.x / g.n_c;
    const int cJ = blockIdx.x % g.n_c;
    const int I = pr.I[p], J = pr.J[p];
    const int aI = g.nao[I], aJ = g.nao[J];
    const int bI = g.nabf[I], bJ = g.nabf[J];
    const int part = blockIdx.z % nsplit;
    const int mu0 = blockIdx.y * TT, nu0 = static_cast<int>(blockIdx.z) / nsplit * TN;
    if (mu0 >= bI || nu0 >= bJ) return;  // every CTA of the cluster
    const int mt = min(TT, bI - mu0), nt = min(TN, bJ - nu0);
    const long long nsup = g.n_sup;
    const long long rI = g.rowc_off[I], rJ = g.rowc_off[J];
    const int tx = threadIdx.x % 16, ty = threadIdx.x / 16;
    const int *cd = g.cdiff;
    const int nc = g.n_c, nao = g.n_ao;
    auto g_at = [&](int pass, int i, int j) -> T {
        return (pass == 0 ? Gp : Gm)[(static_cast<size_t>(cJ) * nao + g.ao_off[I] + i) * nao + g.ao_off[J] + j];
    };
    if (g_smem)
        for (int t = threadIdx.x; t < 2 * aI * MQ; t += 256)
        {
            const int j = t % MQ, i = t / MQ % aI, pass = t / (MQ * aI);
            gs[(pass * g.max_nao + i) * MQ + j] = j < aJ ? g_at(pass, i, j) : T(0);
        }

    T acc[3][RN];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = 0; b < RN; ++b) acc[a][b] = T(0);
    // acc[mu][nu] += sum_j sum_lc A[mu][j][lc] Cs[nu][j][lc]; a warp's rows beyond the tile are skipped
    auto contract = [&](const T *A) {
        for (int j = 0; j < aJ; ++j)
        {
            T cv[RN][LC];
#pragma unroll
            for (int b = 0; b < RN; ++b) load4(Cs + ((tx + 16 * b) * MP + j) * LC, cv[b]);
#pragma unroll
            for (int a = 0; a < 3; ++a)
            {
                if ((ty & ~1) + 16 * a >= mt) continue;
                T ev[LC];
                load4(A + ((ty + 16 * a) * MP + j) * LC, ev);
#pragma unroll
                for (int b = 0; b < RN; ++b)
#pragma unroll
                    for (int l = 0; l < LC; ++l) acc[a][b] += ev[l] * cv[b][l];
            }
        }
    };

    // ---- T1 over this part's columns
    const int nq = (aJ + 3) / 4;
    const long long steps = (nsup + LC - 1) / LC, s0 = steps * part / nsplit, s1 = steps * (part + 1) / nsplit;
    for (long long st = s0; st < s1; ++st)
    {
        const long long l0 = st * LC;
        for (int pass = 0; pass < 2; ++pass)
        {
            const T *Xb = pass == 0 ? Xm : Xp;
            __syncthreads();
            // a row (mu, i) or (nu, j) per thread at a time: its 4 columns are 4 independent loads
#pragma unroll 4
            for (int t = threadIdx.x; t < mt * aI; t += 256)
            {
                const T *src = Xb + (rI + static_cast<long long>(mu0) * aI + t) * nsup + l0;
                const int m = t / aI, i = t - m * aI;
                T v[LC];
#pragma unroll
                for (int l = 0; l < LC; ++l) v[l] = l0 + l < nsup ? src[l] : T(0);
                store4(Xs + (m * MP + i) * LC, v);
            }
            if (pass == 0)
            {
                long long cp[LC];
#pragma unroll
                for (int l = 0; l < LC; ++l)
                {
                    const long long col = l0 + l;
                    const int cL = static_cast<int>(min(col, nsup - 1) / nao);
                    cp[l] = col < nsup ? static_cast<long long>(cd[cL * nc + cJ]) * nao + (col - static_cast<long long>(cL) * nao) : -1;
                }
#pragma unroll 4
                for (int t = threadIdx.x; t < nt * aJ; t += 256)
                {
                    const T *src = Cm + (rJ + static_cast<long long>(nu0) * aJ + t) * nsup;
                    const int n = t / aJ, j = t - n * aJ;
                    T v[LC];
#pragma unroll
                    for (int l = 0; l < LC; ++l) v[l] = cp[l] >= 0 ? src[cp[l]] : T(0);
                    store4(Cs + (n * MP + j) * LC, v);
                }
            }
            __syncthreads();
            // E[m][4 j][lc] (+)= sum_i g[i][4 j] X[m][i][lc]
            for (int t = threadIdx.x; t < mt * nq; t += 256)
            {
                const int m = t / nq, j0 = t % nq * 4;
                T e[4][LC];
#pragma unroll
                for (int j = 0; j < 4; ++j)
#pragma unroll
                    for (int l = 0; l < LC; ++l) e[j][l] = T(0);
                for (int i = 0; i < aI; ++i)
                {
                    T x[LC], gv[4];
                    load4(Xs + (m * MP + i) * LC, x);
                    if (g_smem)
                        load4(gs + (pass * g.max_nao + i) * MQ + j0, gv);
                    else
#pragma unroll
                        for (int j = 0; j < 4; ++j) gv[j] = j0 + j < aJ ? g_at(pass, i, j0 + j) : T(0);
#pragma unroll
                    for (int j = 0; j < 4; ++j)
#pragma unroll
                        for (int l = 0; l < LC; ++l) e[j][l] += gv[j] * x[l];
                }
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    if (j0 + j < aJ)
                    {
                        T *d = Es + (m * MP + j0 + j) * LC;
#pragma unroll
                        for (int l = 0; l < LC; ++l) d[l] = pass == 0 ? e[j][l] : d[l] + e[j][l];
                    }
            }
        }
        __syncthreads();
        contract(Es);
    }
    // ---- T2: sum_{i,j} Xb^I[mu i; (cJ,J) j] * Xa^J[nu j; (c(-RJ), I) i], 4 i at a time in place of the
    // columns, the (pass, i) blocks dealt to the parts in turn
    const long long colJ = static_cast<long long>(cJ) * nao + g.ao_off[J];
    const long long colI = static_cast<long long>(g.cneg[cJ]) * nao + g.ao_off[I];
    const int niq = (aI + LC - 1) / LC;
    for (int u = part; u < 2 * niq; u += nsplit)
    {
        const int pass = u / niq, i0 = u % niq * LC;
        const T *Xb = pass == 0 ? Xm : Xp, *Xa = pass == 0 ? Xp : Xm;
        __syncthreads();
#pragma unroll 4
        for (int t = threadIdx.x; t < mt * aJ; t += 256)
        {
            const int m = t / aJ, j = t - m * aJ;
            const T *src = Xb + (rI + static_cast<long long>(mu0 + m) * aI + i0) * nsup + colJ + j;
            T v[LC];
#pragma unroll
            for (int l = 0; l < LC; ++l) v[l] = i0 + l < aI ? src[l * nsup] : T(0);
            store4(Es + (m * MP + j) * LC, v);
        }
#pragma unroll 4
        for (int t = threadIdx.x; t < nt * aJ; t += 256)
        {
            const int n = t / aJ, j = t - n * aJ;
            const T *src = Xa + (rJ + static_cast<long long>(nu0) * aJ + t) * nsup + colI + i0;
            T v[LC];
#pragma unroll
            for (int l = 0; l < LC; ++l) v[l] = i0 + l < aI ? src[l] : T(0);
            store4(Cs + (n * MP + j) * LC, v);
        }
        __syncthreads();
        contract(Es);
    }
    double *o = out + pr.r_off[p] + static_cast<long long>(cJ) * bI * bJ;
    if (nsplit == 1)
    {
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < RN; ++b)
            {
                const int m = ty + 16 * a, n = tx + 16 * b;
                if (m < mt && n < nt) o[static_cast<long long>(mu0 + m) * bJ + nu0 + n] = static_cast<double>(acc[a][b]);
            }
        return;
    }
    cg::cluster_group cl = cg::this_cluster();
    __syncthreads();
    if (part != 0)
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < RN; ++b) sm[(ty + 16 * a) * TN + tx + 16 * b] = acc[a][b];
    cl.sync();
    if (part == 0)
#pragma unroll
        for (int a = 0; a < 3; ++a)
#pragma unroll
            for (int b = 0; b < RN; ++b)
            {
                const int m = ty + 16 * a, n = tx + 16 * b;
                if (m < mt && n < nt)
                {
                    double v = static_cast<double>(acc[a][b]);
                    for (int k = 1; k < nsplit; ++k) v += static_cast<double>(cl.map_shared_rank(sm, k)[m * TN + n]);
                    o[static_cast<long long>(mu0 + m) * bJ + nu0 + n] = v;
                }
            }
    cl.sync();  // the tiles stay until they are read
}

template <typename T, int RN>
void launch_chi0_simt_rn(const T *Xp, const T *Xm, const T *Cm, const T *Gp, const T *Gm, const Geom &g,
                         const Pairs &pr, double *out, cudaStream_t st)
{
    constexpr size_t cap = 227 * 1024;
    const SimtShape sh = simt_shape<T>(g, RN);
    const bool g_smem = sizeof(T) * (sh.tiles + sh.gs) <= cap;
    const size_t smem = sizeof(T) * (sh.tiles + (g_smem ? sh.gs : 0));
    // the cap once per device (calls of other shapes may run on other host threads)
    static PerDeviceOnce attr;
    attr.run([] {
        GB_CUDA(cudaFuncSetAttribute(k_chi0_simt<T, RN>, cudaFuncAttributeMaxDynamicSharedMemorySize, static_cast<int>(cap)));
    });
    const int tiles_mu = (g.max_nabf + TT - 1) / TT, tiles_nu = (g.max_nabf + sh.tn - 1) / sh.tn;
    // parts of the orbital axis: while the tiles leave SMs idle, up to the portable cluster size and 2
    // steps a part
    int dev = 0, n_sm = 0;
    GB_CUDA(cudaGetDevice(&dev));
    GB_CUDA(cudaDeviceGetAttribute(&n_sm, cudaDevAttrMultiProcessorCount, dev));
    const long long ctas = static_cast<long long>(pr.n_pairs) * g.n_c * tiles_mu * tiles_nu;
    const int nsplit = static_cast<int>(
        std::max<long long>(1, std::min<long long>({8, n_sm / std::max<long long>(ctas, 1), g.n_sup / (2 * LC)})));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(pr.n_pairs * g.n_c, tiles_mu, tiles_nu * nsplit);
    cfg.blockDim = dim3(256);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = nsplit;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    GB_CUDA(cudaLaunchKernelEx(&cfg, k_chi0_simt<T, RN>, Xp, Xm, Cm, Gp, Gm, g, pr, sh, nsplit, g_smem ? 1 : 0, out));
}

// nu per tile: as many as the atoms have (E is formed again for every nu tile), while the tile fits
// shared memory
template <typename T>
void launch_chi0_simt(const T *Xp, const T *Xm, const T *Cm, const T *Gp, const T *Gm, const Geom &g,
                      const Pairs &pr, double *out, cudaStream_t st)
{
    // the sizes taken: a block of G and three operand tiles of 48 rows in shared memory (46 NAOs in FP64, 87 in
    // FP32); these tiles would hold 49 and 99, at which a sum has 20 to 30% more terms
    const size_t na = g.max_nao;
    GB_REQUIRE(sizeof(T) * (na * na + 3 * TT * na * LC) <= 227 * 1024, "atom NAO count too large for the SIMT chi0 kernel");
    auto fits = [&](int rn) { return sizeof(T) * simt_shape<T>(g, rn).tiles <= 227 * 1024; };
    if (g.max_nabf > 96 && fits(9))
        launch_chi0_simt_rn<T, 9>(Xp, Xm, Cm, Gp, Gm, g, pr, out, st);
    else if (g.max_nabf > TT && fits(6))
        launch_chi0_simt_rn<T, 6>(Xp, Xm, Cm, Gp, Gm, g, pr, out, st);
    else
        launch_chi0_simt_rn<T, 3>(Xp, Xm, Cm, Gp, Gm, g, pr, out, st);
}

} // namespace

void launch_chi0_fp64(const double *Xp, const double *Xm, const double *Cm, const double *Gp,
                      const double *Gm, const Geom &g, const Pairs &pr, double *out, cudaStream_t st)
{
    launch_chi0_simt<double>(Xp, Xm, Cm, Gp, Gm, g, pr, out, st);
}

void launch_chi0_fp32(const float *Xp, const float *Xm, const float *Cm, const float *Gp,
                      const float *Gm, const Geom &g, const Pairs &pr, double *out, cudaStream_t st)
{
    launch_chi0_simt<float>(Xp, Xm, Cm, Gp, Gm, g, pr, out, st);
}

} // namespace gb
