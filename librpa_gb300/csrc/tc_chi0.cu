// Tensor-core chi0 path (BF16 split products on tcgen05, FP32 accumulation).
//
// Per (tau, spin), with the algebra of k_chi0_simt.cu:
//  1. X(+-) = C * G_super(+-): one batched split-precision GEMM (k_tc_gemm.cu); the B operand
//     G_super^T is built and split directly from G(R).
//  2. T1 (fused, this file): for each upper atom pair (I, J) and a tile of 128 rows
//     (cell cJ, mu), accumulate in TMEM
//        D[(cJ,mu)][nu] = sum_{pass} sum_{j, K'} E[(cJ,mu)][j, K'] * C^J[nu][j, K']
//        E[(cJ,mu)][j, K'] = sum_i Ga[cJ]_{ij} X_b^I[mu i][shift_cJ(K')]
//     where K' runs over the supercell orbitals (cell R', atom L, orbital l) of C^J's own
//     frame and shift_cJ maps R' -> R' + R_cJ (the T1 term with R_L = R' + R_J).
//     Eight producer warps form E in FP32 on the CUDA cores (packed FP32x2 FMAs, a row and 8 columns
//     a thread), split it into BF16 pieces and write them to TMEM, where the MMAs read A; one lane
//     streams the matching C^J tiles (64 K-elements per row, pre-arranged in HBM) with TMA and issues
//     the tcgen05.mma terms.  K order: 8-column chunk, group of 8 j.
//  3. T2 (small, CUDA cores): D += sum_{i,j} X_b^I[mu i; (cJ,J) j] X_a^J[nu j; (-cJ,I) i].
// Every wait is bounded (tc_common.cuh) and failures surface through a device error flag.
#include <cooperative_groups.h>

#include <algorithm>
#include <map>
#include <mutex>
#include <string>
#include <cstdlib>
#include <vector>

#include "../../include/librpa_gb300.h"
#include "work_schedule.h"
#include "tc_common.cuh"
#include "tc_gemm.h"

namespace gb {

namespace {

using namespace tc;

constexpr int NS = 3;            // BF16 pieces per operand (hi, mid, lo): 6 MMA terms
constexpr int T1_BM = 128;       // rows (cJ, mu) per CTA
constexpr int CW = 8;            // supercell columns per chunk: two groups of 4 columns of one cell each
constexpr int JG = 8;            // j per pipeline stage (JG * CW = 64 = K per stage)
constexpr int T1_MAXB = 8;       // C^J (B tile) ring: up to 8 stages of TMA look-ahead
constexpr int T1_NMAX = 128;     // max N tile (ABFs of one atom, padded to 16)
constexpr int T1_SET = 128;      // producer threads per warpgroup: one row each
constexpr int T1_PRODUCERS = 2 * T1_SET;           // two warpgroups, on alternate chunks
constexpr int T1_DRAIN = T1_PRODUCERS / 32;        // first of the four drain warps
constexpr int T1_ISSUE = T1_DRAIN + 4;             // one lane issues the MMAs and the C^J copies
constexpr int T1_THREADS = T1_PRODUCERS + 256;     // four warpgroups (the last one has three idle warps)
constexpr int T1_TMEM = 512;                       // TMEM columns: accumulators from 0, the A tiles at the end
constexpr int T1_ACOLS = NS * 32;                  // columns of one A tile: 3 pieces x 64 BF16 of K
constexpr int T1_ABASE = T1_TMEM - 2 * T1_ACOLS;   // one A tile per producer warpgroup
constexpr int T1_MAXA = 32;                        // max NAOs per atom
constexpr int T1_CELLS = 32;                       // cells of a row group's shift table in shared memory
constexpr int T1_INFO = 8;                         // ints kept of a row group: pair, cell, I, n_abf(I), n_ao(I)
constexpr int T1_SMEM_MAX = 227 * 1024;
constexpr long long T1_XSLAB = 2LL << 30;          // bytes of row-major X at a time; the contraction reads its re-ordered copy
// Shared memory: nbs x NS B pieces of b_tile bytes | X ring | G blocks | barriers.  b_tile = NT_max * 128
// rounded up to 1024; a G block holds, per 8 j, the 2 n_ao(I) rows q = (pass, i).

// A row group: the n_abf(I) rows mu of one chi0 block (pair (I, J), cell cJ).
struct T1Group
{
    int pair, cell;
};

// A tile: up to 128 consecutive rows of the row groups of one atom J (groups ordered by the NAO
// count of I, then by I, then cell), all contracted with the same C^J operand.
struct T1Work
{
    int J;         // atom of the B operand
    int g0;        // first row group
    int r0;        // first row inside that group
    int nrows;     // valid rows (<= 128)
    int nslot;     // row groups the tile touches
    int kc0, kc1;  // chunks [kc0, kc1) of the supercell axis this CTA contracts
    int split;     // 1: one of several K parts of the tile, added atomically to the output
    int ra;        // most NAOs of an I atom among the tile's row groups (the producers' i range)
};

constexpr int T1_MAXSPEC = 8;    // distinct (NAO, ABF) species with their own B maps
constexpr int T1_KPARTS = 4;     // default K parts per tile (each part a CTA, added into chi0(R) atomically)
constexpr int T1_KPARTS_MAX = 16; // largest K-part count the tuner tries

// C^J B-operand maps, one rank-3 map per (species, piece): dims {ktot, nabf, atoms of the species}.
struct T1Maps
{
    CUtensorMap m[T1_MAXSPEC][3];
    long long ktot[T1_MAXSPEC];
};

struct T1Args
{
    Geom g;
    Pairs pr;
    const float4 *Xt;        // X in 4-column groups (k_x_layout)
    const long long *xoff;   // [n_at] first float4 of each atom there
    const double *G;         // [2][n_c][n_ao][n_ao]
    const int *cadd;         // [n_c*n_c] cadd[a*n_c+b] = cell of R_a + R_b
    const T1Work *work;
    const T1Group *groups;
    const int *spec;           // [n_at] species of each atom
    const int *spec_idx;       // [n_at] index of the atom inside its species
    int n4;                    // 4-column groups of one cell (NAOs rounded up to 4)
    int ng4;                   // of the supercell: n_c * n4
    int b_tile;                // bytes per B piece (1024-aligned)
    int nbs;                   // stages of the B ring (2..T1_MAXB)
    int gq;                    // rows q of the G blocks' parts of 8 j
    int gslot;                 // floats per G block
    int maxcj;                 // most row groups a 128-row tile can touch
    double *out;               // chi0R
    int *err;
};

__device__ __forceinline__ void named_bar_sync(int id, int n)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory");
}

// A = E in TMEM: D(tmem) (+)= A(tmem) * B(smem desc)^T, BF16 inputs, FP32 accumulate.  Row r of A is
// TMEM lane r, each 32-bit column two consecutive K elements.
__device__ __forceinline__ void mma_bf16_ta(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                            uint32_t accumulate)
{
    asm volatile(
        "{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n" ::"r"(
            d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// 16 consecutive 32-bit columns of the warp's 32 TMEM lanes
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&r)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16};" ::"r"(taddr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]),
        "r"(r[10]), "r"(r[11]), "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15])
        : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// X reaches a producer through its own slots of a shared-memory ring, filled by 16-byte asynchronous
// copies T1_XR - 1 blocks of T1_XD rows q ahead: a register ring of that depth does not fit beside E.
constexpr int T1_XD = 4;
constexpr int T1_XR = 3;
// rows q = (pass, i) of X kept for an atom: whole blocks, the last ones zero
__host__ __device__ constexpr int t1_rows(int nao) { return (2 * nao + T1_XD - 1) / T1_XD * T1_XD; }
constexpr int T1_XBYTES = T1_XR * T1_XD * 2 * T1_PRODUCERS * 16;

__device__ __forceinline__ void cp_async16(uint32_t dst, const void *src, bool live)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait()
{
    asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// The place in X a producer's copies have reached: chunk kc, unit un of its j, row q of that unit, and
// the chunk's two 4-column groups (offset of their row 0 from the thread's row, in float4; live: inside
// the supercell and the tile's rows, else zero-filled).
struct T1Cursor
{
    int kc, un, q;
    uint32_t off[2];
    bool live[2];
};

__device__ __forceinline__ float4 lds128(uint32_t addr)
{
    float4 v;
    asm volatile("ld.shared.v4.f32 {%0, %1, %2, %3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr));
    return v;
}

// One row q: E[j][col] += G[q][j] X[q][col], columns in pairs
template <int NJ>
__device__ __forceinline__ void t1_row(uint32_t xs, uint32_t ga, uint32_t gb, float2 (&e)[NJ][CW / 2])
{
    const float4 x0 = lds128(xs), x1 = lds128(xs + T1_PRODUCERS * 16);
    const float2 xp[CW / 2] = {make_float2(x0.x, x0.y), make_float2(x0.z, x0.w), make_float2(x1.x, x1.y),
                               make_float2(x1.z, x1.w)};
#pragma unroll
    for (int jh = 0; jh < (NJ + 3) / 4; ++jh)
    {
        const float4 gg = lds128(jh < 2 ? ga + jh * 16 : gb + (jh - 2) * 16);
        const float gv[4] = {gg.x, gg.y, gg.z, gg.w};
#pragma unroll
        for (int t = 0; t < 4; ++t)
            if (4 * jh + t < NJ)
            {
                const float2 g2 = make_float2(gv[t], gv[t]);
#pragma unroll
                for (int c = 0; c < CW / 2; ++c) e[4 * jh + t][c] = __ffma2_rn(g2, xp[c], e[4 * jh + t][c]);
            }
    }
}

// One unit of a producer thread's work: its row r, one chunk of 8 columns and NJ <= JT consecutive j,
//   E[j][col] = sum_q G[q][j] X[q][col],   q = (pass, i),
// then its 3-piece BF16 split, written to the warpgroup's A tile in TMEM half a stage (4 j) at a time.
//
// Bounds: 128 FP32 FMAs per clock per SM, next to it the shared-memory
// path: a G value loaded serves the thread's 8 columns, an X value its j.  The two warpgroups work on
// alternate chunks, so that the split and the hand-over of one run under the FMAs of the other.
// Measured on one GB300 against two threads a row that wrote E to shared memory, with one drain warp
// issuing everything, the whole chi0 stage: 128 atoms of 13/40 at Gamma 426 -> 289 ms, 48 atoms of 5/20,
// 13/60 and 26/110 528 -> 112 ms, 16 atoms of 13/40 on 3x3x3 k 578 -> 399 ms.  What is left: two producer
// warps per scheduler, 46 of 128 FMAs of E per clock over the kernel (16 atoms), and 49% of the FMA pipe's
// cycles with the split and the drain (ncu, 64 atoms of 13/40 at Gamma).
template <int NJ, typename Fetch>
__device__ __forceinline__ bool t1_unit(uint32_t xring, int &slot, const Fetch &fetch, uint32_t gs,
                                        int gq, int nq, int nhalf, uint32_t atile, uint64_t *full, uint64_t *empty, uint32_t &use,
                                        int lane, int *err)
{
    constexpr uint32_t GQ = JG * 4;  // bytes of a row q of 8 G values
    float2 e[NJ][CW / 2];
#pragma unroll
    for (int j = 0; j < NJ; ++j)
#pragma unroll
        for (int c = 0; c < CW / 2; ++c) e[j][c] = make_float2(0.f, 0.f);
    uint32_t ga = gs, gb = gs + gq * GQ;  // j 0..7 and 8..15
    for (int left = nq; left > 0; left -= T1_XD)
    {
        fetch(slot);  // refills the slot read in the previous round
        cp_async_wait<T1_XR - 1>();
        uint32_t xs = xring + slot * (T1_XD * 2 * T1_PRODUCERS * 16);
        slot = slot + 1 == T1_XR ? 0 : slot + 1;
        // two rows at a time (nq is even): unrolled further, the rows' loads crowd E out of the registers
#pragma unroll 1
        for (int r = min(left, T1_XD); r > 0; r -= 2)
        {
            t1_row<NJ>(xs, ga, gb, e);
            t1_row<NJ>(xs + 2 * T1_PRODUCERS * 16, ga + GQ, gb + GQ, e);
            xs += 4 * T1_PRODUCERS * 16;
            ga += 2 * GQ;
            gb += 2 * GQ;
        }
    }
    // half stages of 4 j x 8 columns (K = 32): the split of one runs under the MMAs of the one before
#pragma unroll
    for (int hs = 0; hs < (NJ + 3) / 4; ++hs)
    {
        if (hs >= nhalf) break;  // the half stages the issue warp counts
        const int h = hs & 1;
        uint32_t wh[16], wm[16], wl[16];  // 16 TMEM columns of each piece
#pragma unroll
        for (int t = 0; t < 4; ++t)
#pragma unroll
            for (int c = 0; c < CW / 2; ++c)
            {
                const int j = hs * 4 + t;
                if (j < NJ)
                    split3_pair(e[j < NJ ? j : 0][c], wh[t * 4 + c], wm[t * 4 + c], wl[t * 4 + c]);
                else
                    wh[t * 4 + c] = wm[t * 4 + c] = wl[t * 4 + c] = 0u;
            }
        // half h of the A tile is free once the MMAs of its previous use are done
        if (!__all_sync(0xffffffffu, mbar_wait_nap<0>(empty + h, (use >> h) & 1)))
        {
            if (lane == 0) atomicExch(err, 201);
            return false;
        }
        use ^= 1u << h;
        tc_fence_after();
        tmem_st16(atile + h * 16, wh);
        tmem_st16(atile + 32 + h * 16, wm);
        tmem_st16(atile + 64 + h * 16, wl);
        tmem_wait_st();
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(full + h);
    }
    return true;
}

// NTC: accumulator columns held by the drain warps (48, 64 or 128: at least the largest N tile).
//
// Both LibRI passes share the B operand C^J, so one A tile carries E(+) + E(-) (pass 0:
// G(+) with X(-), pass 1: G(-) with X(+)) and each K step is contracted once.  Up to NTC = 64
// the three C^J pieces sit on top of each other along N and each K16 step is three MMAs,
// hi x [Ch;Cm;Cl] (N = 3 NT), mid x [Ch;Cm] (N = 2 NT) and lo x Ch (N = NT), landing in three
// accumulator blocks of orders 1, 2^-8 and 2^-16; with NTC = 128 the six products are issued
// one by one into a hi*hi block and a cross-term block.
//
// The A tile goes from the producers' registers to TMEM and is read there by the MMAs: neither the
// 48 KB a stage of E nor its re-reads by the MMAs pass through shared memory, whose bandwidth bounds
// the producers.  TMEM: 512 columns = accumulators (two buffers where they fit, else one) + two A tiles.
// The MMAs and the C^J copies are issued by a warp of their own: issued from a drain warp they cost that
// warp's loop 4900 clocks a stage, which bounded the whole contraction.
//
// Registers: a producer holds up to JT j x 8 columns of E, a drain warp NTC accumulator columns; the
// warpgroups trade registers (setmaxnreg) so that 2 PREG + DREG + CREG = 4 x 128, the launch's share.
template <int NTC>
__global__ void __launch_bounds__(T1_THREADS, 1) k_t1_tc(const __grid_constant__ T1Args a,
                                                         const __grid_constant__ T1Maps maps)
{
    constexpr bool STACKN = NTC <= 64;
    constexpr int NBLK = STACKN ? 3 : 2;           // accumulator blocks per buffer
    constexpr int JT = STACKN ? 16 : 8;            // most j per unit of the producers
    constexpr int PREG = STACKN ? 192 : 160, DREG = NTC == 48 ? 96 : NTC == 64 ? 104 : 168, CREG = NTC == 48 ? 32 : 24;
    static_assert(2 * PREG + DREG + CREG == 4 * 128, "register split of the launch's 128 a thread");
    static_assert(NBLK * NTC <= T1_ABASE, "TMEM budget");
    extern __shared__ __align__(1024) unsigned char smem_raw[];
    unsigned char *bring = reinterpret_cast<unsigned char *>((reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int bstage_bytes = NS * a.b_tile;   // B ring stage
    const int nbs = a.nbs;
    const int gq = a.gq;                      // rows q of a G block's part of 8 j
    unsigned char *xring = bring + nbs * bstage_bytes;
    float *gsm = reinterpret_cast<float *>(xring + T1_XBYTES);
    uint64_t *full = reinterpret_cast<uint64_t *>(gsm + a.maxcj * (a.gslot + T1_CELLS + T1_INFO));  // [set][half] A tile: written
    uint64_t *empty = full + 4;                                              // A tile: MMAs done
    uint64_t *bfull = empty + 4;                                             // B ring: TMA landed
    uint64_t *bempty = bfull + T1_MAXB;                                      // B ring: MMAs done
    uint64_t *accf = bempty + T1_MAXB;
    uint64_t *acce = accf + 2;
    uint64_t *fin = acce + 2;                                                // every issued MMA done
    uint32_t *tmem_slot = reinterpret_cast<uint32_t *>(fin + 1);
    volatile int *drain_stop = reinterpret_cast<volatile int *>(tmem_slot + 1);

    const Geom &g = a.g;
    const T1Work w = a.work[blockIdx.x];
    const int J = w.J;
    const int aJ = g.nao[J], bJ = g.nabf[J];
    const int njg = (aJ + JG - 1) / JG;
    const int NT = (bJ + 15) / 16 * 16;
    const int nab = 2 * NBLK * NT <= T1_ABASE ? 2 : 1;  // accumulator buffers
    const int nc = g.n_c, nao = g.n_ao;
    // the tile's row groups, read once (every later look at them would be a chain of global loads)
    int *ctab = reinterpret_cast<int *>(gsm + a.maxcj * a.gslot);  // [slot][T1_CELLS]
    int *info = ctab + a.maxcj * T1_CELLS;                         // [slot][T1_INFO]
    if (threadIdx.x < static_cast<unsigned>(w.nslot))
    {
        const T1Group gr = a.groups[w.g0 + threadIdx.x];
        const int Ig = a.pr.I[gr.pair];
        int *f = info + threadIdx.x * T1_INFO;
        f[0] = gr.pair;
        f[1] = gr.cell;
        f[2] = Ig;
        f[3] = g.nabf[Ig];
        f[4] = g.nao[Ig];
    }
    // row r of the tile -> (slot of its row group, mu); false beyond the tile's valid rows
    auto row_of = [&](int r, int &slot, int &mu) -> bool {
        slot = mu = 0;
        if (r >= w.nrows) return false;
        int off = w.r0 + r;
        for (int k = 0; k < w.nslot; ++k)
        {
            const int b = info[k * T1_INFO + 3];
            if (off < b)
            {
                slot = k;
                mu = off;
                return true;
            }
            off -= b;
        }
        return false;
    };
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int kc0 = w.kc0, kc1 = w.kc1;
    const int total_stages = (kc1 - kc0) * njg;

    if (threadIdx.x == 0)
    {
        for (int s = 0; s < 4; ++s)
        {
            mbar_init(&full[s], T1_SET / 32);  // one arrival per producer warp
            mbar_init(&empty[s], 1);
        }
        for (int s = 0; s < 2; ++s)
        {
            mbar_init(&accf[s], 1);
            mbar_init(&acce[s], 4);            // one arrival per drain warp
        }
        mbar_init(fin, 1);
        *drain_stop = 0;
        for (int s = 0; s < nbs; ++s)
        {
            mbar_init(&bfull[s], 1);
            mbar_init(&bempty[s], 1);
        }
        fence_barrier_init();
    }
    // the host reads err after the last launch: the CTAs that start after a wait was given up do nothing, where
    // each would run out its own limits
    if (warp == 0) tmem_alloc(tmem_slot, T1_TMEM);
    if (__syncthreads_or(threadIdx.x == 32 && __ldcg(a.err) != 0))
    {
        if (warp == 0) tmem_dealloc(*tmem_slot, T1_TMEM);
        return;
    }
    pdl_trigger();  // T2 may take the SMs that this launch leaves idle
    tc_fence_after();
    const uint32_t tmem = *tmem_slot;

    if (threadIdx.x < T1_PRODUCERS)
    {
        // ---------------- producers: E tiles
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(PREG));
        const int t = threadIdx.x;
        const int set = t / T1_SET;  // chunks kc0 + set, kc0 + set + 2, ...
        int gslot, mu;
        const bool valid = row_of(t % T1_SET, gslot, mu);
        const int *mine = info + gslot * T1_INFO;
        const int cJ = mine[1], I = mine[2], bI = mine[3], aI = mine[4];
        const float4 *xrow = a.Xt + a.xoff[I] + mu;
        // G blocks of the tile's row groups, [slot][j / 8][q = (pass, i)][j % 8] in FP32 (zero rows past
        // 2 a_I, zero past a_J)
        const int nq = 2 * w.ra, per = njg * nq * JG;
#pragma unroll 4
        for (int x = t; x < w.nslot * per; x += T1_PRODUCERS)
        {
            const int s = x / per, e = x - s * per;
            const int *f = info + s * T1_INFO;
            const int Ig = f[2], ag = f[4];
            const int jg = e / (nq * JG), q = e / JG % nq, j = jg * JG + e % JG;
            const int pass = q >= ag, i = pass ? q - ag : q;
            float v = 0.0f;
            if (q < 2 * ag && j < aJ)
                v = static_cast<float>(a.G[((static_cast<size_t>(pass) * nc + f[1]) * nao + g.ao_off[Ig] + i) * nao +
                                           g.ao_off[J] + j]);
            gsm[s * a.gslot + (jg * gq + q) * JG + e % JG] = v;
        }
        // cells of the shifted columns of each row group: R' + R_cJ (kept in shared memory for up to
        // T1_CELLS cells, read once per chunk)
        if (nc <= T1_CELLS)
            for (int e = t; e < w.nslot * nc; e += T1_PRODUCERS)
                ctab[e / nc * T1_CELLS + e % nc] = a.cadd[(e % nc) * nc + info[e / nc * T1_INFO + 1]];
        const int *crow = nc <= T1_CELLS ? ctab + gslot * T1_CELLS : nullptr;
        named_bar_sync(1, T1_PRODUCERS);
        const uint32_t gs = smem_u32(gsm + gslot * a.gslot);
        // units of j: all of an atom of 9 to 14 NAOs at once, 8 at a time otherwise (E of a thread's row
        // and chunk is 14 x 8 registers at most)
        const bool wide = JT == 16 && aJ > 8 && aJ <= 14;
        const int nunit = wide ? 1 : njg;
        T1Cursor cur;
        auto point_at = [&](int kc) {
            cur.kc = kc;
            cur.un = 0;
            cur.q = 0;
#pragma unroll
            for (int h = 0; h < 2; ++h)
            {
                const int g4 = 2 * kc + h;
                cur.off[h] = 0;
                cur.live[h] = valid && kc < kc1 && g4 < a.ng4;
                if (cur.live[h])
                {
                    const int cell = g4 / a.n4, c4 = g4 - cell * a.n4;
                    const int src = crow ? crow[cell] : a.cadd[cell * nc + cJ];
                    cur.off[h] = static_cast<uint32_t>(src * a.n4 + c4) * static_cast<uint32_t>(t1_rows(aI) * bI);
                }
            }
        };
        // copies the next T1_XD rows into the slot before `slot` and moves on (no copy past the last chunk)
        const uint32_t xdst = smem_u32(xring) + t * 16;
        auto fetch = [&](int slot) {
            const uint32_t dst = xdst + (slot == 0 ? T1_XR - 1 : slot - 1) * (T1_XD * 2 * T1_PRODUCERS * 16);
            if (cur.kc < kc1)
            {
#pragma unroll
                for (int h = 0; h < 2; ++h)
                {
                    const bool live = cur.live[h] && cur.q < t1_rows(aI);  // a multiple of T1_XD
                    const float4 *src = xrow + (live ? cur.off[h] + static_cast<uint32_t>(cur.q * bI) : 0u);
                    const int d = live ? bI : 0;
#pragma unroll
                    for (int u = 0; u < T1_XD; ++u) cp_async16(dst + (2 * u + h) * T1_PRODUCERS * 16, src + u * d, live);
                }
                cur.q += T1_XD;
                if (cur.q >= nq)
                {
                    cur.q = 0;
                    if (++cur.un == nunit) point_at(cur.kc + 2);
                }
            }
            cp_async_commit();
        };
        const uint32_t atile = tmem + (static_cast<uint32_t>((warp % 4) * 32) << 16) + T1_ABASE + set * T1_ACOLS;
        point_at(kc0 + set);
        for (int k = 1; k < T1_XR; ++k) fetch(k);
        int slot = 0;
        const uint32_t xown = smem_u32(xring) + t * 16;
        uint32_t use = 3u;  // bit h: phase to wait for before half h of the A tile is written again
        bool ok = true;
        for (int kc = kc0 + set; kc < kc1 && ok; kc += 2)
        {
            for (int un = 0; un < nunit && ok; ++un)
            {
                const int nj = wide ? aJ : min(JG, aJ - un * JG);
                const uint32_t gu = gs + un * (gq * JG * 4);
#define GB_T1_UNIT(NJ) \
    ok = t1_unit<NJ>(xown, slot, fetch, gu, gq, nq, (nj + 3) / 4, atile, full + 2 * set, empty + 2 * set, use, lane, a.err)
                // as many registers of E as j, by half stages of 4
                if (nj <= 2) GB_T1_UNIT(2);
                else if (nj <= 4) GB_T1_UNIT(4);
                else if (nj <= 5) GB_T1_UNIT(5);
                else if (nj <= 8) GB_T1_UNIT(8);
                else if constexpr (JT == 16)
                {
                    if (nj <= 10) GB_T1_UNIT(10);
                    else if (nj <= 12) GB_T1_UNIT(12);
                    else if (nj <= 13) GB_T1_UNIT(13);
                    else GB_T1_UNIT(14);
                }
#undef GB_T1_UNIT
            }
        }
        cp_async_wait<0>();
    }
    else if (warp >= T1_ISSUE)
    {
        // ---------------- issue warp: per stage st, the MMAs of st and the C^J copy of st + nbs - 1
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(CREG));
        if (warp == T1_ISSUE)  // the whole warp, converged: one elected lane issues
        {
            const uint32_t tm = __shfl_sync(0xffffffffu, tmem, 0);
            const uint32_t bbytes = static_cast<uint32_t>(NT) * 64 * 2;  // one piece of a B tile
            const int sp = a.spec[J], zj = a.spec_idx[J];
            const long long ktot = maps.ktot[sp];
            // C^J tiles stream through L2 once per tile: evict them first, keep the X^I rows
            const uint64_t pol_b = l2_policy_evict_first();
            int ts = 0, tph = 1, copied = 0;  // B ring: next stage to fill
            auto issue_tma = [&]() -> bool {
                if (!__all_sync(0xffffffffu, mbar_wait_nap<20>(&bempty[ts], tph)))
                {
                    if (lane == 0) atomicExch(a.err, 202);
                    return false;
                }
                const int x = (kc0 * njg + copied) * 64;  // K offset (kc * njg + jg) * 64
                if (x < 0 || static_cast<long long>(x) + 64 > ktot || (x & 7) != 0)
                {
                    if (lane == 0) atomicExch(a.err, 205);  // coordinate outside the C^J operand: skip the copy
                    return false;
                }
                unsigned char *bst = bring + ts * bstage_bytes;
                if (elect_one())
                {
                    mbar_arrive_expect_tx(&bfull[ts], NS * bbytes);
#pragma unroll
                    for (int p = 0; p < NS; ++p)  // pieces stacked along N: rows [p NT, (p + 1) NT)
                        tma_load_3d_hint(bst + p * bbytes, &maps.m[sp][p], x, 0, zj, &bfull[ts], pol_b);
                }
                __syncwarp();
                ++copied;
                if (++ts == nbs) ts = 0, tph ^= 1;
                return true;
            };
            bool ok = true;
            for (int st = 0; st < nbs - 1 && st < total_stages && ok; ++st) ok = issue_tma();
            int sb = 0, pb = 0, ab = 0, pa = 1, jg = 0, set = 0;
            uint32_t pf = 0;  // bit 2 set + half: phase of that half of the warpgroup's A tile
            const int nhalf = (aJ + 3) / 4;  // half stages of a chunk
            for (int st = 0; st < total_stages && ok; ++st)
            {
                unsigned char *bst = bring + sb * bstage_bytes;
                const uint32_t tb = tm + static_cast<uint32_t>(ab * NBLK * NT);
                const uint64_t db0 = smem_desc_sw128(bst);
                const int nh = min(2, nhalf - 2 * jg);
                for (int h = 0; h < nh && ok; ++h)
                {
                    const int fb = 2 * set + h;
                    if (!__all_sync(0xffffffffu, mbar_wait_nap<50>(&full[fb], (pf >> fb) & 1) &&
                                                     (h != 0 || (mbar_wait_nap<20>(&bfull[sb], pb) &&
                                                                 mbar_wait_nap<20>(&acce[ab], pa)))))
                    {
                        if (lane == 0) atomicExch(a.err, 203);
                        ok = false;
                        break;
                    }
                    pf ^= 1u << fb;
                    tc_fence_after();
                    const uint32_t ta = tm + T1_ABASE + set * T1_ACOLS + h * 16;
                    const uint64_t db = db0 + static_cast<uint64_t>(h * 64 >> 4);
                    if (elect_one())
                    {
                        if constexpr (STACKN)
                        {
                            const uint32_t i3 = idesc_bf16_f32(T1_BM, 3 * NT), i2 = idesc_bf16_f32(T1_BM, 2 * NT),
                                           i1 = idesc_bf16_f32(T1_BM, NT);
#pragma unroll
                            for (int k = 0; k < 2; ++k)  // hi x [Ch;Cm;Cl]
                                mma_bf16_ta(tb, ta + k * 8, db + 2 * k, i3, (h | k) != 0);
#pragma unroll
                            for (int k = 0; k < 2; ++k)  // mid x [Ch;Cm]
                                mma_bf16_ta(tb + NT, ta + 32 + k * 8, db + 2 * k, i2, 1);
#pragma unroll
                            for (int k = 0; k < 2; ++k)  // lo x Ch
                                mma_bf16_ta(tb + 2 * NT, ta + 64 + k * 8, db + 2 * k, i1, 1);
                        }
                        else
                        {
                            const uint32_t idesc = idesc_bf16_f32(T1_BM, NT);
                            const uint32_t t_hh = tb, t_x = tb + NT;
                            const uint64_t dp = static_cast<uint64_t>(bbytes >> 4);  // to the next piece of C^J
#pragma unroll
                            for (int k = 0; k < 2; ++k)
                            {
                                const uint64_t d0 = db + static_cast<uint64_t>(k * 32 >> 4);
                                const uint32_t ah = ta + k * 8, am = ah + 32, al = ah + 64;
                                // cross terms (smallest first) into t_x, hi*hi into t_hh; both restart each stage
                                mma_bf16_ta(t_x, al, d0, idesc, (h | k) != 0);
                                mma_bf16_ta(t_x, ah, d0 + 2 * dp, idesc, 1);
                                mma_bf16_ta(t_x, am, d0 + dp, idesc, 1);
                                mma_bf16_ta(t_x, am, d0, idesc, 1);
                                mma_bf16_ta(t_x, ah, d0 + dp, idesc, 1);
                                mma_bf16_ta(t_hh, ah, d0, idesc, (h | k) != 0);
                            }
                        }
                        mma_commit(&empty[fb]);
                        if (h == nh - 1)
                        {
                            mma_commit(&bempty[sb]);
                            mma_commit(&accf[ab]);
                        }
                    }
                    __syncwarp();
                }
                if (!ok) break;
                if (++sb == nbs) sb = 0, pb ^= 1;
                if (++ab == nab) ab = 0, pa ^= 1;
                if (++jg == njg) jg = 0, set ^= 1;
                if (copied < total_stages) ok = issue_tma();
            }
            // every issued MMA and copy completes before the CTA's TMEM and shared memory are released
            if (elect_one()) mma_commit(fin);
            __syncwarp();
            mbar_wait(fin, 0);
            for (int k = max(0, copied - nbs); k < copied; ++k) mbar_wait(&bfull[k % nbs], (k / nbs) & 1);
        }
    }
    else
    {
        // ---------------- drain warps: per-stage accumulator blocks -> FP32 registers -> chi0R.
        if constexpr (DREG > 128)
            asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(DREG));
        else
            asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(DREG));
        const int wq = warp - T1_DRAIN;
        const uint32_t lane_base = static_cast<uint32_t>(wq * 32) << 16;
        float2 acc[NTC / 2];
#pragma unroll
        for (int c = 0; c < NTC / 2; ++c) acc[c] = make_float2(0.f, 0.f);
        auto pair_of = [](const uint32_t *r, int i) { return make_float2(__uint_as_float(r[i]), __uint_as_float(r[i + 1])); };
        bool ok = true;
        int ab = 0, ph = 0;
        for (int sd = 0; sd < total_stages; ++sd)
        {
            // one warp polls; the others stand at the barrier
            if (wq == 0 && !__all_sync(0xffffffffu, mbar_wait_nap<100>(&accf[ab], ph)) && lane == 0)
            {
                atomicExch(a.err, 204);
                *drain_stop = 1;
            }
            named_bar_sync(2, 128);
            if (*drain_stop)
            {
                ok = false;
                break;
            }
            tc_fence_after();
            const uint32_t tb = tmem + static_cast<uint32_t>(ab * NBLK * NT) + lane_base;
#pragma unroll
            for (int c0 = 0; c0 < NTC; c0 += 8)
            {
                if (c0 < NT)
                {
                    // 8 columns of each block live at a time, added from the smallest order up
                    uint32_t v[8], u[8];
                    tmem_ld8_nowait(tb + (NBLK - 1) * NT + c0, v);
                    if constexpr (STACKN)
                    {
                        uint32_t m[8];
                        tmem_ld8_nowait(tb + NT + c0, m);
                        tmem_ld8_nowait(tb + c0, u);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 8; i += 2)
                            acc[(c0 + i) / 2] = __fadd2_rn(acc[(c0 + i) / 2],
                                                           __fadd2_rn(pair_of(u, i), __fadd2_rn(pair_of(m, i), pair_of(v, i))));
                    }
                    else
                    {
                        tmem_ld8_nowait(tb + c0, u);
                        tmem_wait_ld();
#pragma unroll
                        for (int i = 0; i < 8; i += 2)
                            acc[(c0 + i) / 2] =
                                __fadd2_rn(__fadd2_rn(acc[(c0 + i) / 2], pair_of(v, i)), pair_of(u, i));
                    }
                }
            }
            tc_fence_before();
            __syncwarp();
            if (lane == 0) mbar_arrive(&acce[ab]);
            if (++ab == nab) ab = 0, ph ^= 1;
        }
        int slot, mu;
        if (row_of(wq * 32 + lane, slot, mu) && ok)
        {
            const int *f = info + slot * T1_INFO;
            double *orow = a.out + a.pr.r_off[f[0]] + (static_cast<long long>(f[1]) * f[3] + mu) * bJ;
#pragma unroll
            for (int c = 0; c < NTC; ++c)
                if (c < bJ)
                {
                    const double v = static_cast<double>(c & 1 ? acc[c / 2].y : acc[c / 2].x);
                    if (w.split)
                        atomicAdd(orow + c, v);
                    else
                        orow[c] = v;
                }
        }
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 0) tmem_dealloc(tmem, T1_TMEM);
}

// T2 for one (pair, cJ) and one 64 x 64 tile of its (mu, nu) block:
//   out[mu][nu] += sum_pass sum_{i,j} Xb^I[mu i; (cJ,J) j] * Xa^J[nu j; (-cJ,I) i].
// Grid: x = (pair, cJ) group, y = output tile (CTAs beyond the pair's own block return at once), so that a
// Gamma-only cell, with one group per pair, still spreads over the SMs.  Both operands come from the
// 4-column groups of Xt: a float4 is 4 j of one (mu, i) or 4 i of one (nu, j), and 32 lanes read 512
// contiguous bytes.  A step takes 4 i x 4 j: one float4 of each operand per thread, transposed through
// shared memory to [k = (i, j)][mu] and [k][nu] without bank conflicts, the next step's loads in flight
// meanwhile; each of the tile's (mu, nu) 4 x 4 blocks is one thread's.  Bound by the latency of its steps
// in small cells and by the FP32 pipe in large ones.  Where the tiles leave SMs idle, the steps of one are
// dealt to a cluster of CTAs (z), whose first sums the parts in order through distributed shared memory.
// Tiles are disjoint and each is added once, so the result does not depend on CTA order.  One GB300, a
// launch: 3 atoms of 5/20, 13/60, 26/110 at Gamma 283 -> 107 us by the steps, 42 by the parts; 128 atoms of
// 13/40 1.77 -> 0.73 ms.
constexpr int T2_THREADS = 256;
constexpr int T2_TILE = 64;

__global__ void __launch_bounds__(T2_THREADS) k_t2(const float4 *__restrict__ Xt, const long long *__restrict__ xoff, int n4,
                                                  Geom g, Pairs pr, const T1Group *__restrict__ groups, int tiles,
                                                  double *__restrict__ out)
{
    __shared__ __align__(16) float buf[2][2][16][T2_TILE];  // [operand][step parity][k][row]; the parts' sum
    auto &S1 = buf[0], &S2 = buf[1];
    const int p = groups[blockIdx.x].pair, cJ = groups[blockIdx.x].cell;
    const int I = pr.I[p], J = pr.J[p];
    const int aI = g.nao[I], aJ = g.nao[J], bI = g.nabf[I], bJ = g.nabf[J];
    const int mt0 = static_cast<int>(blockIdx.y) / tiles * T2_TILE, nt0 = static_cast<int>(blockIdx.y) % tiles * T2_TILE;
    if (mt0 >= bI || nt0 >= bJ) return;  // whole CTA: no barrier skipped by part of it
    const int mn = min(T2_TILE, bI - mt0), nn = min(T2_TILE, bJ - nt0);
    // first column group of each atom and the atom's first column inside it
    const int gI = g.ao_off[I] / 4, sI = g.ao_off[I] % 4, gJ = g.ao_off[J] / 4, sJ = g.ao_off[J] % 4;
    const int nI = (sI + aI + 3) / 4, nJ = (sJ + aJ + 3) / 4, steps = 2 * nI * nJ;
    const int nsplit = static_cast<int>(gridDim.z), part = static_cast<int>(blockIdx.z);
    const int st0 = steps * part / nsplit, st1 = steps * (part + 1) / nsplit;
    const int r = threadIdx.x % T2_TILE, s = threadIdx.x / T2_TILE;  // staging: row and i (or j) of the step
    const long long rI = static_cast<long long>(t1_rows(aI)) * bI, rJ = static_cast<long long>(t1_rows(aJ)) * bJ;
    const float4 *XI = Xt + xoff[I] + (static_cast<long long>(cJ) * n4 + gJ) * rI + mt0 + r;
    const float4 *XJ = Xt + xoff[J] + (static_cast<long long>(g.cneg[cJ]) * n4 + gI) * rJ + nt0 + r;
    const float4 zero4 = make_float4(0.f, 0.f, 0.f, 0.f);
    auto load = [&](int st, float4 &v1, float4 &v2) {
        const int pass = st / (nI * nJ), ig = st / nJ % nI, jg = st % nJ;
        const int i = 4 * ig + s - sI, j = 4 * jg + s - sJ;
        // pass 0 contracts X(-) of I with X(+) of J, pass 1 the other way round
        v1 = i >= 0 && i < aI && r < mn ? XI[jg * rI + static_cast<long long>(pass * aI + i) * bI] : zero4;
        v2 = j >= 0 && j < aJ && r < nn ? XJ[ig * rJ + static_cast<long long>((1 - pass) * aJ + j) * bJ] : zero4;
    };
    // one 4 x 4 block of the tile per thread
    const int nb = (nn + 3) / 4;
    const int m0 = static_cast<int>(threadIdx.x) / nb * 4, n0 = static_cast<int>(threadIdx.x) % nb * 4;
    const bool live = m0 < mn;
    float2 acc[4][2];
#pragma unroll
    for (int a = 0; a < 4; ++a) acc[a][0] = acc[a][1] = make_float2(0.f, 0.f);
    float4 v1, v2;
    load(min(st0, steps - 1), v1, v2);
    for (int st = st0; st < st1; ++st)
    {
        float(*A)[T2_TILE] = S1[st & 1], (*B)[T2_TILE] = S2[st & 1];
        A[4 * s][r] = v1.x, A[4 * s + 1][r] = v1.y, A[4 * s + 2][r] = v1.z, A[4 * s + 3][r] = v1.w;
        B[s][r] = v2.x, B[4 + s][r] = v2.y, B[8 + s][r] = v2.z, B[12 + s][r] = v2.w;
        __syncthreads();
        if (st + 1 < st1) load(st + 1, v1, v2);
        if (live)
        {
            // the i and j of this step that lie inside the atoms
            const int ig = st / nJ % nI, jg = st % nJ;
            const int i0 = max(0, sI - 4 * ig), i1 = min(4, sI + aI - 4 * ig), j0 = max(0, sJ - 4 * jg),
                      j1 = min(4, sJ + aJ - 4 * jg);
            for (int i = i0; i < i1; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j)
                {
                    if (j < j0 || j >= j1) continue;
                    const float4 av = *reinterpret_cast<const float4 *>(&A[4 * i + j][m0]);
                    const float4 bv = *reinterpret_cast<const float4 *>(&B[4 * i + j][n0]);
                    const float a4[4] = {av.x, av.y, av.z, av.w};
                    const float2 b0 = make_float2(bv.x, bv.y), b1 = make_float2(bv.z, bv.w);
#pragma unroll
                    for (int a = 0; a < 4; ++a)
                    {
                        const float2 aa = make_float2(a4[a], a4[a]);
                        acc[a][0] = __ffma2_rn(aa, b0, acc[a][0]);
                        acc[a][1] = __ffma2_rn(aa, b1, acc[a][1]);
                    }
                }
        }
    }
    double *o = out + pr.r_off[p] + static_cast<long long>(cJ) * bI * bJ + static_cast<long long>(mt0 + m0) * bJ + nt0 + n0;
    float *tile = &buf[0][0][0][0];  // [T2_TILE][T2_TILE] of a part
    static_assert(sizeof(buf) >= sizeof(float) * T2_TILE * T2_TILE, "a part's tile fits the staging buffers");
    cooperative_groups::cluster_group cl = cooperative_groups::this_cluster();
    pdl_wait();  // T1 has written chi0(R)
    if (nsplit > 1)
    {
        __syncthreads();
        if (live && part != 0)
#pragma unroll
            for (int a = 0; a < 4; ++a)
                *reinterpret_cast<float4 *>(tile + (m0 + a) * T2_TILE + n0) =
                    make_float4(acc[a][0].x, acc[a][0].y, acc[a][1].x, acc[a][1].y);
        cl.sync();
    }
    if (live && part == 0)
#pragma unroll
        for (int a = 0; a < 4; ++a)
        {
            const float v[4] = {acc[a][0].x, acc[a][0].y, acc[a][1].x, acc[a][1].y};
#pragma unroll
            for (int c = 0; c < 4; ++c)
                if (m0 + a < mn && n0 + c < nn)
                {
                    double x = static_cast<double>(v[c]);
                    for (int k = 1; k < nsplit; ++k)
                        x += static_cast<double>(cl.map_shared_rank(tile, k)[(m0 + a) * T2_TILE + n0 + c]);
                    o[static_cast<long long>(a) * bJ + c] += x;
                }
        }
    if (nsplit > 1) cl.sync();  // the tiles stay until they are read
}

// B operand of X = C * Gs: row n = (cL, l), column k = (cK, k'):  Gs^T[n][k] = G[cdiff(cL,cK)][k'][l]
__global__ void k_gsT_split(const double *__restrict__ G, Geom g, long long kpad, __nv_bfloat16 *__restrict__ p0,
                            __nv_bfloat16 *__restrict__ p1, __nv_bfloat16 *__restrict__ p2)
{
    const long long nsup = g.n_sup;
    const int sign = blockIdx.y;
    const long long n_el = nsup * kpad;
    const int nao = g.n_ao, nc = g.n_c;
    for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < n_el;
         t += static_cast<long long>(gridDim.x) * blockDim.x)
    {
        const long long n = t / kpad, k = t % kpad;
        double x = 0.0;
        if (k < nsup)
        {
            const int cL = static_cast<int>(n / nao), l = static_cast<int>(n % nao);
            const int cK = static_cast<int>(k / nao), kk = static_cast<int>(k % nao);
            const int c = g.cdiff[cL * nc + cK];
            x = G[((static_cast<size_t>(sign) * nc + c) * nao + kk) * nao + l];
        }
        const __nv_bfloat16 h = __double2bfloat16(x);
        const double r1 = x - static_cast<double>(__bfloat162float(h));
        const __nv_bfloat16 m = __double2bfloat16(r1);
        const __nv_bfloat16 l = __double2bfloat16(r1 - static_cast<double>(__bfloat162float(m)));
        p0[sign * n_el + t] = h;
        p1[sign * n_el + t] = m;
        p2[sign * n_el + t] = l;
    }
}

// X in the order the T1 producers read it: groups of 4 columns of one cell (n4 = ceil(n_ao / 4) per
// cell, zero past n_ao), atom-major,
//   Xt[xoff[I] + (g4 t1_rows(a_I) + q) b_I + mu] = the 4 columns of X_b[(I, mu, i)], q = (pass, i),
// pass 0 of X(-), pass 1 of X(+), zero rows past 2 a_I.  A warp of producers (32 consecutive rows mu)
// then reads 512 contiguous bytes per q, where row-major X costs it 32 lines.  Grid: x = blocks of 8
// groups, y = atoms (from I0, whose first row is X's) times 32-row tiles of mu, z = blocks of T1_XD rows q;
// bound by HBM (X read and written once, 1% of the contraction's time).
__global__ void __launch_bounds__(256) k_x_layout(const float *__restrict__ X, long long xsign, Geom g, int I0, int n4, int ng4,
                                                  int mu_tiles, const long long *__restrict__ xoff,
                                                  float4 *__restrict__ Xt)
{
    __shared__ float tile[T1_XD][32][33];
    const int I = I0 + blockIdx.y / mu_tiles, mu0 = (blockIdx.y % mu_tiles) * 32;
    const int aI = g.nao[I], bI = g.nabf[I], rows = t1_rows(aI), q0 = blockIdx.z * T1_XD;
    if (mu0 >= bI || q0 >= rows) return;
    const int c = threadIdx.x % 32, r0 = threadIdx.x / 32;
    // the column this thread reads, and the (mu, group) it writes
    const int g4r = blockIdx.x * 8 + c / 4;
    const int ao = (g4r % n4) * 4 + c % 4;
    const bool live = g4r < ng4 && ao < g.n_ao;
    const long long col = static_cast<long long>(g4r / n4) * g.n_ao + ao;
#pragma unroll
    for (int k = 0; k < T1_XD; ++k)
    {
        const int q = q0 + k;
        const bool lq = live && q < 2 * aI;
        const float *src = X + (q < aI ? xsign : 0) + (g.rowc_off[I] - g.rowc_off[I0] + q % aI) * static_cast<long long>(g.n_sup) + col;
#pragma unroll
        for (int r = 0; r < 32; r += 8)
            tile[k][r + r0][c] = lq && mu0 + r + r0 < bI ? src[static_cast<long long>(mu0 + r + r0) * aI * g.n_sup] : 0.0f;
    }
    __syncthreads();
    const int g4w = blockIdx.x * 8 + r0;
    if (g4w >= ng4 || mu0 + c >= bI) return;
    float4 *dst = Xt + xoff[I] + (static_cast<long long>(g4w) * rows + q0) * bI + mu0 + c;
#pragma unroll
    for (int k = 0; k < T1_XD; ++k)
        dst[static_cast<long long>(k) * bI] = make_float4(tile[k][c][4 * r0], tile[k][c][4 * r0 + 1], tile[k][c][4 * r0 + 2],
                                                          tile[k][c][4 * r0 + 3]);
}

// T1 B-operand layout of atom J: row nu, K index ((kc * aJpad + j) * CW + col) for C^J[nu][j][column col
// of chunk kc] (zero beyond the atom's NAOs, the cell's columns and the supercell).
__global__ void k_cb_layout(const double *__restrict__ C, Geom g, int J, int ajp, int n4, int ng4, long long ktot,
                            __nv_bfloat16 *__restrict__ p0, __nv_bfloat16 *__restrict__ p1,
                            __nv_bfloat16 *__restrict__ p2)
{
    const int aJ = g.nao[J], bJ = g.nabf[J];
    const long long n = static_cast<long long>(bJ) * ktot;
    for (long long t = static_cast<long long>(blockIdx.x) * blockDim.x + threadIdx.x; t < n;
         t += static_cast<long long>(gridDim.x) * blockDim.x)
    {
        const int nu = static_cast<int>(t / ktot);
        const long long k = t % ktot;
        const long long kc = k / (static_cast<long long>(ajp) * CW);
        const int rem = static_cast<int>(k % (static_cast<long long>(ajp) * CW));
        const int j = rem / CW, col = rem % CW;
        const int g4 = static_cast<int>(2 * kc + col / 4);
        const int ao = (g4 % n4) * 4 + col % 4;
        double x = 0.0;
        if (j < aJ && g4 < ng4 && ao < g.n_ao)
            x = C[(g.rowc_off[J] + static_cast<long long>(nu) * aJ + j) * g.n_sup + static_cast<long long>(g4 / n4) * g.n_ao + ao];
        const __nv_bfloat16 h = __double2bfloat16(x);
        const double r1 = x - static_cast<double>(__bfloat162float(h));
        const __nv_bfloat16 m = __double2bfloat16(r1);
        const __nv_bfloat16 l = __double2bfloat16(r1 - static_cast<double>(__bfloat162float(m)));
        p0[t] = h;
        p1[t] = m;
        p2[t] = l;
    }
}

} // namespace

struct TcChi0::Impl
{
    Geom g;
    Pairs pr;
    long long kpad = 0;
    int nkc = 0, n4 = 0, ng4 = 0;
    bool t1_simt = false;
    SplitStore csplit, gs;
    DevBuf<float> X, Gf, Cf;
    std::vector<long long> row;  // first row of C of each atom, and their number
    std::vector<int> slab;       // first atom of each slab of X, and the number of atoms
    DevBuf<float4> Xt;
    DevBuf<long long> xoff;
    DevBuf<int> err, cadd;
    DevBuf<T1Work> work;
    DevBuf<T1Group> groups;
    int n_work = 0, n_groups = 0;
    std::vector<int> hI, hJ, nabf_h, nao_h;
    bool all_active = false;  // the uploaded work list covers every (pair, cell)
    bool has_split = false;   // some tiles are K parts that add into chi0(R) atomically
    int n_sm = 0;
    // Row groups of the active (pair, cell) blocks, ordered by J, then I, then cell, and the
    // 128-row tiles over each J's rows; active == nullptr: every block.
    void build_work(const unsigned char *active, cudaStream_t st);
    std::vector<SplitStore> cb;  // per species: C^J of its atoms, stacked
    T1Maps maps{};
    DevBuf<int> spec, spec_idx;
    int b_tile = 0, maxcj = 0, smem = 0, ntc = 64, nbs = 2, gq = 0, gslot = 0;
    // K parts per tile of the contraction.  The tuner times the candidates on the first unscreened
    // contraction of a shape and keeps the fastest for every later call on that shape.
    int kparts = T1_KPARTS;
    bool kparts_forced = false, tuned = false;
    std::string shape_key;
    T1Args t1_args(const double *G, double *chi0R) const;
    void autotune(const double *G, double *chi0R, cudaStream_t st);
    void check(cudaStream_t st) const;
    void launch_t1(const T1Args &a, cudaStream_t st);
    void launch_t2(double *chi0R, cudaStream_t st);
};

namespace {
struct T1Choice
{
    int kparts;
    double ms;
};
std::mutex g_tune_mu;
std::map<std::string, T1Choice> g_tuned;  // shape key -> choice (process-wide)
} // namespace

namespace {
using T1Fn = void (*)(T1Args, T1Maps);
T1Fn t1_kernel(int ntc) { return ntc == 48 ? k_t1_tc<48> : ntc == 64 ? k_t1_tc<64> : k_t1_tc<128>; }
} // namespace

TcChi0::TcChi0(const Geom &g, const Pairs &pr, const double *C, cudaStream_t st) : impl_(std::make_unique<Impl>())
{
    Impl &m = *impl_;
    m.g = g;
    m.pr = pr;
    const long long nsup = g.n_sup;
    m.kpad = (nsup + 63) / 64 * 64;
    m.n4 = (g.n_ao + 3) / 4;
    m.ng4 = g.n_c * m.n4;
    m.nkc = (m.ng4 + 1) / 2;
    const char *env = std::getenv("LIBRPA_GB300_T1");
    m.t1_simt = env && std::string(env) == "simt";
    GB_REQUIRE(g.max_nao <= T1_MAXA, "the tensor-core chi0 kernel supports up to 32 NAOs per atom");
    GB_REQUIRE(g.max_nabf <= T1_NMAX, "the tensor-core chi0 kernel supports up to 128 ABFs per atom");
    m.csplit.alloc(NS, static_cast<size_t>(g.rows_c) * m.kpad);
    split_rows_f64(C, nsup, g.rows_c, static_cast<int>(nsup), static_cast<int>(m.kpad), m.csplit.bufs(), st);
    m.gs.alloc(NS, 2ull * nsup * m.kpad);
    m.err.alloc(1);
    m.err.zero(st);
    // host copies of the small tables (Geom holds device pointers)
    std::vector<int> nao(g.n_at), nabf(g.n_at), cdiff(static_cast<size_t>(g.n_c) * g.n_c);
    GB_CUDA(cudaMemcpyAsync(nao.data(), g.nao, sizeof(int) * g.n_at, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaMemcpyAsync(nabf.data(), g.nabf, sizeof(int) * g.n_at, cudaMemcpyDeviceToHost, st));
    m.row.resize(g.n_at + 1);
    GB_CUDA(cudaMemcpyAsync(m.row.data(), g.rowc_off, sizeof(long long) * g.n_at, cudaMemcpyDeviceToHost, st));
    m.row[g.n_at] = g.rows_c;
    GB_CUDA(cudaMemcpyAsync(cdiff.data(), g.cdiff, sizeof(int) * cdiff.size(), cudaMemcpyDeviceToHost, st));
    std::vector<int> hI(pr.n_pairs), hJ(pr.n_pairs);
    GB_CUDA(cudaMemcpyAsync(hI.data(), pr.I, sizeof(int) * pr.n_pairs, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaMemcpyAsync(hJ.data(), pr.J, sizeof(int) * pr.n_pairs, cudaMemcpyDeviceToHost, st));
    GB_CUDA(cudaStreamSynchronize(st));
    // cadd[a][b] = cell of R_a + R_b: the unique c with cdiff[c][b] == a
    std::vector<int> cadd(cdiff.size(), -1);
    for (int c = 0; c < g.n_c; ++c)
        for (int b = 0; b < g.n_c; ++b) cadd[cdiff[c * g.n_c + b] * g.n_c + b] = c;
    m.cadd.alloc(cadd.size());
    m.cadd.upload(cadd.data(), cadd.size(), st);
    if (m.t1_simt)
    {
        m.X.alloc(2ull * g.rows_c * nsup);
        m.Cf.alloc(static_cast<size_t>(g.rows_c) * nsup);
        launch_d2f(C, m.Cf.get(), g.rows_c * nsup, st);
        m.Gf.alloc(2ull * g.n_c * g.n_ao * g.n_ao);
        return;
    }
    {
        // X is formed for as many atoms at a time as T1_XSLAB bytes hold, at least one
        long long most = 0;
        m.slab.assign(1, 0);
        for (int I = 1; I <= g.n_at; ++I)
        {
            if (I < g.n_at && 8 * nsup * (m.row[I + 1] - m.row[m.slab.back()]) <= T1_XSLAB) continue;
            most = std::max(most, m.row[I] - m.row[m.slab.back()]);
            m.slab.push_back(I);
        }
        m.X.alloc(2ull * most * nsup);
        std::vector<long long> xo(g.n_at);
        long long n = 0;
        for (int I = 0; I < g.n_at; ++I)
        {
            xo[I] = n;
            n += static_cast<long long>(m.ng4) * t1_rows(nao[I]) * nabf[I];
        }
        m.Xt.alloc(n);
        m.xoff.alloc(xo.size());
        m.xoff.upload(xo.data(), xo.size(), st);
        GB_CUDA(cudaStreamSynchronize(st));  // xo goes out of scope
    }
    // T1 B operands grouped by species (same NAO and ABF counts) and their TMA maps
    std::vector<int> ajp(g.n_at), spec(g.n_at), spec_idx(g.n_at);
    std::vector<std::pair<int, int>> species;
    std::vector<int> spec_count;
    for (int J = 0; J < g.n_at; ++J)
    {
        ajp[J] = (nao[J] + JG - 1) / JG * JG;
        const std::pair<int, int> key{nao[J], nabf[J]};
        int sp = -1;
        for (size_t k = 0; k < species.size(); ++k)
            if (species[k] == key) sp = static_cast<int>(k);
        if (sp < 0)
        {
            sp = static_cast<int>(species.size());
            species.push_back(key);
            spec_count.push_back(0);
        }
        GB_REQUIRE(sp < T1_MAXSPEC, "the tensor-core chi0 kernel supports up to 8 atom species");
        spec[J] = sp;
        spec_idx[J] = spec_count[sp]++;
    }
    m.cb.resize(species.size());
    for (size_t sp = 0; sp < species.size(); ++sp)
    {
        const int na = species[sp].first, nb = species[sp].second;
        const int ap = (na + JG - 1) / JG * JG;
        const long long ktot = static_cast<long long>(m.nkc) * ap * CW;
        const long long per_atom = static_cast<long long>(nb) * ktot;
        m.cb[sp].alloc(NS, static_cast<size_t>(per_atom) * spec_count[sp]);
        const SplitBufs b = m.cb[sp].bufs();
        for (int J = 0; J < g.n_at; ++J)
        {
            if (spec[J] != static_cast<int>(sp)) continue;
            const long long o = per_atom * spec_idx[J];
            k_cb_layout<<<static_cast<unsigned>(std::min<long long>((per_atom + 255) / 256, 152LL * 16)), 256, 0, st>>>(
                C, g, J, ap, m.n4, m.ng4, ktot, b.p[0] + o, b.p[1] + o, b.p[2] + o);
            GB_LAUNCH_CHECK();
        }
        const int NT = (nb + 15) / 16 * 16;
        for (int p = 0; p < NS; ++p)
            make_tmap_bf16(&m.maps.m[sp][p], b.p[p], ktot, nb, spec_count[sp], ktot, per_atom, 64, NT);
        m.maps.ktot[sp] = ktot;
    }
    m.spec.alloc(spec.size());
    m.spec.upload(spec.data(), spec.size(), st);
    m.spec_idx.alloc(spec_idx.size());
    m.spec_idx.upload(spec_idx.data(), spec_idx.size(), st);
    m.hI = hI;
    m.hJ = hJ;
    m.nabf_h = nabf;
    m.nao_h = nao;
    {
        int dev = 0;
        GB_CUDA(cudaGetDevice(&dev));
        GB_CUDA(cudaDeviceGetAttribute(&m.n_sm, cudaDevAttrMultiProcessorCount, dev));
    }
    m.work.alloc(static_cast<size_t>(pr.n_pairs) * g.n_c * ((g.max_nabf + T1_BM - 1) / T1_BM + 1) * T1_KPARTS_MAX +
                 8 * static_cast<size_t>(m.n_sm));
    m.groups.alloc(static_cast<size_t>(pr.n_pairs) * g.n_c);
    int ntmax = 16, minb = 1 << 30;
    for (int J = 0; J < g.n_at; ++J)
    {
        ntmax = std::max(ntmax, (nabf[J] + 15) / 16 * 16);
        minb = std::min(minb, nabf[J]);
    }
    m.b_tile = (ntmax * 128 + 1023) / 1024 * 1024;
    m.maxcj = (T1_BM + minb - 1) / minb + 1;
    m.ntc = ntmax <= 48 ? 48 : ntmax <= 64 ? 64 : 128;
    // a G block of the largest atoms; 4 more floats keep the blocks of two groups on different banks
    m.gq = 2 * g.max_nao;
    m.gslot = m.gq * ((g.max_nao + JG - 1) / JG * JG) + 4;
    // shared memory: at least two B stages + the G slots; fewer G slots than a tile of small row
    // groups could touch only shortens such tiles
    const int slot_bytes = (m.gslot + T1_CELLS + T1_INFO) * 4;
    const int base = 1024 + T1_XBYTES + 512;
    const int fit = (T1_SMEM_MAX - base - 2 * NS * m.b_tile) / slot_bytes;
    GB_REQUIRE(fit >= 1, "chi0 tile does not fit shared memory (too many ABFs or NAOs per atom)");
    m.maxcj = std::min(m.maxcj, fit);
    const int fixed = base + m.maxcj * slot_bytes;
    m.nbs = std::min(T1_MAXB, (T1_SMEM_MAX - fixed) / (NS * m.b_tile));
    m.smem = fixed + m.nbs * NS * m.b_tile;
    // the cap, not this shape's own size: contractions of other shapes on other host threads share
    // the kernel, and a smaller value set by one of them would fail this one's launch
    GB_CUDA(cudaFuncSetAttribute(t1_kernel(m.ntc), cudaFuncAttributeMaxDynamicSharedMemorySize, T1_SMEM_MAX));
    // the shape the tuner's choice is kept for: per-atom sizes, cells, pairs, SM count
    {
        std::string key = std::to_string(g.n_c) + ":" + std::to_string(g.n_ao) + ":" + std::to_string(pr.n_pairs) +
                          ":" + std::to_string(m.n_sm) + ":";
        for (int J = 0; J < g.n_at; ++J) key += std::to_string(nao[J]) + "/" + std::to_string(nabf[J]) + ",";
        m.shape_key = key;
        // LIBRPA_GB300_T1_LAUNCH = "wide:<kparts>" fixes the choice (no tuning); "narrow:" reads the same,
        // there is one producer layout
        if (const char *fx = std::getenv("LIBRPA_GB300_T1_LAUNCH"))
        {
            const std::string v(fx);
            const size_t c = v.find(':');
            GB_REQUIRE(c != std::string::npos, "LIBRPA_GB300_T1_LAUNCH must read narrow:<kparts> or wide:<kparts>");
            const std::string lay = v.substr(0, c);
            const int kp = std::atoi(v.c_str() + c + 1);
            GB_REQUIRE((lay == "narrow" || lay == "wide") && kp >= 1 && kp <= T1_KPARTS_MAX,
                       "LIBRPA_GB300_T1_LAUNCH must read narrow:<kparts> or wide:<kparts>, kparts 1-16");
            m.kparts = kp;
            m.kparts_forced = true;
            m.tuned = true;
        }
        std::lock_guard<std::mutex> lk(g_tune_mu);
        auto it = m.tuned ? g_tuned.end() : g_tuned.find(key);
        if (it != g_tuned.end())
        {
            m.kparts = it->second.kparts;
            m.kparts_forced = true;
            m.tuned = true;
        }
    }
    m.build_work(nullptr, st);
    GB_CUDA(cudaStreamSynchronize(st));
}

T1Args TcChi0::Impl::t1_args(const double *G, double *chi0R) const
{
    T1Args a{};
    a.g = g;
    a.pr = pr;
    a.Xt = Xt.get();
    a.xoff = xoff.get();
    a.G = G;
    a.cadd = cadd.get();
    a.work = work.get();
    a.groups = groups.get();
    a.spec = spec.get();
    a.spec_idx = spec_idx.get();
    a.n4 = n4;
    a.ng4 = ng4;
    a.b_tile = b_tile;
    a.nbs = nbs;
    a.gq = gq;
    a.gslot = gslot;
    a.maxcj = maxcj;
    a.out = chi0R;
    a.err = err.get();
    return a;
}

void TcChi0::Impl::launch_t1(const T1Args &a, cudaStream_t st)
{
    t1_kernel(ntc)<<<n_work, T1_THREADS, smem, st>>>(a, maps);
    GB_LAUNCH_CHECK();
}

void TcChi0::Impl::launch_t2(double *chi0R, cudaStream_t st)
{
    const int tiles = (g.max_nabf + T2_TILE - 1) / T2_TILE;
    // parts of a tile's steps while the tiles leave SMs idle, up to the portable cluster size; by the
    // tiles of all blocks, so that a screened call sums a block as the unscreened one does
    const long long ctas = static_cast<long long>(pr.n_pairs) * g.n_c * tiles * tiles;
    const unsigned nsplit = static_cast<unsigned>(std::max<long long>(1, std::min<long long>(8, n_sm / ctas)));
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(n_groups, tiles * tiles, nsplit);
    cfg.blockDim = dim3(T2_THREADS);
    cfg.stream = st;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = 1;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = nsplit;
    // T2 reads what T1 reads and waits for it only to add to chi0(R), so it starts when T1's last CTAs do:
    // beside it where T1 has fewer CTAs than there are SMs, in T1's last wave otherwise.  Before, T1 and T2
    // took turns: a call of 3 atoms at Gamma 5.87 -> 5.31 ms, chi0 of 3 at 3 x 3 x 1 k 6.30 -> 5.73 ms
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = 2;
    GB_CUDA(cudaLaunchKernelEx(&cfg, k_t2, static_cast<const float4 *>(Xt.get()),
                               static_cast<const long long *>(xoff.get()), n4, g, pr,
                               static_cast<const T1Group *>(groups.get()), tiles, chi0R));
}

// Times every candidate count of K parts per tile on this contraction's own inputs, one warm and
// one timed launch each, and keeps the fastest.  T1 and T2 are timed together, since T2 runs beside T1 on
// the SMs that T1 leaves: with T1 alone the tuner took 16 parts at 2 atoms of 13/40 on 2 x 2 x 2 k, which
// left T2 24 SMs and cost 5% of the call.  The candidates write chi0R; the caller's own launch after the
// tuning overwrites it (zeroing it first when tiles are split).
void TcChi0::Impl::autotune(const double *G, double *chi0R, cudaStream_t st)
{
    const T1Args a = t1_args(G, chi0R);
    cudaEvent_t e0, e1;
    GB_CUDA(cudaEventCreate(&e0));
    GB_CUDA(cudaEventCreate(&e1));
    T1Choice best{kparts, 1e30};
    const int kp_cand[] = {1, 2, 4, 8, 16};
    for (int kp : kp_cand)
    {
        if (kp > T1_KPARTS_MAX || kp > nkc) continue;
        kparts = kp;
        kparts_forced = true;
        all_active = false;
        build_work(nullptr, st);
        if (n_work == 0) continue;
        launch_t1(a, st);
        launch_t2(chi0R, st);
        GB_CUDA(cudaEventRecord(e0, st));
        launch_t1(a, st);
        launch_t2(chi0R, st);
        GB_CUDA(cudaEventRecord(e1, st));
        GB_CUDA(cudaEventSynchronize(e1));
        float ms = 0.0f;
        GB_CUDA(cudaEventElapsedTime(&ms, e0, e1));
        if (ms < best.ms) best = T1Choice{kp, ms};
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    check(st);  // launches that gave a wait up time nothing
    kparts = best.kparts;
    kparts_forced = true;
    all_active = false;
    tuned = true;
    build_work(nullptr, st);
    std::lock_guard<std::mutex> lk(g_tune_mu);
    g_tuned[shape_key] = best;
}

void TcChi0::Impl::build_work(const unsigned char *active, cudaStream_t st)
{
    if (!active && all_active) return;
    std::vector<T1Group> grp;
    std::vector<T1Work> tiles;
    std::vector<std::vector<int>> pairs_of(g.n_at);
    for (int p = 0; p < pr.n_pairs; ++p) pairs_of[hJ[p]].push_back(p);
    for (int J = 0; J < g.n_at; ++J)
    {
        // I atoms of one NAO count next to each other, so that most tiles hold row groups of one
        // NAO count and their producers loop over that many orbitals i, not over the largest
        std::sort(pairs_of[J].begin(), pairs_of[J].end(), [&](int x, int y) {
            return nao_h[hI[x]] != nao_h[hI[y]] ? nao_h[hI[x]] < nao_h[hI[y]] : hI[x] < hI[y];
        });
        const int gbeg = static_cast<int>(grp.size());
        for (int p : pairs_of[J])
            for (int c = 0; c < g.n_c; ++c)
                if (!active || active[static_cast<size_t>(p) * g.n_c + c]) grp.push_back({p, c});
        // tiles of 128 rows over the concatenated rows of this J's groups; a tile closes at 128
        // rows or when it touches maxcj row groups (its G slots)
        const int gend = static_cast<int>(grp.size());
        std::vector<int> grows(gend - gbeg);
        for (int gi = gbeg; gi < gend; ++gi) grows[gi - gbeg] = nabf_h[hI[grp[gi].pair]];
        std::vector<sched::RowTile> rt;
        sched::pack_row_tiles(grows.data(), gend - gbeg, gbeg, T1_BM, maxcj, rt);
        for (const sched::RowTile &r : rt)
        {
            GB_REQUIRE(r.nslot <= maxcj, "chi0 tile touches more row groups than its shared-memory G slots");
            int ra_t = 0;
            for (int k = 0; k < r.nslot; ++k) ra_t = std::max(ra_t, nao_h[hI[grp[r.g0 + k].pair]]);
            tiles.push_back(T1Work{J, r.g0, r.r0, r.nrows, r.nslot, 0, nkc, 0, ra_t});
        }
    }
    // launch order: by the I atom of a tile's first row group, so the CTAs resident at one time
    // stream the same X^I rows (the largest operand) through L2
    std::stable_sort(tiles.begin(), tiles.end(), [&](const T1Work &x, const T1Work &y) {
        return hI[grp[x.g0].pair] < hI[grp[y.g0].pair];
    });
    // Every tile contracts the same K range, so the last, partial wave of CTAs leaves SMs idle:
    // its tiles are cut into K parts (added atomically into chi0(R)) when that shortens the
    // makespan.  Every tile is cut into the count that the tuner timed; on a shape that it has not seen
    // (a screened call), into T1_KPARTS where the launch has under 16 waves, finer units for the
    // scheduler.
    has_split = false;
    {
        const std::vector<sched::KPart> plan =
            sched::plan_kparts(static_cast<int>(tiles.size()), n_sm, nkc, kparts, kparts_forced);
        std::vector<T1Work> cut;
        cut.reserve(plan.size());
        for (const sched::KPart &k : plan)
        {
            T1Work u = tiles[k.tile];
            u.kc0 = k.kc0;
            u.kc1 = k.kc1;
            u.split = k.split;
            has_split = has_split || k.split != 0;
            cut.push_back(u);
        }
        tiles.swap(cut);
    }
    n_groups = static_cast<int>(grp.size());
    n_work = static_cast<int>(tiles.size());
    GB_REQUIRE(tiles.size() <= work.size() && grp.size() <= groups.size(), "chi0 work list overflow");
    if (n_groups > 0)
    {
        groups.upload(grp.data(), grp.size(), st);
        work.upload(tiles.data(), tiles.size(), st);
    }
    all_active = active == nullptr;
}

TcChi0::~TcChi0() = default;

void TcChi0::launch_choice(int &narrow, int &kparts) const
{
    narrow = 0;  // one producer layout
    kparts = impl_->kparts;
}

int TcChi0::run(const double *Gs, const double *G, double *chi0R, cudaStream_t st)
{
    (void)Gs;
    return prepare(G, st) + contract(G, chi0R, nullptr, false, st);
}

int TcChi0::prepare(const double *G, cudaStream_t st)
{
    Impl &m = *impl_;
    const Geom &g = m.g;
    const long long nsup = g.n_sup;
    dim3 grid(static_cast<unsigned>(std::min<long long>((nsup * m.kpad + 255) / 256, 152LL * 32)), 2);
    const SplitBufs gb = m.gs.bufs();
    k_gsT_split<<<grid, 256, 0, st>>>(G, g, m.kpad, gb.p[0], gb.p[1], gb.p[2]);
    GB_LAUNCH_CHECK();
    const int mu_tiles = (g.max_nabf + 31) / 32;
    const int n_slab = m.t1_simt ? 1 : static_cast<int>(m.slab.size()) - 1;
    for (int k = 0; k < n_slab; ++k)
    {
        const int I0 = m.t1_simt ? 0 : m.slab[k], I1 = m.t1_simt ? g.n_at : m.slab[k + 1];
        const long long rows = m.row[I1] - m.row[I0];
        SplitMat C = m.csplit.mat(rows, m.kpad, 0);
        for (int i = 0; i < NS; ++i) C.p[i] += m.row[I0] * m.kpad;
        tc_gemm_split(C, m.gs.mat(nsup, m.kpad, nsup * m.kpad), static_cast<int>(rows), static_cast<int>(nsup),
                      static_cast<int>(nsup), 2, m.X.get(), nsup, rows * nsup, false, m.err.get(), st);
        if (m.t1_simt) return 2;
        k_x_layout<<<dim3((m.ng4 + 7) / 8, (I1 - I0) * mu_tiles, t1_rows(g.max_nao) / T1_XD), 256, 0, st>>>(
            m.X.get(), rows * nsup, g, I0, m.n4, m.ng4, mu_tiles, m.xoff.get(), m.Xt.get());
        GB_LAUNCH_CHECK();
    }
    return 1 + 2 * n_slab;
}

int TcChi0::contract(const double *G, double *chi0R, const unsigned char *active, bool zero_first, cudaStream_t st)
{
    Impl &m = *impl_;
    const Geom &g = m.g;
    const long long nsup = g.n_sup;
    int launches = 0;
    if (!m.t1_simt && !active && !m.tuned) m.autotune(G, chi0R, st);
    if (!m.t1_simt) m.build_work(active, st);
    // K-part tiles add into chi0(R), so their rows start from zero; a list of blocks that adds to an earlier
    // one finds its own rows zero and must leave the others alone
    if (zero_first || (!m.t1_simt && !active && m.has_split))
        GB_CUDA(cudaMemsetAsync(chi0R, 0, sizeof(double) * static_cast<size_t>(m.pr.e_total) * g.n_c, st));
    if (m.t1_simt)
    {
        GB_REQUIRE(!active, "block screening needs the tensor-core chi0 kernel");
        const long long ng = static_cast<long long>(g.n_c) * g.n_ao * g.n_ao;
        launch_d2f(G, m.Gf.get(), 2 * ng, st);
        launch_chi0_fp32(m.X.get(), m.X.get() + g.rows_c * nsup, m.Cf.get(), m.Gf.get(), m.Gf.get() + ng, g, m.pr,
                         chi0R, st);
        launches += 2;
    }
    else
    {
        const T1Args a = m.t1_args(G, chi0R);
        if (m.n_work > 0)
        {
            m.launch_t1(a, st);
            m.launch_t2(chi0R, st);
            launches += 2;
        }
    }
    return launches;
}

void TcChi0::check(cudaStream_t st) const { impl_->check(st); }

void TcChi0::Impl::check(cudaStream_t st) const
{
    int herr = 0;
    err.download(&herr, 1, st);
    GB_CUDA(cudaStreamSynchronize(st));
    GB_REQUIRE(herr == 0, "tensor-core chi0 kernel reported wait timeout code " + std::to_string(herr));
}

} // namespace gb
