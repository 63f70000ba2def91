// X = C G of the chi0 contraction formed for some atoms at a time: the re-ordered X is the same whatever the
// slabs, and the row-major X of a large cell stays within its limit.  Prints "ok" or the first failure.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <random>
#include <string>
#include <vector>
#define private public  // the contraction's buffers
#include "../librpa_gb300/csrc/tc_gemm.h"
#undef private
#include "../librpa_gb300/csrc/tc_chi0.cu"

using namespace gb;

#define EXPECT(c)                                        \
    do                                                   \
        if (!(c))                                        \
        {                                                \
            std::printf("line %d: %s\n", __LINE__, #c);  \
            return 1;                                    \
        }                                                \
    while (0)

struct Cell
{
    std::vector<int> nao, nabf;
    Geom g;
    Pairs pr;
    DevBuf<int> d_ao, d_nao, d_nabf, d_cell, d_I, d_J;
    DevBuf<long long> d_row, d_off;
    Cell(std::vector<int> a, std::vector<int> b, cudaStream_t st) : nao(a), nabf(b)
    {
        const int n = static_cast<int>(nao.size());
        std::vector<int> ao(n), pI, pJ, cell0{0};
        std::vector<long long> row(n), off;
        g.n_at = n, g.n_c = 1, g.n_ao = 0, g.rows_c = 0, g.max_nao = 0, g.max_nabf = 0;
        for (int I = 0; I < n; ++I)
        {
            ao[I] = g.n_ao, row[I] = g.rows_c;
            g.n_ao += nao[I], g.rows_c += static_cast<long long>(nao[I]) * nabf[I];
            g.max_nao = std::max(g.max_nao, nao[I]), g.max_nabf = std::max(g.max_nabf, nabf[I]);
        }
        g.n_sup = g.n_ao;
        pr.e_total = 0;
        for (int I = 0; I < n; ++I)
            for (int J = I; J < n; ++J)
            {
                pI.push_back(I), pJ.push_back(J), off.push_back(pr.e_total);
                pr.e_total += static_cast<long long>(nabf[I]) * nabf[J];
            }
        d_ao = to_dev(ao, st), d_nao = to_dev(nao, st), d_nabf = to_dev(nabf, st), d_cell = to_dev(cell0, st);
        d_I = to_dev(pI, st), d_J = to_dev(pJ, st), d_row = to_dev(row, st), d_off = to_dev(off, st);
        g.ao_off = d_ao.get(), g.nao = d_nao.get(), g.nabf = d_nabf.get(), g.rowc_off = d_row.get();
        g.cdiff = g.cneg = d_cell.get();
        pr.n_pairs = static_cast<int>(pI.size()), pr.I = d_I.get(), pr.J = d_J.get(), pr.r_off = pr.e_off = d_off.get();
    }
};

int main()
{
    cudaStream_t st;
    GB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    {
        Cell c({3, 4, 13, 5}, {20, 17, 40, 33}, st);
        std::mt19937 rng(6);
        std::uniform_real_distribution<double> u(-1.0, 1.0);
        std::vector<double> C(c.g.rows_c * c.g.n_sup), G(2ull * c.g.n_ao * c.g.n_ao);
        for (double &x : C) x = u(rng);
        for (double &x : G) x = u(rng);
        auto d_C = to_dev(C, st);
        auto d_G = to_dev(G, st);
        TcChi0 tc(c.g, c.pr, d_C.get(), st);
        TcChi0::Impl &m = *tc.impl_;
        EXPECT((m.slab == std::vector<int>{0, 4}));
        std::vector<float4> one(m.Xt.size()), some(one.size()), clear(one.size(), make_float4(7.f, 7.f, 7.f, 7.f));
        tc.prepare(d_G.get(), st);
        m.Xt.download(one.data(), one.size(), st);
        GB_CUDA(cudaStreamSynchronize(st));
        for (const std::vector<int> &s : {std::vector<int>{0, 1, 2, 3, 4}, std::vector<int>{0, 2, 4}, std::vector<int>{0, 3, 4}})
        {
            m.slab = s;
            m.Xt.upload(clear.data(), clear.size(), st);
            EXPECT(tc.prepare(d_G.get(), st) == 2 * static_cast<int>(s.size()) - 1);
            m.Xt.download(some.data(), some.size(), st);
            tc.check(st);
            EXPECT(std::memcmp(one.data(), some.data(), sizeof(float4) * one.size()) == 0);
        }
    }
    {
        // 48 atoms of 32/128: 2.4 GB of X for all of them
        Cell c(std::vector<int>(48, 32), std::vector<int>(48, 128), st);
        DevBuf<double> d_C(static_cast<size_t>(c.g.rows_c) * c.g.n_sup);
        d_C.zero(st);
        TcChi0 tc(c.g, c.pr, d_C.get(), st);
        EXPECT(tc.impl_->X.bytes() <= (size_t(2) << 30));
    }
    GB_CUDA(cudaStreamDestroy(st));
    std::printf("ok\n");
    return 0;
}
