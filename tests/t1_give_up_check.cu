// After a wait that was given up: the launches that share its error flag do nothing, check() reports the
// code, and the tuner keeps no choice.  Prints "ok" or the first failure.
#include <algorithm>
#include <cstdio>
#include <cstring>
#include <map>
#include <memory>
#include <mutex>
#include <random>
#include <string>
#include <vector>
#define private public  // the contraction's buffers and its error flag
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

int main()
{
    cudaStream_t st;
    GB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    // two atoms in one cell
    const std::vector<int> ao_off{0, 3}, nao{3, 4}, nabf{20, 17}, cell0{0}, pI{0, 0, 1}, pJ{0, 1, 1};
    const std::vector<long long> rowc{0, 60}, off{0, 400, 740};
    auto d_ao = to_dev(ao_off, st), d_nao = to_dev(nao, st), d_nabf = to_dev(nabf, st), d_c = to_dev(cell0, st),
         d_I = to_dev(pI, st), d_J = to_dev(pJ, st);
    auto d_row = to_dev(rowc, st), d_off = to_dev(off, st);
    Geom g;
    g.n_at = 2, g.n_c = 1, g.n_ao = 7, g.n_sup = 7, g.max_nao = 4, g.max_nabf = 20, g.rows_c = 128;
    g.ao_off = d_ao.get(), g.nao = d_nao.get(), g.nabf = d_nabf.get(), g.rowc_off = d_row.get(), g.cdiff = g.cneg = d_c.get();
    Pairs pr;
    pr.n_pairs = 3, pr.I = d_I.get(), pr.J = d_J.get(), pr.r_off = pr.e_off = d_off.get(), pr.e_total = 1029;
    std::mt19937 rng(5);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    std::vector<double> C(128 * 7), G(2 * 49);
    for (double &x : C) x = u(rng);
    for (double &x : G) x = u(rng);
    auto d_C = to_dev(C, st);
    auto d_G = to_dev(G, st);
    DevBuf<double> out(1029);
    std::vector<double> ref(1029), got(1029), marks(1029, 42.0);
    const int seven = 7, zero = 0;
    {
        TcChi0 tc(g, pr, d_C.get(), st);
        tc.run(nullptr, d_G.get(), out.get(), st);
        tc.check(st);
        out.download(ref.data(), ref.size(), st);
        TcChi0::Impl &m = *tc.impl_;
        // the flag is set: no output of the contraction, none of the X product
        m.err.upload(&seven, 1, st);
        out.upload(marks.data(), marks.size(), st);
        std::vector<float> x(m.X.size(), 42.0f), x2(x.size());
        m.X.upload(x.data(), x.size(), st);
        tc.prepare(d_G.get(), st);
        m.launch_t1(m.t1_args(d_G.get(), out.get()), st);
        out.download(got.data(), got.size(), st);
        m.X.download(x2.data(), x2.size(), st);
        GB_CUDA(cudaStreamSynchronize(st));
        EXPECT(got == marks);
        EXPECT(x2 == x);
        std::string what;
        try
        {
            tc.check(st);
        }
        catch (const Error &e)
        {
            what = e.what();
        }
        EXPECT(what.find("code 7") != std::string::npos);
        // cleared: the call runs as before (FP64 additions of K parts in any order)
        m.err.upload(&zero, 1, st);
        tc.run(nullptr, d_G.get(), out.get(), st);
        tc.check(st);
        out.download(got.data(), got.size(), st);
        GB_CUDA(cudaStreamSynchronize(st));
        double top = 0, diff = 0;
        for (size_t i = 0; i < ref.size(); ++i) top = std::max(top, std::fabs(ref[i])), diff = std::max(diff, std::fabs(got[i] - ref[i]));
        EXPECT(top > 0 && diff <= 1e-14 * top);
    }
    EXPECT(g_tuned.size() == 1);
    g_tuned.clear();
    {
        TcChi0 tc(g, pr, d_C.get(), st);
        tc.impl_->err.upload(&seven, 1, st);
        bool thrown = false;
        try
        {
            tc.run(nullptr, d_G.get(), out.get(), st);
        }
        catch (const Error &)
        {
            thrown = true;
        }
        EXPECT(thrown && g_tuned.empty());
    }
    GB_CUDA(cudaStreamDestroy(st));
    std::printf("ok\n");
    return 0;
}
