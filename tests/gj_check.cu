// The Gauss-Jordan solve of W_c in both forms, columns in shared memory and in global memory, on matrices with
// a row-permuted dominant diagonal, with ties, with a zero column and with a NaN.  One line a case:
//   N M staged kind residual bad,  residual = max |A X - B| / (N max |A| max |X|).
#include <cstdio>
#include <random>
#include <vector>

#include "../librpa_gb300/csrc/gw.cu"

using namespace gb;

namespace {

void run(int N, int M, bool staged, int kind, int batch, cudaStream_t st)
{
    std::mt19937 rng(N + 1000 * M + kind);
    std::uniform_real_distribution<double> u(-1.0, 1.0);
    std::vector<double> A(static_cast<size_t>(batch) * N * N), B(static_cast<size_t>(batch) * N * M), X(B.size());
    for (int b = 0; b < batch; ++b)
    {
        double *a = A.data() + static_cast<size_t>(b) * N * N;
        const double d = std::ceil(4.0 * std::sqrt(static_cast<double>(N)));
        for (int i = 0; i < N; ++i)
            for (int j = 0; j < N; ++j)
            {
                const double x = kind == 1 ? std::nearbyint(1.4 * u(rng)) : u(rng);
                a[static_cast<size_t>(i) * N + j] = x + (j == (i * 7 + 3 + b) % N ? d : 0.0);
            }
        if (kind == 2)
            for (int i = 0; i < N; ++i) a[static_cast<size_t>(i) * N + N / 2] = 0.0;
        if (kind == 3) a[static_cast<size_t>(N / 2) * N + N / 3] = std::nan("");
    }
    for (double &x : B) x = u(rng);
    DevBuf<double> dA(A.size()), dB(B.size());
    DevBuf<int> dbad(1);
    dA.upload(A.data(), A.size(), st);
    dB.upload(B.data(), B.size(), st);
    dbad.zero(st);
    if (staged)
        launch_gj_solve(dA.get(), dB.get(), N, M, batch, dbad.get(), st);
    else
    {
        k_gj_solve<false><<<batch * GJ_CL, 256, gj_smem(N, M, false), st>>>(dA.get(), dB.get(), N, M, dbad.get());
        GB_LAUNCH_CHECK();
    }
    int bad = 0;
    dB.download(X.data(), X.size(), st);
    dbad.download(&bad, 1, st);
    GB_CUDA(cudaStreamSynchronize(st));
    double worst = 0.0;
    for (int b = 0; b < batch && kind < 2; ++b)
    {
        const double *a = A.data() + static_cast<size_t>(b) * N * N, *x = X.data() + static_cast<size_t>(b) * N * M,
                     *y = B.data() + static_cast<size_t>(b) * N * M;
        double ma = 0.0, mx = 0.0, r = 0.0;
        for (long long t = 0; t < static_cast<long long>(N) * N; ++t) ma = std::max(ma, std::fabs(a[t]));
        for (long long t = 0; t < static_cast<long long>(N) * M; ++t) mx = std::max(mx, std::fabs(x[t]));
        std::vector<double> row(M);
        for (int i = 0; i < N; ++i)
        {
            for (int j = 0; j < M; ++j) row[j] = -y[static_cast<size_t>(i) * M + j];
            for (int k = 0; k < N; ++k)
                for (int j = 0; j < M; ++j) row[j] += a[static_cast<size_t>(i) * N + k] * x[static_cast<size_t>(k) * M + j];
            for (int j = 0; j < M; ++j) r = !(std::fabs(row[j]) <= r) ? std::fabs(row[j]) : r;
        }
        r /= N * ma * mx;
        worst = !(r <= worst) ? r : worst;
    }
    std::printf("%d %d %d %d %g %d\n", N, M, staged ? 1 : 0, kind, worst, bad);
}

} // namespace

int main()
{
    cudaStream_t st;
    GB_CUDA(cudaStreamCreateWithFlags(&st, cudaStreamNonBlocking));
    const int sizes[][2] = {{1, 1}, {2, 3}, {3, 3}, {31, 2}, {33, 33}, {33, 40}, {101, 101}, {311, 311}};
    for (const auto &s : sizes)
        for (int kind = 0; kind < 4; ++kind)
            for (bool staged : {true, false})
            {
                GB_REQUIRE(gj_smem(s[0], s[1], true) <= GJ_SMEM_MAX, "a case of the staged form");
                run(s[0], s[1], staged, kind, 3, st);
            }
    // sizes that launch_gj_solve itself sends to the form in global memory
    const int wide[][2] = {{312, 312}, {321, 321}, {400, 397}, {640, 640}};
    for (const auto &s : wide)
        for (int kind = 0; kind < 4; ++kind)
        {
            GB_REQUIRE(gj_smem(s[0], s[1], true) > GJ_SMEM_MAX, "a case of the form in global memory");
            run(s[0], s[1], true, kind, 2, st);
        }
    GB_CUDA(cudaStreamDestroy(st));
    return 0;
}
