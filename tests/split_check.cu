// Splits pairs of floats read from a file as the chi0 contraction does: writes the bits of hi, mid and lo of
// each value.
#include <cstdio>
#include <vector>

#include "tc_common.cuh"

__global__ void k_split(const float2 *x, int n, uint32_t *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) gb::tc::split3_pair(x[i], out[3 * i], out[3 * i + 1], out[3 * i + 2]);
}

int main(int argc, char **argv)
{
    if (argc != 3) return 2;
    std::FILE *f = std::fopen(argv[1], "rb");
    if (!f) return 2;
    std::vector<float2> x;
    for (float2 v; std::fread(&v, sizeof(v), 1, f) == 1;) x.push_back(v);
    std::fclose(f);
    const int n = static_cast<int>(x.size());
    float2 *d = nullptr;
    uint32_t *o = nullptr;
    if (n == 0 || cudaMalloc(&d, sizeof(float2) * n) != cudaSuccess || cudaMalloc(&o, 12ull * n) != cudaSuccess) return 1;
    if (cudaMemcpy(d, x.data(), sizeof(float2) * n, cudaMemcpyHostToDevice) != cudaSuccess) return 1;
    k_split<<<(n + 255) / 256, 256>>>(d, n, o);
    std::vector<uint32_t> h(3ull * n);
    if (cudaMemcpy(h.data(), o, 4 * h.size(), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
    f = std::fopen(argv[2], "wb");
    if (!f || std::fwrite(h.data(), 4, h.size(), f) != h.size()) return 2;
    std::fclose(f);
    return 0;
}
