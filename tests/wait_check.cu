// Waits on mbarriers that nothing arrives at: prints, per kind of wait, whether it gave up and after how
// many milliseconds.
#include <cstdio>

#include "tc_common.cuh"

using namespace gb::tc;

constexpr uint32_t LIMIT_MS = 200;

template <uint32_t NAP>
__global__ void k_wait(float *out)
{
    __shared__ uint64_t bar;
    if (threadIdx.x == 0)
    {
        mbar_init(&bar, 1);
        fence_barrier_init();
    }
    __syncthreads();
    const uint64_t t0 = globaltimer_ns();
    const bool done = mbar_wait_nap<NAP>(&bar, 0, LIMIT_MS);
    if (threadIdx.x == 0)
    {
        out[0] = done ? 1.0f : 0.0f;
        out[1] = static_cast<float>((globaltimer_ns() - t0) * 1e-6);
    }
}

int main()
{
    float *out = nullptr, h[2];
    if (cudaMalloc(&out, sizeof(h)) != cudaSuccess) return 1;
    for (int nap : {0, 20, 100})
    {
        (nap == 0 ? k_wait<0> : nap == 20 ? k_wait<20> : k_wait<100>)<<<1, 32>>>(out);
        if (cudaMemcpy(h, out, sizeof(h), cudaMemcpyDeviceToHost) != cudaSuccess) return 1;
        std::printf("%d %g %g\n", nap, h[0], h[1]);
    }
    return 0;
}
