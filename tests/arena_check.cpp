// The arenas of device memory kept between calls (librpa_gb300/csrc/device_arena.cpp) over a stand-in for the
// CUDA runtime with a device of a given capacity.  Prints "ok" or the first failure.
#include "../librpa_gb300/csrc/device_arena.cpp"

#include <condition_variable>
#include <cstdlib>
#include <map>
#include <thread>

namespace {
std::mutex g_dev_mu;
std::map<void *, size_t> g_held;
size_t g_capacity = 0;
constexpr size_t GB = size_t(1) << 30;

size_t held()
{
    size_t n = 0;
    for (const auto &h : g_held) n += h.second;
    return n;
}
} // namespace

extern "C" {
cudaError_t cudaMalloc(void **p, size_t n)
{
    std::lock_guard<std::mutex> lk(g_dev_mu);
    if (held() + n > g_capacity) return cudaErrorMemoryAllocation;
    *p = std::malloc(1);
    g_held[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    std::lock_guard<std::mutex> lk(g_dev_mu);
    if (!g_held.erase(p)) std::abort();  // freed twice, or never allocated
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d)
{
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorName(cudaError_t) { return "error"; }
const char *cudaGetErrorString(cudaError_t) { return "error"; }
}

using namespace gb;

#define EXPECT(c)                                        \
    do                                                   \
        if (!(c))                                        \
        {                                                \
            std::printf("line %d: %s\n", __LINE__, #c);  \
            std::exit(1);                                \
        }                                                \
    while (0)

using Buf = DevBuf<unsigned char>;

// a call that holds `first` bytes and lets them go, then one buffer of `then`
bool fits(size_t first, size_t then)
{
    try
    {
        ArenaScope s(nullptr);
        Buf a(first);
        a.release();
        Buf b(then);
        return true;
    }
    catch (const Error &)
    {
        return false;
    }
}

int main()
{
    // within one call, and after it: what is unused makes room
    g_capacity = 100 * GB;
    EXPECT(fits(60 * GB, 90 * GB));
    EXPECT(fits(60 * GB, 100 * GB));
    EXPECT(!fits(1 * GB, 101 * GB));
    {
        ArenaScope s(nullptr);
    }
    EXPECT(held() <= 4 * GB);
    release_idle_arenas();
    EXPECT(held() == 0);

    // a block is taken again, by this call and the next one
    for (int i = 0; i < 2; ++i)
    {
        ArenaScope s(nullptr);
        Buf a(3 * GB);
        void *p = a.get();
        a.release();
        a.alloc(3 * GB - 1000);
        EXPECT(a.get() == p && held() == 3 * GB);
    }

    // buffers that fit the device fit, whatever sizes went before
    {
        ArenaScope s(nullptr);
        Buf a(100 * GB);
        a.release();
        Buf b(60 * GB), c;
        bool room = true;
        try
        {
            c.alloc(40 * GB);
        }
        catch (const Error &)
        {
            room = false;
        }
        EXPECT(room);
    }
    release_idle_arenas();

    // a call on another thread that holds nothing but unused blocks leaves the device to this one
    std::mutex mu;
    std::condition_variable cv;
    int stage = 0;
    std::thread other([&] {
        ArenaScope s(nullptr);
        Buf small(GB);
        {
            Buf big(60 * GB);
        }
        std::unique_lock<std::mutex> lk(mu);
        stage = 1;
        cv.notify_all();
        cv.wait(lk, [&] { return stage == 2; });
        EXPECT(g_held.count(small.get()) == 1);
    });
    {
        std::unique_lock<std::mutex> lk(mu);
        cv.wait(lk, [&] { return stage == 1; });
    }
    const bool fitted = fits(GB, 90 * GB);
    {
        std::lock_guard<std::mutex> lk(mu);
        stage = 2;
    }
    cv.notify_all();
    other.join();
    EXPECT(fitted);

    // many calls at a time on a device too small for them: some fail, nothing is lost or freed twice
    g_capacity = 60 * GB;
    std::vector<std::thread> pool;
    for (int t = 0; t < 8; ++t)
        pool.emplace_back([t] {
            for (int i = 0; i < 200; ++i) fits((3 + (i * 7 + t) % 9) * GB, (12 - i % 5) * GB);
        });
    for (std::thread &t : pool) t.join();
    EXPECT(held() <= 4 * GB);
    release_idle_arenas();
    EXPECT(held() == 0);
    std::printf("ok\n");
    return 0;
}
