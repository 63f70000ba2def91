// Device memory kept between calls (declared in common.h).
//
// A call that allocates its work buffers with cudaMalloc and frees them with cudaFree pays for both in
// the driver, and cudaFree waits for the whole device, so calls on other host threads run one after the
// other.  Here a call takes an arena for its duration (ArenaScope); a DevBuf made meanwhile on that
// thread takes its memory from the arena and gives it back to it.  One arena serves one call at a time,
// and a call's GPU work is on one stream, so a block given back may be taken again at once: the stream
// orders the two uses.  The scope's end waits for that stream before the arena goes back to the idle
// list.  Buffers that outlive a call (the handler's staged inputs) are made under ArenaPause and owned
// by cudaMalloc as before.
//
// Bounded: idle arenas hold at most kIdleBytes together (a call's largest blocks go back to the driver
// first), a block serves no request that leaves more than kWaste of it unused, an allocation that fails gives
// back all that is unused, in idle arenas and in those of running calls, and tries again, and
// librpa_finalize_global and the destruction of the last handler give the idle ones back too.
// One GB300, a pass: 12 molecules in one batch call 90 -> 45 ms, one molecule 10.0 -> 8.4.
#include <algorithm>
#include <memory>

#include "common.h"

namespace gb {

namespace {
constexpr size_t kIdleBytes = size_t(4) << 30;
constexpr size_t kWaste = size_t(256) << 20;

struct Block
{
    void *p;
    size_t bytes;
    bool used;
};

std::mutex g_arena_mu;  // the two lists below and the blocks of every arena
std::mutex g_free_mu;   // taken first: blocks on their way back to the driver
} // namespace

class DeviceArena
{
public:
    int device = -1;
    std::vector<Block> blocks;

    size_t bytes() const
    {
        size_t n = 0;
        for (const Block &b : blocks) n += b.bytes;
        return n;
    }
    // takes out unused blocks, the largest first, until at most `keep` bytes are held; the caller frees them
    void trim(size_t keep, std::vector<void *> &out)
    {
        std::sort(blocks.begin(), blocks.end(), [](const Block &a, const Block &b) { return a.bytes < b.bytes; });
        size_t held = bytes();
        for (size_t i = blocks.size(); i-- > 0 && held > keep;)
        {
            if (blocks[i].used) continue;
            out.push_back(blocks[i].p);
            held -= blocks[i].bytes;
            blocks.erase(blocks.begin() + static_cast<std::ptrdiff_t>(i));
        }
    }
};

namespace {
// arenas without a call, newest last, and those of running calls; never destroyed, the driver may be gone by then
std::vector<std::unique_ptr<DeviceArena>> &g_idle = *new std::vector<std::unique_ptr<DeviceArena>>;
std::vector<DeviceArena *> &g_running = *new std::vector<DeviceArena *>;
thread_local DeviceArena *t_arena = nullptr;
} // namespace

void release_idle_arenas()
{
    std::lock_guard<std::mutex> fr(g_free_mu);
    std::vector<void *> out;
    {
        std::lock_guard<std::mutex> lk(g_arena_mu);
        for (auto &a : g_idle) a->trim(0, out);
        g_idle.clear();
    }
    for (void *p : out) cudaFree(p);
}

void *device_malloc(size_t bytes)
{
    void *p = nullptr;
    cudaError_t e = cudaMalloc(&p, bytes);
    if (e == cudaErrorMemoryAllocation)
    {
        int dev = -1;
        GB_CUDA(cudaGetDevice(&dev));
        std::lock_guard<std::mutex> fr(g_free_mu);
        // again while there is something to give back: other calls give and take meanwhile
        for (int dry = 0; e == cudaErrorMemoryAllocation && dry < 3;)
        {
            cudaGetLastError();
            std::vector<void *> out;
            {
                std::lock_guard<std::mutex> lk(g_arena_mu);
                for (auto &a : g_idle) a->trim(0, out);
                for (DeviceArena *a : g_running)
                    if (a->device == dev) a->trim(0, out);
            }
            dry += out.empty();
            // a block was given back after the last launch that uses it, on whatever stream of whatever call
            if (!out.empty()) cudaDeviceSynchronize();
            for (void *q : out) cudaFree(q);
            e = cudaMalloc(&p, bytes);
        }
    }
    GB_CUDA(e);
    return p;
}

DeviceArena *current_arena() { return t_arena; }

void *arena_take(DeviceArena *a, size_t bytes)
{
    bytes = std::max<size_t>((bytes + 511) / 512 * 512, 512);
    {
        // the smallest free block that fits without wasting more than its half (small blocks: whatever fits 4 KB)
        std::lock_guard<std::mutex> lk(g_arena_mu);
        const size_t most = std::max<size_t>(bytes + std::min(bytes, kWaste), 4096);
        Block *best = nullptr;
        for (Block &b : a->blocks)
            if (!b.used && b.bytes >= bytes && b.bytes <= most && (!best || b.bytes < best->bytes)) best = &b;
        if (best)
        {
            best->used = true;
            return best->p;
        }
    }
    void *p = device_malloc(bytes);
    std::lock_guard<std::mutex> lk(g_arena_mu);
    a->blocks.push_back({p, bytes, true});
    return p;
}

void arena_give(DeviceArena *a, void *p)
{
    std::lock_guard<std::mutex> lk(g_arena_mu);
    for (Block &b : a->blocks)
        if (b.p == p) b.used = false;
}

ArenaScope::ArenaScope(cudaStream_t st) : st_(st), prev_(t_arena)
{
    int dev = -1;
    GB_CUDA(cudaGetDevice(&dev));
    std::unique_ptr<DeviceArena> a;
    std::lock_guard<std::mutex> lk(g_arena_mu);
    for (size_t i = g_idle.size(); i-- > 0 && !a;)
        if (g_idle[i]->device == dev)
        {
            a = std::move(g_idle[i]);
            g_idle.erase(g_idle.begin() + static_cast<std::ptrdiff_t>(i));
        }
    if (!a) a = std::make_unique<DeviceArena>();
    a->device = dev;
    g_running.push_back(a.get());
    t_arena = a.release();
}

ArenaScope::~ArenaScope()
{
    cudaStreamSynchronize(st_);  // nothing of this call still uses a block (an error was or will be reported)
    std::unique_ptr<DeviceArena> a(t_arena);
    t_arena = prev_;
    std::lock_guard<std::mutex> fr(g_free_mu);
    std::vector<void *> out;
    {
        std::lock_guard<std::mutex> lk(g_arena_mu);
        g_running.erase(std::find(g_running.begin(), g_running.end(), a.get()));
        size_t idle = 0;
        for (const auto &x : g_idle) idle += x->bytes();
        a->trim(idle < kIdleBytes ? kIdleBytes - idle : 0, out);
        g_idle.push_back(std::move(a));
    }
    for (void *p : out) cudaFree(p);
}

ArenaPause::ArenaPause() : prev_(t_arena) { t_arena = nullptr; }
ArenaPause::~ArenaPause() { t_arena = prev_; }

} // namespace gb
