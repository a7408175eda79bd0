// memory.cu -- device memory of the library, with a bounded stock of idle blocks.
//
// On a B200 host cudaMalloc of a block of 1 MiB or more takes 0.4 to 0.8 ms
// and cudaFree 0.3 to 1 ms (single calls up to 10 ms), and building an index
// takes some two dozen blocks: 9 of the 13 ms of building an index over
// 200,000 words and asking it once.  Smaller blocks lie together in chunks of
// 2 MiB, which cost as much whenever their sum passes another one: 0.6 ms more
// for each index of 5,000 x 32 or 16,000 x 8.  Freed blocks of 64 KiB on
// therefore wait, up to kPoolCap bytes and kPoolBlocks of them per process, for
// the next request they fit.
//
//   * A block is handed out again only on its own device, and only after the
//     device has been synchronised, as cudaFree would: a waiting block has no
//     work in flight on any stream, so it may serve any stream and thread.
//   * Blocks of a context that is gone (cudaDeviceReset) are forgotten, not
//     reused: contexts are told apart by their id.
//   * The oldest blocks are freed when the stock is over its bound, all of the
//     device's when an allocation fails, and all on gts_memory_release.
#include <cuda.h>
#include <mutex>
#include <unordered_map>
#include <vector>
#include "index.cuh"

namespace gts {

namespace {

constexpr size_t kPoolMin = (size_t)64 << 10;
constexpr size_t kPoolCap = (size_t)4 << 30;
constexpr size_t kPoolBlocks = 1024;           // a request looks at each
constexpr size_t kPoolLarge = (size_t)1 << 20, kPoolRound = (size_t)2 << 20;

struct Block {
    void *p;
    size_t bytes;
    int dev;
    unsigned long long ctx;
};

struct Pool {
    std::mutex m;
    std::vector<Block> idle;                     // oldest first
    std::unordered_map<void *, Block> live;
    size_t idle_bytes = 0;
};

Pool &pool()
{
    static Pool *p = new Pool;   // lives as long as the process: handles may be freed late
    return *p;
}

// Device and id of the current context (0 when it cannot be told: no reuse
// then).  A thread that has made no CUDA call yet has none: cudaFree(nullptr)
// makes the device's current in it, as a call of the runtime would.
void where(int *dev, unsigned long long *ctx)
{
    *dev = 0;
    *ctx = 0;
    cudaFree(nullptr);
    cudaGetDevice(dev);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static const GetId get_id = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &fn, cudaEnableDefault, &found) != cudaSuccess ||
            found != cudaDriverEntryPointSuccess)
            fn = nullptr;
        cudaGetLastError();
        return (GetId)fn;
    }();
    if (get_id && get_id(nullptr, ctx) != CUDA_SUCCESS) *ctx = 0;
}

// Takes the idle blocks of `dev` (all devices: -1) out of the stock.
std::vector<Block> take_idle(Pool &P, int dev)
{
    std::vector<Block> out, rest;
    for (const Block &b : P.idle) (dev < 0 || b.dev == dev ? out : rest).push_back(b);
    P.idle.swap(rest);
    P.idle_bytes = 0;
    for (const Block &b : P.idle) P.idle_bytes += b.bytes;
    return out;
}

void give_back(const std::vector<Block> &blocks)
{
    int cur = 0;
    cudaGetDevice(&cur);
    for (const Block &b : blocks) {
        int dev;
        unsigned long long ctx;
        cudaSetDevice(b.dev);
        where(&dev, &ctx);
        if (ctx == b.ctx) cudaFree(b.p);   // another context: the block went with its own
    }
    cudaSetDevice(cur);
}

}  // namespace

cudaError_t dev_malloc(void **p, size_t bytes)
{
    *p = nullptr;
    if (bytes < kPoolMin) return cudaMalloc(p, bytes ? bytes : 1);
    const size_t unit = bytes < kPoolLarge ? kPoolMin : kPoolRound;
    const size_t want = (bytes + unit - 1) / unit * unit;
    Block b{nullptr, want, 0, 0};
    where(&b.dev, &b.ctx);
    Pool &P = pool();
    {
        std::lock_guard<std::mutex> lock(P.m);
        size_t best = P.idle.size();
        for (size_t i = 0; i < P.idle.size();) {
            const Block &c = P.idle[i];
            if (c.dev == b.dev && c.ctx != b.ctx) {   // of a context that is gone
                P.idle_bytes -= c.bytes;
                P.idle.erase(P.idle.begin() + (long)i);
                if (best > P.idle.size()) best = P.idle.size();
                continue;
            }
            if (c.dev == b.dev && b.ctx != 0 && c.bytes >= want && c.bytes <= want + want / 4 &&
                (best >= P.idle.size() || c.bytes < P.idle[best].bytes))
                best = i;
            i++;
        }
        if (best < P.idle.size()) {
            b = P.idle[best];
            P.idle_bytes -= b.bytes;
            P.idle.erase(P.idle.begin() + (long)best);
            P.live[b.p] = b;
            *p = b.p;
            return cudaSuccess;
        }
    }
    cudaError_t e = cudaMalloc(&b.p, want);
    if (e != cudaSuccess) {
        std::vector<Block> idle;
        {
            std::lock_guard<std::mutex> lock(P.m);
            idle = take_idle(P, b.dev);
        }
        if (!idle.empty()) {
            cudaGetLastError();
            give_back(idle);
            e = cudaMalloc(&b.p, want);
        }
        if (e != cudaSuccess) return e;
    }
    std::lock_guard<std::mutex> lock(P.m);
    P.live[b.p] = b;
    *p = b.p;
    return cudaSuccess;
}

void dev_free(void *p)
{
    if (!p) return;
    Pool &P = pool();
    Block b{nullptr, 0, 0, 0};
    {
        std::lock_guard<std::mutex> lock(P.m);
        auto it = P.live.find(p);
        if (it != P.live.end()) {
            b = it->second;
            P.live.erase(it);
        }
    }
    if (!b.p) {
        cudaFree(p);
        return;
    }
    int cur = 0, dev;
    unsigned long long ctx;
    cudaGetDevice(&cur);
    if (cur != b.dev) cudaSetDevice(b.dev);
    where(&dev, &ctx);
    std::vector<Block> out;
    if (b.ctx == 0 || ctx != b.ctx || b.bytes > kPoolCap || cudaDeviceSynchronize() != cudaSuccess) {
        if (ctx == b.ctx) cudaFree(p);
    } else {
        std::lock_guard<std::mutex> lock(P.m);
        P.idle.push_back(b);
        P.idle_bytes += b.bytes;
        while (P.idle_bytes > kPoolCap || P.idle.size() > kPoolBlocks) {
            out.push_back(P.idle.front());
            P.idle_bytes -= P.idle.front().bytes;
            P.idle.erase(P.idle.begin());
        }
    }
    if (cur != b.dev) cudaSetDevice(cur);
    if (!out.empty()) give_back(out);
}

}  // namespace gts

extern "C" int gts_memory_release(size_t *bytes)
{
    gts::Pool &P = gts::pool();
    std::vector<gts::Block> idle;
    {
        std::lock_guard<std::mutex> lock(P.m);
        if (bytes) *bytes = P.idle_bytes;
        idle = gts::take_idle(P, -1);
    }
    gts::give_back(idle);
    return GTS_OK;
}
