// Device memory behind DevBuf.  A call of a stage entry point or an index build makes a
// dozen buffers and gives them back at its end; allocating and freeing them took 2-3 ms of
// a 5 ms call (100k reads to NAMs) and of an 11 ms build (100 Mbp).  Freed blocks are kept for the
// next allocation instead, up to a bound, per device and context.
//
// A block is kept only once the device is idle (the synchronisation that cudaFree makes
// too), so a block that is handed out again has no work of any stream left on it.  The
// cache is emptied when an allocation fails and before the free device memory is asked
// for; blocks of a context that is gone are forgotten with it.
#include <cuda_runtime.h>

#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <vector>

#include "host_state.h"

namespace sa {

namespace {

struct Block {
    void* p;
    size_t size;
    int dev;
    unsigned long long ctx;
};

constexpr size_t KEEP_MAX = (size_t)8 << 30;  // per process, and a 32nd of the device

std::mutex g_mu;
std::vector<Block> g_free;                     // oldest first
std::unordered_map<void*, Block> g_live;       // blocks that may be kept
size_t g_kept = 0;
size_t g_bound = 0;                            // set by the first release

using CtxGetCurrent = int (*)(void**);                    // cuCtxGetCurrent(CUcontext*)
using CtxGetId = int (*)(void*, unsigned long long*);     // cuCtxGetId(CUcontext, id)

// The current context's id, which no other context of the process has or had; false when
// it cannot be told (nothing is kept then).
bool current_context(int& dev, unsigned long long& id) {
    static CtxGetCurrent get = nullptr;
    static CtxGetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        cudaDriverEntryPointQueryResult q{};
        void *a = nullptr, *b = nullptr;
        if (cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", &a, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess &&
            cudaGetDriverEntryPointByVersion("cuCtxGetId", &b, 12000, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess) {
            get = reinterpret_cast<CtxGetCurrent>(a);
            get_id = reinterpret_cast<CtxGetId>(b);
        } else {
            cudaGetLastError();
        }
    });
    void* ctx = nullptr;
    return get && get_id && cudaGetDevice(&dev) == cudaSuccess && get(&ctx) == 0 && ctx && get_id(ctx, &id) == 0;
}

// Sizes in steps of an eighth of a power of two, so that calls of nearly one size share
// blocks.
size_t round_size(size_t n) {
    if (n <= 4096) return (n + 511) / 512 * 512;
    size_t step = 512;
    while (step * 16 < n) step *= 2;
    return (n + step - 1) / step * step;
}

size_t keep_bound() {  // of the current device
    size_t mem_free = 0, mem_total = 0;
    return cudaMemGetInfo(&mem_free, &mem_total) == cudaSuccess ? std::min(KEEP_MAX, mem_total / 32) : 0;
}

// g_mu held: gives back the blocks of a context, and forgets those of other contexts of the
// device
void drop_all(int dev, unsigned long long ctx) {
    size_t k = 0;
    for (const Block& b : g_free) {
        if (b.dev != dev) {
            g_free[k++] = b;
            continue;
        }
        if (b.ctx == ctx) cudaFree(b.p);
        g_kept -= b.size;
    }
    g_free.resize(k);
}

}  // namespace

void* dev_alloc(size_t bytes) {
    int dev = 0;
    unsigned long long ctx = 0;
    const size_t size = round_size(bytes);
    bool known = current_context(dev, ctx);
    if (known) {
        std::lock_guard<std::mutex> g(g_mu);
        size_t best = g_free.size();
        for (size_t i = 0; i < g_free.size(); i++) {
            const Block& b = g_free[i];
            if (b.dev == dev && b.ctx == ctx && b.size >= size && b.size <= 2 * size &&
                (best == g_free.size() || b.size < g_free[best].size))
                best = i;
        }
        if (best < g_free.size()) {
            const Block b = g_free[best];
            g_free.erase(g_free.begin() + (std::ptrdiff_t)best);
            g_kept -= b.size;
            g_live[b.p] = b;
            return b.p;
        }
    }
    void* p = nullptr;
    cudaError_t e = cudaMalloc(&p, known ? size : bytes);
    if (e == cudaErrorMemoryAllocation && known) {
        cudaGetLastError();
        dev_trim();
        e = cudaMalloc(&p, bytes);
        known = false;
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        return nullptr;
    }
    if (known) {
        std::lock_guard<std::mutex> g(g_mu);
        g_live[p] = Block{p, size, dev, ctx};
    }
    return p;
}

void dev_free(void* p) {
    if (!p) return;
    Block b{nullptr, 0, 0, 0};
    {
        std::lock_guard<std::mutex> g(g_mu);
        auto it = g_live.find(p);
        if (it != g_live.end()) {
            b = it->second;
            g_live.erase(it);
        }
    }
    int dev = 0;
    unsigned long long ctx = 0;
    if (!b.p || !current_context(dev, ctx) || dev != b.dev || ctx != b.ctx || cudaDeviceSynchronize() != cudaSuccess) {
        cudaFree(p);
        return;
    }
    std::lock_guard<std::mutex> g(g_mu);
    if (!g_bound) g_bound = keep_bound();
    const size_t bound = g_bound;
    if (b.size > bound) {
        cudaFree(p);
        return;
    }
    while (g_kept + b.size > bound && !g_free.empty()) {
        const Block old = g_free.front();
        g_free.erase(g_free.begin());
        g_kept -= old.size;
        if (old.dev == dev && old.ctx == ctx) cudaFree(old.p);
    }
    g_free.push_back(b);
    g_kept += b.size;
}

void dev_trim() {
    int dev = 0;
    unsigned long long ctx = 0;
    if (!current_context(dev, ctx)) return;
    std::lock_guard<std::mutex> g(g_mu);
    drop_all(dev, ctx);
}

}  // namespace sa
