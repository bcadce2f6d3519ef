// Device memory behind DevBuf.  A call of a stage entry point or an index build makes a
// dozen buffers and gives them back at its end; allocating and freeing them took 2-3 ms of
// a 5 ms call (100k reads to NAMs) and of an 11 ms build (100 Mbp).  Freed blocks are kept for the
// next allocation instead (devcache.h), up to a bound.  They are given back when an
// allocation fails, before the free device memory is asked for and by sa_device_trim.
#include <cuda_runtime.h>

#include <algorithm>
#include <mutex>

#include "devcache.h"
#include "host_state.h"

namespace sa {

namespace {

constexpr size_t KEEP_MAX = (size_t)8 << 30;  // per device and context, and a 32nd of the device

using CtxGetCurrent = int (*)(void**);                    // cuCtxGetCurrent(CUcontext*)
using CtxGetId = int (*)(void*, unsigned long long*);     // cuCtxGetId(CUcontext, id)

class CudaBackend : public DevBackend {
public:
    // the context's id, which no other context of the process has or had
    bool place(DevPlace& at) override {
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
        return get && get_id && cudaGetDevice(&at.dev) == cudaSuccess && get(&ctx) == 0 && ctx &&
               get_id(ctx, &at.ctx) == 0;
    }
    void* alloc(size_t bytes) override {
        void* p = nullptr;
        if (cudaMalloc(&p, bytes) == cudaSuccess) return p;
        cudaGetLastError();
        return nullptr;
    }
    void free(void* p) override { cudaFree(p); }
    bool idle() override { return cudaDeviceSynchronize() == cudaSuccess; }
    size_t keep_bound() override {
        size_t mem_free = 0, mem_total = 0;
        return cudaMemGetInfo(&mem_free, &mem_total) == cudaSuccess ? std::min(KEEP_MAX, mem_total / 32) : 0;
    }
};

// lives until the process ends: buffers may be freed by other static objects' destructors
DevCache& cache() {
    static CudaBackend* be = new CudaBackend;
    static DevCache* c = new DevCache(*be);
    return *c;
}

}  // namespace

void* dev_alloc(size_t bytes, bool exact) { return cache().alloc(bytes, exact); }
void dev_free(void* p) { cache().free(p); }
size_t dev_trim() { return cache().trim(); }

}  // namespace sa
