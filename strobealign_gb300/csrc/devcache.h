// Freed device blocks kept for the next allocation, up to a bound, per place: a device and
// one of its contexts.  A place's blocks serve, and make room for, that place alone, so what
// another device or context does neither takes nor loses them.  Blocks of a context that is
// gone are forgotten with it (its memory is, and no later context has its id).
#pragma once
#include <cstddef>
#include <cstdint>
#include <mutex>
#include <unordered_map>
#include <vector>

namespace sa {

struct DevPlace {
    int dev = 0;
    unsigned long long ctx = 0;
    bool operator==(const DevPlace& o) const { return dev == o.dev && ctx == o.ctx; }
};

// The calls a cache makes, each of the calling thread's current device and context.
class DevBackend {
public:
    virtual ~DevBackend() = default;
    virtual bool place(DevPlace& p) = 0;  // false: cannot be told (nothing is kept then)
    virtual void* alloc(size_t bytes) = 0;  // null: no memory
    virtual void free(void* p) = 0;
    virtual bool idle() = 0;         // waits for the device's work
    virtual size_t keep_bound() = 0;  // the most that may be kept at the current place
};

class DevCache {
public:
    explicit DevCache(DevBackend& be) : be_(be) {}
    DevCache(const DevCache&) = delete;
    DevCache& operator=(const DevCache&) = delete;

    // exact: for a buffer that stays (an index, a read arena): a block of its own size.
    // Others may get a quarter more (or 64 KB), so that calls of nearly one size share blocks.
    void* alloc(size_t bytes, bool exact = false) {
        DevPlace at;
        if (!be_.place(at)) return be_.alloc(bytes);
        size_t size = round_to_512(bytes);
        {
            std::lock_guard<std::mutex> g(mu_);
            Pool& pool = pool_of(at);
            // a block that is too large to be kept is not rounded up either
            if (!exact && round_size(bytes) <= pool.bound) size = round_size(bytes);
            const size_t most = exact ? size : size + (size / 4 > SLACK_MIN ? size / 4 : SLACK_MIN);
            size_t best = pool.free.size();
            for (size_t i = 0; i < pool.free.size(); i++)
                if (pool.free[i].size >= size && pool.free[i].size <= most &&
                    (best == pool.free.size() || pool.free[i].size < pool.free[best].size))
                    best = i;
            if (best < pool.free.size()) {
                const Block b = pool.take(best);
                live_[b.p] = Live{b.size, at};
                return b.p;
            }
        }
        void* p = be_.alloc(size);
        if (!p) {
            trim();
            return be_.alloc(bytes);  // not kept when it is freed
        }
        std::lock_guard<std::mutex> g(mu_);
        live_[p] = Live{size, at};
        return p;
    }

    // Waits for the device, as freeing does, so that a kept block has no work left on it.
    void free(void* p) {
        if (!p) return;
        Live l;
        {
            std::lock_guard<std::mutex> g(mu_);
            auto it = live_.find(p);
            if (it != live_.end()) {
                l = it->second;
                live_.erase(it);
            }
        }
        DevPlace at;
        if (!l.size || !be_.place(at) || !(at == l.at) || !be_.idle()) {
            be_.free(p);
            return;
        }
        std::lock_guard<std::mutex> g(mu_);
        Pool& pool = pool_of(at);
        if (l.size > pool.bound) {
            be_.free(p);
            return;
        }
        while (pool.kept + l.size > pool.bound) be_.free(pool.take(0).p);  // the oldest
        pool.free.push_back(Block{p, l.size});
        pool.kept += l.size;
    }

    // Gives back what is kept at the current place; its bytes.
    size_t trim() {
        DevPlace at;
        if (!be_.place(at)) return 0;
        std::lock_guard<std::mutex> g(mu_);
        Pool& pool = pool_of(at);
        const size_t bytes = pool.kept;
        while (!pool.free.empty()) be_.free(pool.take(pool.free.size() - 1).p);
        return bytes;
    }

    // bytes kept at a place; blocks handed out that may be kept, of all places
    size_t kept(const DevPlace& at) {
        std::lock_guard<std::mutex> g(mu_);
        for (const Pool& p : pools_)
            if (p.at == at) return p.kept;
        return 0;
    }
    size_t live() {
        std::lock_guard<std::mutex> g(mu_);
        return live_.size();
    }

    static constexpr size_t SLACK_MIN = 64 << 10;
    static size_t round_to_512(size_t n) { return (n + 511) / 512 * 512; }
    // sizes in steps of an eighth of a power of two
    static size_t round_size(size_t n) {
        if (n <= 4096) return round_to_512(n);
        size_t step = 512;
        while (step * 16 < n) step *= 2;
        return (n + step - 1) / step * step;
    }

private:
    struct Block {
        void* p;
        size_t size;
    };
    struct Live {
        size_t size = 0;
        DevPlace at;
    };
    struct Pool {
        DevPlace at;
        size_t bound = 0, kept = 0;
        std::vector<Block> free;  // oldest first
        Block take(size_t i) {
            const Block b = free[i];
            free.erase(free.begin() + (std::ptrdiff_t)i);
            kept -= b.size;
            return b;
        }
    };
    Pool& pool_of(const DevPlace& at) {  // of the current place
        for (Pool& p : pools_)
            if (p.at == at) return p;
        pools_.emplace_back();
        pools_.back().at = at;
        pools_.back().bound = be_.keep_bound();
        return pools_.back();
    }

    DevBackend& be_;
    std::mutex mu_;
    std::vector<Pool> pools_;
    std::unordered_map<void*, Live> live_;
};

}  // namespace sa
