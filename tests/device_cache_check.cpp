// The cache of freed device blocks over a fake device (no GPU): random allocations and
// frees from two devices, one with two contexts, with bounds small enough to evict all the time.
// Every block is freed exactly once, at its own place or by its context's end, and what
// is kept stays within the place's own bound.
#include <cstdio>
#include <map>
#include <random>

#include "devcache.h"

using namespace sa;

static long errors = 0;
static void check(bool ok, const char* what) {
    if (!ok && errors++ < 20) std::printf("failed: %s\n", what);
}

struct Fake : DevBackend {
    struct Owned {
        DevPlace at;
        size_t bytes;
    };
    DevPlace now;
    bool known = true;
    size_t bound[2] = {40000, 900000}, capacity = 4 << 20;
    std::map<void*, Owned> owned;
    std::map<int, size_t> used;
    uintptr_t next = 0x1000;
    bool place(DevPlace& p) override {
        p = now;
        return known;
    }
    void* alloc(size_t bytes) override {
        if (used[now.dev] + bytes > capacity) return nullptr;
        used[now.dev] += bytes;
        void* p = reinterpret_cast<void*>(next += 0x1000000);
        owned[p] = Owned{now, bytes};
        return p;
    }
    void free(void* p) override {
        auto it = owned.find(p);
        check(it != owned.end(), "a block is freed once");
        if (it == owned.end()) return;
        used[it->second.at.dev] -= it->second.bytes;
        owned.erase(it);
    }
    bool idle() override { return true; }
    size_t keep_bound() override { return bound[now.dev]; }
};

int main() {
    const DevPlace places[3] = {{0, 1}, {0, 2}, {1, 3}};
    Fake f;
    DevCache c(f);
    std::mt19937 rng(1);
    struct Held {
        void* p;
        size_t bytes;
        int place;
    };
    std::vector<Held> held;
    long reused = 0;
    for (int it = 0; it < 200000; it++) {
        const int x = (int)(rng() % 3);
        f.now = places[x];
        const bool untold = rng() % 50 == 0;
        f.known = !untold;
        if (rng() % 2 && held.size() < 60) {
            // up to beyond either bound
            const size_t bytes = 1 + rng() % (rng() % 20 ? 9000 : 500000);
            const uintptr_t before = f.next;
            const bool exact = rng() % 3 == 0;
            void* p = c.alloc(bytes, exact);
            if (p) {
                reused += f.next == before;
                check(f.owned.count(p) == 1, "a block that is handed out is allocated");
                check(f.owned[p].at == places[x], "a block serves its own place");
                const size_t size = f.owned[p].bytes;
                check(size >= bytes, "a block is large enough");
                if (exact) check(size < bytes + 512, "a block that stays is no larger than asked for");
                else check(size <= DevCache::round_size(bytes) * 5 / 4 ||
                               size <= DevCache::round_size(bytes) + DevCache::SLACK_MIN,
                           "a block is not much larger than asked for");
                for (const Held& h : held) check(h.p != p, "a block is handed out once");
                held.push_back(Held{p, bytes, x});
            }
        } else if (!held.empty()) {
            const size_t i = rng() % held.size();
            // mostly where it was allocated
            if (rng() % 10) f.now = places[held[i].place];
            c.free(held[i].p);
            held[i] = held.back();
            held.pop_back();
        }
        f.known = true;
        for (const DevPlace& p : places) check(c.kept(p) <= f.bound[p.dev], "what is kept stays within the bound");
        // nothing is lost: every allocated block is held by the user or kept
        size_t kept = 0, owned = 0, user = 0;
        for (const DevPlace& p : places) kept += c.kept(p);
        for (const auto& o : f.owned) owned += o.second.bytes;
        for (const Held& h : held) user += f.owned[h.p].bytes;
        check(owned == kept + user, "every block is in use or kept");
        if (it % 5000 == 4999) {
            f.now = places[x];
            const size_t others = kept - c.kept(places[x]);
            c.trim();
            check(c.kept(places[x]) == 0, "a trim gives back all of its place");
            size_t rest = 0;
            for (const DevPlace& p : places) rest += c.kept(p);
            check(rest == others, "a trim leaves other places alone");
        }
    }
    for (const Held& h : held) {
        f.now = places[h.place];
        c.free(h.p);
    }
    for (const DevPlace& p : places) {
        f.now = p;
        c.trim();
    }
    check(f.owned.empty() && c.live() == 0, "all is given back at the end");
    // an allocation that does not fit gives back what is kept and tries again
    f.now = places[2];
    f.capacity = 100000;
    c.free(c.alloc(60000));
    check(c.kept(places[2]) > 0, "a block is kept");
    void* p = c.alloc(99000);
    check(p != nullptr && c.kept(places[2]) == 0, "kept blocks make room");
    check(c.alloc(2000) == nullptr, "no memory is reported");
    c.free(p);
    check(f.owned.empty(), "the block that took the retry is given back");
    std::printf("reused %ld errors %ld\n", reused, errors);
    return errors || reused < 1000;
}
