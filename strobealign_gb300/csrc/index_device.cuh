// Device-side StrobemerIndex probes (src/index.rs:127-338, src/partition.rs).
// All lookups are functions of the sorted table only, so any lower-bound search
// returns the reference's partition point.
#pragma once
#include "sa_internal.h"

namespace sa {

__device__ __forceinline__ uint64_t rs_hash(const RefRandstrobe& r) { return r.hash_offset & HASH_MASK; }

// 16-byte vectorised load of one table entry
__device__ __forceinline__ RefRandstrobe load_rs(const RefRandstrobe* rs, uint64_t i) {
    ulonglong2 v = __ldg(reinterpret_cast<const ulonglong2*>(rs) + i);
    RefRandstrobe r;
    r.hash_offset = v.x;
    r.position = (uint32_t)v.y;
    r.ref_index = (uint32_t)(v.y >> 32);
    return r;
}

__device__ __forceinline__ uint64_t load_hash(const RefRandstrobe* rs, uint64_t i) {
    return __ldg(reinterpret_cast<const unsigned long long*>(rs) + 2 * i) & HASH_MASK;
}

// get_masked_from (src/index.rs:159-197); returns UINT64_MAX when absent
__device__ __forceinline__ uint64_t idx_get_masked_from(const DevIndex& ix, uint64_t hash, uint64_t mask,
                                                        bool has_start, uint64_t start) {
    const uint64_t masked = hash & mask;
    const uint64_t top = hash >> (64 - ix.bits);
    ulonglong2 b;
    if ((top & 1) == 0) {
        b = __ldg(reinterpret_cast<const ulonglong2*>(ix.buckets + top));
    } else {
        b.x = __ldg(reinterpret_cast<const unsigned long long*>(ix.buckets) + top);
        b.y = __ldg(reinterpret_cast<const unsigned long long*>(ix.buckets) + top + 1);
    }
    uint64_t ps = has_start ? start : b.x, pe = b.y;
    if (ps >= pe) return UINT64_MAX;
    uint64_t len = pe - ps;
    if (len < 4) {
        for (uint64_t i = 0; i < len; i++) {
            uint64_t h = load_hash(ix.rs, ps + i) & mask;
            if (h == masked) return ps + i;
            if (h > masked) return UINT64_MAX;
        }
        return UINT64_MAX;
    }
    uint64_t lo = 0, hi = len;
    while (lo < hi) {
        uint64_t mid = lo + (hi - lo) / 2;
        if ((load_hash(ix.rs, ps + mid) & mask) < masked) lo = mid + 1;
        else hi = mid;
    }
    if (lo < len && (load_hash(ix.rs, ps + lo) & mask) == masked) return ps + lo;
    return UINT64_MAX;
}

// get_count (src/index.rs:272-295)
__device__ __forceinline__ uint32_t idx_get_count(const DevIndex& ix, uint64_t position, uint64_t mask) {
    uint64_t key = load_hash(ix.rs, position);
    uint64_t masked = key & mask;
    uint64_t top = key >> (64 - ix.bits);
    uint64_t pe = __ldg(reinterpret_cast<const unsigned long long*>(ix.buckets) + top + 1);
    if (pe - position < 8) {
        uint32_t c = 1;
        for (uint64_t p = position + 1; p < pe; p++) {
            if ((load_hash(ix.rs, p) & mask) == masked) c++;
            else break;
        }
        return c;
    }
    uint64_t lo = 0, hi = pe - position;
    while (lo < hi) {
        uint64_t mid = lo + (hi - lo) / 2;
        if ((load_hash(ix.rs, position + mid) & mask) <= masked) lo = mid + 1;
        else hi = mid;
    }
    return (uint32_t)lo;
}

__device__ __forceinline__ uint64_t idx_full_forward(const DevIndex& ix, uint64_t h) {
    return idx_get_masked_from(ix, h, HASH_MASK, false, 0);
}

// is_too_frequent_forward (src/index.rs:298-307): guarded by the index's own cutoff
__device__ __forceinline__ bool idx_too_frequent_forward(const DevIndex& ix, uint64_t pos, uint32_t cutoff) {
    if (pos + ix.filter_cutoff < ix.n) return load_hash(ix.rs, pos) == load_hash(ix.rs, pos + cutoff);
    return false;
}

// is_too_frequent (src/index.rs:309-323)
__device__ __forceinline__ bool idx_too_frequent(const DevIndex& ix, uint64_t pos, uint32_t cutoff, uint64_t hash_rc) {
    if (idx_too_frequent_forward(ix, pos, cutoff)) return true;
    uint64_t rc = idx_full_forward(ix, hash_rc);
    if (rc != UINT64_MAX) {
        if (idx_too_frequent_forward(ix, rc, cutoff)) return true;
        uint64_t c = (uint64_t)idx_get_count(ix, pos, HASH_MASK) + idx_get_count(ix, rc, HASH_MASK);
        return c > cutoff;
    }
    return false;
}

// is_too_frequent_partial (src/index.rs:325-337)
__device__ __forceinline__ bool idx_too_frequent_partial(const DevIndex& ix, uint64_t pos, uint32_t cutoff) {
    if (pos + cutoff < ix.n)
        return (load_hash(ix.rs, pos) & ix.p.main_mask) == (load_hash(ix.rs, pos + cutoff) & ix.p.main_mask);
    return false;
}

// get_count_full (src/index.rs:254-263)
__device__ __forceinline__ uint32_t idx_count_full(const DevIndex& ix, uint64_t pos, uint64_t hash_rc) {
    uint64_t rc = idx_full_forward(ix, hash_rc);
    uint32_t r = rc == UINT64_MAX ? 0 : idx_get_count(ix, rc, HASH_MASK);
    return r + idx_get_count(ix, pos, HASH_MASK);
}

// ------------------------------------------------------------------ latency-parallel probes
// The same answers as idx_full_forward / idx_too_frequent (and, for a hash that is not
// there, idx_get_masked_from / idx_too_frequent_partial) above with fewer dependent memory
// rounds and fewer sectors: a bucket of up to 8 entries is read with independent loads
// instead of a binary search (the lower bound is the number of smaller keys), larger ones
// narrow 8-ary; a hash's repeat test looks first at the entry after it, which those
// loads hold (the table is sorted: no equal neighbour, no run of `cutoff`; a bucket's last
// entry has its neighbour in the next bucket, where only a partial lookup's run can go on, and
// only under a mask shorter than the bucket number), and the reverse complement is looked
// up only for hashes that are there.  Random 32-byte sectors bound the lookups: 1.4 M reads
// of 150 nt on a 310 Mbp human-shaped index took 5.1 ms with both orientations and the
// entries a cutoff further read for every hash, 3.8 ms now.
// bucket range [ps, pe) of a full hash (same directory reads as idx_get_masked_from)
__device__ __forceinline__ void idx_bucket(const DevIndex& ix, uint64_t hash, uint64_t& ps, uint64_t& pe) {
    const uint64_t top = hash >> (64 - ix.bits);
    if ((top & 1) == 0) {
        ulonglong2 b = __ldg(reinterpret_cast<const ulonglong2*>(ix.buckets + top));
        ps = b.x;
        pe = b.y;
    } else {
        ps = __ldg(reinterpret_cast<const unsigned long long*>(ix.buckets) + top);
        pe = __ldg(reinterpret_cast<const unsigned long long*>(ix.buckets) + top + 1);
    }
}

// narrow [lo, hi) to at most 8 entries around the lower bound of key, 8-ary
__device__ __forceinline__ void idx_narrow(const DevIndex& ix, uint64_t key, uint64_t& lo, uint64_t& hi) {
    while (hi - lo > 8) {
        const uint64_t len = hi - lo;
        uint64_t piv[7];
        uint64_t hv[7];
#pragma unroll
        for (int t = 0; t < 7; t++) {
            piv[t] = lo + len * (uint64_t)(t + 1) / 8;
            hv[t] = load_hash(ix.rs, piv[t]);
        }
        uint64_t nlo = lo, nhi = hi;
#pragma unroll
        for (int t = 0; t < 7; t++) {
            if (hv[t] < key) nlo = piv[t] + 1;
        }
#pragma unroll
        for (int t = 6; t >= 0; t--) {
            if (hv[t] >= key) nhi = piv[t];
        }
        // the lower bound lies in [nlo, nhi]; keep one entry past the range so that an
        // equal key at nhi is seen
        lo = nlo;
        hi = nhi < hi ? nhi + 1 : hi;
    }
}

// The entries [lo, hi) of a bucket (hi - lo <= 8), masked; absent ones are UINT64_MAX.
struct Entries8 {
    uint64_t h[8];
};
__device__ __forceinline__ Entries8 idx_load8(const DevIndex& ix, uint64_t lo, uint64_t hi) {
    Entries8 e;
    const uint32_t len = (uint32_t)(hi - lo);
#pragma unroll
    for (int t = 0; t < 8; t++) e.h[t] = (uint32_t)t < len ? load_hash(ix.rs, lo + t) : UINT64_MAX;
    return e;
}

// The first of len entries that equals key under mask (len when none does), and whether
// the one after it does too.
__device__ __forceinline__ uint32_t idx_find8(const Entries8& e, uint32_t len, uint64_t key, uint64_t mask,
                                              bool& next_eq) {
    uint32_t lt = 0, eq = 0;
#pragma unroll
    for (int t = 0; t < 8; t++) {
        const uint64_t h = e.h[t] & mask;
        lt += (uint32_t)t < len && h < key;
        eq += (uint32_t)t < len && h == key;
    }
    next_eq = eq > 1;
    return eq ? lt : len;
}

// One orientation's lookup of a full hash: its first entry (UINT64_MAX when absent) and the
// number of its entries (1, or `many` when the next entry has the hash too: not counted).
// e, len: the bucket's entries when it has no more than 8 (whole), for a partial lookup.
__device__ __forceinline__ uint64_t idx_lookup8(const DevIndex& ix, uint64_t hash, bool& many, Entries8& e,
                                                uint64_t& start, uint32_t& len, bool& whole) {
    const uint64_t key = hash & HASH_MASK;
    uint64_t ps, pe;
    idx_bucket(ix, hash, ps, pe);
    uint64_t lo = ps, hi = ps < pe ? pe : ps;
    whole = hi - lo <= 8;
    if (!whole) idx_narrow(ix, key, lo, hi);
    len = (uint32_t)(hi - lo);
    start = lo;
    e = idx_load8(ix, lo, hi);
    const uint32_t at = idx_find8(e, len, key, HASH_MASK, many);
    if (at == len) return UINT64_MAX;
    // the entry after a narrowed range's last one may have the hash
    if (at + 1 == len && hi < pe) many = load_hash(ix.rs, lo + len) == key;
    return lo + at;
}

// full lookup of h with is_too_frequent (src/index.rs:309-323) using the reverse-complement
// hash hrc; pos = UINT64_MAX when absent, then with `partial` the lookup under main_mask
// with is_too_frequent_partial (src/index.rs:325-337).  found_partial tells which.
__device__ __forceinline__ void idx_full_probe(const DevIndex& ix, uint64_t h, uint64_t hrc, uint32_t cutoff,
                                               bool partial, uint64_t& pos, bool& filtered, bool& found_partial) {
    Entries8 e;
    uint64_t start;
    uint32_t len;
    bool many, whole;
    filtered = found_partial = false;
    const bool always = cutoff == 0;  // an entry is then too frequent by itself
    pos = idx_lookup8(ix, h, many, e, start, len, whole);
    if (pos == UINT64_MAX) {
        if (!partial) return;
        const uint64_t mask = ix.p.main_mask;
        bool next_eq = true;  // whether a run of cutoff entries can start at pos
        if (whole) {
            const uint32_t at = idx_find8(e, len, h & mask, mask, next_eq);
            if (at == len) return;
            pos = start + at;
            // a mask that leaves out leading bits of the bucket number: the run goes on in
            // the next bucket
            if (at + 1 == len && (~mask >> (64 - ix.bits)) != 0) next_eq = true;
        } else {
            pos = idx_get_masked_from(ix, h, mask, false, 0);
            if (pos == UINT64_MAX) return;
        }
        found_partial = true;
        filtered = (next_eq || always) && idx_too_frequent_partial(ix, pos, cutoff);
        return;
    }
    // is_too_frequent: either orientation's run reaches the cutoff, or both together pass it
    if ((many || always) && idx_too_frequent_forward(ix, pos, cutoff)) {
        filtered = true;
        return;
    }
    bool many_rc;
    const uint64_t rc = idx_lookup8(ix, hrc, many_rc, e, start, len, whole);
    if (rc == UINT64_MAX) return;
    if ((many_rc || always) && idx_too_frequent_forward(ix, rc, cutoff)) {
        filtered = true;
        return;
    }
    const uint64_t c = (uint64_t)(many ? idx_get_count(ix, pos, HASH_MASK) : 1) +
                       (many_rc ? idx_get_count(ix, rc, HASH_MASK) : 1);
    filtered = c > cutoff;
}

}  // namespace sa
