// NAM finding on the GPU: the reference's get_nams_by_chaining (src/nam.rs:138-166)
// for a whole batch of reads, one launch per stage:
//
//   k_seed          warp per read: canonical syncmers + forward / reverse-complement
//                   randstrobes (src/seeding/{syncmers,strobes,mod}.rs)
//   k_probe         warp per read, a randstrobe per lane: index probes with the repeat
//                   filter (src/hit.rs)
//   k_hits          warp per read: hits, global and local rescue, orientation choice
//                   (src/hit.rs, src/chainer.rs:205-216)
//   k_anchors       warp per read: anchors counted and written (src/chainer.rs:304-384)
//   segmented sort  (ref_id, ref_start, query_start) packed in a u64 key
//   k_chain_long_prep, k_chain_big, k_chain_long   orientations of over 96 anchors, their
//                   position clusters scored apart, beside k_chain4
//   k_chain4        warp per eight read orientations: anchor sort and dedup, collinear
//                   chaining DP with the reference's early-break rules evaluated as a
//                   prefix max over the candidates (four lanes per orientation), chain
//                   extraction
//                   (src/chainer.rs:85-180, 386-449)
//   k_nam_compact   warp per read: NAM ids in push order, stable sort by score
//                   (src/nam.rs:168-170); reads with more than 32 NAMs through a
//                   segmented stable sort and k_nam_gather
//
// Floating point follows the reference exactly: f32 with explicit round-to-nearest
// intrinsics (no contraction) and log2(d + 1) from a table built with the host's
// log2f, the function the reference calls.
#include <cub/cub.cuh>
#include <type_traits>

#include <cmath>
#include <mutex>
#include <string>

#include "index_device.cuh"
#include "pipeline.h"

namespace sa {

namespace {

constexpr uint32_t FULL = 0xffffffffu;
constexpr int WARPS_PER_BLOCK = 8;

__device__ __forceinline__ uint32_t lane_id() { return threadIdx.x & 31; }
__device__ __forceinline__ uint32_t lanemask_lt() { return (1u << lane_id()) - 1; }

// A, C, G, T or U, in either case: 0 to 3; anything else 4
__device__ __forceinline__ uint32_t nt_code(uint8_t c) {
    const uint32_t u = c & 0xdfu, x = u - 'A';
    return x < 32 && ((0x180045u >> x) & 1) ? ((u >> 1) ^ (u >> 2)) & 3 : 4;
}

// ------------------------------------------------------------------ seeding
// A read packed 2 bits per base (base i at bits 2(i % 32) of word i / 32) with one
// N flag bit per base, so that any window of up to 32 bases comes out in O(1).
__device__ __forceinline__ uint64_t spread_bits(uint32_t v) {
    uint64_t x = v;
    x = (x | (x << 16)) & 0x0000FFFF0000FFFFULL;
    x = (x | (x << 8)) & 0x00FF00FF00FF00FFULL;
    x = (x | (x << 4)) & 0x0F0F0F0F0F0F0F0FULL;
    x = (x | (x << 2)) & 0x3333333333333333ULL;
    x = (x | (x << 1)) & 0x5555555555555555ULL;
    return x;
}
__device__ __forceinline__ uint64_t window_bits(const uint64_t* packed, uint32_t q) {
    const uint32_t* w = reinterpret_cast<const uint32_t*>(packed) + (q >> 4);
    const uint32_t sh = 2 * (q & 15), w1 = w[1];
    return (uint64_t)__funnelshift_r(w1, w[2], sh) << 32 | __funnelshift_r(w[0], w1, sh);
}
__device__ __forceinline__ uint32_t window_n(const uint32_t* nflags, uint32_t q) {
    const uint32_t w = q >> 5;
    return (uint32_t)((((uint64_t)nflags[w + 1] << 32) | nflags[w]) >> (q & 31));
}
__device__ __forceinline__ uint64_t low_mask(uint32_t bits) { return bits >= 64 ? ~0ULL : (1ULL << bits) - 1; }
// the n-base window w (base 0 in the low bits) as the reference encodes it: forward
// with the first base most significant, reverse complement with the first base least
__device__ __forceinline__ void kmer_codes(uint64_t w, uint32_t n, uint64_t& fw, uint64_t& rc) {
    const uint64_t m = low_mask(2 * n);
    w &= m;
    rc = ~w & m;
    uint64_t r = __brevll(w);
    r = ((r >> 1) & 0x5555555555555555ULL) | ((r & 0x5555555555555555ULL) << 1);
    fw = r >> (64 - 2 * n);
}

// src/seeding/syncmers.rs:171-237: a syncmer at p requires an N-free k-mer window
// and the (t-1)-th of its k-s+1 s-mer hashes to equal their minimum.
// Bound by the instructions issued. The bases are packed for 32 words at a time by a lane
// each; the windows' minima take log2 steps; the k-mers of syncmers are hashed once their
// positions are gathered, by full warps; and the syncmers stay in shared memory, unless a
// read has more than SEED_SYNCMERS (104, what the warp's 2 KB leave room for), whose
// syncmers all go to global memory. 100,000 reads of 150 nt take 0.207 ms; 0.300 ms (2850
// warp instructions a read) with a shuffle per window position, each chunk's few syncmers
// hashed at once and the syncmers in global memory.
constexpr uint32_t SEED_SYNCMERS = 104;
// CHECKED (offsets supplied by a caller, not built here): a read whose offsets are
// decreasing, end past `total` or span more than MAX_READ_LEN gets the count
// UINT32_MAX in both orientations and is not touched otherwise.
template <bool CHECKED>
__global__ void __launch_bounds__(256) k_seed(const uint8_t* __restrict__ seq, const uint64_t* __restrict__ off,
                                              uint32_t n, SeedParams p, uint64_t* syn_hash, uint32_t* syn_pos,
                                              uint64_t* qr_hash, uint64_t* qr_hash_rc, uint32_t* qr_start,
                                              uint32_t* qr_end, uint64_t total, uint32_t* n_rs) {
    extern __shared__ uint8_t smem[];
    // per warp: packed bases and N flags (MAX_READ_LEN / 32 + 2 words each), then syncmers
    constexpr uint32_t WORDS = MAX_READ_LEN / 32 + 2;
    static_assert(WORDS * 12 + SEED_SYNCMERS * 12 <= MAX_READ_LEN && WORDS % 2 == 0, "a warp's shared memory");
    uint64_t* packed = reinterpret_cast<uint64_t*>(smem + (threadIdx.x / 32) * MAX_READ_LEN);
    uint32_t* nflags = reinterpret_cast<uint32_t*>(packed + WORDS);
    uint64_t* sh_hash = reinterpret_cast<uint64_t*>(nflags + WORDS);
    uint32_t* sh_pos = reinterpret_cast<uint32_t*>(sh_hash + SEED_SYNCMERS);
    const uint32_t lane = lane_id();
    const uint32_t span = p.k - p.s, step = 32 - span, all = (uint32_t)low_mask(span + 1);
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; r < n; r += nwarps) {
        const uint64_t o = off[r];
        if (CHECKED) {
            const uint64_t e = off[r + 1];
            if (e < o || e > total || e - o > MAX_READ_LEN) {
                if (lane == 0) {
                    n_rs[2 * r] = UINT32_MAX;
                    n_rs[2 * r + 1] = UINT32_MAX;
                }
                continue;
            }
        }
        const uint32_t L = (uint32_t)(off[r + 1] - o);
        const uint32_t nwords = (L + 31) / 32;
        for (uint32_t w0 = 0; w0 <= nwords; w0 += 32) {
            uint32_t b0 = 0, b1 = 0, bn = 0;
            const uint32_t wn = nwords + 1 - w0 < 32 ? nwords + 1 - w0 : 32;
            for (uint32_t w = 0; w < wn; w++) {
                const uint32_t i = (w0 + w) * 32 + lane;
                const uint32_t cc = i < L ? nt_code(seq[o + i]) : 0;
                const uint32_t v0 = __ballot_sync(FULL, cc & 1), v1 = __ballot_sync(FULL, cc & 2);
                const uint32_t vn = __ballot_sync(FULL, cc > 3);
                if (lane == w) {
                    b0 = v0;
                    b1 = v1;
                    bn = vn;
                }
            }
            if (lane < wn) {
                packed[w0 + lane] = spread_bits(b0) | (spread_bits(b1) << 1);
                nflags[w0 + lane] = bn;
            }
        }
        __syncwarp();
        uint32_t nsyn = 0;
        for (uint32_t c = 0; L >= p.k && c + p.k <= L; c += step) {
            const uint32_t q = c + lane;
            bool v = q + p.s <= L;
            uint64_t fw = 0, rc = 0;
            if (v) {
                v = (window_n(nflags, q) & (uint32_t)low_mask(p.s)) == 0;
                kmer_codes(window_bits(packed, q), p.s, fw, rc);
            }
            const uint64_t hs = v ? xxh64_u64(fw < rc ? fw : rc) : 0;
            const uint32_t good = __ballot_sync(FULL, v) >> lane;
            // the window's minimum (lanes >= step: not used)
            uint64_t mn = hs;
            uint32_t len = 1;
            for (; 2 * len <= span + 1; len *= 2) {
                const uint64_t h = __shfl_down_sync(FULL, mn, len);
                mn = h < mn ? h : mn;
            }
            if (len <= span) {
                const uint64_t h = __shfl_down_sync(FULL, mn, span + 1 - len);
                mn = h < mn ? h : mn;
            }
            const uint64_t ht = p.t - 1 <= span ? __shfl_down_sync(FULL, hs, p.t - 1) : 0;
            const bool is_syn = lane < step && q + p.k <= L && (good & all) == all && ht == mn;
            const uint32_t bal = __ballot_sync(FULL, is_syn);
            if (is_syn) {
                const uint32_t idx = nsyn + __popc(bal & lanemask_lt());
                if (idx < SEED_SYNCMERS) sh_pos[idx] = q;
                else syn_pos[o + idx] = q;
            }
            nsyn += __popc(bal);
        }
        __syncwarp();
        const bool in_shared = nsyn <= SEED_SYNCMERS;
        if (!in_shared)
            for (uint32_t i = lane; i < SEED_SYNCMERS; i += 32) syn_pos[o + i] = sh_pos[i];
        uint32_t* spos = in_shared ? sh_pos : syn_pos + o;
        uint64_t* shash = in_shared ? sh_hash : syn_hash + o;
        __syncwarp();
        for (uint32_t i = lane; i < nsyn; i += 32) {
            const uint32_t pos = spos[i];
            uint64_t kf, kr;
            kmer_codes(window_bits(packed, pos), p.k, kf, kr);
            shash[i] = xxh64_u64(kf < kr ? kf : kr);
            spos[i] = (pos << 1) | (uint32_t)(kf <= kr);
        }
        __syncwarp();
        const uint32_t nr = L < p.w_max ? 0 : nsyn;
        // forward randstrobes (src/seeding/strobes.rs:145-176)
        for (uint32_t i = lane; i < nr; i += 32) {
            uint64_t h1 = shash[i];
            uint32_t p1 = spos[i];
            uint32_t pos1 = p1 >> 1;
            uint32_t best = UINT32_MAX;
            uint64_t h2 = h1;
            uint32_t p2 = p1;
            for (uint32_t j = i + p.w_min; j <= i + p.w_max && j < nsyn; j++) {
                uint32_t pj = spos[j];
                if ((pj >> 1) > pos1 + p.max_dist) break;
                uint64_t hj = shash[j];
                const uint32_t ones = __popcll((h1 ^ hj) & p.q);
                if (ones < best) { best = ones; h2 = hj; p2 = pj; }
            }
            uint64_t f1 = p1 & 1, f2 = p2 & 1;
            qr_hash[o + i] = randstrobe_hash(h1, h2, f1, f2, p);
            qr_hash_rc[o + i] = randstrobe_hash(h2, h1, f1 ^ 1, f2 ^ 1, p);
            qr_start[o + i] = pos1;
            qr_end[o + i] = (p2 >> 1) + p.k;
        }
        // reverse-complement randstrobes from the reversed syncmer list (src/seeding/mod.rs:53-73)
        for (uint32_t ir = lane; ir < nr; ir += 32) {
            uint32_t i = nsyn - 1 - ir;
            uint64_t h1 = shash[i];
            uint32_t p1 = spos[i];
            uint32_t pos1 = L - (p1 >> 1) - p.k;
            uint32_t f1 = (p1 & 1) ^ 1;
            uint32_t best = UINT32_MAX;
            uint64_t h2 = h1;
            uint32_t pos2 = pos1, f2 = f1;
            for (uint32_t d = p.w_min; d <= p.w_max && d <= i; d++) {
                uint32_t j = i - d;
                uint32_t pj = spos[j];
                uint32_t posj = L - (pj >> 1) - p.k;
                if (posj > pos1 + p.max_dist) break;
                uint64_t hj = shash[j];
                const uint32_t ones = __popcll((h1 ^ hj) & p.q);
                if (ones < best) { best = ones; h2 = hj; pos2 = posj; f2 = (pj & 1) ^ 1; }
            }
            qr_hash[total + o + ir] = randstrobe_hash(h1, h2, f1, f2, p);
            qr_hash_rc[total + o + ir] = randstrobe_hash(h2, h1, f1 ^ 1, f2 ^ 1, p);
            qr_start[total + o + ir] = pos1;
            qr_end[total + o + ir] = pos2 + p.k;
        }
        if (lane == 0) {
            n_rs[2 * r] = nr;
            n_rs[2 * r + 1] = nr;
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ hits
struct HitsCounts {
    uint32_t fnf = 0, ff = 0, ffound = 0, pnf = 0, pf = 0, pfound = 0, rescued = 0;
};

__device__ __forceinline__ uint32_t warp_sum(uint32_t v) {
    for (int d = 16; d > 0; d >>= 1) v += __shfl_xor_sync(FULL, v, d);
    return v;
}

// count used by rescue_least_frequent (src/hit.rs:96-107), cached per hit
__device__ __forceinline__ uint32_t hit_count(const DevIndex& ix, uint64_t pos, uint32_t info, uint64_t hash_rc) {
    if (info & 2) return idx_get_count(ix, pos, ix.p.main_mask);
    return idx_count_full(ix, pos, hash_rc);
}

// rescue_least_frequent (src/hit.rs:88-125) over hits [s, e) of one read-orientation.
// Whole warp participates; returns the number rescued (valid in all lanes).
__device__ uint32_t warp_rescue_least_frequent(const DevIndex& ix, uint32_t s, uint32_t e, uint32_t to_rescue,
                                               uint32_t threshold, const uint64_t* hit_pos, uint32_t* hit_info,
                                               uint32_t* cache, const uint64_t* rs_hash_rc) {
    for (uint32_t h = s + lane_id(); h < e; h += 32) {
        if (cache[h] == 0xffffffffu) {
            uint32_t info = hit_info[h];
            cache[h] = hit_count(ix, hit_pos[h], info, rs_hash_rc[info >> 3]);
        }
    }
    __syncwarp();
    uint32_t rescued = 0;
    if (lane_id() == 0) {
        // stable ascending sort by count == pick (count, index) in lexicographic order
        uint32_t pc = 0, pi = 0;
        bool have_prev = false;
        for (uint32_t t = 0; t < to_rescue; t++) {
            uint32_t bc = 0xffffffffu, bi = 0xffffffffu;
            for (uint32_t h = s; h < e; h++) {
                uint32_t c = cache[h];
                if (c > threshold) continue;
                if (have_prev && (c < pc || (c == pc && h <= pi))) continue;
                if (c < bc || (c == bc && h < bi)) { bc = c; bi = h; }
            }
            if (bi == 0xffffffffu) break;
            uint32_t info = hit_info[bi];
            rescued += (info >> 2) & 1;
            hit_info[bi] = info & ~4u;
            pc = bc;
            pi = bi;
            have_prev = true;
        }
    }
    __syncwarp();
    return __shfl_sync(FULL, rescued, 0);
}

// Per-randstrobe index probes of find_hits' first pass (src/hit.rs:143-187), ahead of
// k_hits: lanes run over both orientations' randstrobes of a read together, each lane
// one probe with the latency-parallel lookups.  Writes, per randstrobe slot, the table
// position (UINT64_MAX if absent) and PROBE_* flags; k_hits compacts them in place.  Bound by
// the latency of random table sectors: five blocks an SM in 48 registers (four in 57: 100,000
// reads spend 1.62 ms in the NAM stage instead of 1.59; six in 40 spill: 1.63).
constexpr uint32_t PROBE_FULL = 1, PROBE_PARTIAL = 2, PROBE_FILTERED = 4;

__global__ void __launch_bounds__(256, 5) k_probe(DevIndex ix, const uint64_t* __restrict__ off, uint32_t n,
                                               uint64_t total, uint32_t mcs, const uint64_t* __restrict__ qr_hash,
                                               const uint64_t* __restrict__ qr_hash_rc,
                                               const uint32_t* __restrict__ n_rs, uint64_t* __restrict__ hit_pos,
                                               uint32_t* __restrict__ hit_info) {
    const uint32_t lane = lane_id();
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    const uint32_t cutoff = ix.filter_cutoff;
    for (uint32_t r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; r < n; r += nwarps) {
        const uint64_t o = off[r];
        const uint32_t n0 = n_rs[2 * r], n1 = n_rs[2 * r + 1];
        for (uint32_t j = lane; j < n0 + n1; j += 32) {
            const uint32_t ori = j >= n0;
            const uint64_t slot = ori * total + o + (j - ori * n0);
            const uint64_t h = qr_hash[slot];
            uint64_t pos;
            bool filtered, partial;
            idx_full_probe(ix, h, qr_hash_rc[slot], cutoff, mcs == SA_MCS_ALWAYS, pos, filtered, partial);
            uint32_t flags = 0;
            if (pos != UINT64_MAX)
                flags = (partial ? PROBE_PARTIAL : PROBE_FULL) | (filtered ? PROBE_FILTERED : 0u);
            hit_pos[slot] = pos;
            hit_info[slot] = flags;
        }
    }
}

// find_hits (src/hit.rs:129-333) for both orientations of each read, then the
// orientation heuristic (src/chainer.rs:205-216, src/hit.rs:76-81).  The first pass
// reads k_probe's per-slot answers.  Counts come from ballots, and the walk over filtered
// stretches, hit after hit on one lane, is entered only when some stretch is long enough
// (1.4 M reads: 4.0 ms with six warp sums per orientation and the walk for every read, 2.2 ms).
__global__ void __launch_bounds__(256) k_hits(DevIndex ix, const uint64_t* __restrict__ off, uint32_t n,
                                              uint64_t total, uint32_t mcs, uint32_t rescue_distance,
                                              const uint64_t* qr_hash, const uint64_t* qr_hash_rc,
                                              const uint32_t* qr_start, const uint32_t* qr_end,
                                              const uint32_t* n_rs, uint64_t* hit_pos, uint32_t* hit_info,
                                              uint32_t* cache, uint32_t* n_hits, uint8_t* orient,
                                              NamDetailsRec* details) {
    const uint32_t lane = lane_id();
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    const uint32_t cutoff = ix.filter_cutoff;
    for (uint32_t r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; r < n; r += nwarps) {
        const uint64_t o = off[r];
        HitsCounts hc[2];
        for (int ori = 0; ori < 2; ori++) {
            const uint64_t b = ori * total + o;
            const uint32_t nr = n_rs[2 * r + ori];
            uint32_t nh = 0;
            HitsCounts d;  // the same in every lane: counted by ballots
            const bool do_full = mcs != SA_MCS_FIRST_STROBE;
            // pass 1: full lookups (with partial fallback under MCS always), probed by
            // k_probe; compacted in place (a slot is written only after every lane of
            // the round has read its own)
            if (do_full) {
                for (uint32_t c = 0; c < nr; c += 32) {
                    uint32_t i = c + lane;
                    uint32_t fl = 0;
                    uint64_t pos = UINT64_MAX;
                    if (i < nr) {
                        fl = hit_info[b + i];
                        pos = hit_pos[b + i];
                    }
                    const bool filtered = fl & PROBE_FILTERED, partial = fl & PROBE_PARTIAL;
                    const bool is_hit = fl & (PROBE_FULL | PROBE_PARTIAL);
                    const uint32_t in = __ballot_sync(FULL, i < nr), full = __ballot_sync(FULL, fl & PROBE_FULL),
                                   part = __ballot_sync(FULL, partial), filt = __ballot_sync(FULL, filtered);
                    d.ff += __popc(full & filt);
                    d.ffound += __popc(full & ~filt);
                    d.fnf += __popc(in & ~full);
                    if (mcs == SA_MCS_ALWAYS) {
                        d.pf += __popc(part & filt);
                        d.pfound += __popc(part & ~filt);
                        d.pnf += __popc(in & ~full & ~part);
                    }
                    const uint32_t bal = full | part;
                    __syncwarp();
                    if (is_hit) {
                        uint32_t idx = nh + __popc(bal & lanemask_lt());
                        hit_pos[b + idx] = pos;
                        hit_info[b + idx] = (i << 3) | (filtered ? 4u : 0u) | (partial ? 2u : 0u) | 1u;
                    }
                    nh += __popc(bal);
                }
            }
            bool partial_pass = mcs == SA_MCS_FIRST_STROBE || (mcs == SA_MCS_RESCUE && d.ff + d.ffound == 0);
            if (partial_pass) {
                for (uint32_t c = 0; c < nr; c += 32) {
                    uint32_t i = c + lane;
                    bool is_hit = false, filtered = false;
                    uint64_t pos = UINT64_MAX;
                    if (i < nr) {
                        pos = idx_get_masked_from(ix, qr_hash[b + i], ix.p.main_mask, false, 0);
                        if (pos != UINT64_MAX) {
                            is_hit = true;
                            filtered = idx_too_frequent_partial(ix, pos, cutoff);
                        }
                    }
                    uint32_t bal = __ballot_sync(FULL, is_hit);
                    const uint32_t in = __ballot_sync(FULL, i < nr), filt = __ballot_sync(FULL, filtered);
                    d.pf += __popc(bal & filt);
                    d.pfound += __popc(bal & ~filt);
                    d.pnf += __popc(in & ~bal);
                    if (is_hit) {
                        uint32_t idx = nh + __popc(bal & lanemask_lt());
                        hit_pos[b + idx] = pos;
                        hit_info[b + idx] = (i << 3) | (filtered ? 4u : 0u) | 2u | 1u;
                    }
                    nh += __popc(bal);
                }
            }
            __syncwarp();
            // rescue (src/hit.rs:270-304)
            uint32_t total_hits = d.pf + d.pfound + d.ff + d.ffound;
            uint32_t nonrep = d.ffound + d.pfound;
            float frac = total_hits > 0 ? __fdiv_rn(__uint2float_rn(nonrep), __uint2float_rn(total_hits)) : 1.0f;
            if (rescue_distance > 0) {
                // counts of the hits that a rescue may look at, none known yet
                bool counts_ready = false;
                auto ready = [&]() {
                    if (!counts_ready)
                        for (uint32_t h = lane; h < nh; h += 32) cache[b + h] = 0xffffffffu;
                    counts_ready = true;
                    __syncwarp();
                };
                if (frac < 0.7f && nonrep < 5) {
                    ready();
                    d.rescued += warp_rescue_least_frequent(ix, 0, nh, 5, 1000, hit_pos + b, hit_info + b, cache + b,
                                                            qr_hash_rc + b);
                }
                // most reads have no filtered stretch to rescue: tested for all hits at once
                // (the walk below reads hit after hit)
                bool stretch = false;
                {
                    uint32_t last = 0, lq = 0;
                    for (uint32_t c = 0; c < nh; c += 32) {
                        const uint32_t h = c + lane;
                        uint32_t qs = 0;
                        bool unf = false;
                        if (h < nh) {
                            const uint32_t info = hit_info[b + h];
                            qs = qr_start[b + (info >> 3)];
                            unf = !(info & 4);
                        }
                        const uint32_t um = __ballot_sync(FULL, unf), lower = um & lanemask_lt();
                        const uint32_t pq = __shfl_sync(FULL, qs, lower ? 31 - __clz(lower) : 0);
                        stretch = stretch || __any_sync(FULL, unf && qs > (lower ? pq : last) + rescue_distance);
                        const uint32_t lu = __shfl_sync(FULL, qs, um ? 31 - __clz(um) : 0);
                        if (um) last = lu;
                        lq = __shfl_sync(FULL, qs, (nh - 1 < c + 31 ? nh - 1 - c : 31));
                    }
                    if (nh > 0 && lq - last > rescue_distance) stretch = true;
                }
                if (stretch) ready();
                // local rescue over filtered stretches (src/hit.rs:232-268); an interval is
                // processed as soon as it is found, which only touches hits already scanned
                uint32_t scan = 0, last_unf = 0, first_f = 0;
                while (stretch) {
                    uint32_t is = 0, ie = 0, tr = 0, found = 0;
                    if (lane == 0) {
                        while (scan < nh) {
                            uint32_t h = scan++;
                            uint32_t info = hit_info[b + h];
                            if (info & 4) continue;
                            uint32_t qs = qr_start[b + (info >> 3)];
                            bool iv = qs > last_unf + rescue_distance;
                            if (iv) { is = first_f; ie = h; tr = (qs - last_unf) / rescue_distance; found = 1; }
                            last_unf = qs;
                            first_f = h + 1;
                            if (iv) break;
                        }
                        if (!found && scan == nh && nh > 0 && scan != 0xffffffffu) {
                            uint32_t lq = qr_start[b + (hit_info[b + nh - 1] >> 3)];
                            uint32_t diff = lq - last_unf;
                            if (diff > rescue_distance) { is = first_f; ie = nh; tr = diff / rescue_distance; found = 1; }
                            scan = 0xffffffffu;
                        }
                    }
                    found = __shfl_sync(FULL, found, 0);
                    if (!found) break;
                    is = __shfl_sync(FULL, is, 0);
                    ie = __shfl_sync(FULL, ie, 0);
                    tr = __shfl_sync(FULL, tr, 0);
                    d.rescued += warp_rescue_least_frequent(ix, is, ie, tr, 10000, hit_pos + b, hit_info + b,
                                                            cache + b, qr_hash_rc + b);
                }
            }
            hc[ori] = d;
            if (lane == 0) n_hits[2 * r + ori] = nh;
        }
        if (lane == 0) {
            uint32_t t0 = hc[0].ffound + hc[0].ff, t1 = hc[1].ffound + hc[1].ff;
            bool b0 = t0 >= t1 * 2 && t0 > t1 + 5;
            bool b1 = t1 >= t0 * 2 && t1 > t0 + 5;
            uint8_t m = b0 ? 1 : b1 ? 2 : 3;
            orient[r] = m;
            NamDetailsRec dr;
            dr.full_not_found = hc[0].fnf + hc[1].fnf;
            dr.full_filtered = hc[0].ff + hc[1].ff;
            dr.full_found = hc[0].ffound + hc[1].ffound;
            dr.partial_not_found = hc[0].pnf + hc[1].pnf;
            dr.partial_filtered = hc[0].pf + hc[1].pf;
            dr.partial_found = hc[0].pfound + hc[1].pfound;
            dr.rescued = hc[0].rescued + hc[1].rescued;
            dr.n_randstrobes = n_rs[2 * r] + n_rs[2 * r + 1];
            dr.n_anchors = 0;
            dr.n_nams = 0;
            dr.both_orientations = m == 3;
            details[r] = dr;
        }
        __syncwarp();
    }
}

// ------------------------------------------------------------------ anchors
// Anchor keys: (ref_id, ref_start, query_start) packed so that integer order is the
// reference's anchor order (src/chainer.rs:228).
struct AnchorPack {
    uint32_t qbits, pbits;
    __device__ __forceinline__ uint64_t key(uint32_t ref_id, uint32_t ref_start, uint32_t qs) const {
        return ((uint64_t)ref_id << (pbits + qbits)) | ((uint64_t)ref_start << qbits) | qs;
    }
};

// add_to_anchors_full / add_to_anchors_partial (src/chainer.rs:304-366) are split into
// run_head (one lane, the first 32 entries of a run) and warp_run_anchors (the rest).
//
// A hit's run of equal-hash table entries: its first entry and hash (full hits:
// the entry found; partial hits: get_masked_from with the forward main mask).  False
// when a partial hit has no entry under that mask.
__device__ __forceinline__ bool hit_run(const DevIndex& ix, uint64_t pos, uint32_t info, uint64_t hash,
                                        uint64_t& start, uint64_t& fh) {
    if (info & 2) {
        start = idx_get_masked_from(ix, hash, ix.p.fwd_main_mask, true, pos);
        if (start == UINT64_MAX) return false;
        fh = load_rs(ix.rs, start).hash_offset & ix.p.fwd_main_mask;
    } else {
        start = pos;
        fh = load_hash(ix.rs, pos);
    }
    return true;
}

// The first 32 entries of a run by one lane (hit_anchors' loop): anchors to out (if
// not null), their count, the running minimum length difference (full hits).  True
// when the run ended within them; otherwise the warp continues from start + 32.
__device__ __forceinline__ bool run_head(const DevIndex& ix, uint64_t start, uint64_t fh, bool partial, uint32_t qs,
                                         uint32_t qe, AnchorPack ap, uint64_t* out, uint32_t& cnt, uint32_t& minld) {
    const uint32_t k = ix.p.k, ql = qe - qs;
    cnt = 0;
    minld = 0xffffffffu;
    const uint64_t end = start + 32 < ix.n ? start + 32 : ix.n;
    for (uint64_t i = start; i < end; i++) {
        const RefRandstrobe rr = load_rs(ix.rs, i);
        if (partial) {
            if ((rr.hash_offset & ix.p.fwd_main_mask) != fh) return true;
            if (out) out[cnt] = ap.key(rr.ref_index, rr.position, qs);
            cnt++;
        } else {
            if (rs_hash(rr) != fh) return true;
            const uint32_t rl = (uint32_t)(rr.hash_offset & 0xff) + k;
            const uint32_t ld = ql > rl ? ql - rl : rl - ql;
            if (ld <= minld) {
                if (out) {
                    out[cnt] = ap.key(rr.ref_index, rr.position, qs);
                    out[cnt + 1] = ap.key(rr.ref_index, rr.position + rl - k, qe - k);
                }
                cnt += 2;
                minld = ld;
            }
        }
    }
    return end == ix.n;
}

// hit_anchors for one run by the whole warp (arguments uniform across the warp): lanes
// take consecutive entries; the running-minimum length filter of full hits becomes a
// prefix minimum over the lanes carried between 32-entry slices.
__device__ uint32_t warp_run_anchors(const DevIndex& ix, uint64_t start, uint64_t fh, bool partial, uint32_t qs,
                                     uint32_t qe, AnchorPack ap, uint64_t* out, uint32_t carry) {
    const uint32_t lane = lane_id(), k = ix.p.k, ql = qe - qs;
    uint32_t cnt = 0;
    for (uint64_t c = start;; c += 32) {
        const uint64_t i = c + lane;
        bool valid = false;
        RefRandstrobe rr{};
        if (i < ix.n) {
            rr = load_rs(ix.rs, i);
            valid = partial ? (rr.hash_offset & ix.p.fwd_main_mask) == fh : rs_hash(rr) == fh;
        }
        // the table is sorted: the run's entries are a prefix of the lanes
        const uint32_t vb = __ballot_sync(FULL, valid);
        if (partial) {
            if (valid && out) out[cnt + lane] = ap.key(rr.ref_index, rr.position, qs);
            cnt += __popc(vb);
        } else {
            const uint32_t rl = valid ? (uint32_t)(rr.hash_offset & 0xff) + k : 0;
            const uint32_t ld = valid ? (ql > rl ? ql - rl : rl - ql) : 0xffffffffu;
            uint32_t incl = ld;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t y = __shfl_up_sync(FULL, incl, d);
                if (lane >= (uint32_t)d) incl = min(incl, y);
            }
            uint32_t excl = __shfl_up_sync(FULL, incl, 1);
            if (lane == 0) excl = 0xffffffffu;
            const bool o = valid && ld <= min(carry, excl);
            const uint32_t ob = __ballot_sync(FULL, o);
            if (o && out) {
                const uint32_t p = cnt + 2 * __popc(ob & lanemask_lt());
                out[p] = ap.key(rr.ref_index, rr.position, qs);
                out[p + 1] = ap.key(rr.ref_index, rr.position + rl - k, qe - k);
            }
            cnt += 2 * __popc(ob);
            carry = min(carry, __shfl_sync(FULL, incl, 31));
        }
        if (vb != FULL) break;
    }
    return cnt;
}

__device__ __forceinline__ uint32_t warp_excl_scan(uint32_t v, uint32_t& total) {
    uint32_t x = v;
    for (int d = 1; d < 32; d <<= 1) {
        uint32_t y = __shfl_up_sync(FULL, x, d);
        if (lane_id() >= (uint32_t)d) x += y;
    }
    total = __shfl_sync(FULL, x, 31);
    return x - v;
}

// The anchors of each read orientation (src/chainer.rs:304-384): counted, then written to the
// next free range of the anchor array while the table entries are still in the L1 (a launch
// each for counts and anchors read the table's random sectors twice: 11.2 KB of DRAM per read
// on a human-sized index; 6.0 ms for 1.4 M reads, 4.6 ms now).  The ranges' order does not
// matter to the stages after.  Past the array's capacity nothing is written; *cursor then
// tells what it takes. Five blocks an SM in 48 registers: the NAM stage of 100,000 reads takes
// 1.60 ms, with four in 64 registers 1.62 ms; six gain nothing more.
__global__ void __launch_bounds__(256, 5) k_anchors(DevIndex ix, const uint64_t* __restrict__ off, uint32_t n,
                                                 uint64_t total, const uint64_t* qr_hash, const uint32_t* qr_start,
                                                 const uint32_t* qr_end, const uint64_t* hit_pos,
                                                 const uint32_t* hit_info, const uint32_t* n_hits,
                                                 const uint8_t* orient, uint32_t* hit_anchors_n, uint64_t* seg_count,
                                                 uint64_t* seg_off, unsigned long long* cursor, uint64_t* anchors,
                                                 uint64_t capacity, AnchorPack ap, NamDetailsRec* details) {
    const uint32_t lane = lane_id();
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; r < n; r += nwarps) {
        const uint64_t o = off[r];
        const uint8_t m = orient[r];
        uint32_t read_total = 0;
        for (int ori = 0; ori < 2; ori++) {
            const uint64_t b = ori * total + o;
            const uint32_t nh = (m >> ori) & 1 ? n_hits[2 * r + ori] : 0;
            uint32_t sum = 0;
            uint64_t base = 0;
            // pass 0 counts, pass 1 writes; the counts of up to 32 hits stay in registers
            uint32_t info = 0, qs = 0, qe = 0, cnt = 0;
            uint64_t start = 0, fh = 0;
            bool has_run = false;
            for (int pass = 0; pass < 2 && nh; pass++) {
                uint64_t acc = base;
                for (uint32_t c = 0; c < nh; c += 32) {
                    const uint32_t h = c + lane;
                    if (pass == 0 || nh > 32) {
                        has_run = false;
                        cnt = 0;
                        if (h < nh) {
                            info = hit_info[b + h];
                            if (!(info & 4)) {
                                const uint32_t ri = info >> 3;
                                qs = qr_start[b + ri];
                                qe = (info & 2) ? qs + ix.p.k : qr_end[b + ri];
                                has_run = hit_run(ix, hit_pos[b + h], info, qr_hash[b + ri], start, fh);
                                if (pass) cnt = hit_anchors_n[b + h];
                            }
                        }
                    }
                    uint32_t tot = 0, ex = 0;
                    if (pass) ex = warp_excl_scan(cnt, tot);
                    uint64_t* out = pass ? anchors + acc + ex : nullptr;
                    // each lane its run's first 32 entries; longer runs continue with the
                    // whole warp, one hit at a time
                    uint32_t head = 0, minld = 0xffffffffu;
                    bool is_long = false;
                    if (has_run) is_long = !run_head(ix, start, fh, info & 2, qs, qe, ap, out, head, minld);
                    for (uint32_t lm = __ballot_sync(FULL, is_long); lm; lm &= lm - 1) {
                        const int L = __ffs(lm) - 1;
                        const uint32_t hL = __shfl_sync(FULL, head, L);
                        const uint32_t rest = warp_run_anchors(
                            ix, __shfl_sync(FULL, start, L) + 32, __shfl_sync(FULL, fh, L),
                            __shfl_sync(FULL, info, L) & 2, __shfl_sync(FULL, qs, L), __shfl_sync(FULL, qe, L), ap,
                            pass ? anchors + acc + __shfl_sync(FULL, ex, L) + hL : nullptr, __shfl_sync(FULL, minld, L));
                        if (lane == (uint32_t)L) head += rest;
                    }
                    if (!pass) {
                        cnt = head;
                        if (nh > 32 && has_run) hit_anchors_n[b + h] = cnt;
                        else if (nh > 32 && h < nh && !(info & 4)) hit_anchors_n[b + h] = 0;
                        warp_excl_scan(cnt, tot);
                        sum += tot;
                    }
                    acc += tot;
                }
                if (pass == 0) {
                    if (lane == 0 && sum) base = atomicAdd(cursor, (unsigned long long)sum);
                    base = __shfl_sync(FULL, base, 0);
                    if (sum == 0 || base + sum > capacity) break;
                }
            }
            if (lane == 0) {
                seg_count[2 * r + ori] = sum;
                seg_off[2 * r + ori] = base;
            }
            read_total += sum;
        }
        if (lane == 0) details[r].n_anchors = read_total;
    }
}

// ------------------------------------------------------------------ chaining
struct ChainCtx {
    ChainParams cp;
    uint32_t k;
    const float* lut;
    // fl(mx / mn) > max_diagonal_ratio without the division, for integers below 2^24
    // (whose float conversions are exact): with R = M * 2^e (M the 24-bit significand),
    // the quotient rounds above R exactly when mx / mn exceeds the midpoint
    // (2M + 1) * 2^(e - 1), or reaches it when M is odd (ties go to even).  That is
    // mx * 2^(1 - e) > mn * (2M + 1) in 64-bit integers.  ratio_exact is false when R
    // does not fit this form; the division is used then.
    bool ratio_exact;
    bool ratio_strict;
    uint32_t ratio_shift;
    uint64_t ratio_num;
};

// fl(mx / mn) > R, as the reference computes it in f32 (0 / 0 is NaN: false)
__device__ __forceinline__ bool ratio_above(uint32_t mx, uint32_t mn, const ChainCtx& c) {
    if (c.ratio_exact) {
        const uint64_t lhs = (uint64_t)mx << c.ratio_shift, rhs = (uint64_t)mn * c.ratio_num;
        return mx != 0 && (c.ratio_strict ? lhs > rhs : lhs >= rhs);
    }
    return __fdiv_rn(__uint2float_rn(mx), __uint2float_rn(mn)) > c.cp.max_diagonal_ratio;
}

// compute_score (src/chainer.rs:286-302)
__device__ __forceinline__ float chain_score(uint32_t dq, uint32_t dr, const ChainCtx& c) {
    uint32_t dd = dr > dq ? dr - dq : dq - dr;
    uint32_t dg = dq < dr ? dq : dr;
    float score = __uint2float_rn(c.k < dg ? c.k : dg);
    uint32_t dg2 = dg > c.k ? dg - c.k : 0;
    float lin = __fadd_rn(__fmul_rn(c.cp.diag_diff_penalty, __uint2float_rn(dd)),
                          __fmul_rn(c.cp.gap_length_penalty, __uint2float_rn(dg2)));
    float lg = dd >= 1 ? __ldg(c.lut + (dd < LOG2_LUT_SIZE ? dd : LOG2_LUT_SIZE - 1)) : 0.0f;
    return __fsub_rn(score, __fadd_rn(lin, __fmul_rn(0.5f, lg)));
}

// Stable LSD radix sort of anchor indices idx[0..m) by score (dp[idx]) descending, by
// one warp: four 8-bit passes over an order-preserving key, each a warp-ordered stable
// counting scatter (rank among equal digits of a 32-slice from __match_any_sync).
// idx and tmp are ping-pong buffers; the sorted order ends in tmp.
__device__ __forceinline__ uint32_t desc_key(float s) {
    const uint32_t b = __float_as_uint(s == 0.0f ? 0.0f : s);
    return ~((b & 0x80000000u) ? ~b : (b | 0x80000000u));  // ascending key = descending score
}

__device__ void warp_radix_sort_desc(uint32_t* idx, uint32_t* tmp, uint32_t m, const float* dp, uint32_t* hist) {
    const uint32_t lane = lane_id();
    uint32_t* src = idx;
    uint32_t* dst = tmp;
    for (int pass = 0; pass < 4; pass++) {
        const int sh = 8 * pass;
        for (uint32_t t = lane; t < 256; t += 32) hist[t] = 0;
        __syncwarp();
        for (uint32_t c = lane; c < m; c += 32) atomicAdd(&hist[(desc_key(dp[src[c]]) >> sh) & 255], 1u);
        __syncwarp();
        // exclusive scan of the 256 counters, 8 per lane
        uint32_t v[8], sum = 0;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            v[k] = hist[lane * 8 + k];
            sum += v[k];
        }
        uint32_t incl = sum;
        for (int d = 1; d < 32; d <<= 1) {
            const uint32_t y = __shfl_up_sync(FULL, incl, d);
            if (lane >= (uint32_t)d) incl += y;
        }
        uint32_t run = incl - sum;
#pragma unroll
        for (int k = 0; k < 8; k++) {
            hist[lane * 8 + k] = run;
            run += v[k];
        }
        __syncwarp();
        for (uint32_t c0 = 0; c0 < m; c0 += 32) {
            const uint32_t c = c0 + lane;
            const bool in = c < m;
            const uint32_t x = in ? src[c] : 0;
            const uint32_t dg = in ? (desc_key(dp[x]) >> sh) & 255 : 256 + lane;
            const uint32_t peers = __match_any_sync(FULL, dg);
            const uint32_t base = in ? hist[dg] : 0;
            __syncwarp();
            if (in) {
                dst[base + __popc(peers & lanemask_lt())] = x;
                // the highest lane of each digit group advances the digit's offset
                if ((peers >> lane) == 1u) hist[dg] = base + __popc(peers);
            }
            __syncwarp();
        }
        uint32_t* t = src;
        src = dst;
        dst = t;
    }
    // four passes: the result is back in idx; copy it to tmp for the caller
    for (uint32_t c = lane; c < m; c += 32) tmp[c] = idx[c];
}

// extract_chains (src/chainer.rs:386-449) for one read orientation (segment sg, anchors
// b .. b + N of the deduplicated list) by the whole warp; best_score is the segment's
// best chain score.  hist: this warp's 256 shared counters; scratch: one word per anchor.
//
// The reference walks the candidates' chains in order of score and drops a chain that
// meets an anchor which an earlier walk marked.  The predecessors make a forest, every
// walk ends at its tree's root, and a walk marks all its anchors but the first.  So a
// tree's root is marked by the first candidate in order that is not the root itself;
// that candidate meets no mark, and every later one is marked or meets one at the root at
// the latest.  A tree therefore keeps that one chain, and the root alone as a chain of its
// own if it is a candidate and comes before it.  So there is no order to walk in: the
// roots, each tree's first candidate (a maximum per root), and only the kept chains are
// sorted and walked, 32 at a time.  Tandem arrays leave hundreds of chains per orientation:
// walked one after another, 5,200 anchors with 512 chains took 2.2 M cycles (1.1 ms, the
// kernel's length).
__device__ void chain_extract(const uint64_t* dedup, const float* dp, const uint32_t* pred, uint32_t* aux,
                              uint64_t total_anchors, unsigned long long* scratch, uint64_t b, uint32_t N, uint32_t sg,
                              float best_score, const AnchorPack& ap, const ChainCtx& cc, NamRec* nam_out,
                              uint32_t* nam_seg_count, uint64_t* anc_out, uint64_t* anc_start, uint32_t* hist) {
    const uint32_t lane = lane_id();
    const uint64_t qmask = (1ULL << ap.qbits) - 1, pmask = (1ULL << ap.pbits) - 1;
    const float valid_score = __fmul_rn(best_score, cc.cp.valid_score_threshold);
    constexpr uint32_t NO = 0xffffffffu;
    uint32_t* kept = aux + b;
    uint32_t* sorted = aux + total_anchors + b;
    uint32_t* root = aux + 2 * total_anchors + b;
    unsigned long long* first = scratch + b;
    // larger = earlier in the reference's order: by score, ties by anchor order
    auto order_key = [](uint32_t i, float score) { return ((uint64_t)~desc_key(score) << 32) | (NO - i); };
    // predecessors come before their successors: roots 32 anchors at a time, a
    // predecessor within the 32 by pointer jumping
    for (uint32_t c = 0; c < N; c += 32) {
        const uint32_t i = c + lane;
        const uint32_t p = i < N ? pred[b + i] : NO;
        uint32_t r = p == NO ? i : p;  // an anchor on i's way to the root
#pragma unroll
        for (int d = 0; d < 5; d++) {
            const uint32_t up = __shfl_sync(FULL, r, r >= c ? r - c : lane);
            if (r >= c) r = up;
        }
        if (r < c) r = root[r];
        if (i < N) {
            root[i] = r;
            first[i] = 0;
        }
        __syncwarp();
    }
    for (uint32_t i = lane; i < N; i += 32) {
        const float s = dp[b + i];
        const uint32_t r = root[i];
        if (s >= valid_score && r != i) atomicMax(&first[r], (unsigned long long)order_key(i, s));
    }
    __syncwarp();
    uint32_t K = 0;
    for (uint32_t c = 0; c < N; c += 32) {
        const uint32_t i = c + lane;
        bool take = false;
        if (i < N) {
            const float s = dp[b + i];
            const uint32_t r = root[i];
            if (s >= valid_score) {
                const uint64_t f = __ldcg(&first[r]), key = order_key(i, s);
                take = i == r ? key > f : key == f;
            }
        }
        const uint32_t bal = __ballot_sync(FULL, take);
        if (take) kept[K + __popc(bal & lanemask_lt())] = i;
        K += __popc(bal);
    }
    __syncwarp();
    // by score, descending, ties in anchor order (a stable sort)
    if (K <= 32) {
        const uint32_t ci = lane < K ? kept[lane] : 0;
        const float s = lane < K ? dp[b + ci] : 0.0f;
        uint32_t rank = 0;
        for (uint32_t u = 0; u < K; u++) {
            const float su = __shfl_sync(FULL, s, u);
            rank += (su > s) || (su == s && u < lane);
        }
        if (lane < K) sorted[rank] = ci;
    } else {
        warp_radix_sort_desc(kept, sorted, K, dp + b, hist);
    }
    __syncwarp();
    // kept chains share no anchor but a root that is also a chain of its own: 2 slots
    // per anchor suffice (3 are there)
    uint64_t* ao = anc_out ? anc_out + 3 * b : nullptr;
    uint32_t acur = 0;
    for (uint32_t c = 0; c < K; c += 32) {
        const uint32_t x = c + lane;
        uint32_t n = 0, i = 0;
        if (x < K) {
            i = sorted[x];
            const uint64_t ki = dedup[b + i];
            uint32_t matching = cc.k, cov = (uint32_t)((ki >> ap.qbits) & pmask);
            uint64_t kj = ki;
            n = 1;
            // a root that is followed by its tree's chain stands alone: it has no predecessor
            for (uint32_t j = pred[b + i]; j != NO;) {
                kj = dedup[b + j];
                j = pred[b + j];
                n++;
                const uint32_t rs = (uint32_t)((kj >> ap.qbits) & pmask), d = cov > rs ? cov - rs : 0;
                matching += d < cc.k ? d : cc.k;
                cov = rs;
            }
            NamRec nr;
            nr.nam_id = x;
            nr.query_start = (uint32_t)(kj & qmask);
            nr.query_end = (uint32_t)(ki & qmask) + cc.k;
            nr.ref_start = cov;
            nr.ref_end = (uint32_t)((ki >> ap.qbits) & pmask) + cc.k;
            nr.matching_bases = matching;
            nr.ref_id = (uint32_t)(ki >> (ap.pbits + ap.qbits));
            nr.score = __fadd_rn(dp[b + i], __fmul_rn(__uint2float_rn(n), cc.cp.matches_weight));
            nr.is_revcomp = sg & 1;
            nr.n_anchors = n;
            nam_out[b + x] = nr;
        }
        if (ao) {
            uint32_t tot;
            const uint32_t at = acur + warp_excl_scan(n, tot);
            if (x < K) {
                anc_start[b + x] = 3 * b + at;
                uint32_t j = i;
                for (uint32_t t = 0; t < n; t++) {
                    ao[at + t] = dedup[b + j];
                    j = pred[b + j];
                }
            }
            acur += tot;
        }
    }
    if (lane == 0) nam_seg_count[sg] = K;
    __syncwarp();
}

// extract_chains (src/chainer.rs:386-449) for the eight orientations of a grouped warp at
// once: group g (lanes 4g .. 4g+3) collects its orientation's candidates, and its first
// lane orders them (insertion into the sorted list: a stable sort by score, descending)
// and walks the chains, so the eight walks' dependent loads overlap instead of running
// one orientation after another.  nmax bounds every group's anchor count; sg == ~0u
// marks a group without an orientation.
__device__ void group_chain_extract(const uint64_t* dedup, const float* dp, const uint32_t* pred, uint32_t* aux,
                                    uint64_t total_anchors, uint64_t b, uint32_t N, uint32_t nmax, uint32_t sg,
                                    float best_score, const AnchorPack& ap, const ChainCtx& cc, NamRec* nam_out,
                                    uint32_t* nam_seg_count, uint64_t* anc_out, uint64_t* anc_start) {
    const uint32_t lane = lane_id(), gl = lane % 4, gsh = lane - gl;
    const uint64_t qmask = (1ULL << ap.qbits) - 1, pmask = (1ULL << ap.pbits) - 1;
    const bool has = sg != 0xffffffffu && N > 0;
    const float valid_score = __fmul_rn(best_score, cc.cp.valid_score_threshold);
    uint32_t* cand = aux + b;
    uint32_t* sorted_c = aux + total_anchors + b;
    uint32_t M = 0;
    for (uint32_t c = 0; c < nmax; c += 4) {
        const uint32_t i = c + gl;
        const bool in = has && i < N;
        const bool take = in && dp[b + i] >= valid_score;
        const uint32_t bal = (__ballot_sync(FULL, take) >> gsh) & 15u;
        if (take) cand[M + __popc(bal & ((1u << gl) - 1))] = i;
        M += __popc(bal);
    }
    __syncwarp();
    // used flags of the group's anchors (at most CHAIN_GROUP_MAX = 96) in three words
    uint32_t u0 = 0, u1 = 0, u2 = 0;
    auto is_used = [&](uint32_t j) -> bool {
        const uint32_t w = j < 32 ? u0 : j < 64 ? u1 : u2;
        return (w >> (j & 31)) & 1;
    };
    auto set_used = [&](uint32_t j) {
        const uint32_t m = 1u << (j & 31);
        if (j < 32) u0 |= m;
        else if (j < 64) u1 |= m;
        else u2 |= m;
    };
    if (has && gl == 0) {
        // candidates arrive in anchor order; each goes after every entry scoring at least
        // as much, so equal scores keep anchor order
        for (uint32_t t = 0; t < M; t++) {
            const uint32_t ci = cand[t];
            const float sc = dp[b + ci];
            uint32_t pos = t;
            while (pos > 0 && dp[b + sorted_c[pos - 1]] < sc) {
                sorted_c[pos] = sorted_c[pos - 1];
                pos--;
            }
            sorted_c[pos] = ci;
        }
        uint32_t nn = 0;
        NamRec* outp = nam_out + b;
        uint64_t* ao = anc_out ? anc_out + 3 * b : nullptr;
        uint32_t acur = 0;
        for (uint32_t c = 0; c < M; c++) {
            const uint32_t i = sorted_c[c];
            if (is_used(i)) continue;
            uint32_t j = i;
            bool overlaps = false;
            uint32_t nanch = 1;
            const uint64_t ki = dedup[b + i];
            if (ao) ao[acur] = ki;
            uint32_t matching = cc.k;
            uint32_t cov = (uint32_t)((ki >> ap.qbits) & pmask);
            while (pred[b + j] != 0xffffffffu) {
                j = pred[b + j];
                if (is_used(j)) {
                    overlaps = true;
                    break;
                }
                const uint64_t kj = dedup[b + j];
                if (ao) ao[acur + nanch] = kj;
                nanch++;
                set_used(j);
                const uint32_t rsj = (uint32_t)((kj >> ap.qbits) & pmask);
                const uint32_t d = cov > rsj ? cov - rsj : 0;
                matching += d < cc.k ? d : cc.k;
                cov = rsj;
            }
            if (overlaps) continue;
            const uint64_t kf2 = dedup[b + j];
            NamRec nr;
            nr.nam_id = nn;
            nr.query_start = (uint32_t)(kf2 & qmask);
            nr.query_end = (uint32_t)(ki & qmask) + cc.k;
            nr.ref_start = (uint32_t)((kf2 >> ap.qbits) & pmask);
            nr.ref_end = (uint32_t)((ki >> ap.qbits) & pmask) + cc.k;
            nr.matching_bases = matching;
            nr.ref_id = (uint32_t)(ki >> (ap.pbits + ap.qbits));
            nr.score = __fadd_rn(dp[b + i], __fmul_rn(__uint2float_rn(nanch), cc.cp.matches_weight));
            nr.is_revcomp = sg & 1;
            nr.n_anchors = nanch;
            if (anc_start) anc_start[b + nn] = 3 * b + acur;
            acur += nanch;
            outp[nn++] = nr;
        }
        nam_seg_count[sg] = nn;
    }
    if (sg != 0xffffffffu && N == 0 && gl == 0) nam_seg_count[sg] = 0;
    __syncwarp();
}

// The read orientations that have anchors (only the better orientation of a read gets
// anchors, src/chainer.rs:205-216, so about half are empty), for k_chain4: those with
// at most CHAIN_GROUP_MAX anchors in `list`, taken eight per warp, the others in
// `long_list`, one per warp; key / long_key receive their anchor counts (the lists
// are then ordered by them).  The ranges of those with
// more than CHAIN_SORT_SMALL anchors go to sort_begin / sort_end for a segmented sort;
// k_chain4 sorts the others itself.  n_list: [0] listed, [1] sort ranges, [2] long.
constexpr uint32_t CHAIN_SORT_SMALL = 256;
constexpr uint32_t CHAIN_GROUP_MAX = 96;

__global__ void k_seg_list(const uint64_t* seg_count, const uint64_t* seg_off, uint32_t nseg, uint32_t* list,
                           uint32_t* long_list, uint32_t* n_list, uint64_t* sort_begin, uint64_t* sort_end,
                           uint32_t* key, uint32_t* long_key) {
    const uint32_t lane = lane_id();
    const uint32_t step = gridDim.x * blockDim.x;
    for (uint32_t base = (blockIdx.x * blockDim.x + threadIdx.x) & ~31u; base < nseg; base += step) {
        const uint32_t sg = base + lane;
        const uint64_t cnt = sg < nseg ? seg_count[sg] : 0;
        const bool lng = cnt > CHAIN_GROUP_MAX, shrt = cnt > 0 && !lng, big = cnt > CHAIN_SORT_SMALL;
        const uint32_t bs = __ballot_sync(FULL, shrt), bl = __ballot_sync(FULL, lng), bb = __ballot_sync(FULL, big);
        uint32_t as = 0, al = 0, ab = 0;
        if (lane == 0 && bs) as = atomicAdd(n_list, (uint32_t)__popc(bs));
        if (lane == 0 && bb) ab = atomicAdd(n_list + 1, (uint32_t)__popc(bb));
        if (lane == 0 && bl) al = atomicAdd(n_list + 2, (uint32_t)__popc(bl));
        as = __shfl_sync(FULL, as, 0);
        ab = __shfl_sync(FULL, ab, 0);
        al = __shfl_sync(FULL, al, 0);
        if (shrt) {
            list[as + __popc(bs & lanemask_lt())] = sg;
            key[as + __popc(bs & lanemask_lt())] = (uint32_t)cnt;
        }
        if (lng) {
            long_list[al + __popc(bl & lanemask_lt())] = sg;
            long_key[al + __popc(bl & lanemask_lt())] = cnt < 0xffffffffull ? (uint32_t)cnt : 0xffffffffu;
        }
        if (big) {
            const uint32_t k = ab + __popc(bb & lanemask_lt());
            const uint64_t o = seg_off[sg];
            sort_begin[k] = o;
            sort_end[k] = o + cnt;
        }
    }
}

// Ascending bitonic sort of R * 32 keys held R per lane (element r * 32 + lane in v[r]).
template <int R>
__device__ __forceinline__ void warp_bitonic_sort(uint64_t (&v)[R]) {
    const uint32_t lane = lane_id();
#pragma unroll
    for (uint32_t k = 2; k <= 32 * R; k <<= 1) {
#pragma unroll
        for (uint32_t j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                // partners in two registers of one lane; the direction depends on r only
                const int jr = (int)(j >> 5);
#pragma unroll
                for (int r = 0; r < R; r++) {
                    if (r & jr) continue;
                    const int r2 = r | jr;
                    const bool asc = ((32u * r) & k) == 0;
                    const uint64_t lo = v[r] < v[r2] ? v[r] : v[r2], hi = v[r] < v[r2] ? v[r2] : v[r];
                    v[r] = asc ? lo : hi;
                    v[r2] = asc ? hi : lo;
                }
            } else {
                const bool lower = (lane & j) == 0;
#pragma unroll
                for (int r = 0; r < R; r++) {
                    const uint64_t p = __shfl_xor_sync(FULL, v[r], j);
                    const bool asc = ((32 * r + lane) & k) == 0;
                    const bool take_min = lower == asc;
                    v[r] = take_min ? (p < v[r] ? p : v[r]) : (p > v[r] ? p : v[r]);
                }
            }
        }
    }
}

// Sort the cnt <= 32 * R keys at keys[0..cnt) (one read orientation's anchors, in the
// order k_anchors wrote them) and write the distinct ones back in order; returns their
// number (src/chainer.rs:228-229).
template <int R>
__device__ __forceinline__ uint32_t warp_sort_dedup(uint64_t* keys, uint32_t cnt) {
    const uint32_t lane = lane_id();
    uint64_t v[R];
#pragma unroll
    for (int r = 0; r < R; r++) v[r] = 32 * r + lane < cnt ? keys[32 * r + lane] : ~0ULL;
    warp_bitonic_sort<R>(v);
    uint32_t bal[R];
#pragma unroll
    for (int r = 0; r < R; r++) {
        uint64_t prev = __shfl_up_sync(FULL, v[r], 1);
        if (r > 0) {
            const uint64_t last = __shfl_sync(FULL, v[r > 0 ? r - 1 : 0], 31);
            if (lane == 0) prev = last;
        }
        const uint32_t e = 32 * r + lane;
        bal[r] = __ballot_sync(FULL, e < cnt && (e == 0 || prev != v[r]));
    }
    __syncwarp();
    uint32_t n = 0;
#pragma unroll
    for (int r = 0; r < R; r++) {
        if ((bal[r] >> lane) & 1u) keys[n + __popc(bal[r] & lanemask_lt())] = v[r];
        n += __popc(bal[r]);
    }
    return n;
}

// Chaining (src/chainer.rs:128-176 and 386-449) for NG = 8 read orientations per warp.
// The anchor sort and the deduplication run over the whole warp, one orientation after
// the other.  The DP is serial over a read orientation's anchors;
// the candidates j of anchor i (back to max_lookback) are scored in parallel and an
// exclusive prefix max over them reproduces the reference's downward scan with its
// ">=" updates and its stops (a different reference or a gap >= max_ref_gap ends the
// scan; an update on the same diagonal ends it after that candidate).  The DP runs for
// the NG orientations at once, one group of CG = 4 lanes each, four candidates at a
// time (most anchors stop at the first candidate: the one before on the same
// diagonal).  The orientations come from k_seg_list (those with up to CHAIN_GROUP_MAX
// anchors; longer ones: k_chain_long); nam_seg_count of those without anchors is zeroed
// before the launch.
//
// RING: max_lookback < 64, so the predecessors of anchor i (and their scores) come
// from a 64-entry ring in shared memory per orientation, written as anchors are
// scored, instead of global memory (this takes the store-to-load round trip out of
// each serial step).
constexpr uint32_t CG = 4;                   // lanes per orientation in the grouped DP
constexpr uint32_t NG = 32 / CG;             // orientations per warp
constexpr uint32_t GMASK = (1u << CG) - 1;  // one group's ballot bits
constexpr uint32_t CHAIN_WARPS = 4;          // warps per block (shared rings: 28 KB per block)

template <bool RING>
__device__ __forceinline__ void chain_candidates(uint32_t j, bool in, const uint64_t* dedup, const float* dp,
                                                 uint64_t b, const uint64_t* ring_key, const float* ring_dp,
                                                 uint32_t ri, uint32_t rsi, uint32_t qi, uint32_t max_ref_gap,
                                                 const ChainCtx& cc, const AnchorPack& ap, bool& hard, bool& valid,
                                                 bool& diag, float& val) {
    const uint64_t qmask = (1ULL << ap.qbits) - 1, pmask = (1ULL << ap.pbits) - 1;
    hard = valid = diag = false;
    val = 0.0f;
    if (!in) return;
    const uint64_t kj = RING ? ring_key[j & 63] : dedup[b + j];
    const uint32_t rj = (uint32_t)(kj >> (ap.pbits + ap.qbits)), rsj = (uint32_t)((kj >> ap.qbits) & pmask),
                   qj = (uint32_t)(kj & qmask);
    if (rj != ri) {
        hard = true;
    } else if (qi >= qj) {
        const uint32_t dq = qi - qj, dr = rsi - rsj;
        if (dr >= max_ref_gap) {
            hard = true;
        } else {
            const uint32_t mx = dq > dr ? dq : dr, mn = dq < dr ? dq : dr;
            if (!ratio_above(mx, mn, cc)) {
                valid = true;
                diag = dq == dr;
                val = __fadd_rn(RING ? ring_dp[j & 63] : dp[b + j], chain_score(dq, dr, cc));
            }
        }
    }
}

// The lookback DP of collinear_chaining (src/chainer.rs:85-180) over anchors [c0, c1)
// of one read orientation (its anchors at dedup[b ..]) by the whole warp, for a
// max_lookback of 64 or more (warp_chain_regs otherwise): 32 predecessors per step, the
// early-break rules as a prefix max over the lanes.
// Predecessors never go below c0 (earlier anchors lie max_ref_gap or more behind, or
// on another reference, and end the reference's scan without contributing).  With
// recheck, (best_score, best_index, best_key) is the running best over all anchors
// before c0 and is updated as the reference updates it (strict >); without, the
// best-index re-check (:150-165) is left out.
__device__ void warp_chain_range(const uint64_t* dedup, float* dp, uint32_t* pred, uint64_t b, uint32_t c0, uint32_t c1,
                                 uint32_t floor, uint32_t max_ref_gap, const ChainCtx& cc, const AnchorPack& ap,
                                 bool recheck, float& best_score, uint32_t& best_index, uint64_t& best_key) {
    const uint32_t lane = lane_id();
    const uint64_t qmask = (1ULL << ap.qbits) - 1, pmask = (1ULL << ap.pbits) - 1;
    const float kf = __uint2float_rn(cc.k);
    uint64_t next_key = c0 < c1 ? dedup[b + c0] : 0;
    for (uint32_t i = c0; i < c1; i++) {
        const uint64_t ki = next_key;
        if (i + 1 < c1) next_key = dedup[b + i + 1];
        const uint32_t ri = (uint32_t)(ki >> (ap.pbits + ap.qbits)), rsi = (uint32_t)((ki >> ap.qbits) & pmask),
                       qi = (uint32_t)(ki & qmask);
        uint32_t lookup_end = i > cc.cp.max_lookback ? i - cc.cp.max_lookback : 0;
        if (lookup_end < floor) lookup_end = floor;
        float cur = kf;
        uint32_t cur_pred = 0xffffffffu;
        bool stop = false;
        for (uint32_t base = 0; !stop && base < i - lookup_end; base += 32) {
            const uint32_t t = base + lane;
            const bool in = t < i - lookup_end;
            const uint32_t j = i - 1 - t;
            bool hard, valid, diag;
            float val;
            chain_candidates<false>(j, in, dedup, dp, b, nullptr, nullptr, ri, rsi, qi, max_ref_gap, cc, ap, hard,
                                    valid, diag, val);
            // the common case: the first candidate updates and lies on the same diagonal,
            // which ends the scan (the prefix max below would find the same)
            if (__ballot_sync(FULL, lane == 0 && valid && diag && val >= cur)) {
                cur = __shfl_sync(FULL, val, 0);
                cur_pred = i - 1 - base;
                break;
            }
            const uint32_t hb = __ballot_sync(FULL, hard);
            const uint32_t lim = hb ? (uint32_t)(__ffs(hb) - 1) : 32;
            if (lane >= lim) valid = false;
            float incl = valid ? val : -INFINITY;
            for (int d = 1; d < 32; d <<= 1) {
                const float y = __shfl_up_sync(FULL, incl, d);
                if (lane >= (uint32_t)d) incl = fmaxf(incl, y);
            }
            float excl = __shfl_up_sync(FULL, incl, 1);
            if (lane == 0) excl = -INFINITY;
            const bool upd = valid && val >= fmaxf(cur, excl);
            const uint32_t ub = __ballot_sync(FULL, upd);
            const uint32_t sb = __ballot_sync(FULL, upd && diag);
            uint32_t reach = lim;
            if (sb) {
                reach = (uint32_t)__ffs(sb);
                stop = true;
            }
            if (hb) stop = true;
            const uint32_t um = ub & (reach >= 32 ? FULL : ((1u << reach) - 1));
            if (um) {
                const uint32_t last = 31 - __clz(um);
                cur = __shfl_sync(FULL, val, last);
                cur_pred = i - 1 - (base + last);
            }
        }
        if (recheck && best_index != 0xffffffffu) {
            const uint64_t kb = best_key;
            const uint32_t rb = (uint32_t)(kb >> (ap.pbits + ap.qbits)), rsb = (uint32_t)((kb >> ap.qbits) & pmask),
                           qb = (uint32_t)(kb & qmask);
            if (rb == ri && qi > qb) {
                const uint32_t dq = qi - qb, dr = rsi - rsb;
                const uint32_t mx = dq > dr ? dq : dr, mn = dq < dr ? dq : dr;
                if (dr < max_ref_gap && dr > 0 && !ratio_above(mx, mn, cc)) {
                    const float ns = __fadd_rn(best_score, chain_score(dq, dr, cc));
                    if (ns > cur) {
                        cur = ns;
                        cur_pred = best_index;
                    }
                }
            }
        }
        if (lane == 0) {
            dp[b + i] = cur;
            pred[b + i] = cur_pred;
        }
        if (recheck && cur > best_score) {
            best_score = cur;
            best_index = i;
            best_key = ki;
        }
        if (!recheck && cur > best_score) best_score = cur;  // the range's maximum
        __syncwarp();
    }
}

// One predecessor pair's share of chain_candidates without the predecessor's score:
// chain_score, or -inf where the pair is no candidate; both anchors on one reference.
__device__ __forceinline__ float pair_score(uint32_t rsi, uint32_t qi, uint32_t rsj, uint32_t qj, bool in,
                                            uint32_t max_ref_gap, const ChainCtx& cc, bool& diag) {
    const uint32_t dq = qi - qj, dr = rsi - rsj;
    const uint32_t mx = dq > dr ? dq : dr, mn = dq < dr ? dq : dr;
    const bool ok = in && qi >= qj && dr < max_ref_gap && !ratio_above(mx, mn, cc);
    diag = ok && dq == dr;
    return ok ? chain_score(dq, dr, cc) : -INFINITY;
}

// Slots as bits (a: slots 0-31, c: slots 32-63) in scan order of anchor i: the predecessor
// at distance t (anchor i - 1 - t, slot (i - 1 - t) & 63) at bit 63 - t.
__device__ __forceinline__ uint64_t scan_order(uint32_t i, bool a, bool c) {
    const uint64_t m = __ballot_sync(FULL, a) | ((uint64_t)__ballot_sync(FULL, c) << 32);
    const uint32_t rot = 63 - ((i - 1) & 63);
    return rot ? (m << rot) | (m >> (64 - rot)) : m;
}

// The outcome of anchor i's predecessor scan (src/chainer.rs:98-147) from the candidates'
// chain scores, lane l holding those of slots l (vA) and l + 32 (vB), -inf for no
// candidate; diag marks those on the anchor's diagonal, in scan order.  A candidate whose
// gap ends the reference's scan is simply none (positions are sorted, so none after it
// could count).  Without one on the same diagonal the result is the maximum, ties to the
// farthest; with one, it ends the scan if it reaches the maximum (checked first) or the
// maximum over the nearer ones (a prefix maximum).  Scores below k never update and all
// others are positive, so their bits order as integers (redux).
__device__ __forceinline__ void scan_outcome(uint32_t i, float vA, float vB, uint64_t diag, float kf, float& cur,
                                             uint32_t& cur_pred) {
    const uint32_t lane = lane_id();
    const float M = __uint_as_float(__reduce_max_sync(FULL, __float_as_uint(fmaxf(fmaxf(vA, vB), 0.0f))));
    cur = kf;
    cur_pred = 0xffffffffu;
    if (!(M >= kf)) return;
    if (diag) {
        uint32_t t = (uint32_t)__clzll((long long)diag);
        uint32_t slot = (i - 1 - t) & 63;
        float v = __shfl_sync(FULL, slot & 32 ? vB : vA, slot & 31);
        bool stopped = v >= M;
        if (!stopped) {
            // does a same-diagonal candidate reach the maximum over the nearer ones?
            // each lane has one candidate at distance r and one at r + 32
            const uint32_t r = (i - 1 - lane) & 31;
            const bool near_b = (i - 1 - r) & 32;
            const float near = near_b ? vB : vA, far = near_b ? vA : vB;
            float pn = near, pf = far;
#pragma unroll
            for (uint32_t d = 1; d < 32; d <<= 1) {
                const float yn = __shfl_sync(FULL, pn, (lane + d) & 31), yf = __shfl_sync(FULL, pf, (lane + d) & 31);
                if (r >= d) {
                    pn = fmaxf(pn, yn);
                    pf = fmaxf(pf, yf);
                }
            }
            const float all_near = __shfl_sync(FULL, pn, (i - 32) & 31);  // the lane with r = 31
            float en = __shfl_sync(FULL, pn, (lane + 1) & 31), ef = __shfl_sync(FULL, pf, (lane + 1) & 31);
            if (r == 0) en = ef = -INFINITY;
            ef = fmaxf(ef, all_near);
            const uint32_t un = __ballot_sync(FULL, ((diag >> (63 - r)) & 1) && near >= fmaxf(kf, en));
            const uint32_t uf = __ballot_sync(FULL, ((diag >> (31 - r)) & 1) && far >= fmaxf(kf, ef));
            if (un | uf) {
                // the nearest one's lane to bit 31
                const uint32_t m = un ? un : uf;
                t = __clz(__funnelshift_l(m, m, 31 - ((i - 1) & 31))) + (un ? 0 : 32);
                slot = (i - 1 - t) & 63;
                v = __shfl_sync(FULL, slot & 32 ? vB : vA, slot & 31);
                stopped = true;
            }
        }
        if (stopped) {
            cur = v;
            cur_pred = i - 1 - t;
            return;
        }
    }
    cur = M;
    const uint64_t eq = scan_order(i, vA == M, vB == M);
    cur_pred = i - 1 - (uint32_t)(64 - __ffsll((long long)eq));
}

// The best-index re-check (:150-165) of an anchor (its key, position and query start)
// against the running best: whether it applies, and the score it gives.
__device__ __forceinline__ bool recheck_score(uint64_t key, uint32_t rs, uint32_t q, uint64_t best_key,
                                              float best_score, uint32_t max_ref_gap, const ChainCtx& cc,
                                              const AnchorPack& ap, float& ns) {
    const uint64_t pmask = (1ULL << ap.pbits) - 1;
    const uint32_t rsb = (uint32_t)((best_key >> ap.qbits) & pmask),
                   qb = (uint32_t)best_key & (uint32_t)((1ULL << ap.qbits) - 1);
    const uint32_t dq = q - qb, dr = rs - rsb;
    if (dr >= max_ref_gap || dr == 0 || q <= qb) return false;
    if ((best_key >> (ap.pbits + ap.qbits)) != (key >> (ap.pbits + ap.qbits))) return false;
    if (ratio_above(dq > dr ? dq : dr, dq < dr ? dq : dr, cc)) return false;
    ns = __fadd_rn(best_score, chain_score(dq, dr, cc));
    return true;
}

// warp_chain_range with the re-check, for max_lookback < 64, the predecessors in
// registers: slot j & 63 of the last 64 anchors, two per lane; used where a cluster is
// scored again from an anchor on.
__device__ void warp_chain_regs(const uint64_t* dedup, float* dp, uint32_t* pred, uint64_t b, uint32_t c0, uint32_t c1,
                                uint32_t floor, uint32_t max_ref_gap, const ChainCtx& cc, const AnchorPack& ap,
                                float& best_score, uint32_t& best_index, uint64_t& best_key) {
    const uint32_t lane = lane_id();
    const uint64_t pmask = (1ULL << ap.pbits) - 1;
    const uint32_t qmask = (uint32_t)((1ULL << ap.qbits) - 1);
    const float kf = __uint2float_rn(cc.k);
    const uint32_t lookback = cc.cp.max_lookback;
    auto ref_of = [&](uint64_t k) { return (uint32_t)((k >> ap.qbits) & pmask); };
    uint32_t rsA = 0, qA = 0, rsB = 0, qB = 0;
    float dA = 0.0f, dB = 0.0f;
    if (c0 > floor) {
        // resuming inside a cluster: the anchors before c0 from memory
        const uint32_t jA = c0 - 1 - ((c0 - 1 - lane) & 63), jB = c0 - 1 - ((c0 - 33 - lane) & 63);
        if ((int32_t)(jA - floor) >= 0 && jA < c0) {
            const uint64_t k = dedup[b + jA];
            rsA = ref_of(k);
            qA = (uint32_t)k & qmask;
            dA = dp[b + jA];
        }
        if ((int32_t)(jB - floor) >= 0 && jB < c0) {
            const uint64_t k = dedup[b + jB];
            rsB = ref_of(k);
            qB = (uint32_t)k & qmask;
            dB = dp[b + jB];
        }
    }
    for (uint32_t i = c0; i < c1; i++) {
        const uint64_t ki = dedup[b + i];
        const uint32_t rsi = ref_of(ki), qi = (uint32_t)ki & qmask;
        uint32_t span = i > lookback ? lookback : i;
        if (span > i - floor) span = i - floor;
        bool gA, gB;
        const float sA = pair_score(rsi, qi, rsA, qA, ((i - 1 - lane) & 63) < span, max_ref_gap, cc, gA);
        const float sB = pair_score(rsi, qi, rsB, qB, ((i - 33 - lane) & 63) < span, max_ref_gap, cc, gB);
        float cur, ns;
        uint32_t cur_pred;
        scan_outcome(i, __fadd_rn(dA, sA), __fadd_rn(dB, sB), scan_order(i, gA, gB), kf, cur, cur_pred);
        if (best_index != 0xffffffffu &&
            recheck_score(ki, rsi, qi, best_key, best_score, max_ref_gap, cc, ap, ns) && ns > cur) {
            cur = ns;
            cur_pred = best_index;
        }
        if (lane == 0) {
            dp[b + i] = cur;
            pred[b + i] = cur_pred;
        }
        if (lane == (i & 31)) {
            if (i & 32) {
                rsB = rsi;
                qB = qi;
                dB = cur;
            } else {
                rsA = rsi;
                qA = qi;
                dA = cur;
            }
        }
        if (cur > best_score) {
            best_score = cur;
            best_index = i;
            best_key = ki;
        }
    }
    __syncwarp();
}

// The first anchor of [lo, hi) (one cluster) where the best-index re-check
// (src/chainer.rs:150-165) would change the DP values dp holds from scoring the cluster
// without it; hi when there is none.  Up to that anchor both scorings agree, so the
// running best (best_score / best_index / best_key, strict > updates as the reference
// makes them) is a prefix maximum, taken 32 anchors at a time by a shuffle scan; the
// re-check's test runs on every anchor at once.  On return the running best is the one
// before the returned anchor.
__device__ uint32_t recheck_first_fire(const uint64_t* dedup, const float* dp, uint64_t b, uint32_t lo, uint32_t hi,
                                       uint32_t max_ref_gap, const ChainCtx& cc, const AnchorPack& ap,
                                       float& best_score, uint32_t& best_index, uint64_t& best_key) {
    const uint32_t lane = lane_id();
    const uint64_t qmask = (1ULL << ap.qbits) - 1, pmask = (1ULL << ap.pbits) - 1;
    for (uint32_t c = lo; c < hi; c += 32) {
        const uint32_t i = c + lane;
        const bool in = i < hi;
        const float d = in ? dp[b + i] : -INFINITY;
        const uint64_t k = in ? dedup[b + i] : 0;
        // inclusive prefix (maximum, first index reaching it) over the lanes
        float pv = d;
        uint32_t pi = i;
        for (uint32_t s = 1; s < 32; s <<= 1) {
            const float v2 = __shfl_up_sync(FULL, pv, s);
            const uint32_t i2 = __shfl_up_sync(FULL, pi, s);
            if (lane >= s && v2 >= pv) {
                pv = v2;
                pi = i2;
            }
        }
        // the running best before anchor i: the carry, then lanes < lane
        float ev = __shfl_up_sync(FULL, pv, 1);
        uint32_t ei = __shfl_up_sync(FULL, pi, 1);
        if (lane == 0) ev = -INFINITY;
        float bs = best_score;
        uint32_t bi = best_index;
        bool from_chunk = false;
        if (ev > bs) {
            bs = ev;
            bi = ei;
            from_chunk = true;
        }
        const uint64_t kc = __shfl_sync(FULL, k, from_chunk ? ei - c : 0);
        const uint64_t bk = from_chunk ? kc : best_key;
        bool fire = false;
        if (in && bi != 0xffffffffu) {
            const uint32_t ri = (uint32_t)(k >> (ap.pbits + ap.qbits)), rsi = (uint32_t)((k >> ap.qbits) & pmask),
                           qi = (uint32_t)(k & qmask);
            const uint32_t rb = (uint32_t)(bk >> (ap.pbits + ap.qbits)), rsb = (uint32_t)((bk >> ap.qbits) & pmask),
                           qb = (uint32_t)(bk & qmask);
            if (rb == ri && qi > qb) {
                const uint32_t dq = qi - qb, dr = rsi - rsb;
                const uint32_t mx = dq > dr ? dq : dr, mn = dq < dr ? dq : dr;
                if (dr < max_ref_gap && dr > 0 && !ratio_above(mx, mn, cc))
                    fire = __fadd_rn(bs, chain_score(dq, dr, cc)) > d;
            }
        }
        const uint32_t fb = __ballot_sync(FULL, fire);
        if (fb) {
            const int f = __ffs(fb) - 1;
            best_score = __shfl_sync(FULL, bs, f);
            best_index = __shfl_sync(FULL, bi, f);
            best_key = __shfl_sync(FULL, bk, f);
            return c + (uint32_t)f;
        }
        // the whole chunk: carry its maximum on
        const float v31 = __shfl_sync(FULL, pv, 31);
        const uint32_t i31 = __shfl_sync(FULL, pi, 31);
        const uint64_t k31 = __shfl_sync(FULL, k, (i31 - c) & 31);
        if (v31 > best_score) {
            best_score = v31;
            best_index = i31;
            best_key = k31;
        }
    }
    return hi;
}

// The same for a small cluster [c0, c1) by one thread, without the re-check; returns
// the cluster's maximum.
__device__ float lane_chain_range(const uint64_t* dedup, float* dp, uint32_t* pred, uint64_t b, uint32_t c0,
                                  uint32_t c1, uint32_t max_ref_gap, const ChainCtx& cc, const AnchorPack& ap) {
    const uint64_t qmask = (1ULL << ap.qbits) - 1, pmask = (1ULL << ap.pbits) - 1;
    const float kf = __uint2float_rn(cc.k);
    float mx = 0.0f;
    for (uint32_t i = c0; i < c1; i++) {
        const uint64_t ki = dedup[b + i];
        const uint32_t rsi = (uint32_t)((ki >> ap.qbits) & pmask), qi = (uint32_t)(ki & qmask);
        uint32_t lookup_end = i > cc.cp.max_lookback ? i - cc.cp.max_lookback : 0;
        if (lookup_end < c0) lookup_end = c0;
        float cur = kf;
        uint32_t cur_pred = 0xffffffffu;
        for (uint32_t j = i; j-- > lookup_end;) {
            // one reference within a cluster: the reference's ref_id break cannot fire
            const uint64_t kj = dedup[b + j];
            const uint32_t rsj = (uint32_t)((kj >> ap.qbits) & pmask), qj = (uint32_t)(kj & qmask);
            if (qi < qj) continue;
            const uint32_t dq = qi - qj, dr = rsi - rsj;
            if (dr >= max_ref_gap) break;
            const uint32_t a = dq > dr ? dq : dr, m = dq < dr ? dq : dr;
            if (ratio_above(a, m, cc)) continue;
            const float ns = __fadd_rn(dp[b + j], chain_score(dq, dr, cc));
            if (ns >= cur) {
                cur = ns;
                cur_pred = j;
                if (dq == dr) break;
            }
        }
        dp[b + i] = cur;
        pred[b + i] = cur_pred;
        if (cur > mx) mx = cur;
    }
    return mx;
}


// Sort (orientations up to CHAIN_SORT_SMALL anchors, whose keys are still unsorted in
// the dedup buffer) or take the segmented sort's output, and deduplicate
// (src/chainer.rs:228-229) the anchors [b, e) of one read orientation into
// dedup[b ..]; returns the count.  The whole warp.
__device__ __forceinline__ uint32_t orientation_dedup(const uint64_t* sorted, uint64_t* dedup, uint64_t b, uint64_t e) {
    const uint32_t lane = lane_id();
    const uint32_t cnt = (uint32_t)(e - b);
    if (cnt <= CHAIN_SORT_SMALL) {
        if (cnt <= 32) return warp_sort_dedup<1>(dedup + b, cnt);
        if (cnt <= 64) return warp_sort_dedup<2>(dedup + b, cnt);
        if (cnt <= 128) return warp_sort_dedup<4>(dedup + b, cnt);
        return warp_sort_dedup<8>(dedup + b, cnt);
    }
    uint32_t N = 0;
    for (uint64_t c = b; c < e; c += 32) {
        const uint64_t i = c + lane;
        bool keep = false;
        uint64_t key = 0;
        if (i < e) {
            key = sorted[i];
            keep = i == b || sorted[i - 1] != key;
        }
        const uint32_t bal = __ballot_sync(FULL, keep);
        if (keep) dedup[b + N + __popc(bal & lanemask_lt())] = key;
        N += __popc(bal);
    }
    return N;
}

// Long read orientations (more than CHAIN_GROUP_MAX anchors), before k_chain4.  Anchors
// sorted by (reference, position) fall into clusters: a new one starts where the
// reference changes or the position jumps by max_ref_gap or more.  A predecessor scan
// never crosses into an earlier cluster (the reference's scan breaks there or skips
// without contributing), so a cluster's DP depends on the others only through the
// best-index re-check (src/chainer.rs:150-165), which can change a score only once the
// cluster holds the running best, a strict maximum over all earlier anchors.  So the
// clusters are scored at once: the small ones without the re-check, here, the large ones
// both without it and with their own running best (k_chain_big).  k_chain_long then takes
// them in order.  A cluster scored without the re-check whose maximum beats the running best
// of those before it is scored again from the first anchor where the re-check fires
// (recheck_first_fire); a large one whose own running best was ahead by then has its scores
// already (a cluster of thousands of anchors would otherwise run its serial DP twice).
//
// k_chain_long_prep: a warp per long orientation u: the dedup, the cluster starts
// (aux[b ..]), and the clusters of up to lane_max anchors scored a thread each (maxima
// at aux[T + b ..] as floats); the larger ones are queued as (u, cluster) items for
// k_chain_big, a block each.  long_n[u] / long_c[u]: anchors after dedup, clusters.
__global__ void __launch_bounds__(128) k_chain_long_prep(const uint64_t* __restrict__ off, const uint64_t* seg_off,
                                                         const uint64_t* seg_count, const uint64_t* sorted, uint64_t* dedup, float* dp,
                                                         uint32_t* pred, uint32_t* aux, uint64_t total_anchors,
                                                         AnchorPack ap, ChainCtx cc, const uint32_t* long_list,
                                                         uint32_t n_long, uint32_t* long_n, uint32_t* long_c,
                                                         uint32_t* big_items, uint32_t* n_big, uint32_t lane_max) {
    const uint32_t lane = lane_id();
    const uint64_t pmask = (1ULL << ap.pbits) - 1;
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t u = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; u < n_long; u += nwarps) {
        const uint32_t sg = long_list[u];
        const uint64_t b = seg_off[sg], e = b + seg_count[sg];
        const uint32_t N = orientation_dedup(sorted, dedup, b, e);
        __syncwarp();
        const uint32_t read_len = (uint32_t)(off[(sg >> 1) + 1] - off[sg >> 1]);
        const uint32_t max_ref_gap = cc.cp.max_ref_gap ? cc.cp.max_ref_gap : read_len;
        uint32_t* cstart = aux + b;
        float* cmax = reinterpret_cast<float*>(aux + total_anchors + b);
        uint32_t C = 0;
        for (uint32_t c = 0; c < N; c += 32) {
            const uint32_t i = c + lane;
            bool st = false;
            if (i < N) {
                if (i == 0) {
                    st = true;
                } else {
                    const uint64_t ki = dedup[b + i], kp = dedup[b + i - 1];
                    st = (ki >> (ap.pbits + ap.qbits)) != (kp >> (ap.pbits + ap.qbits)) ||
                         (uint32_t)((ki >> ap.qbits) & pmask) - (uint32_t)((kp >> ap.qbits) & pmask) >= max_ref_gap;
                }
            }
            const uint32_t bal = __ballot_sync(FULL, st);
            if (st) cstart[C + __popc(bal & lanemask_lt())] = i;
            C += __popc(bal);
        }
        __syncwarp();
        for (uint32_t c0 = 0; c0 < C; c0 += 32) {
            const uint32_t c = c0 + lane;
            bool big = false;
            if (c < C) {
                const uint32_t lo = cstart[c], hi = c + 1 < C ? cstart[c + 1] : N;
                big = hi - lo > lane_max;
                if (!big) cmax[c] = lane_chain_range(dedup, dp, pred, b, lo, hi, max_ref_gap, cc, ap);
            }
            const uint32_t bal = __ballot_sync(FULL, big);
            uint32_t at = 0;
            if (lane == 0 && bal) at = atomicAdd(n_big, (uint32_t)__popc(bal));
            at = __shfl_sync(FULL, at, 0);
            if (big) {
                const uint32_t x = at + __popc(bal & lanemask_lt());
                big_items[2 * x] = u;
                big_items[2 * x + 1] = c;
            }
        }
        if (lane == 0) {
            long_n[u] = N;
            long_c[u] = C;
        }
        __syncwarp();
    }
}

// What k_chain_big leaves of a large cluster at aux[2T + b + its first anchor ..] besides
// the maximum at aux[T + b + cluster].
struct BigCluster {
    uint32_t best_index;  // the first anchor that reaches the maximum
    uint32_t fire;        // the first anchor whose score the cluster's own re-check changed (~0u: none)
    float fire_best;      // the maximum before that anchor
};

// The queued large clusters for max_lookback < 64, a block each (their maxima into
// aux[T + b + cluster]), scored twice side by side: by the first warp with the re-check
// against the cluster's own running best (dp, pred), by the second without it (plain: the
// score's bits, the predecessor).  The first is the reference's score of every anchor if the
// best of the clusters before is already beaten when the re-check first changes a score
// (BigCluster::fire), and in any case up to that anchor; otherwise the second is from there
// on, until the cluster beats that best.  Neither bounds the other: a score that the
// re-check raised can end the scan of a later anchor on the same diagonal before a better
// predecessor, so that with it the cluster's maximum is lower.
//
// A cluster is one serial chain of anchors and the kernel lasts as long as its longest
// cluster (a tandem repeat's: thousands of anchors), so what counts is a scoring warp's
// instructions from one anchor's score to the next.  The other three warps prepare, 32 anchors
// ahead in shared memory, everything that does not depend on scores: the pair scores
// (gap, ratio test, chain_score) against the 64 anchors before, and which of them lie on
// the same diagonal.  A scoring warp holds those anchors' scores two per lane.
//
// The longest clusters of 53k-read parts on a 310 Mbp human-shaped genome (up to 3,100
// anchors): 0.34 ms a launch on average, 0.56 at most, with the first scoring alone; with the
// whole DP in one warp 1.06 and 1.69 ms, and 1.1 and 1.9 ms with the predecessors in shared
// memory.  The second scoring makes a launch a tenth longer (parts of 185k reads: 0.56 ->
// 0.62 ms on average, with cold caches) and spares k_chain_long serial work (0.43 -> 0.41,
// at most 0.73 -> 0.52); 200k pairs to PAF take 19.0 ms, 19.3 with the first alone.
constexpr uint32_t BIG_CHUNK = 32, BIG_SCORING = 2, BIG_WARPS = 5;

__global__ void __launch_bounds__(32 * BIG_WARPS) k_chain_big(const uint64_t* __restrict__ off, const uint64_t* seg_off,
                                                   const uint64_t* __restrict__ dedup, float* dp, uint32_t* pred,
                                                   uint2* plain, uint32_t* aux, uint64_t total_anchors, AnchorPack ap, ChainCtx cc,
                                                   const uint32_t* long_list, const uint32_t* long_n,
                                                   const uint32_t* long_c, const uint32_t* big_items,
                                                   const uint32_t* n_big) {
    __shared__ float s_pair[2][BIG_CHUNK][64];
    __shared__ uint64_t s_diag[2][BIG_CHUNK];  // the same-diagonal candidates in scan order
    __shared__ uint2 s_near[2][BIG_CHUNK];     // the nearest one: its distance, its pair score
    __shared__ uint2 s_pos[2][BIG_CHUNK];      // the anchor's reference position and query start
    __shared__ uint64_t s_key[128];  // anchor j's key in slot j & 127
    const uint32_t lane = lane_id(), w = threadIdx.x / 32;
    const uint64_t pmask = (1ULL << ap.pbits) - 1;
    const uint32_t qmask = (uint32_t)((1ULL << ap.qbits) - 1);
    const float kf = __uint2float_rn(cc.k);
    const uint32_t lookback = cc.cp.max_lookback;
    const uint32_t nb = *n_big;
    for (uint32_t x = blockIdx.x; x < nb; x += gridDim.x) {
        const uint32_t u = big_items[2 * x], c = big_items[2 * x + 1];
        const uint32_t sg = long_list[u], N = long_n[u], C = long_c[u];
        const uint64_t seg_b = seg_off[sg];
        const uint32_t* cstart = aux + seg_b;
        const uint32_t lo = cstart[c], n = (c + 1 < C ? cstart[c + 1] : N) - lo;
        const uint64_t b = seg_b + lo;  // anchors 0 .. n of the cluster
        const uint32_t read_len = (uint32_t)(off[(sg >> 1) + 1] - off[sg >> 1]);
        const uint32_t max_ref_gap = cc.cp.max_ref_gap ? cc.cp.max_ref_gap : read_len;
        // pair scores of chunk q's anchors, by the warps from w0 on
        auto prepare = [&](uint32_t q, uint32_t w0) {
            for (uint32_t a = w - w0; a < BIG_CHUNK; a += BIG_WARPS - w0) {
                const uint32_t i = q * BIG_CHUNK + a;
                if (i >= n) break;
                const uint64_t ki = s_key[i & 127];
                const uint32_t rsi = (uint32_t)((ki >> ap.qbits) & pmask), qi = (uint32_t)ki & qmask;
                const uint32_t span = i < lookback ? i : lookback;
                bool g[2];
#pragma unroll
                for (uint32_t h = 0; h < 2; h++) {
                    const uint32_t t = (i - 1 - lane - 32 * h) & 63;
                    const uint64_t kj = s_key[(i - 1 - t) & 127];
                    s_pair[q & 1][a][lane + 32 * h] =
                        pair_score(rsi, qi, (uint32_t)((kj >> ap.qbits) & pmask), (uint32_t)kj & qmask, t < span,
                                   max_ref_gap, cc, g[h]);
                }
                const uint64_t d = scan_order(i, g[0], g[1]);
                __syncwarp();
                if (lane == 0) {
                    const uint32_t t = d ? (uint32_t)__clzll((long long)d) : 63;
                    s_diag[q & 1][a] = d;
                    s_near[q & 1][a] =
                        make_uint2(t, __float_as_uint(d ? s_pair[q & 1][a][(i - 1 - t) & 63] : -INFINITY));
                    s_pos[q & 1][a] = make_uint2(rsi, qi);
                }
            }
        };
        __syncthreads();  // the cluster before is done with the shared buffers
        for (uint32_t j = threadIdx.x; j < 2 * BIG_CHUNK; j += blockDim.x)
            if (j < n) s_key[j] = dedup[b + j];
        __syncthreads();
        prepare(0, 0);
        __syncthreads();
        float best_score = 0.0f, fire_best = 0.0f;
        uint32_t best_index = 0xffffffffu, best_pos = 0, fire = 0xffffffffu;
        uint64_t best_key = 0;
        float dA = 0.0f, dB = 0.0f;
        const uint32_t chunks = (n + BIG_CHUNK - 1) / BIG_CHUNK;
        // Chunk q's scores.  Most anchors take the nearest candidate on their diagonal.  Its
        // score dj is fetched an anchor ahead (it is the last one's only for distance 0), so
        // that path needs one addition, one comparison and one vote from the last anchor's
        // score to this one's.
        auto score = [&](auto recheck, uint32_t q, uint32_t m) -> uint32_t {
            const uint32_t i0 = q * BIG_CHUNK;
            const bool high = q & 1;
            float sA = s_pair[q & 1][0][lane], sB = s_pair[q & 1][0][lane + 32];
            uint2 near = s_near[q & 1][0];
            uint2 pos = s_pos[q & 1][0];
            uint32_t slot = (i0 - 1 - near.x) & 63;
            float dj = __shfl_sync(FULL, slot & 32 ? dB : dA, slot & 31);
            uint32_t my_pred = 0xffffffffu;
            for (uint32_t a = 0; a < m; a++) {
                const uint32_t i = i0 + a;
                const float v0 = __fadd_rn(dj, __uint_as_float(near.y));  // -inf without one
                const float vA = __fadd_rn(dA, sA), vB = __fadd_rn(dB, sB);
                const uint32_t t0 = near.x;
                const uint2 here = pos;
                const uint32_t a1 = a + 1 < m ? a + 1 : a;
                sA = s_pair[q & 1][a1][lane];
                sB = s_pair[q & 1][a1][lane + 32];
                near = s_near[q & 1][a1];
                pos = s_pos[q & 1][a1];
                slot = (i - near.x) & 63;
                dj = __shfl_sync(FULL, slot & 32 ? dB : dA, slot & 31);
                float cur = v0, ns = 0.0f;
                uint32_t cur_pred = i - 1 - t0;
                bool again = false;
                // the re-check's score needs only the best before
                if constexpr (decltype(recheck)::value)
                    again = here.x - best_pos < max_ref_gap && best_index != 0xffffffffu &&
                            recheck_score(s_key[i & 127], here.x, here.y, best_key, best_score, max_ref_gap, cc, ap,
                                          ns);
                if (__any_sync(FULL, vA > v0 || vB > v0) || !(v0 >= kf))
                    scan_outcome(i, vA, vB, s_diag[q & 1][a], kf, cur, cur_pred);
                if (again && ns > cur) {
                    cur = ns;
                    cur_pred = best_index;
                    if (fire == 0xffffffffu) {
                        fire = i;
                        fire_best = best_score;
                    }
                }
                if (lane == a) {
                    if (high) dB = cur;
                    else dA = cur;
                    my_pred = cur_pred == 0xffffffffu ? cur_pred : lo + cur_pred;
                }
                if (near.x == 0) dj = cur;
                if constexpr (decltype(recheck)::value) {
                    if (cur > best_score) {
                        best_score = cur;
                        best_index = i;
                        best_pos = here.x;
                        best_key = s_key[i & 127];
                    }
                }
            }
            return my_pred;
        };
        for (uint32_t q = 0; q < chunks; q++) {
            const uint32_t i0 = q * BIG_CHUNK, m = n - i0 < BIG_CHUNK ? n - i0 : BIG_CHUNK;
            if (w >= BIG_SCORING) {
                // the keys of chunk q + 2 take the slots of chunk q - 2
                const uint32_t j = (q + 2) * BIG_CHUNK + lane;
                uint64_t kn = 0;
                if (w == BIG_SCORING && j < n) kn = dedup[b + j];
                if (q + 1 < chunks) prepare(q + 1, BIG_SCORING);
                if (w == BIG_SCORING && j < n) s_key[j & 127] = kn;
            } else if (w == 0) {
                const uint32_t my_pred = score(std::true_type{}, q, m);
                if (lane < m) {
                    dp[b + i0 + lane] = q & 1 ? dB : dA;
                    pred[b + i0 + lane] = my_pred;
                }
            } else {
                const uint32_t my_pred = score(std::false_type{}, q, m);
                if (lane < m) plain[b + i0 + lane] = make_uint2(__float_as_uint(q & 1 ? dB : dA), my_pred);
            }
            __syncthreads();
        }
        if (threadIdx.x == 0) {
            // a large cluster has at least three anchors (lane_max >= 2)
            uint32_t* info = aux + 2 * total_anchors + b;
            info[0] = lo + best_index;
            info[1] = fire == 0xffffffffu ? fire : lo + fire;
            info[2] = __float_as_uint(fire_best);
            reinterpret_cast<float*>(aux + total_anchors + seg_b)[c] = best_score;
        }
    }
}

// The queued large clusters for longer lookbacks, a warp each, without the re-check.
__global__ void __launch_bounds__(128) k_chain_big_far(const uint64_t* __restrict__ off, const uint64_t* seg_off,
                                                       const uint64_t* dedup, float* dp, uint32_t* pred, uint32_t* aux,
                                                       uint64_t total_anchors, AnchorPack ap, ChainCtx cc,
                                                       const uint32_t* long_list, const uint32_t* long_n,
                                                       const uint32_t* long_c, const uint32_t* big_items,
                                                       const uint32_t* n_big) {
    const uint32_t lane = lane_id();
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    const uint32_t nb = *n_big;
    for (uint32_t x = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; x < nb; x += nwarps) {
        const uint32_t u = big_items[2 * x], c = big_items[2 * x + 1];
        const uint32_t sg = long_list[u], N = long_n[u], C = long_c[u];
        const uint64_t b = seg_off[sg];
        const uint32_t* cstart = aux + b;
        const uint32_t lo = cstart[c], hi = c + 1 < C ? cstart[c + 1] : N;
        const uint32_t read_len = (uint32_t)(off[(sg >> 1) + 1] - off[sg >> 1]);
        const uint32_t max_ref_gap = cc.cp.max_ref_gap ? cc.cp.max_ref_gap : read_len;
        float mx = 0.0f;
        uint32_t bi = 0xffffffffu;
        uint64_t bk = 0;
        warp_chain_range(dedup, dp, pred, b, lo, hi, lo, max_ref_gap, cc, ap, false, mx, bi, bk);
        if (lane == 0) reinterpret_cast<float*>(aux + total_anchors + b)[c] = mx;
        __syncwarp();
    }
}

// A long orientation per warp, its clusters scored by k_chain_long_prep (without the
// re-check) and k_chain_big: in order, the clusters whose maximum beats the running best
// and those whose own re-check changed a score, then the chains.  A kernel apart from
// k_chain4: the rings there take the shared memory that the L1 needs here (the walks are
// chains of dependent loads; 300-500 cycles an anchor from L2).
template <bool RING>
__global__ void __launch_bounds__(128) k_chain_long(const uint64_t* __restrict__ off, const uint64_t* seg_off,
                                                    uint64_t* dedup, float* dp, uint32_t* pred, uint32_t* aux,
                                                    uint64_t total_anchors, unsigned long long* scratch,
                                                    const uint2* plain, AnchorPack ap, ChainCtx cc, NamRec* nam_out,
                                                    uint32_t* nam_seg_count, uint64_t* anc_out,
                                                    uint64_t* anc_start, const uint32_t* long_list, uint32_t n_long,
                                                    const uint32_t* long_n, const uint32_t* long_c,
                                                    uint32_t lane_max) {
    __shared__ uint32_t hist[4 * 256];
    constexpr uint32_t NONE = 0xffffffffu;
    const uint32_t lane = lane_id(), wib = threadIdx.x / 32;
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t u = blockIdx.x * (blockDim.x / 32) + wib; u < n_long; u += nwarps) {
        const uint32_t sg = long_list[u], N = long_n[u];
        const uint64_t b = seg_off[sg];
        const uint32_t read_len = (uint32_t)(off[(sg >> 1) + 1] - off[sg >> 1]);
        const uint32_t max_ref_gap = cc.cp.max_ref_gap ? cc.cp.max_ref_gap : read_len;
        const uint32_t* cstart = aux + b;
        const float* cmax = reinterpret_cast<const float*>(aux + total_anchors + b);
        const uint32_t* info = aux + 2 * total_anchors + b;
        const uint32_t C = long_c[u];
        float best_score = 0.0f;
        uint32_t best_index = NONE;
        uint64_t best_key = 0;
        for (uint32_t c0 = 0; c0 < C; c0 += 32) {
            const uint32_t c = c0 + lane;
            const float m = c < C ? cmax[c] : -INFINITY;
            const uint32_t my_lo = c < C ? cstart[c] : 0, my_hi = c + 1 < C ? cstart[c + 1] : N;
            const bool my_big = RING && c < C && my_hi - my_lo > lane_max;
            const uint32_t my_fire = my_big ? info[my_lo + 1] : NONE;
            uint32_t from = 0;
            for (;;) {
                const bool rec =
                    c < C && lane >= from && (best_index == NONE || m > best_score || my_fire != NONE);
                const uint32_t bal = __ballot_sync(FULL, rec);
                if (!bal) break;
                const uint32_t l = __ffs(bal) - 1;
                from = l + 1;
                const uint32_t lo = __shfl_sync(FULL, my_lo, l), hi = __shfl_sync(FULL, my_hi, l);
                uint32_t i0;
                if (__shfl_sync(FULL, my_big, l)) {
                    i0 = __shfl_sync(FULL, my_fire, l);
                    if (i0 == NONE || best_index == NONE || __uint_as_float(info[lo + 2]) > best_score) {
                        // every score of the cluster stands
                        const float cm = __shfl_sync(FULL, m, l);
                        if (cm > best_score) {
                            best_score = cm;
                            best_index = info[lo];
                            best_key = dedup[b + best_index];
                        }
                        continue;
                    }
                    // an earlier cluster held the running best when the re-check fired: from
                    // there on the scores are those without it
                    for (uint32_t i = i0 + lane; i < hi; i += 32) {
                        const uint2 s = plain[b + i];
                        dp[b + i] = __uint_as_float(s.x);
                        pred[b + i] = s.y;
                    }
                    __syncwarp();
                } else {
                    i0 = lo;
                }
                // the values scored without the re-check stand up to the first anchor
                // where it would fire; only the rest is scored again
                i0 = recheck_first_fire(dedup, dp, b, i0, hi, max_ref_gap, cc, ap, best_score, best_index, best_key);
                if (i0 < hi) {
                    if (RING)
                        warp_chain_regs(dedup, dp, pred, b, i0, hi, lo, max_ref_gap, cc, ap, best_score, best_index,
                                        best_key);
                    else
                        warp_chain_range(dedup, dp, pred, b, i0, hi, lo, max_ref_gap, cc, ap, true, best_score,
                                         best_index, best_key);
                }
            }
        }
        __syncwarp();
        chain_extract(dedup, dp, pred, aux, total_anchors, scratch, b, N, sg, best_score, ap, cc, nam_out,
                      nam_seg_count, anc_out, anc_start, hist + wib * 256);
    }
}

template <bool RING>
__global__ void __launch_bounds__(32 * CHAIN_WARPS, 8) k_chain4(const uint64_t* __restrict__ off, uint32_t n, const uint64_t* seg_off,
                                                const uint64_t* seg_count, const uint64_t* sorted, uint64_t* dedup, float* dp, uint32_t* pred,
                                                uint32_t* aux, uint64_t total_anchors, AnchorPack ap, ChainCtx cc,
                                                NamRec* nam_out, uint32_t* nam_seg_count, uint64_t* anc_out,
                                                uint64_t* anc_start, const uint32_t* seg_list, uint32_t n_list) {
    __shared__ uint64_t ring_key_s[RING ? CHAIN_WARPS * NG * 64 : 1];
    __shared__ float ring_dp_s[RING ? CHAIN_WARPS * NG * 64 : 1];
    const uint32_t lane = lane_id(), g = lane / CG, gl = lane % CG, gsh = CG * g;
    const uint32_t wib = threadIdx.x / 32;
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    const uint64_t qmask = (1ULL << ap.qbits) - 1, pmask = (1ULL << ap.pbits) - 1;
    const float kf = __uint2float_rn(cc.k);
    constexpr uint32_t NONE = 0xffffffffu;
    // units of NG orientations.  Lane q holds the q-th orientation's segment, anchor count
    // after dedup and first anchor.
    const uint32_t n_units = (n_list + NG - 1) / NG;
    for (uint32_t u = blockIdx.x * (blockDim.x / 32) + wib; u < n_units; u += nwarps) {
        uint32_t my_sg = NONE;
        {
            const uint32_t l = NG * u + lane;
            if (lane < NG && l < n_list) my_sg = seg_list[l];
        }
        // dedup (src/chainer.rs:228-229), one orientation after the other
        uint32_t my_n = 0;
        uint64_t my_b = 0;
        for (uint32_t q = 0; q < NG; q++) {
            const uint32_t sg = __shfl_sync(FULL, my_sg, q);
            if (sg == NONE) continue;
            const uint64_t b = seg_off[sg], e = b + seg_count[sg];
            const uint32_t N = orientation_dedup(sorted, dedup, b, e);
            if (lane == q) {
                my_n = N;
                my_b = b;
            }
        }
        __syncwarp();
        const uint32_t nmax = __reduce_max_sync(FULL, my_n);
        {
            // grouped DP: group g scores the g-th orientation
            const uint32_t sg = __shfl_sync(FULL, my_sg, g);
            const uint32_t N = __shfl_sync(FULL, my_n, g);
            const uint64_t b = __shfl_sync(FULL, my_b, g);
            uint64_t* ring_key = ring_key_s + (RING ? (wib * NG + g) * 64 : 0);
            float* ring_dp = ring_dp_s + (RING ? (wib * NG + g) * 64 : 0);
            const uint32_t read_len = sg != NONE ? (uint32_t)(off[(sg >> 1) + 1] - off[sg >> 1]) : 0;
            const uint32_t max_ref_gap = cc.cp.max_ref_gap ? cc.cp.max_ref_gap : read_len;
            float best_score = 0.0f;
            uint32_t best_index = 0xffffffffu;
            uint64_t best_key = 0;
            uint64_t next_key = N ? dedup[b] : 0;
            for (uint32_t i = 0; i < nmax; i++) {
                const bool act = i < N;
                const uint64_t ki = next_key;
                if (act && i + 1 < N) next_key = dedup[b + i + 1];
                const uint32_t ri = (uint32_t)(ki >> (ap.pbits + ap.qbits)), rsi = (uint32_t)((ki >> ap.qbits) & pmask),
                               qi = (uint32_t)(ki & qmask);
                const uint32_t lookup_end = i > cc.cp.max_lookback ? i - cc.cp.max_lookback : 0;
                const uint32_t span = act ? i - lookup_end : 0;  // candidates j = i-1 .. lookup_end
                float cur = kf;
                uint32_t cur_pred = 0xffffffffu;
                bool more = span > 0;
                for (uint32_t base = 0; __any_sync(FULL, more); base += CG) {
                    const uint32_t t = base + gl;
                    const bool in = more && t < span;
                    const uint32_t j = i - 1 - t;
                    bool hard, valid, diag;
                    float val;
                    chain_candidates<RING>(j, in, dedup, dp, b, ring_key, ring_dp, ri, rsi, qi, max_ref_gap, cc, ap,
                                           hard, valid, diag, val);
                    const uint32_t hb = (__ballot_sync(FULL, hard) >> gsh) & GMASK;
                    const uint32_t lim = hb ? (uint32_t)(__ffs(hb) - 1) : CG;  // lanes >= lim are not reached
                    if (gl >= lim) valid = false;
                    // exclusive prefix max of val over valid lanes in scan order
                    float incl = valid ? val : -INFINITY;
                    for (uint32_t d = 1; d < CG; d <<= 1) {
                        const float y = __shfl_up_sync(FULL, incl, d, CG);
                        if (gl >= d) incl = fmaxf(incl, y);
                    }
                    float excl = __shfl_up_sync(FULL, incl, 1, CG);
                    if (gl == 0) excl = -INFINITY;
                    const bool upd = valid && val >= fmaxf(cur, excl);
                    const uint32_t ub = (__ballot_sync(FULL, upd) >> gsh) & GMASK;
                    const uint32_t sb = (__ballot_sync(FULL, upd && diag) >> gsh) & GMASK;
                    uint32_t reach = lim;
                    bool stop = hb != 0;
                    if (sb) {
                        reach = (uint32_t)__ffs(sb);
                        stop = true;
                    }
                    const uint32_t um = ub & (reach >= CG ? GMASK : ((1u << reach) - 1));
                    const uint32_t last = um ? 31 - __clz(um) : 0;
                    const float lv = __shfl_sync(FULL, val, last, CG);
                    if (more && um) {
                        cur = lv;
                        cur_pred = i - 1 - (base + last);
                    }
                    if (stop || base + CG >= span) more = false;
                }
                // re-check of the best chain end (src/chainer.rs:150-165)
                if (act && best_index != 0xffffffffu) {
                    const uint64_t kb = best_key;
                    const uint32_t rb = (uint32_t)(kb >> (ap.pbits + ap.qbits)),
                                   rsb = (uint32_t)((kb >> ap.qbits) & pmask), qb = (uint32_t)(kb & qmask);
                    if (rb == ri && qi > qb) {
                        const uint32_t dq = qi - qb, dr = rsi - rsb;
                        const uint32_t mx = dq > dr ? dq : dr, mn = dq < dr ? dq : dr;
                        if (dr < max_ref_gap && dr > 0 && !ratio_above(mx, mn, cc)) {
                            const float ns = __fadd_rn(best_score, chain_score(dq, dr, cc));
                            if (ns > cur) {
                                cur = ns;
                                cur_pred = best_index;
                            }
                        }
                    }
                }
                if (act && gl == 0) {
                    dp[b + i] = cur;
                    pred[b + i] = cur_pred;
                    if (RING) {
                        ring_key[i & 63] = ki;
                        ring_dp[i & 63] = cur;
                    }
                }
                if (act && cur > best_score) {
                    best_score = cur;
                    best_index = i;
                    best_key = ki;
                }
                __syncwarp();
            }
            // the eight extractions side by side, a group each
            __syncwarp();
            group_chain_extract(dedup, dp, pred, aux, total_anchors, b, N, nmax, sg, best_score, ap, cc, nam_out,
                                nam_seg_count, anc_out, anc_start);
        }
    }
}

// NAM ids in push order (forward chains first), then a stable sort by score,
// descending (src/nam.rs:168-170; the tie shuffle is applied by the host policy)
// Order-preserving u32 key of a NAM score; -0 and +0 map to one key, as they compare
// equal in the reference's sort.
__device__ __forceinline__ uint32_t score_key(float s) {
    const uint32_t b = __float_as_uint(s == 0.0f ? 0.0f : s);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

__device__ __forceinline__ uint64_t nam_anchor_src(const uint64_t* anc_start, const uint64_t* seg_off, uint32_t r,
                                                   uint32_t c0, uint32_t t) {
    return t < c0 ? anc_start[seg_off[2 * r] + t] : anc_start[seg_off[2 * r + 1] + t - c0];
}

// NAM ids in push order (forward chains, then reverse) and the stable sort by score,
// descending (src/nam.rs:168-170), warp per read.  Up to 32 NAMs: ranks from the
// warp's scores by shuffles.  More: the NAMs go to tmp in push order with sort keys,
// and the read is listed for the segmented stable sort and k_nam_gather.
__global__ void __launch_bounds__(256) k_nam_compact(uint32_t n, const uint64_t* seg_off, const NamRec* scratch,
                                                     const uint32_t* nam_seg_count, const uint64_t* nam_off,
                                                     NamRec* out, NamDetailsRec* details,
                                                     const uint64_t* anc_start, uint64_t* anc_src,
                                                     uint64_t* anc_count, NamRec* tmp, uint32_t* keys,
                                                     uint32_t* vals, uint32_t* long_reads, uint64_t* long_begin,
                                                     uint64_t* long_end, uint32_t* n_long) {
    const uint32_t lane = lane_id();
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t r = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; r < n; r += nwarps) {
        const uint32_t c0 = nam_seg_count[2 * r], c1 = nam_seg_count[2 * r + 1], c = c0 + c1;
        const NamRec* s0 = scratch + seg_off[2 * r];
        const NamRec* s1 = scratch + seg_off[2 * r + 1];
        const uint64_t ob = nam_off[r];
        if (lane == 0) details[r].n_nams = c;
        if (c <= 32) {
            NamRec nr{};
            float s = 0.0f;
            if (lane < c) {
                nr = lane < c0 ? s0[lane] : s1[lane - c0];
                s = nr.score;
            }
            uint32_t rank = 0;
            for (uint32_t u = 0; u < c; u++) {
                const float su = __shfl_sync(FULL, s, u);
                rank += (su > s) || (su == s && u < lane);
            }
            if (lane < c) {
                nr.nam_id = lane;
                out[ob + rank] = nr;
                if (anc_src) {
                    anc_src[ob + rank] = nam_anchor_src(anc_start, seg_off, r, c0, lane);
                    anc_count[ob + rank] = nr.n_anchors;
                }
            }
        } else {
            for (uint32_t t = lane; t < c; t += 32) {
                NamRec nr = t < c0 ? s0[t] : s1[t - c0];
                nr.nam_id = t;
                tmp[ob + t] = nr;
                keys[ob + t] = score_key(nr.score);
                vals[ob + t] = t;
            }
            if (lane == 0) {
                const uint32_t i = atomicAdd(n_long, 1u);
                long_reads[i] = r;
                long_begin[i] = ob;
                long_end[i] = ob + c;
            }
        }
    }
}

// the sorted order of each listed read applied: out[ob + rank] = tmp[ob + perm[rank]]
__global__ void __launch_bounds__(256) k_nam_gather(uint32_t n_long, const uint32_t* long_reads,
                                                    const uint64_t* seg_off, const uint32_t* nam_seg_count,
                                                    const uint64_t* nam_off, const NamRec* tmp, const uint32_t* perm,
                                                    NamRec* out, const uint64_t* anc_start, uint64_t* anc_src,
                                                    uint64_t* anc_count) {
    const uint32_t lane = lane_id();
    const uint32_t nwarps = gridDim.x * (blockDim.x / 32);
    for (uint32_t i = blockIdx.x * (blockDim.x / 32) + threadIdx.x / 32; i < n_long; i += nwarps) {
        const uint32_t r = long_reads[i];
        const uint32_t c0 = nam_seg_count[2 * r], c = c0 + nam_seg_count[2 * r + 1];
        const uint64_t ob = nam_off[r];
        for (uint32_t k = lane; k < c; k += 32) {
            const uint32_t t = perm[ob + k];
            const NamRec nr = tmp[ob + t];
            out[ob + k] = nr;
            if (anc_src) {
                anc_src[ob + k] = nam_anchor_src(anc_start, seg_off, r, c0, t);
                anc_count[ob + k] = nr.n_anchors;
            }
        }
    }
}

__global__ void k_nam_counts(uint32_t n, const uint32_t* nam_seg_count, uint64_t* nam_count) {
    for (uint32_t r = blockIdx.x * blockDim.x + threadIdx.x; r < n; r += gridDim.x * blockDim.x)
        nam_count[r] = (uint64_t)nam_seg_count[2 * r] + nam_seg_count[2 * r + 1];
}

// each NAM's anchors, from the chaining scratch into one array in NAM output order
__global__ void k_nam_anchor_gather(uint64_t total_nams, const uint64_t* src, const uint64_t* dst_off,
                                    const uint64_t* sparse, uint64_t* dense) {
    for (uint64_t t = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; t < total_nams;
         t += (uint64_t)gridDim.x * blockDim.x) {
        const uint64_t s = src[t], d = dst_off[t], c = dst_off[t + 1] - d;
        for (uint64_t u = 0; u < c; u++) dense[d + u] = sparse[s + u];
    }
}

inline unsigned warps_grid(uint64_t items) {
    uint64_t blocks = (items + WARPS_PER_BLOCK - 1) / WARPS_PER_BLOCK;
    if (blocks > sm_count() * 32) blocks = sm_count() * 32;
    return (unsigned)(blocks ? blocks : 1);
}

uint32_t ceil_log2(uint64_t v) {
    uint32_t b = 0;
    while ((1ULL << b) < v) b++;
    return b;
}

template <class T>
void cub_excl_sum(NamWorkspace& ws, const T* in, T* out, uint64_t n, cudaStream_t st) {
    size_t tmp = 0;
    cub::DeviceScan::ExclusiveSum(nullptr, tmp, in, out, (int64_t)n, st);
    ws.cub_tmp.reserve(tmp);
    cub::DeviceScan::ExclusiveSum(ws.cub_tmp.p, tmp, in, out, (int64_t)n, st);
}

}  // namespace

uint32_t run_seeding(const SeedParams& sp, uint32_t n, uint64_t total, NamWorkspace& ws, cudaStream_t st,
                     KernelTimers* kt) {
    KernelTimers none;
    if (!kt) kt = &none;
    ws.syn_hash.reserve(total);
    ws.syn_pos.reserve(total);
    ws.qr_hash.reserve(2 * total);
    ws.qr_hash_rc.reserve(2 * total);
    ws.qr_start.reserve(2 * total);
    ws.qr_end.reserve(2 * total);
    ws.n_rs.reserve(2 * (size_t)n);
    size_t smem = WARPS_PER_BLOCK * MAX_READ_LEN;
    kt->begin(KS_SEED, st);
    k_seed<false><<<warps_grid(n), 32 * WARPS_PER_BLOCK, smem, st>>>(ws.seq.p, ws.off.p, n, sp, ws.syn_hash.p,
                                                                     ws.syn_pos.p, ws.qr_hash.p, ws.qr_hash_rc.p,
                                                                     ws.qr_start.p, ws.qr_end.p, total, ws.n_rs.p);
    kt->end(st);
    SA_CUDA(cudaGetLastError());
    return 1;
}

// Syncmer scratch of the allocation-free seeding entry point: hashes (8 bytes per
// base) then positions (4 bytes per base) for at most
// SA_RANDSTROBES_NOALLOC_MAX_BASES bases.  One copy per device, shared by every
// call on that device.  Nothing in it needs to start at zero: each read writes
// its own syncmer slots before reading them.
static __device__ __align__(256) uint8_t g_seed_scratch[(size_t)SA_RANDSTROBES_NOALLOC_MAX_BASES * 12];

void run_seeding_noalloc(const SeedParams& sp, const uint8_t* seq, const uint64_t* off, uint32_t n, uint64_t total,
                         uint64_t* qr_hash, uint64_t* qr_hash_rc, uint32_t* qr_start, uint32_t* qr_end,
                         uint32_t* counts, cudaStream_t st) {
    if (total > SA_RANDSTROBES_NOALLOC_MAX_BASES)
        throw Error(SA_ERR_INVALID, "batch has " + std::to_string(total) + " bases; the allocation-free seeding "
                                    "entry point takes at most " +
                                        std::to_string((uint64_t)SA_RANDSTROBES_NOALLOC_MAX_BASES));
    // scratch address per device and CUDA context, looked up by the first call on that
    // device in that context (a context created anew, e.g. after cudaDeviceReset,
    // looks it up again instead of using a stale address)
    constexpr int MAX_DEVICES = 64;
    using CtxGetCurrent = int (*)(void**);  // cuCtxGetCurrent(CUcontext*)
    static std::mutex mu;
    static CtxGetCurrent ctx_current = nullptr;
    static void* scratch_ctx[MAX_DEVICES] = {};
    static uint8_t* scratch[MAX_DEVICES] = {};
    int dev = 0;
    SA_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= MAX_DEVICES) throw Error(SA_ERR_CUDA, "device ordinal out of range");
    uint8_t* base;
    {
        std::lock_guard<std::mutex> g(mu);
        if (!ctx_current) {
            cudaDriverEntryPointQueryResult q{};
            SA_CUDA(cudaGetDriverEntryPointByVersion("cuCtxGetCurrent", reinterpret_cast<void**>(&ctx_current), 12000,
                                                     cudaEnableDefault, &q));
            if (q != cudaDriverEntryPointSuccess || !ctx_current)
                throw Error(SA_ERR_CUDA, "cuCtxGetCurrent is not available");
        }
        void* ctx = nullptr;
        if (ctx_current(&ctx) != 0) throw Error(SA_ERR_CUDA, "cuCtxGetCurrent failed");
        if (!ctx || !scratch[dev] || scratch_ctx[dev] != ctx) {
            // binds (or creates) the device's primary context and loads the kernel, so
            // that later calls only launch
            cudaFuncAttributes fa;
            SA_CUDA(cudaFuncGetAttributes(&fa, k_seed<true>));
            if (ctx_current(&ctx) != 0 || !ctx) throw Error(SA_ERR_CUDA, "no current CUDA context");
        }
        if (!scratch[dev] || scratch_ctx[dev] != ctx) {
            uint8_t* p = nullptr;
            SA_CUDA(cudaGetSymbolAddress((void**)&p, g_seed_scratch));
            scratch[dev] = p;
            scratch_ctx[dev] = ctx;
        }
        base = scratch[dev];
    }
    if (!n) return;
    if (!off || !counts || (total && (!seq || !qr_hash || !qr_hash_rc || !qr_start || !qr_end)))
        throw Error(SA_ERR_INVALID, "null device pointer");
    uint64_t* syn_hash = reinterpret_cast<uint64_t*>(base);
    uint32_t* syn_pos = reinterpret_cast<uint32_t*>(base + (size_t)SA_RANDSTROBES_NOALLOC_MAX_BASES * 8);
    const size_t smem = WARPS_PER_BLOCK * MAX_READ_LEN;
    k_seed<true><<<warps_grid(n), 32 * WARPS_PER_BLOCK, smem, st>>>(seq, off, n, sp, syn_hash, syn_pos, qr_hash,
                                                                    qr_hash_rc, qr_start, qr_end, total, counts);
    SA_CUDA(cudaGetLastError());
}

uint32_t run_nam_pipeline(const DevIndex& ix, const DevRefs& refs, const NamConfig& cfg, uint32_t n, uint64_t total,
                          uint32_t max_contig_len, uint32_t n_contigs, NamWorkspace& ws, cudaStream_t st,
                          KernelTimers* kt) {
    (void)refs;
    KernelTimers none;
    if (!kt) kt = &none;
    uint32_t launches = 0;
    if (!ws.log2_lut.p) {
        std::vector<float> lut(LOG2_LUT_SIZE);
        for (uint32_t d = 0; d < LOG2_LUT_SIZE; d++) lut[d] = std::log2((float)d + 1.0f);
        ws.log2_lut.reserve(LOG2_LUT_SIZE);
        SA_CUDA(cudaMemcpy(ws.log2_lut.p, lut.data(), LOG2_LUT_SIZE * sizeof(float), cudaMemcpyHostToDevice));
    }
    AnchorPack ap;
    ap.qbits = ceil_log2((uint64_t)MAX_READ_LEN + 1);
    ap.pbits = ceil_log2((uint64_t)max_contig_len + 1);
    uint32_t rbits = ceil_log2((uint64_t)n_contigs);
    if (ap.qbits + ap.pbits + rbits > 64) throw Error(SA_ERR_INVALID, "contig count/length too large for anchor keys");
    launches += run_seeding(ix.p, n, total, ws, st, kt);
    ws.hit_pos.reserve(2 * total);
    ws.hit_info.reserve(2 * total);
    ws.hit_count_cache.reserve(2 * total);
    ws.n_hits.reserve(2 * (size_t)n);
    ws.orient.reserve(n);
    ws.details.reserve(n);
    kt->begin(KS_HITS, st);
    if (cfg.mcs != SA_MCS_FIRST_STROBE) {
        k_probe<<<warps_grid(n), 32 * WARPS_PER_BLOCK, 0, st>>>(ix, ws.off.p, n, total, cfg.mcs, ws.qr_hash.p,
                                                                ws.qr_hash_rc.p, ws.n_rs.p, ws.hit_pos.p,
                                                                ws.hit_info.p);
        launches++;
    }
    k_hits<<<warps_grid(n), 32 * WARPS_PER_BLOCK, 0, st>>>(
        ix, ws.off.p, n, total, cfg.mcs, cfg.rescue_distance, ws.qr_hash.p, ws.qr_hash_rc.p, ws.qr_start.p,
        ws.qr_end.p, ws.n_rs.p, ws.hit_pos.p, ws.hit_info.p, ws.hit_count_cache.p, ws.n_hits.p, ws.orient.p,
        ws.details.p);
    kt->end(st);
    launches++;
    ws.hit_anchors.reserve(2 * total);
    ws.seg_count.reserve(2 * (size_t)n + 1);
    ws.seg_off.reserve(2 * (size_t)n + 1);
    // seg_list: short list [0, 2n), long list [2n, 4n), counts at 4n
    ws.seg_list.reserve(4 * (size_t)n + 4);
    ws.sort_begin.reserve(2 * (size_t)n);
    ws.sort_end.reserve(2 * (size_t)n);
    uint32_t* const long_list = ws.seg_list.p + 2 * (size_t)n;
    uint32_t* const list_counts = ws.seg_list.p + 4 * (size_t)n;
    ws.seg_key.reserve(4 * (size_t)n);
    ws.seg_key_alt.reserve(4 * (size_t)n);
    ws.seg_sorted.reserve(4 * (size_t)n);
    unsigned long long* const cursor = reinterpret_cast<unsigned long long*>(ws.seg_count.p + 2 * (size_t)n);
    uint64_t total_anchors = 0;
    uint32_t n_list[3] = {0, 0, 0};
    // about 40 anchors per 150 nt read of a human-sized genome
    ws.anchors.reserve(std::max<uint64_t>(ws.anchors.n, total / 3 + 64 * (uint64_t)n));
    for (;;) {
        SA_CUDA(cudaMemsetAsync(cursor, 0, 8, st));
        SA_CUDA(cudaMemsetAsync(list_counts, 0, 12, st));
        kt->begin(KS_ANCHORS, st);
        k_anchors<<<warps_grid(n), 32 * WARPS_PER_BLOCK, 0, st>>>(
            ix, ws.off.p, n, total, ws.qr_hash.p, ws.qr_start.p, ws.qr_end.p, ws.hit_pos.p, ws.hit_info.p, ws.n_hits.p,
            ws.orient.p, ws.hit_anchors.p, ws.seg_count.p, ws.seg_off.p, cursor, ws.anchors.p, ws.anchors.n, ap,
            ws.details.p);
        kt->end(st);
        k_seg_list<<<warps_grid((2 * (uint64_t)n + 31) / 32), 32 * WARPS_PER_BLOCK, 0, st>>>(
            ws.seg_count.p, ws.seg_off.p, 2 * n, ws.seg_list.p, long_list, list_counts, ws.sort_begin.p, ws.sort_end.p,
            ws.seg_key.p, ws.seg_key.p + 2 * (size_t)n);
        launches += 2;
        SA_CUDA(cudaMemcpyAsync(&total_anchors, cursor, 8, cudaMemcpyDeviceToHost, st));
        SA_CUDA(cudaMemcpyAsync(n_list, list_counts, 12, cudaMemcpyDeviceToHost, st));
        SA_CUDA(cudaStreamSynchronize(st));
        if (total_anchors <= ws.anchors.n) break;
        ws.anchors.reserve(total_anchors);  // did not fit: once more with room for all
    }
    ws.anchors_sorted.reserve(total_anchors);
    if (n_list[1]) {
        // orientations with more than CHAIN_SORT_SMALL anchors; k_chain4 sorts the rest
        size_t tmp = 0;
        kt->begin(KS_SORT, st);
        cub::DeviceSegmentedSort::SortKeys(nullptr, tmp, ws.anchors.p, ws.anchors_sorted.p, (int64_t)total_anchors,
                                           (int64_t)n_list[1], ws.sort_begin.p, ws.sort_end.p, st);
        ws.cub_tmp.reserve(tmp);
        cub::DeviceSegmentedSort::SortKeys(ws.cub_tmp.p, tmp, ws.anchors.p, ws.anchors_sorted.p,
                                           (int64_t)total_anchors, (int64_t)n_list[1], ws.sort_begin.p, ws.sort_end.p,
                                           st);
        kt->end(st);
        launches++;
    }
    // read orientations by anchor count, largest first: the eight orientations of a
    // grouped warp then have similar counts (the warp runs as many steps as its largest
    // one), and the long orientations start first
    const uint32_t* short_list = ws.seg_list.p;
    const uint32_t* long_sorted = long_list;
    {
        size_t tmp = 0, t2 = 0;
        if (n_list[0] > 1)
            cub::DeviceRadixSort::SortPairsDescending(nullptr, tmp, ws.seg_key.p, ws.seg_key_alt.p, ws.seg_list.p,
                                                      ws.seg_sorted.p, (int64_t)n_list[0], 0, 8, st);
        if (n_list[2] > 1)
            cub::DeviceRadixSort::SortPairsDescending(nullptr, t2, ws.seg_key.p, ws.seg_key_alt.p, ws.seg_list.p,
                                                      ws.seg_sorted.p, (int64_t)n_list[2], 0, 32, st);
        ws.cub_tmp.reserve(std::max(tmp, t2));
        kt->begin(KS_NAMS_OTHER, st);
        if (n_list[0] > 1) {
            cub::DeviceRadixSort::SortPairsDescending(ws.cub_tmp.p, tmp, ws.seg_key.p, ws.seg_key_alt.p,
                                                      ws.seg_list.p, ws.seg_sorted.p, (int64_t)n_list[0], 0, 8, st);
            short_list = ws.seg_sorted.p;
            launches++;
        }
        if (n_list[2] > 1) {
            const size_t o = 2 * (size_t)n;
            cub::DeviceRadixSort::SortPairsDescending(ws.cub_tmp.p, t2, ws.seg_key.p + o, ws.seg_key_alt.p + o,
                                                      long_list, ws.seg_sorted.p + o, (int64_t)n_list[2], 0, 32, st);
            long_sorted = ws.seg_sorted.p + o;
            launches++;
        }
        kt->end(st);
    }
    ws.dp.reserve(total_anchors);
    ws.pred.reserve(total_anchors);
    ws.aux.reserve(3 * total_anchors);
    ws.nam_scratch.reserve(total_anchors);
    ws.nam_seg_count.reserve(2 * (size_t)n);
    ChainCtx cc{cfg.cp, ix.p.k, ws.log2_lut.p, false, true, 0, 0};
    {
        // R = M * 2^e with M the 24-bit significand of a normal positive float
        const float R = cfg.cp.max_diagonal_ratio;
        int ex = 0;
        const float fr = std::frexp(R, &ex);  // R = fr * 2^ex, fr in [0.5, 1)
        if (std::isfinite(R) && R > 0.0f && fr != 0.0f) {
            const uint64_t M = (uint64_t)std::ldexp((double)fr, 24);  // exact: 24 significant bits
            const int e = ex - 24;
            const int shift = 1 - e;
            if (M >= (1u << 23) && M < (1u << 24) && shift >= 0 && shift <= 30) {
                cc.ratio_exact = true;
                cc.ratio_strict = (M & 1) == 0;
                cc.ratio_shift = (uint32_t)shift;
                cc.ratio_num = 2 * M + 1;
            }
        }
    }
    kt->begin(KS_CHAIN, st);
    SA_CUDA(cudaMemsetAsync(ws.nam_seg_count.p, 0, 2 * (size_t)n * sizeof(uint32_t), st));
    const uint64_t chain_units = ((uint64_t)n_list[0] + NG - 1) / NG;
    const unsigned chain_grid = (unsigned)std::max<uint64_t>(
        1, std::min<uint64_t>((chain_units + CHAIN_WARPS - 1) / CHAIN_WARPS, sm_count() * 64));
    if (cfg.nam_anchors) {
        ws.anc_sparse.reserve(3 * total_anchors + 1);
        ws.anc_start.reserve(total_anchors + 1);
    }
    uint64_t* const anc_out = cfg.nam_anchors ? ws.anc_sparse.p : nullptr;
    uint64_t* const anc_start = cfg.nam_anchors ? ws.anc_start.p : nullptr;
    // The long orientations' kernels last as long as the longest cluster's serial chain,
    // with most of the device idle: they run beside the short ones' k_chain4.
    uint32_t* const long_n = ws.seg_key_alt.p;
    uint32_t* const long_c = ws.seg_key_alt.p + 2 * (size_t)n;
    // a large cluster has three words of BigCluster at its first anchors
    const uint32_t lane_max = std::max<uint32_t>(2, cfg.chain_lane_max);
    const bool ring = cfg.cp.max_lookback < 64;
    if (n_list[2]) {
        const uint64_t cap = total_anchors / (lane_max + 1) + 1;
        ws.chain_big.reserve(2 * cap + 2);
        const cudaStream_t sl = ws.side.fork(st);
        SA_CUDA(cudaMemsetAsync(ws.chain_big.p, 0, 4, sl));
        const unsigned pgrid = (unsigned)std::min<uint64_t>(((uint64_t)n_list[2] + 3) / 4, sm_count() * 16);
        k_chain_long_prep<<<pgrid, 128, 0, sl>>>(ws.off.p, ws.seg_off.p, ws.seg_count.p, ws.anchors_sorted.p, ws.anchors.p, ws.dp.p,
                                                 ws.pred.p, ws.aux.p, total_anchors, ap, cc, long_sorted, n_list[2],
                                                 long_n, long_c, ws.chain_big.p + 2, ws.chain_big.p, lane_max);
        const unsigned bgrid = (unsigned)(sm_count() * 8);
        // the sorted anchors have been copied out: their room for the scores without the
        // re-check, then for the extraction
        uint2* const plain = reinterpret_cast<uint2*>(ws.anchors_sorted.p);
        if (ring)
            k_chain_big<<<bgrid, 32 * BIG_WARPS, 0, sl>>>(ws.off.p, ws.seg_off.p, ws.anchors.p, ws.dp.p, ws.pred.p,
                                                          plain, ws.aux.p, total_anchors, ap, cc, long_sorted, long_n,
                                                          long_c, ws.chain_big.p + 2, ws.chain_big.p);
        else
            k_chain_big_far<<<bgrid, 128, 0, sl>>>(ws.off.p, ws.seg_off.p, ws.anchors.p, ws.dp.p, ws.pred.p, ws.aux.p,
                                                   total_anchors, ap, cc, long_sorted, long_n, long_c,
                                                   ws.chain_big.p + 2, ws.chain_big.p);
        (ring ? k_chain_long<true> : k_chain_long<false>)<<<pgrid, 128, 0, sl>>>(
            ws.off.p, ws.seg_off.p, ws.anchors.p, ws.dp.p, ws.pred.p, ws.aux.p, total_anchors,
            reinterpret_cast<unsigned long long*>(ws.anchors_sorted.p), plain, ap, cc, ws.nam_scratch.p,
            ws.nam_seg_count.p, anc_out, anc_start, long_sorted, n_list[2], long_n, long_c, lane_max);
        launches += 3;
    }
    if (n_list[0]) {
        (ring ? k_chain4<true> : k_chain4<false>)<<<chain_grid, 32 * CHAIN_WARPS, 0, st>>>(
            ws.off.p, n, ws.seg_off.p, ws.seg_count.p, ws.anchors_sorted.p, ws.anchors.p, ws.dp.p, ws.pred.p, ws.aux.p,
            total_anchors, ap, cc, ws.nam_scratch.p, ws.nam_seg_count.p, anc_out, anc_start, short_list, n_list[0]);
        launches++;
    }
    if (n_list[2]) ws.side.join(st);
    kt->end(st);
    ws.nam_count.reserve((size_t)n + 1);
    ws.nam_off.reserve((size_t)n + 1);
    kt->begin(KS_NAMS_OTHER, st);
    k_nam_counts<<<(n + 255) / 256 + 1, 256, 0, st>>>(n, ws.nam_seg_count.p, ws.nam_count.p);
    SA_CUDA(cudaMemsetAsync(ws.nam_count.p + n, 0, 8, st));
    cub_excl_sum(ws, ws.nam_count.p, ws.nam_off.p, (uint64_t)n + 1, st);
    kt->end(st);
    launches += 2;
    uint64_t total_nams = 0;
    SA_CUDA(cudaMemcpyAsync(&total_nams, ws.nam_off.p + n, 8, cudaMemcpyDeviceToHost, st));
    SA_CUDA(cudaStreamSynchronize(st));
    ws.nams.reserve(total_nams);
    if (cfg.nam_anchors) {
        ws.nam_anc_src.reserve(total_nams + 1);
        ws.nam_anc_off.reserve(total_nams + 1);
    }
    ws.nam_tmp.reserve(total_nams);
    ws.nam_keys.reserve(2 * total_nams);
    ws.nam_vals.reserve(2 * total_nams);
    ws.long_reads.reserve((size_t)n + 1);
    ws.long_begin.reserve((size_t)n);
    ws.long_end.reserve((size_t)n);
    kt->begin(KS_NAMS_OTHER, st);
    SA_CUDA(cudaMemsetAsync(ws.long_reads.p + n, 0, 4, st));
    k_nam_compact<<<warps_grid(n), 32 * WARPS_PER_BLOCK, 0, st>>>(
        n, ws.seg_off.p, ws.nam_scratch.p, ws.nam_seg_count.p, ws.nam_off.p, ws.nams.p, ws.details.p,
        cfg.nam_anchors ? ws.anc_start.p : nullptr, cfg.nam_anchors ? ws.nam_anc_src.p : nullptr,
        cfg.nam_anchors ? ws.nam_anc_off.p : nullptr, ws.nam_tmp.p, ws.nam_keys.p, ws.nam_vals.p,
        ws.long_reads.p, ws.long_begin.p, ws.long_end.p, ws.long_reads.p + n);
    launches++;
    uint32_t n_long = 0;
    SA_CUDA(cudaMemcpyAsync(&n_long, ws.long_reads.p + n, 4, cudaMemcpyDeviceToHost, st));
    SA_CUDA(cudaStreamSynchronize(st));
    if (n_long) {
        uint32_t* keys_out = ws.nam_keys.p + total_nams;
        uint32_t* perm = ws.nam_vals.p + total_nams;
        size_t tmp = 0;
        cub::DeviceSegmentedSort::StableSortPairsDescending(nullptr, tmp, ws.nam_keys.p, keys_out, ws.nam_vals.p,
                                                            perm, (int64_t)total_nams, (int64_t)n_long,
                                                            ws.long_begin.p, ws.long_end.p, st);
        ws.cub_tmp.reserve(tmp);
        cub::DeviceSegmentedSort::StableSortPairsDescending(ws.cub_tmp.p, tmp, ws.nam_keys.p, keys_out,
                                                            ws.nam_vals.p, perm, (int64_t)total_nams,
                                                            (int64_t)n_long, ws.long_begin.p, ws.long_end.p, st);
        k_nam_gather<<<warps_grid(n_long), 32 * WARPS_PER_BLOCK, 0, st>>>(
            n_long, ws.long_reads.p, ws.seg_off.p, ws.nam_seg_count.p, ws.nam_off.p, ws.nam_tmp.p, perm, ws.nams.p,
            cfg.nam_anchors ? ws.anc_start.p : nullptr, cfg.nam_anchors ? ws.nam_anc_src.p : nullptr,
            cfg.nam_anchors ? ws.nam_anc_off.p : nullptr);
        launches += 2;
    }
    kt->end(st);
    ws.anchor_qbits = ap.qbits;
    ws.anchor_pbits = ap.pbits;
    ws.last_total_nam_anchors = 0;
    if (cfg.nam_anchors) {
        // counts -> offsets in place, then the gather
        SA_CUDA(cudaMemsetAsync(ws.nam_anc_off.p + total_nams, 0, 8, st));
        ws.nam_count.reserve(total_nams + 1);
        SA_CUDA(cudaMemcpyAsync(ws.nam_count.p, ws.nam_anc_off.p, (total_nams + 1) * 8, cudaMemcpyDeviceToDevice, st));
        cub_excl_sum(ws, ws.nam_count.p, ws.nam_anc_off.p, total_nams + 1, st);
        uint64_t tot = 0;
        SA_CUDA(cudaMemcpyAsync(&tot, ws.nam_anc_off.p + total_nams, 8, cudaMemcpyDeviceToHost, st));
        SA_CUDA(cudaStreamSynchronize(st));
        ws.nam_anc.reserve(tot + 1);
        if (total_nams)
            k_nam_anchor_gather<<<(unsigned)std::min<uint64_t>((total_nams + 255) / 256, sm_count() * 16), 256, 0, st>>>(
                total_nams, ws.nam_anc_src.p, ws.nam_anc_off.p, ws.anc_sparse.p, ws.nam_anc.p);
        launches += 3;
        ws.last_total_nam_anchors = tot;
    }
    SA_CUDA(cudaGetLastError());
    ws.last_total_nams = total_nams;
    return launches;
}

}  // namespace sa
