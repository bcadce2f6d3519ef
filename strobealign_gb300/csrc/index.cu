// GPU construction of the StrobemerIndex (src/indexer.rs:18-253) and batched
// lookups (src/index.rs:127-338).
//
// Build: (1) one thread per reference position tests the canonical open-syncmer
// condition on the 2-bit reference (the reference never holds N: wildcards are
// pseudo-random bases, src/packed_seq.rs:50-59, so a syncmer is a pure function of
// its k-mer window); (2) the flagged positions are compacted in order; (3) one
// thread per syncmer picks its partner among the next w_min..w_max syncmers of the
// same contig within max_dist (src/seeding/strobes.rs:145-176); (4) a radix sort on
// the full 128-bit (hash_offset, position, ref_index) key reproduces the reference's
// sorted order exactly; (5) the bucket directory and the repeat cutoff are derived
// from the sorted table.
#include <cub/cub.cuh>
#include <cuda/std/tuple>
#include <thrust/iterator/counting_iterator.h>

#include "host_state.h"
#include "index_device.cuh"

namespace sa {

namespace {

// 2-bit base i of a contig (LSB-first packing)
__device__ __forceinline__ uint64_t bases_le(const uint64_t* w, uint64_t i, uint32_t nb) {
    // nb <= 32 bases starting at i, packed little-endian (base i in bits 0..1)
    uint64_t wi = i >> 5;
    uint32_t sh = (uint32_t)(i & 31) * 2;
    uint64_t v = w[wi] >> sh;
    if (sh + 2 * nb > 64) v |= w[wi + 1] << (64 - sh);
    return nb == 32 ? v : (v & ((1ULL << (2 * nb)) - 1));
}

// reverse the order of the 2-bit groups of a 64-bit word
__device__ __forceinline__ uint64_t rev2(uint64_t x) {
    x = __brevll(x);
    return ((x >> 1) & 0x5555555555555555ULL) | ((x & 0x5555555555555555ULL) << 1);
}

// canonical value of the nb-mer at i: min(forward, reverse complement)
// (src/seeding/syncmers.rs:186-199, 217-221)
__device__ __forceinline__ uint64_t canonical(const uint64_t* w, uint64_t i, uint32_t nb, bool* is_fwd) {
    uint64_t le = bases_le(w, i, nb);
    uint64_t fwd = rev2(le) >> (64 - 2 * nb);
    uint64_t mask = nb == 32 ? ~0ULL : ((1ULL << (2 * nb)) - 1);
    uint64_t rc = (~le) & mask;
    if (is_fwd) *is_fwd = fwd <= rc;
    return fwd < rc ? fwd : rc;
}

__device__ __forceinline__ uint32_t find_contig(const uint64_t* cstart, uint32_t n, uint64_t g) {
    uint32_t lo = 0, hi = n;  // last c with cstart[c] <= g
    while (hi - lo > 1) {
        uint32_t mid = (lo + hi) / 2;
        if (cstart[mid] <= g) lo = mid;
        else hi = mid;
    }
    return lo;
}

// Open-syncmer flag of every reference position: the (t-1)-th of the k-mer's k-s+1 s-mer
// hashes equals their minimum.  A warp takes 32 consecutive s-mers at a time, one hash
// per lane, and shuffles give each of the first 32 - (k - s) lanes the hashes of its
// k-mer, so a position costs 32 / (32 - (k - s)) hashes instead of k - s + 1.  Its
// FLAG_RUN windows are consecutive: the contig is searched for once, and lanes past its
// end step on from there.  Bound by the hash's 64-bit multiplies and the shuffles: 100 Mbp
// (k 20, s 16) take 0.77 ms; a thread per position with its five hashes and its own
// contig search took 1.96 ms.
constexpr uint32_t FLAG_RUN = 16;

__global__ void __launch_bounds__(256) k_syncmer_flags(const uint64_t* words, const uint64_t* word_off,
                                                       const uint32_t* clen, const uint64_t* cstart, uint32_t ncontig,
                                                       uint64_t total, SeedParams p, uint8_t* flags) {
    const uint32_t lane = threadIdx.x & 31, span = p.k - p.s, step = 32 - span;
    const uint64_t run = (uint64_t)step * FLAG_RUN, nruns = (total + run - 1) / run;
    const uint64_t nwarps = (uint64_t)gridDim.x * (blockDim.x / 32);
    for (uint64_t w = blockIdx.x * (uint64_t)(blockDim.x / 32) + threadIdx.x / 32; w < nruns; w += nwarps) {
        uint32_t c = find_contig(cstart, ncontig, w * run);
        uint64_t c0 = cstart[c], c1 = cstart[c + 1];
        for (uint32_t x = 0; x < FLAG_RUN; x++) {
            const uint64_t g = w * run + (uint64_t)x * step + lane;
            while (g >= c1 && c + 1 < ncontig) {
                c++;
                c0 = c1;
                c1 = cstart[c + 1];
            }
            const uint64_t pos = g - c0, left = c1 > g ? c1 - g : 0;
            const uint64_t h = left >= p.s && left ? xxh64_u64(canonical(words + word_off[c], pos, p.s, nullptr)) : 0;
            uint64_t mn = h, ht = p.t == 1 ? h : 0;
            for (uint32_t d = 1; d <= span; d++) {
                const uint64_t y = __shfl_down_sync(0xffffffffu, h, d);
                mn = y < mn ? y : mn;
                if (d == p.t - 1) ht = y;
            }
            // left >= k: the k-mer's s-mers are those of lanes lane .. lane + span
            if (lane < step && left) flags[g] = left >= p.k && ht == mn;
        }
    }
}

struct SyncmerRec {
    uint64_t hash;
    uint32_t pos;
    uint32_t contig_fwd;  // contig << 1 | is_forward
};

__global__ void k_syncmer_info(const uint64_t* words, const uint64_t* word_off, const uint64_t* cstart,
                               uint32_t ncontig, const uint64_t* gpos, const uint64_t* count, SeedParams p,
                               SyncmerRec* out) {
    uint64_t n = *count;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t g = gpos[i];
        uint32_t c = find_contig(cstart, ncontig, g);
        uint64_t pos = g - cstart[c];
        bool fwd;
        uint64_t v = canonical(words + word_off[c], pos, p.k, &fwd);
        out[i] = SyncmerRec{xxh64_u64(v), (uint32_t)pos, (c << 1) | (fwd ? 1u : 0u)};
    }
}

// src/seeding/strobes.rs:145-176 + src/indexer.rs:239-250
__global__ void k_ref_randstrobes(const SyncmerRec* sy, const uint64_t* count, SeedParams p, RefRandstrobe* out) {
    uint64_t n = *count;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        SyncmerRec s1 = sy[i];
        uint32_t c = s1.contig_fwd >> 1;
        uint64_t maxpos = (uint64_t)s1.pos + p.max_dist;
        uint64_t best = UINT64_MAX;
        SyncmerRec s2 = s1;
        for (uint64_t j = i + p.w_min; j <= i + p.w_max && j < n; j++) {
            SyncmerRec cj = sy[j];
            if ((cj.contig_fwd >> 1) != c) break;
            if (cj.pos > maxpos) break;
            uint64_t ones = (uint64_t)__popcll((s1.hash ^ cj.hash) & p.q);
            if (ones < best) {
                best = ones;
                s2 = cj;
            }
        }
        uint64_t h = randstrobe_hash(s1.hash, s2.hash, s1.contig_fwd & 1, s2.contig_fwd & 1, p);
        uint64_t off = (uint8_t)(s2.pos - s1.pos);
        out[i] = RefRandstrobe{(h & HASH_MASK) | off, s1.pos, c};
    }
}

struct RsDecomposer {
    __host__ __device__ ::cuda::std::tuple<uint64_t&, uint32_t&, uint32_t&> operator()(RefRandstrobe& r) const {
        return {r.hash_offset, r.position, r.ref_index};
    }
};

// One pass over the sorted table for everything derived from it:
//
// * the bucket directory exactly as src/indexer.rs:82-124 fills it: bucket_starts[0] = 0,
//   and for x >= 1 the first position p >= 1 that starts a new hash with top bits >= x (N
//   if none).  Entry 0 only ever starts bucket 0, so when the smallest hash has top
//   bits t > 0, buckets 1..t begin at the end of its run;
// * the histogram of the run lengths of equal hashes (src/indexer.rs:82-137), capped at
//   101 (a run's walk stops there), and the number of distinct hashes in hist[102];
// * the largest position and reference index (extent[0], extent[1]).
//
// Bound by the table's bytes.  Nearly all runs have one entry: they are counted in
// registers, the others in shared counters, so that the global counters take a block's
// sum instead of two 64-bit additions per run on the same two addresses.  20 M entries
// (320 MB): 0.15 ms, 2.1 TB/s; directory, histogram and extent took 13.8 ms as three
// kernels, 13.6 of them in those additions.
__global__ void __launch_bounds__(256) k_table_scan(const RefRandstrobe* rs, uint64_t n, uint32_t bits,
                                                    uint64_t* buckets, unsigned long long* hist,
                                                    unsigned int* extent) {
    __shared__ unsigned int s_hist[103];
    __shared__ unsigned int s_ext[2];
    for (uint32_t t = threadIdx.x; t < 103; t += blockDim.x) s_hist[t] = 0;
    if (threadIdx.x < 2) s_ext[threadIdx.x] = 0;
    __syncthreads();
    const uint64_t nb = (1ULL << bits) + 1;
    const uint64_t h0 = n ? rs_hash(rs[0]) : 0;
    unsigned int mp = 0, mr = 0, starts = 0, ones = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i <= n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t h = 0, hp = 0;
        if (i < n) {
            const RefRandstrobe e = load_rs(rs, i);
            h = rs_hash(e);
            mp = max(mp, e.position);
            mr = max(mr, e.ref_index);
        }
        if (i > 0) hp = load_hash(rs, i - 1);
        if (i > 0 && i < n && h == hp) continue;  // not the start of a new hash
        int64_t lo, hi;
        if (i == 0) {
            lo = -1;
            hi = n == 0 ? (int64_t)nb - 1 : 0;
        } else {
            lo = hp == h0 ? 0 : (int64_t)(hp >> (64 - bits));
            hi = i == n ? (int64_t)nb - 1 : (int64_t)(h >> (64 - bits));
        }
        for (int64_t x = lo + 1; x <= hi; x++) buckets[x] = i;
        if (i < n) {
            uint32_t c = 1;
            while (c < 101 && i + c < n && load_hash(rs, i + c) == h) c++;
            starts++;
            if (c == 1) ones++;
            else atomicAdd(&s_hist[c], 1u);
        }
    }
    for (int d = 16; d > 0; d >>= 1) {
        mp = max(mp, __shfl_xor_sync(0xffffffffu, mp, d));
        mr = max(mr, __shfl_xor_sync(0xffffffffu, mr, d));
        starts += __shfl_xor_sync(0xffffffffu, starts, d);
        ones += __shfl_xor_sync(0xffffffffu, ones, d);
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&s_ext[0], mp);
        atomicMax(&s_ext[1], mr);
        atomicAdd(&s_hist[102], starts);
        atomicAdd(&s_hist[1], ones);
    }
    __syncthreads();
    if (threadIdx.x < 2) atomicMax(extent + threadIdx.x, s_ext[threadIdx.x]);
    for (uint32_t t = threadIdx.x; t < 103; t += blockDim.x)
        if (s_hist[t]) atomicAdd(&hist[t], (unsigned long long)s_hist[t]);
}

__global__ void k_lookup(DevIndex ix, const uint64_t* hashes, uint64_t n, int kind, int64_t* out_pos,
                         uint32_t* out_count) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t mask = kind == 0 ? HASH_MASK : kind == 1 ? ix.p.main_mask : ix.p.fwd_main_mask;
        uint64_t pos = idx_get_masked_from(ix, hashes[i], mask, false, 0);
        out_pos[i] = pos == UINT64_MAX ? -1 : (int64_t)pos;
        if (out_count) out_count[i] = pos == UINT64_MAX ? 0 : idx_get_count(ix, pos, mask);
    }
}

__global__ void k_extent(const RefRandstrobe* rs, uint64_t n, unsigned int* out) {
    unsigned int mp = 0, mr = 0;
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += (uint64_t)gridDim.x * blockDim.x) {
        mp = max(mp, rs[i].position);
        mr = max(mr, rs[i].ref_index);
    }
    atomicMax(out, mp);
    atomicMax(out + 1, mr);
}

inline unsigned grid_for(uint64_t n, unsigned block) {
    uint64_t g = (n + block - 1) / block;
    if (g > sm_count() * 64) g = sm_count() * 64;
    return (unsigned)(g == 0 ? 1 : g);
}

// eight blocks of 256 threads fill an SM; a block's sums go to the global counters once
inline unsigned scan_grid(uint64_t n) { return std::min(grid_for(n, 256), (unsigned)sm_count() * 8); }

}  // namespace

void build_index_gpu(const std::vector<Contig>& contigs, const SeedParams& sp, uint32_t bits, double filter_fraction,
                     sa_index& idx, cudaStream_t st) {
    const uint32_t nc = (uint32_t)contigs.size();
    std::vector<uint64_t> word_off(nc), cstart(nc + 1, 0);
    std::vector<uint32_t> clen(nc);
    uint64_t nwords = 0;
    for (uint32_t c = 0; c < nc; c++) {
        word_off[c] = nwords;
        nwords += contigs[c].words.size() + 1;  // one guard word per contig
        clen[c] = (uint32_t)contigs[c].len;
        cstart[c + 1] = cstart[c] + contigs[c].len;
    }
    const uint64_t total = cstart[nc];
    DevBuf<uint64_t> d_words, d_woff, d_cstart;
    DevBuf<uint32_t> d_clen;
    d_words.reserve(nwords);
    d_woff.reserve(nc);
    d_cstart.reserve(nc + 1);
    d_clen.reserve(nc);
    {
        std::vector<uint64_t> hw(nwords, 0);
        for (uint32_t c = 0; c < nc; c++)
            std::copy(contigs[c].words.begin(), contigs[c].words.end(), hw.begin() + word_off[c]);
        SA_CUDA(cudaMemcpyAsync(d_words.p, hw.data(), nwords * 8, cudaMemcpyHostToDevice, st));
        SA_CUDA(cudaMemcpyAsync(d_woff.p, word_off.data(), nc * 8, cudaMemcpyHostToDevice, st));
        SA_CUDA(cudaMemcpyAsync(d_cstart.p, cstart.data(), (nc + 1) * 8, cudaMemcpyHostToDevice, st));
        SA_CUDA(cudaMemcpyAsync(d_clen.p, clen.data(), nc * 4, cudaMemcpyHostToDevice, st));
        SA_CUDA(cudaStreamSynchronize(st));
    }
    // (1) syncmer flags
    DevBuf<uint8_t> d_flags;
    d_flags.reserve(total);
    if (total)
        k_syncmer_flags<<<grid_for((total + 13) / 14, 256), 256, 0, st>>>(d_words.p, d_woff.p, d_clen.p, d_cstart.p, nc,
                                                                           total, sp, d_flags.p);
    // (2) compaction in position order
    DevBuf<uint64_t> d_gpos, d_count;
    d_gpos.reserve(total + 1);
    d_count.reserve(1);
    SA_CUDA(cudaMemsetAsync(d_count.p, 0, 8, st));
    if (total) {
        size_t tmp = 0;
        thrust::counting_iterator<uint64_t> it(0);
        cub::DeviceSelect::Flagged(nullptr, tmp, it, d_flags.p, d_gpos.p, d_count.p, (int64_t)total, st);
        DevBuf<uint8_t> d_tmp;
        d_tmp.reserve(tmp);
        cub::DeviceSelect::Flagged(d_tmp.p, tmp, it, d_flags.p, d_gpos.p, d_count.p, (int64_t)total, st);
    }
    uint64_t nsy = 0;
    SA_CUDA(cudaMemcpyAsync(&nsy, d_count.p, 8, cudaMemcpyDeviceToHost, st));
    SA_CUDA(cudaStreamSynchronize(st));
    d_flags.release();
    // (3) syncmers -> randstrobes (one per syncmer, src/seeding/strobes.rs:216-238)
    DevBuf<SyncmerRec> d_sy;
    d_sy.reserve(nsy);
    if (nsy) k_syncmer_info<<<grid_for(nsy, 256), 256, 0, st>>>(d_words.p, d_woff.p, d_cstart.p, nc, d_gpos.p, d_count.p, sp, d_sy.p);
    d_gpos.release();
    DevBuf<RefRandstrobe> d_unsorted;
    d_unsorted.reserve(nsy, true);
    if (nsy) k_ref_randstrobes<<<grid_for(nsy, 256), 256, 0, st>>>(d_sy.p, d_count.p, sp, d_unsorted.p);
    SA_CUDA(cudaStreamSynchronize(st));
    SA_CUDA(cudaGetLastError());
    d_sy.release();
    // (4) sort on (hash_offset, position, ref_index).  The radix sort is stable and the
    // randstrobes come by (ref_index, position), so the reference index needs no pass, a
    // single contig's positions none either, and several contigs' positions only those
    // bits that the longest contig has: 11 passes of 8 bits for contigs below 2^24 nt
    // and 8 for one contig, of the 16 that the whole 128-bit key takes (240 us each for
    // 20 M entries: 2.66 ms of passes for 24 contigs, 3.68 ms before).
    idx.rs.reserve(nsy, true);
    if (nsy) {
        uint32_t max_len = 0;
        for (uint32_t c = 0; c < nc; c++) max_len = std::max(max_len, clen[c]);
        const int pos_bits = nc > 1 ? 32 - __builtin_clz(max_len | 1u) : 0;
        cub::DoubleBuffer<RefRandstrobe> db(d_unsorted.p, idx.rs.p);
        auto sort_bits = [&](void* tmp, size_t& bytes, int b0, int b1) {
            SA_CUDA(cub::DeviceRadixSort::SortKeys(tmp, bytes, db, (int64_t)nsy, RsDecomposer{}, b0, b1, st));
        };
        size_t tp = 0, th = 0;
        if (pos_bits) sort_bits(nullptr, tp, 32, 32 + pos_bits);
        sort_bits(nullptr, th, 64, 128);
        DevBuf<uint8_t> d_tmp;
        d_tmp.reserve(std::max(tp, th));
        if (pos_bits) sort_bits(d_tmp.p, tp, 32, 32 + pos_bits);
        sort_bits(d_tmp.p, th, 64, 128);
        SA_CUDA(cudaStreamSynchronize(st));
        if (db.Current() != idx.rs.p) {
            std::swap(d_unsorted.p, idx.rs.p);
            std::swap(d_unsorted.n, idx.rs.n);
        }
    }
    d_unsorted.release();
    // (5) bucket directory and filter cutoff
    uint64_t nb = (1ULL << bits) + 1;
    idx.buckets.reserve(nb, true);
    DevBuf<unsigned long long> d_hist;  // the histogram, then the two extents
    d_hist.reserve(104);
    SA_CUDA(cudaMemsetAsync(d_hist.p, 0, 104 * 8, st));
    k_table_scan<<<scan_grid(nsy + 1), 256, 0, st>>>(idx.rs.p, nsy, bits, idx.buckets.p, d_hist.p,
                                                      reinterpret_cast<unsigned int*>(d_hist.p + 103));
    unsigned long long hist[104];
    SA_CUDA(cudaMemcpyAsync(hist, d_hist.p, sizeof(hist), cudaMemcpyDeviceToHost, st));
    SA_CUDA(cudaStreamSynchronize(st));
    SA_CUDA(cudaGetLastError());
    uint64_t unique = hist[102];
    // counts of repeated hashes sorted descending; the entry at index_cutoff, clamped
    uint64_t n_rep = 0;
    for (int c = 2; c <= 101; c++) n_rep += hist[c];
    uint64_t index_cutoff = (uint64_t)((double)unique * filter_fraction);
    uint64_t cutoff;
    if (index_cutoff < n_rep) {
        // value v with (#counts >= v) > index_cutoff >= (#counts > v); bin 101 stands for >= 101
        uint64_t above = 0;
        cutoff = 2;
        for (int c = 101; c >= 2; c--) {
            above += hist[c];
            if (above > index_cutoff) { cutoff = (uint64_t)c; break; }
        }
    } else if (n_rep > 0) {
        cutoff = 101;
        for (int c = 2; c <= 101; c++)
            if (hist[c]) { cutoff = (uint64_t)c; break; }
    } else {
        cutoff = 30;
    }
    if (cutoff < 30) cutoff = 30;
    if (cutoff > 100) cutoff = 100;
    idx.filter_cutoff = (uint32_t)cutoff;
    idx.bits = bits;
    idx.n = nsy;
    idx.sp = sp;
    idx.max_pos = (uint32_t)hist[103];
    idx.n_refs_seen = nsy ? (uint32_t)(hist[103] >> 32) + 1 : 1;
}

void index_extent_gpu(const sa_index& idx, uint32_t& max_pos, uint32_t& max_ref, cudaStream_t st) {
    DevBuf<unsigned int> d;
    d.reserve(2);
    SA_CUDA(cudaMemsetAsync(d.p, 0, 8, st));
    if (idx.n) k_extent<<<grid_for(idx.n, 256), 256, 0, st>>>(idx.rs.p, idx.n, d.p);
    unsigned int h[2];
    SA_CUDA(cudaMemcpyAsync(h, d.p, 8, cudaMemcpyDeviceToHost, st));
    SA_CUDA(cudaStreamSynchronize(st));
    max_pos = h[0];
    max_ref = h[1];
}

void lookup_batch_gpu(const sa_index& idx, const uint64_t* hashes, size_t n, int kind, int64_t* out_pos,
                      uint32_t* out_count, cudaStream_t st) {
    if (n == 0) return;
    DevBuf<uint64_t> d_h;
    DevBuf<int64_t> d_p;
    DevBuf<uint32_t> d_c;
    d_h.reserve(n);
    d_p.reserve(n);
    if (out_count) d_c.reserve(n);
    SA_CUDA(cudaMemcpyAsync(d_h.p, hashes, n * 8, cudaMemcpyHostToDevice, st));
    k_lookup<<<grid_for(n, 256), 256, 0, st>>>(idx.view(), d_h.p, n, kind, d_p.p, out_count ? d_c.p : nullptr);
    SA_CUDA(cudaGetLastError());
    SA_CUDA(cudaMemcpyAsync(out_pos, d_p.p, n * 8, cudaMemcpyDeviceToHost, st));
    if (out_count) SA_CUDA(cudaMemcpyAsync(out_count, d_c.p, n * 4, cudaMemcpyDeviceToHost, st));
    SA_CUDA(cudaStreamSynchronize(st));
}

}  // namespace sa
