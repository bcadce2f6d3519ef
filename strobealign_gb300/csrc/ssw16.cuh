// SSW's end searches (ext/ssw/ssw.c:818-888) in packed 16-bit scores: two of the
// library's lanes per thread, one in each half of every register, so that a DPX
// instruction updates two cells.
//
// Layout.  A task's striped query (ext/ssw/ssw.c:163-596: segLen = ceil(L / 16) rows per
// lane in byte mode, ceil(L / 8) in word mode) is cut into 16 pieces of consecutive rows (a
// byte lane, or half a word lane), two per thread: thread t of a group of eight holds
// piece 2t in the low halves and piece 2t + 1 in the high halves.  The pieces form a
// wavefront over the reference columns: piece v works on column s - v at step s, takes from
// piece v - 1 its last row's H and the F / lazy-F raise that enters its rows, and hands on
// its own.  For the high half that is the thread's own low half of the step before; only
// the low half's inputs come by shuffle.  (Four threads a task with pieces twice as long
// spend fewer instructions per cell but last longer per step, and the longest windows set a
// launch's length: 36,000 tasks of 150 nt took 1.72 ms against 1.06 ms.)
//
// The recurrences are those of the warp-per-task kernel: F restarts at each lane, the
// lazy-F pass is the raise H = max(H, G - row * gap_extend) with G = max(F leaving the lane
// above, G of the lane above - segLen * gap_extend), E takes H before the raise (exact for
// gap_open > gap_extend).
//
// Scores are scaled by 32; the low five bits of a row's key hold 31 - row, so one
// instruction per two cells tracks a piece's column maximum and its first row.  Every
// piece keeps the first column that reached its own maximum.  The pass's result needs no
// more: the library's maximum is the largest of the pieces', its column the first one among
// the pieces that have it, and its row the first among those.  The reverse pass ends at
// the first column whose maximum equals the forward score; that is the same thing unless
// a piece goes beyond that score (the library's E can miss a path in one direction), and
// such a task is queued for the warp-per-task kernel.
//
// Columns before a piece's first and after its last run on a code whose scores are all
// lowest: H, E and F stay 0 before, and cannot reach the maximum again after, so there is
// no test for activity in the loop.
//
// Bound by the integer ALUs: nine instructions for two cells (a DPX add-max runs at the rate
// of its 32-bit form) and about 60 per step of a piece.  60,000 tasks of 100-300 nt (3.1 G
// cells to score, forward and reverse): 3.85 ms; in 32 bits, a warp per task above 192 nt
// and eight threads below, 17.5 ms.  8,700 tasks of 150 nt: 0.48 ms, 0.85 ms before.
#pragma once
#include <type_traits>

#include "ssw16.h"

namespace sa {

namespace {

constexpr uint32_t FULLM = 0xffffffffu;
constexpr int KEY_BITS = 5;
constexpr uint32_t ROW_BITS = 0x001f001fu;
constexpr uint32_t CODE_NONE = 5;       // no column here
constexpr uint32_t NO_BASE = 256;       // its index in the code table (CODE_TABLE uint4)
constexpr int CODE_TABLE = 17;
constexpr int T16 = 8;                  // threads per task
constexpr int SSW16_WARPS = 2;          // per block

__host__ __device__ constexpr uint32_t pack2(int v) { return (uint32_t)(uint16_t)(int16_t)v * 0x10001u; }

struct Gaps {
    uint32_t neg_open, neg_ext;  // packed, scaled, negated
    int ext;                     // scaled
    __device__ __forceinline__ uint32_t no() const { return neg_open; }
    __device__ __forceinline__ uint32_t ne() const { return neg_ext; }
    __device__ __forceinline__ int e() const { return ext; }
};
// the default penalties (12, 1) as constants: each row's raise is then one instruction
struct DefaultGaps {
    __host__ __device__ static constexpr uint32_t no() { return pack2(-(12 << KEY_BITS)); }
    __host__ __device__ static constexpr uint32_t ne() { return pack2(-(1 << KEY_BITS)); }
    __host__ __device__ static constexpr int e() { return 1 << KEY_BITS; }
};

struct End16 {
    int score, ref, read, cols;
    bool beyond;  // reverse pass: a piece went beyond the terminate score
};

__device__ __forceinline__ uint32_t add2(uint32_t a, uint32_t b) { return __vadd2(a, b); }
__device__ __forceinline__ uint32_t max2(uint32_t a, uint32_t b) { return __vmaxs2(a, b); }
__device__ __forceinline__ uint32_t addmax2(uint32_t a, uint32_t b, uint32_t c) { return __viaddmax_s16x2(a, b, c); }

// One pass for every group of the warp (those not running have rlen = 0).  n: the rows of
// the group's lanes (byte mode), or of the first halves of its lanes of seg rows (word
// mode); they sit in the last n of the NB registers, the d0 before them unused.  Only the
// first SKIP rows test for that: 0 when every group of the warp uses all registers, 4 when
// none leaves out more.
// AHEAD: the columns' codes and the first rows' profiles are read a step ahead, lane 0's
// base two steps ahead. A warp that is alone on its scheduler waits for each of these reads
// in every step otherwise (waves of 14 to 500 tasks of 150 nt: 97 to 180 us, 140 to 245
// before). Where other warps fill the waits it only costs registers: with the base alone
// read ahead, 140 for 127 at 20 rows and 188 for 152 at 32, and 60,000 tasks of 100-300 nt
// lost 5 %.
template <int NB, bool BYTE, int SKIP, bool AHEAD, class GP>
__device__ __forceinline__ End16 wave16(const uint8_t* r, int rlen, bool r_rev, int qlen, bool check_term,
                                        int terminate, int bias, GP gp, const uint4* prof, const uint8_t* code, int n,
                                        int seg, int d0) {
    constexpr int T = T16, V = 2 * T, NW = (NB + 7) / 8;
    constexpr bool SPLIT = !BYTE;  // two pieces per lane
    constexpr uint32_t STEP = NW * 32, NONE = CODE_NONE * STEP;  // a code's profile, in uint4
    constexpr bool CONST = std::is_same_v<GP, DefaultGaps>;
    const int lane = threadIdx.x & 31, gl = lane % T;
    uint32_t H[NB], E[NB];
#pragma unroll
    for (int j = 0; j < NB; j++) H[j] = E[j] = 0;
    const bool odd = SPLIT && (seg & 1);
    // G loses a gap extension per row: over a lane (piece), and over the unused registers
    const uint32_t g_rows = SPLIT ? ((uint32_t)(uint16_t)(-n * gp.e()) | ((uint32_t)(uint16_t)(-(seg - n) * gp.e()) << 16))
                                  : pack2(-n * gp.e());
    const uint32_t g_skip = pack2(d0 * gp.e());
    uint32_t hO = 0, xO = 0, gO = 0, fO = 0, hd = 0;
    uint32_t b_lo = NONE, b_hi = NONE;  // the columns' codes as profile offsets
    uint32_t bk = ROW_BITS, key_lo = 31, key_hi = 31;
    int col_lo = 0, col_hi = 0;
    int limit = rlen, cols = rlen;
    const int dir = r_rev ? -1 : 1;
    const uint8_t* rp = r + (r_rev ? rlen - 1 : 0);
    uint32_t b_next = gl == 0 && rlen > 0 ? code[*rp] * STEP : NONE;
    // AHEAD: b_lo, b_hi and the first rows' profiles are this step's already
    uint32_t base_next = NO_BASE;
    uint4 L_next, U_next;
    if (AHEAD) {
        b_lo = b_next;
        L_next = prof[b_lo];
        U_next = prof[6 * STEP + b_hi];
        rp += dir;
        b_next = rlen > 1 ? code[*rp] * STEP : NONE;
        rp += dir;
        if (rlen > 2) base_next = *rp;
    }
    int steps = __reduce_max_sync(FULLM, limit ? limit + V - 1 : 0);
    const int thr = ((BYTE && !check_term ? 255 - bias : terminate) << KEY_BITS);
    for (int s = 0; s < steps; s++) {
        const uint32_t w = __shfl_up_sync(FULLM, __byte_perm(hO, xO, 0x7632), 1, T);
        uint32_t bin = __shfl_up_sync(FULLM, b_hi, 1, T);
        if (!AHEAD) {
            b_hi = b_lo;
            if (gl == 0) {
                bin = b_next;
                rp += dir;
                b_next = s + 1 < rlen ? code[*rp] * STEP : NONE;
            }
            b_lo = bin;
        }
        const uint32_t win = gl == 0 ? 0 : w;
        const uint32_t hin = __byte_perm(win, hO, 0x5410);
        uint32_t gb = __byte_perm(win, SPLIT ? gO : xO, 0x5432);
        uint32_t diag = hd;
        hd = hin;
        uint32_t F = SPLIT ? fO << 16 : 0;
        gO = add2(gb, g_rows);
        if (SKIP) gb = add2(gb, g_skip);
        const uint4* pl = prof + b_lo;
        const uint4* ph = prof + 6 * STEP + b_hi;
        uint32_t k = 0;
        uint32_t f_last = 0;
        uint32_t gj = gb;
        uint4 L, U;
        if (AHEAD) {
            L = L_next;
            U = U_next;
            b_hi = b_lo;
            b_lo = gl == 0 ? b_next : bin;
            b_next = code[base_next] * STEP;
            rp += dir;
            base_next = s + 3 < rlen ? *rp : NO_BASE;
            L_next = prof[b_lo];
            U_next = prof[6 * STEP + b_hi];
        }
#pragma unroll
        for (int j = 0; j < NB; j++) {
            if ((j & 7) == 0 && (j > 0 || !AHEAD)) {
                L = pl[(j >> 3) * 32];
                U = ph[(j >> 3) * 32];
            }
            if (j >= SKIP || j >= d0) {
                const uint32_t lw = (&L.x)[(j >> 1) & 3], uw = (&U.x)[(j >> 1) & 3];
                const uint32_t sc = __byte_perm(lw, uw, (j & 1) ? 0x7632 : 0x5410);
                const uint32_t A = addmax2(diag, sc, E[j]);    // max(H(diag) + score, E)
                const uint32_t u = addmax2(A, gp.no(), 0);     // max(A - gap_open, 0)
                const uint32_t Hp = max2(A, F);                // H before the raise
                if (SPLIT && j == NB - 1) f_last = F;
                E[j] = addmax2(E[j], gp.ne(), addmax2(F, gp.no(), u));
                F = addmax2(F, gp.ne(), u);
                uint32_t Hr;
                if constexpr (CONST) Hr = addmax2(gb, pack2(-j * GP::e()), Hp);
                else Hr = max2(gj, Hp);
                k = addmax2(Hr, pack2(31 - j), k);
                diag = H[j];
                H[j] = Hr;
            }
            // the raise's row offset counts the unused registers too (g_skip)
            if (!CONST) gj = add2(gj, gp.ne());
        }
        hO = H[NB - 1];
        fO = F;
        if (SPLIT && odd) {
            // the lane's second piece has a row less
            hO = __byte_perm(hO, H[NB >= 2 ? NB - 2 : 0], 0x7610);
            fO = __byte_perm(F, f_last, 0x7610);
        }
        xO = max2(fO, gO);
        // pieces that passed their maximum
        const uint32_t nb = max2(bk, k), ch = nb ^ bk;
        if (ch & 0xffffu) {
            key_lo = k;
            col_lo = s;
        }
        if (ch >> 16) {
            key_hi = k >> 16;
            col_hi = s;
        }
        bk = nb | ROW_BITS;
        if ((s & 7) == 7 && (BYTE || check_term)) {
            // byte overflow ends the pass; the terminate score ends it after its column
            const bool lo = (int)(bk & 0xffffu) >= thr, hi = (int)(bk >> 16) >= thr;
            int at = limit;
            if (BYTE && !check_term) {
                if (lo || hi) at = 0;
            } else {
                if (lo) at = min(at, col_lo - 2 * gl + 1);
                if (hi) at = min(at, col_hi - 2 * gl);
            }
#pragma unroll
            for (int o = 1; o < T; o <<= 1) at = min(at, __shfl_xor_sync(FULLM, at, o, T));
            if (limit && !at) cols = min(s + 1, rlen);
            limit = at;
            steps = min(steps, __reduce_max_sync(FULLM, limit ? limit + V - 1 : 0));
        }
    }
    // the largest score, then the first column, then the first row
    auto cand = [&](int score, int col, int key, int piece) -> unsigned long long {
        const int row = (SPLIT ? (piece >> 1) * seg + (piece & 1) * n : piece * n) + 31 - (key & 31) - d0;
        return ((unsigned long long)score << 52) | ((unsigned long long)(0xffffffffu - (uint32_t)col) << 20) |
               (unsigned long long)(0xfffff - row);
    };
    const int s_lo = (int)(bk & 0xffffu) >> KEY_BITS, s_hi = (int)(bk >> 16) >> KEY_BITS;
    unsigned long long best = s_lo ? cand(s_lo, col_lo - 2 * gl, (int)key_lo, 2 * gl) : 0;
    if (s_hi) {
        const unsigned long long o = cand(s_hi, col_hi - 2 * gl - 1, (int)key_hi, 2 * gl + 1);
        best = o > best ? o : best;
    }
#pragma unroll
    for (int o = 1; o < T; o <<= 1) {
        const unsigned long long x = __shfl_xor_sync(FULLM, best, o, T);
        best = x > best ? x : best;
    }
    End16 e;
    const int mx = (int)(best >> 52);
    const int col = (int)(0xffffffffu - (uint32_t)(best >> 20)), row = 0xfffff - (int)(best & 0xfffff);
    e.score = BYTE && mx + bias >= 255 ? 255 : mx;
    e.beyond = check_term && mx > terminate;
    e.ref = mx ? (r_rev ? rlen - 1 - col : col) : (BYTE ? -1 : 0);
    e.read = mx ? min(row, qlen - 1) : 0;
    e.cols = limit ? limit : cols;
    return e;
}

// The striped profile of this thread's two pieces for a pass with NB registers per piece:
// codes A, C, G, T, other, none.
template <int NB, bool BYTE>
__device__ __forceinline__ void profile16(const uint8_t* q, int qlen, bool q_rev, int match, int mismatch, uint4* prof,
                                          const uint8_t* code, int n, int seg, int d0) {
    constexpr int NW = (NB + 7) / 8;
    const int gl = (threadIdx.x & 31) % T16;
    for (int half = 0; half < 2; half++) {
        const int piece = 2 * gl + half;
        for (int w = 0; w < NW; w++) {
            // the rows' query codes, 6 for padding (score 0), 5 for a row the lane does not have
            int c[8];
#pragma unroll
            for (int x = 0; x < 8; x++) {
                const int jl = 8 * w + x - d0;
                c[x] = 6;
                if (8 * w + x < NB && jl >= 0) {
                    const int row = BYTE ? piece * n + jl : (piece >> 1) * seg + (piece & 1) * n + jl;
                    if (!BYTE && (piece & 1) * n + jl >= seg) c[x] = 5;
                    else if (row < qlen) c[x] = code[q_rev ? q[qlen - 1 - row] : q[row]];
                }
            }
            for (int b = 0; b <= (int)CODE_NONE; b++) {
                uint32_t v[8];
#pragma unroll
                for (int x = 0; x < 8; x++) {
                    const int sv = b == (int)CODE_NONE ? -512 : c[x] == 6 ? 0 : c[x] == 5 ? -256
                                   : c[x] == b && b < 4 ? match : -mismatch;
                    v[x] = (uint32_t)(uint16_t)(int16_t)(sv * (1 << KEY_BITS));
                }
                prof[((half * 6 + b) * NW + w) * 32] =
                    make_uint4(v[0] | v[1] << 16, v[2] | v[3] << 16, v[4] | v[5] << 16, v[6] | v[7] << 16);
            }
        }
    }
}

// A pass of the groups that run: with NB registers per piece where that is enough for
// the warp's longest lane (the next size otherwise, MAXNB at last), the profiles of their
// pieces, then the wavefront.
template <int NB, int MAXNB, bool BYTE, bool AHEAD, class GP>
__device__ __forceinline__ End16 pass16(bool run, const uint8_t* q, int qlen, bool q_rev, const uint8_t* r, int rlen,
                                        bool r_rev, bool check_term, int terminate, int match, int mismatch, int bias,
                                        GP gp, uint4* prof, const uint8_t* code, int n, int seg, int nmax, int nmin) {
    if constexpr (NB < MAXNB) {
        constexpr int NEXT = NB == 8 ? 10 : NB == 10 ? 12 : NB + 4;
        if (NB - nmin > 4 || nmax > NB)
            return pass16<NEXT, MAXNB, BYTE, AHEAD, GP>(run, q, qlen, q_rev, r, rlen, r_rev, check_term, terminate,
                                                        match, mismatch, bias, gp, prof, code, n, seg, nmax, nmin);
    }
    const int d0 = run ? NB - n : 0;
    if (run) profile16<NB, BYTE>(q, qlen, q_rev, match, mismatch, prof, code, n, seg, d0);
#define SA_W16(S) \
    wave16<NB, BYTE, S, AHEAD, GP>(r, run ? rlen : 0, r_rev, qlen, check_term, terminate, bias, gp, prof, code, n, seg, \
                                   d0)
    if constexpr (std::is_same_v<GP, DefaultGaps>) {
        if (nmin == NB) return SA_W16(0);
        if (NB < MAXNB || NB - nmin <= 4) return SA_W16(4);
    }
    if constexpr (NB == MAXNB) return SA_W16(NB);
#undef SA_W16
}

template <int MAXNB, bool BYTE, bool AHEAD, class GP>
__device__ __forceinline__ End16 pass16(bool run, const uint8_t* q, int qlen, bool q_rev, const uint8_t* r, int rlen,
                                        bool r_rev, bool check_term, int terminate, int match, int mismatch, int bias,
                                        GP gp, uint4* prof, const uint8_t* code) {
    if (qlen <= 0) run = false;
    End16 z;
    z.score = 0;
    z.ref = BYTE ? -1 : 0;
    z.read = qlen - 1;
    z.cols = 0;
    z.beyond = false;
    if (!__any_sync(FULLM, run)) return z;
    const int seg = !run ? 0 : BYTE ? (qlen + 15) / 16 : (qlen + 7) / 8;
    const int n = BYTE ? seg : (seg + 1) / 2;
    const int nmax = __reduce_max_sync(FULLM, n), nmin = __reduce_min_sync(FULLM, run ? n : nmax);
    // other gap penalties: one size, all rows tested
    constexpr int FIRST = std::is_same_v<GP, DefaultGaps> ? 8 : MAXNB;
    const End16 e = pass16<FIRST, MAXNB, BYTE, AHEAD, GP>(run, q, qlen, q_rev, r, rlen, r_rev, check_term, terminate,
                                                          match, mismatch, bias, gp, prof, code, n, seg, nmax, nmin);
    return run ? e : z;
}

// A lower bound of the score ssw.c's striped passes reach (in either striping), from
// the NAM's diagonal: the best local path over the T diagonals around d0 with at most one
// gap of up to 3 bases, one diagonal per thread of the group (all 32 threads enter).  Such
// a path is a lower bound of the passes' H: every H takes the diagonal term; a gap entered
// from a cell reached diagonally is counted by E (computed from H before the lazy-F raise,
// which already holds the diagonal term) or by F (exact after the lazy-F loop); only a path
// that goes F then E could be missed, and none is used.  When the bound reaches
// 255 - bias, the byte pass must overflow, so the task can run its word pass directly with
// the same results.  Returns the group's bound (0 when the group does not run).
template <int T>
__device__ __forceinline__ int diag_bound(bool run, const uint8_t* q, int qlen, const uint8_t* r, int rlen, int d0,
                                          int match, int mismatch, int go, int ge, int gl, const uint8_t* code) {
    constexpr int NEG = -(1 << 28);
    const int rows = __reduce_max_sync(FULLM, run ? qlen : 0);
    const int delta = d0 + gl - T / 2;
    int A = NEG, B = NEG, best = 0;
    int h1 = NEG, h2 = NEG, h3 = NEG;  // A on this diagonal 1, 2, 3 rows back (h1 = A(i - 1))
    for (int i = 0; i < rows; i++) {
        const bool in = run && i < qlen;
        const int j = i + delta;
        int s = NEG;
        if (in && j >= 0 && j < rlen) {
            const int qc = code[q[i]], rc = code[r[j]];
            s = (qc == rc && qc < 4) ? match : -mismatch;
        }
        // entries into this diagonal after one gap: deletion from a lower diagonal
        // (lane - g, row i - 1), insertion from a higher one (lane + g, row i - 1 - g)
        const int d1 = __shfl_up_sync(FULLM, h1, 1, T), d2 = __shfl_up_sync(FULLM, h1, 2, T),
                  d3 = __shfl_up_sync(FULLM, h1, 3, T);
        const int i1 = __shfl_down_sync(FULLM, h2, 1, T), i2 = __shfl_down_sync(FULLM, h3, 2, T);
        int x = NEG;
        if (gl >= 1) x = max(x, d1 - go);
        if (gl >= 2) x = max(x, d2 - go - ge);
        if (gl >= 3) x = max(x, d3 - go - 2 * ge);
        if (gl + 1 < T) x = max(x, i1 - go);
        if (gl + 2 < T) x = max(x, i2 - go - ge);
        if (s == NEG) {
            A = NEG;
            B = NEG;
        } else {
            A = max(A, 0) + s;
            B = max(B, x) + s;
            best = max(best, max(A, B));
        }
        h3 = h2;
        h2 = h1;
        h1 = A;
    }
#pragma unroll
    for (int o = T / 2; o; o >>= 1) best = max(best, __shfl_xor_sync(FULLM, best, o, T));
    return run ? best : 0;
}

// PAIR: a block's two warps share four tasks, the first for the byte passes, the second
// for the word passes: the forward passes of a task run at once, whether the byte pass
// overflows or not.  More work but less latency, for launches that leave SMs idle: 140
// rescue tasks (windows of up to 600 columns) 0.15 ms; 0.21 ms without the reads
// ahead, 0.35 ms with the passes one after the other.
template <int NB, bool PAIR, class GP>
__global__ void __launch_bounds__(32 * SSW16_WARPS, NB > 20 ? 4 : 6)
    k_ssw16(SswTask* tasks, const uint32_t* order, uint32_t n_tasks, const PrepRec* prep, const uint8_t* arena,
            AlignScores sc, GP gp, int bias, uint32_t* counters, uint32_t qmax, uint32_t* redo, uint32_t* n_redo,
            int32_t* hscratch) {
    constexpr int T = T16, NW = (NB + 7) / 8, G = 32 / T;
    extern __shared__ __align__(16) uint4 s16_smem[];
    __shared__ uint32_t s_base;
    __shared__ End16 s_end[2][G];
    // the code table, then each warp's profiles
    uint8_t* code = reinterpret_cast<uint8_t*>(s16_smem);
    for (int i = threadIdx.x; i < 256; i += blockDim.x) {
        const char u = (char)(i & 0xdf);
        code[i] = i >= 128 ? 4 : u == 'A' || u == 'U' ? 0 : u == 'C' ? 1 : u == 'G' ? 2 : u == 'T' ? 3 : 4;
    }
    if (threadIdx.x == 0) code[NO_BASE] = CODE_NONE;
    __syncthreads();
    const int lane = threadIdx.x & 31, gi = lane / T, gl = lane % T, wib = threadIdx.x / 32;
    uint4* prof = s16_smem + CODE_TABLE + wib * (2 * 6 * NW * 32) + lane;
    unsigned long long* cells = reinterpret_cast<unsigned long long*>(counters + 8);
    for (;;) {
        uint32_t base = 0;
        if (PAIR) {
            __syncthreads();
            if (threadIdx.x == 0) s_base = atomicAdd(&counters[30], (uint32_t)G);
            __syncthreads();
            base = s_base;
        } else {
            if (lane == 0) base = atomicAdd(&counters[30], (uint32_t)G);
            base = __shfl_sync(FULLM, base, 0);
        }
        if (base >= n_tasks) break;
        const uint32_t li = base + gi;
        uint32_t ti = 0;
        bool have = li < n_tasks;
        int qlen = 0, wlen = 0;
        uint32_t d0 = NO_DIAG;
        const uint8_t* q = arena;
        if (have) {
            ti = order ? order[li] : li;
            const PrepRec& pr = prep[tasks[ti].job];
            have = pr.qlen <= qmax;  // longer reads: another kernel's task
            if (have) {
                qlen = (int)pr.qlen;
                wlen = (int)pr.wlen;
                q = arena + pr.arena_off;
                d0 = pr.diag;
            }
        }
        const uint8_t* r = q + qlen;
        // a byte pass that must overflow is skipped: the word pass alone gives the same
        // results (the task's diagonal bound reaches 255 - bias).  Where the two run side by
        // side, the bound would only come before both (22 us at 150 nt).
        const bool try_bound = !PAIR && have && d0 != NO_DIAG && qlen * (int)sc.match >= 255 - bias;
        bool certain = false;
        if (!PAIR && __any_sync(FULLM, try_bound))
            certain = diag_bound<T>(try_bound, q, qlen, r, wlen, (int)d0, sc.match, sc.mismatch, sc.gap_open,
                                    sc.gap_extend, gl, code) >= 255 - bias;
        // forward: byte, word on overflow (ext/ssw/ssw.c:840-862)
        End16 e, ew;
        if (!PAIR || wib == 0)
            e = pass16<NB, true, PAIR, GP>(have && !certain, q, qlen, false, r, wlen, false, false, 0, sc.match,
                                           sc.mismatch, bias, gp, prof, code);
        if (!PAIR || wib == 1)
            ew = pass16<NB, false, PAIR, GP>(have && (PAIR || certain || e.score == 255), q, qlen, false, r, wlen,
                                             false, false, 0, sc.match, sc.mismatch, bias, gp, prof, code);
        if (PAIR) {
            if (gl == 0) s_end[wib][gi] = wib ? ew : e;
            __syncthreads();
            e = s_end[0][gi];
            ew = s_end[1][gi];
        }
        const bool word = have && (certain || e.score == 255);
        const unsigned long long c_fb = certain ? 0 : (unsigned long long)qlen * e.cols;
        const unsigned long long c_fw = PAIR || word ? (unsigned long long)qlen * ew.cols : 0;
        if (word) e = ew;
        // reverse pass over read[0..=read_end1] and ref[0..=ref_end1] (ext/ssw/ssw.c:870-888)
        const bool rev = have && e.ref >= 0;
        End16 b;
        if (!PAIR || wib == 0)
            b = pass16<NB, true, PAIR, GP>(rev && !word, q, e.read + 1, true, r, e.ref + 1, true, true, e.score,
                                           sc.match, sc.mismatch, bias, gp, prof, code);
        if (!PAIR || wib == 1) {
            const End16 bw = pass16<NB, false, PAIR, GP>(rev && word, q, e.read + 1, true, r, e.ref + 1, true, true,
                                                         e.score, sc.match, sc.mismatch, bias, gp, prof, code);
            if (word) b = bw;
        }
        if (!rev) {
            b.score = 0;
            b.ref = -1;
            b.read = e.read;
            b.cols = 0;
            b.beyond = false;
        }
        // the warp of the task's mode has its reverse pass
        const bool mine = have && (!PAIR || wib == (int)word);
        // Both ends known, equally long spans whose diagonal alone scores score1: banded_sw
        // would find that diagonal (its first band holds it; a cell of it above the
        // diagonal's own prefix sum would make a path better than score1, and its
        // traceback takes the diagonal on ties).  The passes miss only paths with an
        // insertion next to a deletion, which within that band cost no less than the
        // mismatches they replace if mismatch <= gap_open + gap_extend.
        const int ql = b.read + 1, qs = e.read - b.read, rs = b.ref;
        const bool even = mine && rev && e.score <= b.score && !b.beyond && e.ref - rs + 1 == ql &&
                          (int)sc.mismatch <= (int)sc.gap_open + (int)sc.gap_extend;
        int same = 0;
        for (int i = gl; even && i < ql; i += T) {
            const int c = code[q[qs + i]];
            same += c < 4 && c == code[r[rs + i]];
        }
#pragma unroll
        for (int o = 1; o < T; o <<= 1) same += __shfl_xor_sync(FULLM, same, o, T);
        const bool ungapped = even && same * (int)sc.match - (ql - same) * (int)sc.mismatch == e.score;
        if (mine && gl == 0) {
            SswTask& tk = tasks[ti];
            tk.score1 = e.score;
            tk.ref_end1 = e.ref;
            tk.read_end1 = e.read;
            tk.word = word;
            tk.ref_begin1 = b.ref;
            tk.read_begin1 = e.read - b.read;
            tk.flag = e.score > b.score ? 2 : 0;
            if (ungapped) {
                // as k_band_small leaves a task: its CIGAR after the rows' words
                const uint64_t at = prep[tk.job].h_off + 4 * (uint64_t)ql;
                hscratch[at] = ql << 4;
                tk.band_width = 1;
                tk.raw_len = 1;
                tk.raw_off = at;
            }
            if (b.beyond) redo[atomicAdd(n_redo, 1u)] = ti;
            const unsigned long long c_r = (unsigned long long)(e.read + 1) * b.cols;
            if (c_fb) atomicAdd(cells + 1, c_fb);
            if (c_fw) atomicAdd(cells + 2, c_fw);
            if (c_r) atomicAdd(cells + (word ? 4 : 3), c_r);
        }
        __syncwarp();
    }
}

inline bool ssw16_default_gaps(const AlignScores& sc) { return sc.gap_open == 12 && sc.gap_extend == 1; }

inline Gaps other_gaps(const AlignScores& sc) {
    return Gaps{pack2(-((int)sc.gap_open << KEY_BITS)), pack2(-((int)sc.gap_extend << KEY_BITS)),
                (int)sc.gap_extend << KEY_BITS};
}

template <int NB, bool PAIR, class GP>
void launch_one(const Ssw16Args& a, GP gp) {
    constexpr int NW = (NB + 7) / 8, G = 32 / T16;
    const size_t smem = (CODE_TABLE + (size_t)SSW16_WARPS * 2 * 6 * NW * 32) * sizeof(uint4);
    SA_CUDA(cudaFuncSetAttribute(k_ssw16<NB, PAIR, GP>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const uint64_t per_block = (uint64_t)(PAIR ? 1 : SSW16_WARPS) * G;
    const uint64_t blocks = std::min<uint64_t>((a.n_tasks + per_block - 1) / per_block, sm_count() * 32);
    k_ssw16<NB, PAIR, GP><<<(unsigned)std::max<uint64_t>(1, blocks), 32 * SSW16_WARPS, smem, a.st>>>(
        a.tasks, a.order, a.n_tasks, a.prep, a.arena, a.sc, gp, a.bias, a.counters, a.qmax, a.redo, a.n_redo,
        a.hscratch);
}

template <bool PAIR>
void launch_sizes(const Ssw16Args& a, uint32_t longest) {
    if (ssw16_default_gaps(a.sc)) {
        if (longest <= 192) launch_one<12, PAIR>(a, DefaultGaps{});
        else if (longest <= 320) launch_one<20, PAIR>(a, DefaultGaps{});
        else launch_one<32, PAIR>(a, DefaultGaps{});
    } else {
        // Other gap penalties take the row offsets at run time, with one register size for
        // up to 192 nt and one beyond, and never the paired form.  All of them measured faster
        // than the 32-bit kernels (whole alignment calls, match/mismatch/open/extend): 100
        // tasks of 150 nt 1/4/6/1 1.47 -> 0.81 ms, 2/4/8/2 1.58 -> 1.05, 4/6/10/2 1.56 ->
        // 1.02, 5/4/20/3 1.56 -> 1.01; 3,000 of 100-300 nt 4.8 -> 3.6, 5.3 -> 2.9, 5.2 -> 4.2,
        // 5.2 -> 4.2; 20,000 9.5 -> 4.5, 13.7 -> 4.5, 15.3 -> 6.2, 14.9 -> 8.4 ms.
        if (longest <= 192) launch_one<12, false>(a, other_gaps(a.sc));
        else launch_one<32, false>(a, other_gaps(a.sc));
    }
}

}  // namespace

}  // namespace sa
