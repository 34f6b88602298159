// Exact k-clique count (4 <= k <= 7) by bit-matrix induced subgraphs (sm_100a).
//
// On the degree-ordered copy (id 0 = largest degree) every k-clique is
// counted once, at its largest id v0 (its member of smallest degree).  The
// other members lie in L = N<(v0) = {u in N(v0) : u < v0}: the first lo(v0)
// entries of v0's sorted row, which the orientation keeps short (at most
// 668 on R-MAT 2^20 with 16M edges although the largest degree is 64,337).
// With L sorted, the subgraph induced on L is a bit matrix R: row i has bit
// j (j < i) set iff L[j] is a neighbour of L[i].  A k-clique at v0 is then a
// (k-1)-clique of R taken in decreasing index order:
//
//   k = 4:  sum_i  sum_{j in R_i}  |R_i & R_j|
//   k = 5:  sum_i  sum_{j in R_i}  sum_{l in R_i & R_j}  |R_i & R_j & R_l|
//
// and so on; the innermost level is a popcount, never an enumeration.  The
// exact schedule plan of K_k (all restrictions v_b < v_a, level-1 units
// v1 < v0) counts the same cliques at the same roots, so root ranges and
// shards agree between the two paths.
//
// Two kernels split the roots by lo(v0):
//  * clique_warp_kernel: a warp per root with lo(v0) <= kWarpD (rows of at
//    most two words, in the warp's slice of shared memory).  It meets the
//    larger roots too and lists them by size;
//  * clique_cta_kernel: a CTA per listed root, longest lists first, one root
//    at a time (neighbouring ids have lists of like length, so a CTA that
//    took 32 ids at once was the whole tail of a small graph's count).
//    v0's list is staged into shared memory by one bulk copy (cp.async.bulk,
//    completion on an mbarrier, waits bounded); the matrix is in shared
//    memory when it fits and in a per-CTA slice of global scratch otherwise
//    (lo(v0) up to 2048).
//
// Building row i intersects N<(L[i]) with L[0, i).  Three ways, chosen per
// row:
//  * L[i] has a bitmap row: lanes take j and test bit L[j] of that row (one
//    load each, four words or rows in flight); the warp's ballot is one word
//    of R_i;
//  * scan: lanes read consecutive entries of N<(L[i]), four loads each in
//    flight, and look them up in a hash table of L in shared memory (one or
//    two probes; a binary search of L was 7 to 9);
//  * probe: when N<(L[i]) is much longer than i, lanes take j and
//    binary-search L[j] in it; the ballot is one word of R_i.
//
// Counting.  f_F(M) = number of F-cliques of a bit matrix M; a root adds
// f_{K-1} of its own.  f_3(M) = sum over set bits (a, b) of |M_a & M_b|: the
// set bits of all rows are compacted into a per-warp queue (ballot + popc)
// and every lane takes one (a, b), so rows with few bits leave no lane idle.
// For K >= 5 the matrix is first compacted to the members of a row: bit
// (a, b) of C is bit (pos a, pos b) of R for the positions of R_i's set bits.
// C's rows are as short as row i's clique neighbourhood (|R_i| / 32 words
// instead of lo(v0) / 32), and for |R_i| <= kSubD one lane holds a whole
// M_a & M_b in registers and walks the levels below it alone (lane_dfs).
// Rows with more set bits are compacted by the whole CTA into the part of
// the matrix region the root left free.  On R-MAT 2^18 (avg. degree 58) the
// 5-clique spent 126 of 129 ms walking full-length rows, a warp per (i, j).
//
// Neither kernel waits on another CTA.  The only inter-CTA traffic is the
// root cursors, the root lists and the total.
#include <algorithm>

#include "engine.hpp"

namespace gat {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kMaxD = kCliqueMaxLower;  // longest lower list (64 words a row)
constexpr int kMaxWords = kMaxD / 32;
constexpr int kWarpD = 64;              // roots up to this go to the warp kernel
constexpr int kWarpPitch = 3;           // row pitch of the warp kernel's matrix
constexpr int kWarpThreads = 256;
constexpr int kCtaThreads = kCliqueCtaThreads;
constexpr int kCtaWarps = kCtaThreads / 32;
constexpr int kQueue = 64;
constexpr int kRootChunk = 32;            // most root ids per cursor grab
constexpr unsigned kWaitLimit = 1u << 24;  // mbarrier polls before giving up
constexpr int kSubD = 96;                 // members of a warp's compacted matrix
constexpr int kSubWords = kSubD / 32;     // its row pitch (odd: lanes of different
static_assert(kSubWords % 2 == 1, "");    // rows hit different banks)
constexpr uint16_t kNone = 0xFFFF;

// Matrix words in shared memory: two CTAs fit an SM in both forms.
template <int K>
constexpr int row_smem_words() {
    return K == 4 ? 17 * 1024 : 13 * 1024;
}

__device__ __forceinline__ int words_below(int q) { return (q + 31) >> 5; }

// Row pitch for a root with d lower neighbours: words of the longest row,
// made odd so lanes reading rows of different candidates hit different banks.
__host__ __device__ __forceinline__ int row_pitch(int d) { return ((d + 31) >> 5) | 1; }

__device__ __forceinline__ unsigned lanemask_lt() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_lt;" : "=r"(m));
    return m;
}

__device__ __forceinline__ int ceil_log2(int x) { return x <= 1 ? 1 : 32 - __clz(x - 1); }

// Hash table of a sorted list's elements: slot -> 5 bits of the element's
// hash above the 11 bits of its index (a slot of another element is told
// from them without reading the list), kNone empty, at most half full.
static_assert(kMaxD <= 2048, "an index takes 11 bits");

__device__ __forceinline__ unsigned hash_of(int32_t x) { return (unsigned)x * 0x9E3779B1u; }
// 5 hash bits that do not choose the slot, never all ones (kNone is free)
__device__ __forceinline__ unsigned hash_tag(unsigned h) { return min(h & 31u, 30u); }

__device__ __forceinline__ void hash_add(uint16_t *T, int bits, int32_t x, int index) {
    const unsigned mask = (1u << bits) - 1u, hx = hash_of(x);
    const unsigned short e = (unsigned short)(hash_tag(hx) << 11 | (unsigned)index);
    unsigned h = hx >> (32 - bits);
    while (atomicCAS(reinterpret_cast<unsigned short *>(T + h), (unsigned short)kNone, e) != kNone)
        h = (h + 1) & mask;
}

// Index of x in L, or -1.
__device__ __forceinline__ int hash_find(const uint16_t *T, int bits, const int32_t *L,
                                         int32_t x) {
    const unsigned mask = (1u << bits) - 1u, hx = hash_of(x), tag = hash_tag(hx);
    unsigned h = hx >> (32 - bits);
    for (;;) {
        const unsigned e = T[h];
        if (e == kNone) return -1;
        if ((e >> 11) == tag && L[e & 2047u] == x) return (int)(e & 2047u);
        h = (h + 1) & mask;
    }
}

// Membership of x in the sorted global list b[0, n): branch-free search.
__device__ __forceinline__ bool contains(const int32_t *b, int n, int32_t x) {
    if (n <= 0) return false;
    int lo = 0, len = n;
    while (len > 1) {
        const int h = len >> 1;
        lo = (__ldg(b + lo + h) <= x) ? lo + h : lo;
        len -= h;
    }
    return __ldg(b + lo) == x;
}

struct CliqueArgs {
    const int64_t *off;
    const int32_t *adj;  // rows padded: 4 readable ints past the last entry
    const int64_t *lo_off;
    const int32_t *hub_slot;  // null: no bitmaps
    const uint32_t *bitmaps;
    int64_t bitmap_words;
    int64_t v_begin, v_end;   // roots holding the units [u_begin, u_end)
    int64_t u_begin, u_end;   // level-1 units (v0, L[i]) numbered by lo_off
    DevCounters *ctr;
    CliqueAux *aux;
    uint32_t *rows;       // CTA kernel: per-CTA matrix for roots too large for
    int64_t rows_stride;  // shared memory (null when none is)
    int32_t *lists;       // kCliqueLists root lists, by length of lower list
    int64_t list_at[kCliqueLists];
};

__device__ __forceinline__ int32_t lower_degree(const CliqueArgs &a, int64_t v) {
    return (int32_t)(a.lo_off[v + 1] - a.lo_off[v]);
}

// Rows [*r0, *r1) of root v0 (d rows) are units of this launch: unit
// lo_off[v0] + i is (v0, L[i]), and its cliques are row i's.
__device__ __forceinline__ void unit_rows(const CliqueArgs &a, int64_t v0, int d, int *r0,
                                          int *r1) {
    const int64_t lb = a.lo_off[v0];
    *r0 = (int)max((int64_t)0, a.u_begin - lb);
    *r1 = (int)min((int64_t)d, a.u_end - lb);
}

// Words [0, words_below(i)) of R_i = { j < i : L[j] in N(L[i]) } for a row
// without a bitmap.  One warp; T: hash table of L.
// STATS adds the intersection's list bytes 4 (|N<(L[i])| + i).
template <bool STATS>
__device__ void scan_row(const CliqueArgs &a, const int32_t *L, int i, uint32_t *Ri,
                         const uint16_t *T, int bits, int lane, unsigned long long &bytes) {
    const int nw = words_below(i);
    const int32_t u = L[i];
    const int64_t o = a.off[u];
    const int32_t nu = lower_degree(a, u);
    if (STATS && lane == 0) bytes += 4ull * (unsigned)(nu + i);
    const int32_t *N = a.adj + o;
    if ((long long)i * ceil_log2(nu + 1) * 8 < nu) {
        // probe: few candidates against a long list
        for (int w = 0; w < nw; w++) {
            const int j = (w << 5) + lane;
            const bool f = j < i && contains(N, nu, L[j]);
            const unsigned word = __ballot_sync(kFull, f);
            if (lane == 0) Ri[w] = word;
        }
        return;
    }
    for (int w = lane; w < nw; w += 32) Ri[w] = 0u;
    __syncwarp();
    // lanes on consecutive entries, four loads a lane in flight
    constexpr int kAhead = 4;
    for (int q = lane; q < nu; q += 32 * kAhead) {
        int32_t xs[kAhead];
#pragma unroll
        for (int t = 0; t < kAhead; t++) xs[t] = q + 32 * t < nu ? __ldg(N + q + 32 * t) : -1;
#pragma unroll
        for (int t = 0; t < kAhead; t++) {
            if (xs[t] < 0) continue;
            const int j = hash_find(T, bits, L, xs[t]);
            if (j >= 0 && j < i) atomicOr(Ri + (j >> 5), 1u << (j & 31));
        }
    }
    __syncwarp();
}

// The same for a row with bitmap `slot`.  One warp.
template <bool STATS>
__device__ __forceinline__ void bitmap_row(const CliqueArgs &a, const int32_t *L, int i, int slot,
                                           uint32_t *Ri, int lane, unsigned long long &bytes) {
    const int nw = words_below(i);
    const uint32_t *bm = a.bitmaps + (int64_t)slot * a.bitmap_words;
    constexpr int kAhead = 4;
    for (int w0 = 0; w0 < nw; w0 += kAhead) {
        uint32_t f[kAhead];
#pragma unroll
        for (int t = 0; t < kAhead; t++) {
            const int j = ((w0 + t) << 5) + lane;
            const int32_t y = j < i ? L[j] : 0;
            f[t] = j < i ? __ldg(bm + (y >> 5)) >> (y & 31) : 0u;
        }
#pragma unroll
        for (int t = 0; t < kAhead; t++) {
            const unsigned word = __ballot_sync(kFull, f[t] & 1u);
            if (lane == 0 && w0 + t < nw) Ri[w0 + t] = word;
        }
    }
    if (STATS && lane == 0) bytes += 8ull * (unsigned)i;
}

// sum over w < n of popc(m[w] & r[w])
__device__ __forceinline__ unsigned pop_and(const uint32_t *m, const uint32_t *r, int n) {
    unsigned c = 0;
    for (int w = 0; w < n; w++) c += __popc(m[w] & r[w]);
    return c;
}

// The last level: lanes take the set bits q of m[0, nw) and add
// popc(m & R_q) over R_q's words.  Q: the warp's queue (kQueue entries).
__device__ unsigned long long last_level(const uint32_t *m, int nw, const uint32_t *R, int pitch,
                                         int32_t *Q, int lane, unsigned long long &words) {
    unsigned long long c = 0;
    int nq = 0;
    for (int w = 0; w < nw; w++) {
        const uint32_t x = m[w];
        if (x == 0u) continue;
        if ((x >> lane) & 1u) Q[nq + __popc(x & lanemask_lt())] = (w << 5) + lane;
        nq += __popc(x);
        if (nq >= 32) {
            __syncwarp();
            const int q = Q[lane];
            const int n = words_below(q);
            c += pop_and(m, R + (int64_t)q * pitch, n);
            words += (unsigned)n;
            const int rest = nq - 32;
            const int32_t moved = lane < rest ? Q[32 + lane] : 0;
            __syncwarp();
            if (lane < rest) Q[lane] = moved;
            nq = rest;
            __syncwarp();
        }
    }
    __syncwarp();
    if (lane < nq) {
        const int q = Q[lane];
        const int n = words_below(q);
        c += pop_and(m, R + (int64_t)q * pitch, n);
        words += (unsigned)n;
    }
    __syncwarp();
    return c;
}

// Cliques continuing from mask m[0, nw) with DEPTH more levels walked by the
// whole warp before the last one.  stack: DEPTH buffers of kMaxWords words.
template <int DEPTH>
__device__ unsigned long long walk(const uint32_t *m, int nw, const uint32_t *R, int pitch,
                                   uint32_t *stack, int32_t *Q, int lane,
                                   unsigned long long &words) {
    if constexpr (DEPTH == 0) {
        return last_level(m, nw, R, pitch, Q, lane, words);
    } else {
        unsigned long long c = 0;
        for (int w = 0; w < nw; w++) {
            uint32_t x = m[w];
            while (x != 0u) {
                const int j = (w << 5) + __ffs(x) - 1;
                x &= x - 1;
                const int n2 = words_below(j);
                const uint32_t *Rj = R + (int64_t)j * pitch;
                unsigned any = 0;
                for (int t = lane; t < n2; t += 32) {
                    const uint32_t y = m[t] & Rj[t];
                    stack[t] = y;
                    any |= y;
                }
                words += (unsigned)(lane < n2 ? (n2 - lane + 31) / 32 : 0);
                // a mask with no bits cannot continue
                if (__any_sync(kFull, any != 0u)) {
                    __syncwarp();
                    c += walk<DEPTH - 1>(stack, n2, R, pitch, stack + kMaxWords, Q, lane, words);
                }
                __syncwarp();
            }
        }
        return c;
    }
}

// f_{D+2} of the members of mask m, walked by one lane: M's rows are W words
// (zero above the diagonal), m in registers.
template <int D, int W>
__device__ __forceinline__ unsigned lane_dfs(const uint32_t (&m)[W], const uint32_t *M, int pitch,
                                             unsigned long long &words) {
    unsigned c = 0;
    if constexpr (D == 0) {
#pragma unroll
        for (int w = 0; w < W; w++) c += __popc(m[w]);
    } else {
#pragma unroll
        for (int w = 0; w < W; w++) {
            uint32_t x = m[w];
            while (x != 0u) {
                const uint32_t *r = M + ((w << 5) + __ffs(x) - 1) * pitch;
                x &= x - 1;
                uint32_t m2[W];
#pragma unroll
                for (int t = 0; t < W; t++) m2[t] = t <= w ? m[t] & r[t] : 0u;
                words += w + 1;
                c += lane_dfs<D - 1, W>(m2, M, pitch, words);
            }
        }
    }
    return c;
}

// A warp's queue of set bits (a, b) of a matrix's rows.
struct PairQueue {
    int32_t *Q;  // kQueue entries: a << 11 | b   (a, b < 2048)
    int n = 0;
};

// Value of one queue entry: |M_a & M_b| over any length of row ...
struct PopPair {
    const uint32_t *M;
    int pitch;
    __device__ __forceinline__ unsigned operator()(int32_t e, unsigned long long &words) const {
        const int b = e & 2047, n = words_below(b);
        words += (unsigned)n;
        return pop_and(M + (int64_t)(e >> 11) * pitch, M + (int64_t)b * pitch, n);
    }
};
// ... or the cliques of D more members below (a, b) in rows of W words.
template <int D, int W>
struct DfsPair {
    const uint32_t *M;
    int pitch;
    __device__ __forceinline__ unsigned operator()(int32_t e, unsigned long long &words) const {
        const uint32_t *ra = M + (e >> 11) * pitch, *rb = M + (e & 2047) * pitch;
        uint32_t m[W];
#pragma unroll
        for (int w = 0; w < W; w++) m[w] = ra[w] & rb[w];
        words += W;
        return lane_dfs<D, W>(m, M, pitch, words);
    }
};

template <class Value>
__device__ __forceinline__ void pairs_push_row(PairQueue &pq, const uint32_t *row, int i,
                                               const Value &value, int lane,
                                               unsigned long long &c, unsigned long long &words) {
    const int nw = words_below(i);
    for (int w = 0; w < nw; w++) {
        const uint32_t x = row[w];
        if (x == 0u) continue;
        if ((x >> lane) & 1u)
            pq.Q[pq.n + __popc(x & lanemask_lt())] = (i << 11) | ((w << 5) + lane);
        pq.n += __popc(x);
        if (pq.n >= 32) {
            __syncwarp();
            c += value(pq.Q[lane], words);
            const int rest = pq.n - 32;
            const int32_t moved = lane < rest ? pq.Q[32 + lane] : 0;
            __syncwarp();
            if (lane < rest) pq.Q[lane] = moved;
            pq.n = rest;
            __syncwarp();
        }
    }
}

template <class Value>
__device__ __forceinline__ void pairs_flush(PairQueue &pq, const Value &value, int lane,
                                            unsigned long long &c, unsigned long long &words) {
    __syncwarp();
    if (lane < pq.n) c += value(pq.Q[lane], words);
    pq.n = 0;
    __syncwarp();
}

// Positions of the set bits of row[0, nw), in order, into pos; returns how
// many there are (nothing is written past `most`).  One warp.
__device__ __forceinline__ int set_positions(const uint32_t *row, int nw, uint16_t *pos, int most,
                                             int lane) {
    int n = 0;
    for (int w = 0; w < nw; w++) {
        const uint32_t x = row[w];
        const int at = n + __popc(x & lanemask_lt());
        if (((x >> lane) & 1u) && at < most) pos[at] = (uint16_t)((w << 5) + lane);
        n += __popc(x);
    }
    return n;
}

// A warp's room for one compacted matrix.
struct SubSmem {
    uint32_t C[kSubD * kSubWords];
    uint16_t pos[kSubD];
};

// f_F of the members of R's row r: compacted to their own matrix and counted
// a lane per set bit; members beyond kSubD are walked in R by the whole warp.
template <int F>
__device__ __forceinline__ unsigned long long sub_count(const uint32_t *R, int pitch, int r,
                                                        SubSmem &S, uint32_t *stack, int32_t *Q,
                                                        int lane, unsigned long long &words) {
    const uint32_t *row = R + (int64_t)r * pitch;
    const int nw = words_below(r);
    const int n = set_positions(row, nw, S.pos, kSubD, lane);
    if (n < F) return 0;
    if (n > kSubD) return walk<F - 2>(row, nw, R, pitch, stack, Q, lane, words);
    for (int t = lane; t < n * kSubWords; t += 32) S.C[t] = 0u;
    __syncwarp();
    for (int w = 0; (w << 5) < n - 1; w++) {
        const int col = (w << 5) + lane;
        const int p = col < n ? S.pos[col] : 0;
        const int pw = p >> 5, pb = p & 31;
        // rows a > 32 w have columns of this word below them
        for (int a = (w << 5) + 1; a < n; a++) {
            const uint32_t x = R[(int64_t)S.pos[a] * pitch + pw];
            const unsigned word = __ballot_sync(kFull, col < a && ((x >> pb) & 1u));
            if (lane == 0) S.C[a * kSubWords + w] = word;
        }
    }
    __syncwarp();
    unsigned long long c = 0;
    PairQueue pq;
    pq.Q = Q;
    const DfsPair<F - 3, kSubWords> value{S.C, kSubWords};
    for (int a = F - 2; a < n; a++)
        pairs_push_row(pq, S.C + a * kSubWords, a, value, lane, c, words);
    pairs_flush(pq, value, lane, c, words);
    return c;
}

__device__ __forceinline__ void flush_totals(const CliqueArgs &a, unsigned long long c,
                                             unsigned long long bytes, bool stats, int lane) {
    for (int o = 16; o > 0; o >>= 1) {
        c += __shfl_xor_sync(kFull, c, o);
        if (stats) bytes += __shfl_xor_sync(kFull, bytes, o);
    }
    if (lane == 0) {
        if (c) atomicAdd(&a.ctr->result, c);
        if (stats && bytes) atomicAdd(&a.ctr->bytes, bytes);
    }
}

// ---------------------------------------------------------------- warp kernel

constexpr int kWarpHashBits = 7;  // 128 slots for at most kWarpD elements
static_assert((1 << kWarpHashBits) >= 2 * kWarpD, "hash at most half full");

struct WarpSmem {
    int32_t L[kWarpD];
    int32_t slot[kWarpD];
    uint32_t R[kWarpD * kWarpPitch];
    int32_t Q[kQueue];
    uint16_t T[1 << kWarpHashBits];
};

// The list a larger root goes to: 0 up to 128 lower neighbours, then 256,
// 512 and the rest.
__device__ __forceinline__ int list_of(int d) { return d <= 128 ? 0 : d <= 256 ? 1 : d <= 512 ? 2 : 3; }

// The matrix of a root with d <= kWarpD lower neighbours, rows [0, r1) of
// kWarpPitch words, zero above the diagonal.  One warp.
template <bool STATS>
__device__ __forceinline__ void build_small(const CliqueArgs &a, WarpSmem &S, int r1, int lane,
                                            unsigned long long &bytes) {
    constexpr int kAhead = 4;
    for (int i = lane; i < r1; i += 32)
        S.slot[i] = a.hub_slot != nullptr ? __ldg(a.hub_slot + S.L[i]) : -1;
    __syncwarp();
    // rows with bitmaps, four at a time; the others are cleared
    unsigned plain0 = 0, plain1 = 0;  // rows without: bit i of plain0 | plain1
    for (int i0 = 0; i0 < r1; i0 += kAhead) {
        for (int w = 0; w < 2; w++) {
            const int j = (w << 5) + lane;
            uint32_t f[kAhead];
#pragma unroll
            for (int t = 0; t < kAhead; t++) {
                const int i = i0 + t;
                f[t] = 0u;
                if (i < r1 && j < i && S.slot[i] >= 0) {
                    const int32_t y = S.L[j];
                    f[t] = __ldg(a.bitmaps + (int64_t)S.slot[i] * a.bitmap_words + (y >> 5)) >>
                           (y & 31);
                }
            }
#pragma unroll
            for (int t = 0; t < kAhead; t++) {
                const unsigned word = __ballot_sync(kFull, f[t] & 1u);
                if (lane == 0 && i0 + t < r1) S.R[(i0 + t) * kWarpPitch + w] = word;
            }
        }
    }
    for (int i = lane; i < r1; i += 32) {
        const bool plain = S.slot[i] < 0 && i > 0;
        if (STATS && !plain) bytes += 8ull * (unsigned)i;
        if (i < 32)
            plain0 |= plain ? 1u << i : 0u;
        else
            plain1 |= plain ? 1u << (i - 32) : 0u;
    }
    plain0 = __reduce_or_sync(kFull, plain0);
    plain1 = __reduce_or_sync(kFull, plain1);
    if ((plain0 | plain1) == 0u) {
        __syncwarp();
        return;
    }
    for (int t = lane; t < (1 << kWarpHashBits); t += 32) S.T[t] = kNone;
    __syncwarp();
    for (int t = lane; t < r1; t += 32) hash_add(S.T, kWarpHashBits, S.L[t], t);
    __syncwarp();
    while ((plain0 | plain1) != 0u) {
        const int i = plain0 != 0u ? __ffs(plain0) - 1 : 32 + __ffs(plain1) - 1;
        if (plain0 != 0u)
            plain0 &= plain0 - 1;
        else
            plain1 &= plain1 - 1;
        scan_row<STATS>(a, S.L, i, S.R + i * kWarpPitch, S.T, kWarpHashBits, lane, bytes);
    }
}

// A warp per root v0 of [v_begin, v_end) with K-1 <= lo(v0) <= kWarpD; root
// ids are handed out `chunk` at a time.  Roots with longer lists go to the
// CTA kernel's lists.
template <int K, bool STATS>
__global__ void __launch_bounds__(kWarpThreads) clique_warp_kernel(const CliqueArgs a, int chunk) {
    __shared__ WarpSmem wsmem[kWarpThreads / 32];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    WarpSmem &S = wsmem[wid];
    unsigned long long c = 0, bytes = 0, words = 0;
    PairQueue pq;
    pq.Q = S.Q;
    const DfsPair<K - 4, 2> value{S.R, kWarpPitch};
    for (;;) {
        unsigned long long r0 = 0;
        if (lane == 0) r0 = atomicAdd(&a.aux->warp_cursor, (unsigned long long)chunk);
        r0 = __shfl_sync(kFull, r0, 0);
        const int64_t base = a.v_begin + (int64_t)r0;
        if (base >= a.v_end) break;
        const int64_t v = base + lane;
        const int32_t dl = lane < chunk && v < a.v_end ? lower_degree(a, v) : 0;
        if (dl > kWarpD) {
            const int b = list_of(dl);
            a.lists[a.list_at[b] + (int64_t)atomicAdd(&a.aux->listed[b], 1ull)] = (int32_t)v;
        }
        unsigned mine = __ballot_sync(kFull, dl >= K - 1 && dl <= kWarpD);
        while (mine != 0u) {
            const int r = __ffs(mine) - 1;
            mine &= mine - 1;
            const int64_t v0 = base + r;
            const int d = __shfl_sync(kFull, dl, r);
            int r0, r1;
            unit_rows(a, v0, d, &r0, &r1);
            r0 = max(r0, K - 2);  // row i needs K-2 members below it
            if (r0 >= r1) continue;
            const int32_t *src = a.adj + a.off[v0];
            for (int t = lane; t < r1; t += 32) S.L[t] = __ldg(src + t);
            if (STATS && lane == 0) bytes += 4ull * (unsigned)r1;
            __syncwarp();
            build_small<STATS>(a, S, r1, lane, bytes);
            for (int i = r0; i < r1; i++)
                pairs_push_row(pq, S.R + i * kWarpPitch, i, value, lane, c, words);
            pairs_flush(pq, value, lane, c, words);
        }
    }
    if (STATS) bytes += 8ull * words;
    flush_totals(a, c, bytes, STATS, lane);
}

// ----------------------------------------------------------------- CTA kernel

__device__ __forceinline__ unsigned smem_u32(const void *p) {
    return (unsigned)__cvta_generic_to_shared(p);
}

constexpr int kCtaHashBits = 12;  // 4096 slots for at most kMaxD elements
static_assert((1 << kCtaHashBits) >= 2 * kMaxD, "hash at most half full");

// The build's tables and the count's are never live together.
struct CtaBuild {
    int32_t slot[kMaxD];
    alignas(16) uint16_t T[1 << kCtaHashBits];
    uint16_t plain[kMaxD];  // rows without a bitmap
};
template <int K>
struct CtaCount {
    SubSmem sub[K > 4 ? kCtaWarps : 1];
    uint32_t stack[K > 5 ? kCtaWarps : 1][(K > 5 ? K - 5 : 1) * kMaxWords];
    uint16_t big[K > 4 ? kMaxD : 2];  // rows of more than kSubD members
    uint16_t pos[K > 4 ? kMaxD : 2];  // the members of the one in hand
};
template <int K>
struct CtaSmem {
    alignas(16) int32_t Lbuf[2][kMaxD + 8];  // lists of the root in hand and the
                                             // next, from 16-byte boundaries
    alignas(16) uint32_t R[row_smem_words<K>()];
    union {
        CtaBuild build;
        CtaCount<K> count;
    };
    int32_t Q[kCtaWarps][kQueue];
    alignas(8) unsigned long long bar;
    int32_t root[2], degree[2];
    int64_t begin[2];
    int64_t listed[kCliqueLists];
    int next_build, next_count, nbig, nplain;
};

// Bulk copy of src[0, n_ints) (16-byte aligned, n_ints a multiple of 4) into
// shared memory, completion counted on the mbarrier.  One thread.
__device__ __forceinline__ void bulk_stage(void *dst, const int32_t *src, int n_ints,
                                           unsigned long long *bar) {
    const unsigned bytes = (unsigned)n_ints * 4u;
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)),
                 "r"(bytes)
                 : "memory");
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::
            "r"(smem_u32(dst)),
        "l"(src), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

__device__ __forceinline__ bool mbar_test(unsigned long long *bar, unsigned parity) {
    unsigned ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

// Polls the mbarrier phase at most `limit` times.
__device__ __forceinline__ bool mbar_wait(unsigned long long *bar, unsigned parity,
                                          unsigned limit) {
    for (unsigned t = 0; t < limit; t++)
        if (mbar_test(bar, parity)) return true;
    return false;
}

// Whether a root's matrix sits in shared memory.  For K >= 5 it leaves half
// of the region free, so that every compacted matrix of it fits; a longer
// root's matrix is read from global scratch and the whole region is free.
__host__ __device__ constexpr bool rows_local(int k, int d) {
    const int64_t need = (int64_t)d * (((d + 31) >> 5) | 1);
    return k == 4 ? need <= row_smem_words<4>() : 2 * need <= row_smem_words<5>();
}

// Row r of the root's matrix has more than kSubD members: the whole CTA
// compacts them to a matrix in `region` and its warps count it.
template <int K>
__device__ __forceinline__ void count_big_row(CtaSmem<K> &S, const uint32_t *R, int pitch, int r,
                                              uint32_t *region, int room, int wid, int lane,
                                              unsigned long long &c, unsigned long long &words) {
    const uint32_t *row = R + (int64_t)r * pitch;
    const int nw = words_below(r);
    // every warp counts the words before its own and lists its own words' bits
    int n = 0;
    for (int w = 0; w < nw; w++) {
        const uint32_t x = row[w];
        if (w % kCtaWarps == wid && ((x >> lane) & 1u))
            S.count.pos[n + __popc(x & lanemask_lt())] = (uint16_t)((w << 5) + lane);
        n += __popc(x);
    }
    const int cp = row_pitch(n);
    if (n * cp > room) {
        // no room for the compacted matrix: the warps share the row's members
        __syncthreads();
        for (int a = wid; a < n; a += kCtaWarps) {
            const int j = S.count.pos[a];
            const int n2 = words_below(j);
            const uint32_t *Rj = R + (int64_t)j * pitch;
            uint32_t *m = region + wid * kMaxWords;
            for (int t = lane; t < n2; t += 32) m[t] = row[t] & Rj[t];
            __syncwarp();
            c += walk<K - 5>(m, n2, R, pitch, S.count.stack[K > 5 ? wid : 0], S.Q[wid], lane,
                             words);
            __syncwarp();
        }
        __syncthreads();
        return;
    }
    __syncthreads();
    for (int w = 0; (w << 5) < n; w++) {
        const int col = (w << 5) + lane;
        const int p = col < n ? S.count.pos[col] : 0;
        const int pw = p >> 5, pb = p & 31;
        for (int a = (w << 5) + 1 + wid; a < n; a += kCtaWarps) {
            const uint32_t x = R[(int64_t)S.count.pos[a] * pitch + pw];
            const unsigned word = __ballot_sync(kFull, col < a && ((x >> pb) & 1u));
            if (lane == 0) region[a * cp + w] = word;
        }
    }
    if (threadIdx.x == 0) S.next_count = kCtaWarps;
    __syncthreads();
    PairQueue pq;
    pq.Q = S.Q[wid];
    const PopPair value{region, cp};
    // members in decreasing order: the longest rows first
    for (int t = wid;;) {
        const int a = n - 1 - t;
        if (a < K - 3) break;
        if constexpr (K == 5)
            pairs_push_row(pq, region + a * cp, a, value, lane, c, words);
        else
            c += sub_count<K - 3>(region, cp, a, S.count.sub[wid], S.count.stack[wid], S.Q[wid],
                                  lane, words);
        int nx = 0;
        if (lane == 0) nx = atomicAdd(&S.next_count, 1);
        t = __shfl_sync(kFull, nx, 0);
    }
    if constexpr (K == 5) pairs_flush(pq, value, lane, c, words);
    __syncthreads();
}

// A CTA per listed root (lo(v0) > kWarpD), longest lists first.
template <int K, bool STATS>
__global__ void __launch_bounds__(kCtaThreads, 2) clique_cta_kernel(const CliqueArgs a) {
    extern __shared__ __align__(16) unsigned char csmem[];
    CtaSmem<K> &S = *reinterpret_cast<CtaSmem<K> *>(csmem);
    constexpr int kRegion = row_smem_words<K>();
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned long long c = 0, bytes = 0, words = 0;
    unsigned phase = 0;
    if (threadIdx.x == 0) {
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(smem_u32(&S.bar)) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (threadIdx.x < kCliqueLists) S.listed[threadIdx.x] = (int64_t)a.aux->listed[threadIdx.x];
    __syncthreads();
    uint32_t *grows = a.rows != nullptr ? a.rows + (int64_t)blockIdx.x * a.rows_stride : nullptr;
    // Takes the next listed root (root -1: none left) and starts staging its
    // list: L = adj[begin, begin + degree) from the 16-byte boundary below.
    // One thread, while the CTA builds and counts the root before it: the
    // chain of reads to the list is as long as a small root's count.
    auto fetch = [&](int buf) {
        int64_t at = (int64_t)atomicAdd(&a.aux->cta_cursor, 1ull);
        int b = kCliqueLists - 1;
        for (; b >= 0; b--) {
            const int64_t n = S.listed[b];
            if (at < n) break;
            at -= n;
        }
        S.root[buf] = -1;
        if (b < 0) return;
        const int64_t v = a.lists[a.list_at[b] + at];
        const int64_t o = a.off[v];
        const int d = lower_degree(a, v);
        S.root[buf] = (int32_t)v;
        S.begin[buf] = o;
        S.degree[buf] = d;
        if (d > kMaxD) return;  // reported below
        const int64_t a0 = o & ~3ll, a1 = (o + d + 3) & ~3ll;
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
        bulk_stage(S.Lbuf[buf], a.adj + a0, (int)(a1 - a0), &S.bar);
    };
    if (threadIdx.x == 0) fetch(0);
    for (int buf = 0;; buf ^= 1) {
        __syncthreads();  // the root in hand is known; the last one is done
        const int64_t v0 = S.root[buf];
        if (v0 < 0) break;
        const int64_t o0 = S.begin[buf];
        const int d = S.degree[buf];
        const int32_t *L = S.Lbuf[buf] + (o0 & 3ll);
        // rows below r1 are built; rows [r0, r1) are counted
        int r0, r1;
        unit_rows(a, v0, d, &r0, &r1);
        r0 = max(r0, K - 2);
        const int pitch = row_pitch(d);
        const bool local = rows_local(K, d);
        if (d > kMaxD || (!local && grows == nullptr)) {
            // the host sizes the row scratch for the graph's longest list
            if (threadIdx.x == 0) atomicOr(&a.ctr->error, GAT_DEVERR_SCRATCH);
            if (d <= kMaxD) mbar_wait(&S.bar, phase, kWaitLimit);  // its list is under way
            break;
        }
        if (threadIdx.x == 0) {
            S.next_build = kCtaWarps;
            S.next_count = kCtaWarps;
            S.nbig = 0;
            S.nplain = 0;
        }
        // at most an eighth full up to 512 elements: one probe settles nearly
        // every lookup, and a warp repeats it for its slowest lane
        const int bits = min(kCtaHashBits, 32 - __clz(8 * d - 1));
        for (int t = threadIdx.x; t < (1 << bits) / 8; t += kCtaThreads)
            reinterpret_cast<uint4 *>(S.build.T)[t] = make_uint4(~0u, ~0u, ~0u, ~0u);
        const bool ok = mbar_wait(&S.bar, phase, kWaitLimit);
        phase ^= 1u;
        if (__syncthreads_or(!ok)) {
            // the copy did not complete: report, let it land, stop
            if (threadIdx.x == 0) {
                atomicOr(&a.ctr->error, GAT_DEVERR_WAIT);
                mbar_wait(&S.bar, phase ^ 1u, kWaitLimit);
            }
            break;
        }
        if (r0 >= r1) {
            if (threadIdx.x == kCtaThreads - 32) fetch(buf ^ 1);
            continue;
        }
        if (STATS && threadIdx.x == 0) bytes += 4ull * (unsigned)d;
        for (int t = threadIdx.x; t < r1; t += kCtaThreads) {
            const int32_t u = L[t];
            const int slot = a.hub_slot != nullptr ? __ldg(a.hub_slot + u) : -1;
            S.build.slot[t] = slot;
            if (slot < 0 && t > 0) S.build.plain[atomicAdd(&S.nplain, 1)] = (uint16_t)t;
            hash_add(S.build.T, bits, u, t);
        }
        __syncthreads();
        if (threadIdx.x == kCtaThreads - 32) fetch(buf ^ 1);
        __syncwarp();
        // Written out for the shared and the global matrix: the compiler then
        // knows which loads are shared-memory loads.
        auto build_and_count = [&](uint32_t *R) {
            for (int i = wid; i < r1; i += kCtaWarps) {
                const int slot = S.build.slot[i];
                if (slot >= 0)
                    bitmap_row<STATS>(a, L, i, slot, R + (int64_t)i * pitch, lane, bytes);
            }
            for (int t = wid; t < S.nplain;) {
                const int i = S.build.plain[t];
                scan_row<STATS>(a, L, i, R + (int64_t)i * pitch, S.build.T, bits, lane, bytes);
                if (lane == 0) t = atomicAdd(&S.next_build, 1);
                t = __shfl_sync(kFull, t, 0);
            }
            __syncthreads();
            if constexpr (K == 4) {
                PairQueue pq;
                pq.Q = S.Q[wid];
                const PopPair value{R, pitch};
                for (int i = r0 + wid; i < r1;) {
                    pairs_push_row(pq, R + (int64_t)i * pitch, i, value, lane, c, words);
                    if (lane == 0) i = r0 + atomicAdd(&S.next_count, 1);
                    i = __shfl_sync(kFull, i, 0);
                }
                pairs_flush(pq, value, lane, c, words);
            } else {
                for (int t = wid; r1 - 1 - t >= r0;) {
                    const int i = r1 - 1 - t;
                    const uint32_t *Ri = R + (int64_t)i * pitch;
                    int n = 0;
                    for (int w = lane; w < words_below(i); w += 32) n += __popc(Ri[w]);
                    n = __reduce_add_sync(kFull, n);
                    if (n > kSubD) {
                        if (lane == 0) S.count.big[atomicAdd(&S.nbig, 1)] = (uint16_t)i;
                    } else if (n >= K - 2) {
                        c += sub_count<K - 2>(R, pitch, i, S.count.sub[wid],
                                              S.count.stack[K > 5 ? wid : 0], S.Q[wid], lane,
                                              words);
                    }
                    if (lane == 0) t = atomicAdd(&S.next_count, 1);
                    t = __shfl_sync(kFull, t, 0);
                }
                __syncthreads();
                uint32_t *region = local ? S.R + d * pitch : S.R;
                const int room = local ? kRegion - d * pitch : kRegion;
                const int nbig = S.nbig;
                for (int t = 0; t < nbig; t++)
                    count_big_row<K>(S, R, pitch, S.count.big[t], region, room, wid, lane, c,
                                     words);
            }
        };
        if (local)
            build_and_count(S.R);
        else
            build_and_count(grows);
    }
    if (STATS) bytes += 8ull * words;
    flush_totals(a, c, bytes, STATS, lane);
}

constexpr int32_t kShortLists = 8;  // longest lower list
constexpr int kShortChunk = 8;

template <int K, bool STATS>
cudaError_t launch_k(const CliqueArgs &a, int32_t max_lower, int warp_grid, int cta_grid,
                     cudaStream_t st) {
    cudaError_t e;
    // ids per grab: up to 32 are looked at in one go, but no more than 1/32 of
    // a warp's share: neighbouring ids have lists of like length, and the
    // long ones must spread over the grid.  Where all lists are short there is
    // little to spread, and a grab costs more than the ids in it: a share, up
    // to kShortChunk (Barabasi-Albert 200,000 x 1: 0.150 ms a count with a grab
    // an id, 0.04 so; 2^20 x 4, 5-cliques: 0.76 at 3 ids, 0.83 at 32)
    const bool few = max_lower <= kShortLists;
    const int64_t share =
        (a.v_end - a.v_begin) / (int64_t(warp_grid) * (kWarpThreads / 32) * (few ? 1 : 32));
    const int chunk =
        (int)std::min<int64_t>(std::max<int64_t>(share, 1), few ? kShortChunk : kRootChunk);
    clique_warp_kernel<K, STATS><<<warp_grid, kWarpThreads, 0, st>>>(a, chunk);
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
    const size_t cs = sizeof(CtaSmem<K>);
    if ((e = cudaFuncSetAttribute(clique_cta_kernel<K, STATS>,
                                  cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cs)) !=
        cudaSuccess)
        return e;
    clique_cta_kernel<K, STATS><<<cta_grid, kCtaThreads, cs, st>>>(a);
    return cudaGetLastError();
}

template <int K, bool STATS>
void occupancy_k(int &warp_occ, int &cta_occ) {
    warp_occ = cta_occ = 0;
    const size_t cs = sizeof(CtaSmem<K>);
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&warp_occ, clique_warp_kernel<K, STATS>,
                                                      kWarpThreads, 0) != cudaSuccess)
        warp_occ = 0;
    if (cudaFuncSetAttribute(clique_cta_kernel<K, STATS>,
                             cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cs) != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&cta_occ, clique_cta_kernel<K, STATS>,
                                                      kCtaThreads, cs) != cudaSuccess)
        cta_occ = 0;
}

// Roots a list can hold: lists 0 .. 3 have lower lists longer than 64, 128,
// 256 and 512 entries.
int64_t list_room(int b, int64_t lo_total) { return lo_total / ((int64_t(kWarpD) << b) + 1) + 1; }

}  // namespace

int64_t clique_rows_words(int k, int32_t max_lower) {
    return rows_local(k, max_lower) ? 0 : (int64_t)max_lower * row_pitch(max_lower);
}

int64_t clique_list_ints(int64_t lo_total) {
    int64_t n = 0;
    for (int b = 0; b < kCliqueLists; b++) n += list_room(b, lo_total);
    return n;
}

void clique_blocks_per_sm(int k, bool stats, int *warp_occ, int *cta_occ) {
    int w = 0, c = 0;
    switch (k * 2 + (stats ? 1 : 0)) {
        case 8: occupancy_k<4, false>(w, c); break;
        case 9: occupancy_k<4, true>(w, c); break;
        case 10: occupancy_k<5, false>(w, c); break;
        case 11: occupancy_k<5, true>(w, c); break;
        case 12: occupancy_k<6, false>(w, c); break;
        case 13: occupancy_k<6, true>(w, c); break;
        case 14: occupancy_k<7, false>(w, c); break;
        case 15: occupancy_k<7, true>(w, c); break;
        default: break;
    }
    *warp_occ = w;
    *cta_occ = c;
}

cudaError_t launch_clique(const CliqueLaunch &L, cudaStream_t st) {
    const DevGraphView &g = L.g;
    if (g.lo_off == nullptr) return cudaErrorInvalidValue;
    cudaError_t e;
    if ((e = cudaMemsetAsync(L.ctr, 0, sizeof(DevCounters), st)) != cudaSuccess ||
        (e = cudaMemsetAsync(L.aux, 0, sizeof(CliqueAux), st)) != cudaSuccess)
        return e;
    CliqueArgs a{g.off, g.adj, g.lo_off, g.bitmaps ? g.hub_slot : nullptr, g.bitmaps, g.bitmap_words,
                 L.v_begin, L.v_end, L.u_begin, L.u_end, L.ctr, L.aux, L.rows, L.rows_stride,
                 L.lists, {}};
    for (int b = 1; b < kCliqueLists; b++)
        a.list_at[b] = a.list_at[b - 1] + list_room(b - 1, g.lo_total);
    if (L.v_end <= L.v_begin) return cudaSuccess;
    switch (L.k * 2 + (L.stats ? 1 : 0)) {
        case 8: return launch_k<4, false>(a, g.max_lower, L.warp_grid, L.cta_grid, st);
        case 9: return launch_k<4, true>(a, g.max_lower, L.warp_grid, L.cta_grid, st);
        case 10: return launch_k<5, false>(a, g.max_lower, L.warp_grid, L.cta_grid, st);
        case 11: return launch_k<5, true>(a, g.max_lower, L.warp_grid, L.cta_grid, st);
        case 12: return launch_k<6, false>(a, g.max_lower, L.warp_grid, L.cta_grid, st);
        case 13: return launch_k<6, true>(a, g.max_lower, L.warp_grid, L.cta_grid, st);
        case 14: return launch_k<7, false>(a, g.max_lower, L.warp_grid, L.cta_grid, st);
        case 15: return launch_k<7, true>(a, g.max_lower, L.warp_grid, L.cta_grid, st);
        default: return cudaErrorInvalidValue;
    }
}

}  // namespace gat
