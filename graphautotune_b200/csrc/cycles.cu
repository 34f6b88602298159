// Exact 4-cycle count by wedge aggregation in shared memory (sm_100a).
//
// Every 4-cycle is counted once, at its smallest vertex v0 together with the
// vertex x opposite v0: its other two vertices are common neighbours of v0
// and x above v0.  So
//   count = sum_{v0} sum_{x > v0} C(c(v0, x), 2),
//   c(v0, x) = |{ v1 in N(v0) : v1 > v0, x in N(v1) }|   (x > v0 too).
// On the degree-ordered copy (id 0 = largest degree) v0 is the cycle's
// highest-degree vertex and every v1 has degree <= deg(v0), so the wedges
// v0 - v1 - x number at most the sum over edges of the smaller endpoint's
// degree.
//
// A root's wedge endpoints x are tallied on chip, never in global memory:
//
//  * c4_light_kernel: a warp per root (roots of degree below the heavy
//    threshold).  Lanes take the root's upper neighbours v1, find where
//    N(v1) rises above v0 and add up the wedges W.  With few of them
//    the warp takes the lists end to end into an open-addressing table of
//    its own in shared memory (key x, count c), then read every slot once, add C(c, 2)
//    and clear it.  A root with more wedges is appended to a deferred list.
//  * c4_root_kernel: a CTA per root, for the heavy roots and the deferred
//    ones, largest degree first.  Segment starts (N(v1) above v0) are found
//    once; with few wedges they go to a CTA-wide table as above, otherwise
//    the ids above v0 are swept in windows of consecutive x whose counters
//    fill the shared-memory region, each as wide as its x's degree asks for
//    (Window).  Per window each list advances from its cursor to the window's
//    end, warps stream the long segments and the short ones are flattened
//    (each_entry), the counters are incremented with shared atomics, and the
//    window's counters are read, summed as C(c, 2) and cleared before the
//    next window.  Once the wedges left fit the CTA table, the lists'
//    remainders go through the table in one pass.
//
// Bound: on chip.  On R-MAT 2^18 DRAM is at 0.2% and L2 at 8% of their peaks
// and issue slots are 55% busy; barriers and list loads stall a warp about
// equally (3.3 and 3.1 per instruction).  A shared atomic of 32 random counters
// takes 4.4 wavefronts, and a root's barriers and chains of dependent reads cost
// more than its counting for all but the largest thousand.  R-MAT 2^20 (5.65e9
// wedges) on a B200, ms per CTA: roots of a million wedges and more 5.1 (76% of
// all wedges), others 3.3, reading counters out 2, finding segments 1.3, tables
// 1.5; the light kernel 0.25.  One count: 21.4 ms with a search per entry, 16-bit
// windows and a lane per list in the light kernel, now 12.1; R-MAT 2^18 3.2 ->
// 2.04, Barabasi-Albert 60,000 x 9 0.66 -> 0.23.
//
// Neither kernel waits on another CTA; the deferred list is written by the
// first launch and read by the second, ordered on the stream.
#include <cub/cub.cuh>

#include <algorithm>
#include <limits>
#include <type_traits>

#include "engine.hpp"

namespace gat {
namespace {

constexpr int32_t kEmpty = 0;  // wedge endpoints lie above their root, so no key is 0
constexpr int kWarpSlots = 1024;          // per-warp table slots
constexpr int kWarpBits = 10;
static_assert((1 << kWarpBits) == kWarpSlots, "table size is a power of two");
// Most wedges of a warp's root: probes get long as the table fills (a warp
// repeats one for its slowest lane), and a CTA costs about 3 us a root.  At
// 1/4, 1/2 and 3/4 of the slots G(5,000, 20) took 76, 85 and 115 us a count,
// G(30,000, 20) 201, 126 and 139, Barabasi-Albert 20,000 x 9 135, 141 and 212.
// Where the roots are few the CTAs have the time, so a quarter up to
// kFewRoots vertices (G(5,000, 20) 76 us a count against 86, R-MAT 2^13 89
// against 99) and three eighths beyond (G(30,000, 20) 153 against 201).
constexpr int64_t kFewRoots = 8192;
constexpr int warp_wedges(int64_t V) { return V <= kFewRoots ? kWarpSlots / 4 : kWarpSlots * 3 / 8; }
constexpr int kLightBlock = 256;          // 8 warps
// The root kernel in two shapes.  Two CTAs of 512 threads per SM hide one
// root's barriers and chains of reads behind the other's (R-MAT 2^18: 2.2 ms
// against 2.8 with one of 1,024); on a small graph the largest roots alone
// are the count's time and take 1,024 threads (R-MAT 2^14: 0.119 ms against
// 0.146).
template <int BLOCK>
struct RootShape {
    static constexpr int kCtas = 1024 / BLOCK;              // per SM
    static constexpr int kSlots = 16 * BLOCK;               // CTA table slots
    static constexpr int kWedges = kSlots / 2;              // at most half full
    static constexpr int kRegionBytes = 192 * BLOCK;        // counters or table
    static constexpr int kRegionWords = kRegionBytes / 4;
    static_assert(kSlots * 8 <= kRegionBytes, "table fits in the region");
    static_assert((kSlots & (kSlots - 1)) == 0, "slots are a power of two");
};

__device__ __forceinline__ unsigned long long pairs_of(unsigned long long c) {
    return c * (c - 1) / 2;
}

// First index i of the sorted a[0, n) with a[i] > x (one thread alone).
__device__ __forceinline__ int32_t upper_index(const int32_t *a, int32_t n, int32_t x) {
    int32_t lo = 0;
    while (n > 0) {
        const int32_t h = n >> 1;
        const bool right = a[lo + h] <= x;
        lo = right ? lo + h + 1 : lo;
        n = right ? n - h - 1 : h;
    }
    return lo;
}

// Where N(v1) rises above v0, a neighbour of v1 below it: among v1's lower
// neighbours, which a degree order keeps few.
__device__ __forceinline__ int32_t above(const int32_t *nb, const int64_t *lo_off, int32_t v1,
                                         int32_t v0) {
    return upper_index(nb, (int32_t)(lo_off[v1 + 1] - lo_off[v1]), v0);
}

__device__ __forceinline__ unsigned slot_of(int32_t x, int bits) {
    return ((unsigned)x * 0x9E3779B1u) >> (32 - bits);
}

// Adds one occurrence of x to an open-addressing table of 2^bits slots that
// is never more than half full.  The probe is bounded by the table size (it
// cannot run out by construction; running out would flag an error).
__device__ __forceinline__ void table_add(int32_t *key, uint32_t *cnt, int bits, int32_t x,
                                          unsigned long long *error) {
    const unsigned mask = (1u << bits) - 1u;
    unsigned h = slot_of(x, bits);
    for (unsigned probes = 0; probes <= mask; probes++) {
        const int32_t k = reinterpret_cast<volatile int32_t *>(key)[h];
        if (k == x) {
            atomicAdd(&cnt[h], 1u);
            return;
        }
        if (k == kEmpty) {
            const int32_t old = atomicCAS(&key[h], kEmpty, x);
            if (old == kEmpty || old == x) {
                atomicAdd(&cnt[h], 1u);
                return;
            }
        }
        h = (h + 1) & mask;
    }
    atomicOr(error, GAT_DEVERR_TABLE);
}

// One window of ids and its counters.  c(v0, x) <= deg(x), and on the
// degree-ordered copy degrees only fall along the ids, so a counter needs as
// many bits as the degree at the window's start: 32, 16, 8, 4 or 2.  A window
// has two parts, ids below `split` with 1 << shift1 bits each and the others
// with the next smaller width, so that one window reaches well past the hubs:
// on R-MAT 2^20 two windows hold all ids of degree 2 and more (175,000 ids
// in the first), where 16-bit counters alone took eleven of 98,304.  The
// windows of the hubs all start at id 0, so that they end at the same ids for
// every root and the rows' positions there are looked up once per count
// (kMarks of them) instead of searched for by every root.
constexpr int kMarks = 2;
struct Window {
    int32_t split, hi;
    int shift1, shift2;    // log2 of the counter widths
    unsigned add1, add2;   // bit of x's counter = (x << shift) + add
    int words1, words;     // of the first part, and of both
};

struct Degrees {
    int32_t bound[4];  // first id of degree below 2^16, 2^8, 2^4, 2^2
    int32_t limit;     // ids from here on have degree below 2: never opposite
};

template <int BLOCK>
__host__ __device__ __forceinline__ Window window_from(const Degrees &a, int32_t lo) {
    constexpr int64_t kBits = int64_t(RootShape<BLOCK>::kRegionBytes) * 8;
    int s = 5, next = 0;  // counter width at lo, and the bound it ends at
    while (next < 4 && lo >= a.bound[next]) {
        s--;
        next++;
    }
    Window w;
    w.shift1 = s;
    w.shift2 = s > 1 ? s - 1 : 1;
    auto least = [](int64_t x, int64_t y) { return x < y ? x : y; };
    // one width where it holds all the rest
    const bool rest = ((int64_t(a.limit) - lo) << s) <= kBits;
    const int64_t end1 = next < 4 && !rest ? least(a.bound[next], a.limit) : a.limit;
    const int64_t split = least(end1, lo + (kBits >> s));
    w.split = (int32_t)split;
    w.words1 = (int)((((split - lo) << s) + 31) >> 5);
    int64_t hi = split;
    if (split == end1 && end1 < a.limit) {
        const int64_t end2 = next + 1 < 4 ? least(a.bound[next + 1], a.limit) : a.limit;
        const int64_t most = split + ((kBits - int64_t(w.words1) * 32) >> w.shift2);
        hi = end2 < split ? split : least(end2, most);
    }
    w.hi = (int32_t)hi;
    w.words = w.words1 + (int)((((hi - split) << w.shift2) + 31) >> 5);
    w.add1 = 0u - ((unsigned)lo << w.shift1);
    w.add2 = (unsigned)w.words1 * 32u - ((unsigned)w.split << w.shift2);
    return w;
}

struct LightArgs {
    const int64_t *off;
    const int32_t *adj;
    const int64_t *lo_off;
    int64_t v_begin, v_end;
    DevCounters *ctr;
    C4Aux *aux;
    int32_t *deferred;
    int32_t V;
    int32_t mark[kMarks];  // window ends (V: none), and where every row passes
    int32_t *marks;        // them: kMarks x V positions
    int32_t most;          // wedges of a root that its warp counts itself
    int32_t chunk;         // roots a grab
};

// A warp per root of [v_begin, v_end), handed out one at a time, or, where the
// warps get many each, up to kMostRoots: on trees the grabs were a fifth of the
// count (Barabasi-Albert 200,000 x 1).
constexpr int64_t kRootShare = 16;  // grabs a warp, about
constexpr int64_t kMostRoots = 8;
constexpr size_t kLightSmem = size_t(kLightBlock / 32) * kWarpSlots * 8;

template <bool STATS>
__global__ void __launch_bounds__(kLightBlock) c4_light_kernel(const LightArgs a) {
    extern __shared__ __align__(16) unsigned char lsmem[];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    int32_t *key = reinterpret_cast<int32_t *>(lsmem) + w * 2 * kWarpSlots;
    uint32_t *cnt = reinterpret_cast<uint32_t *>(key + kWarpSlots);
    for (int i = lane; i < kWarpSlots; i += 32) {
        key[i] = kEmpty;
        cnt[i] = 0;
    }
    __syncwarp();
    for (int m = 0; m < kMarks; m++)
        if (a.mark[m] < a.V)
            for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < a.V;
                 v += (int64_t)gridDim.x * blockDim.x) {
                const int64_t o = a.off[v];
                a.marks[(int64_t)m * a.V + v] =
                    upper_index(a.adj + o, (int32_t)(a.off[v + 1] - o), a.mark[m] - 1);
            }
    unsigned long long part = 0, bytes = 0;
    for (;;) {
        unsigned long long r = 0;
        if (lane == 0) r = atomicAdd(&a.aux->light_cursor, (unsigned long long)a.chunk);
        r = __shfl_sync(0xffffffffu, r, 0);
        const int64_t first = a.v_begin + (int64_t)r;
        if (first >= a.v_end) break;
        const int64_t last = min(first + a.chunk, a.v_end);
        for (int64_t v0 = first; v0 < last; v0++) {
            const int64_t o0 = a.off[v0];
            const int32_t d0 = (int32_t)(a.off[v0 + 1] - o0);
            const int32_t lo0 = (int32_t)(a.lo_off[v0 + 1] - a.lo_off[v0]);
            if (d0 - lo0 < 2) continue;  // a cycle needs two neighbours above v0
            // This lane's upper neighbour of a group of 32: where its list rises
            // above v0, and how many entries that leaves.
            auto segment = [&](int i, int64_t &at) -> int32_t {
                if (i >= d0) return 0;
                const int32_t v1 = a.adj[o0 + i];
                const int64_t o1 = a.off[v1];
                const int32_t d1 = (int32_t)(a.off[v1 + 1] - o1);
                const int32_t s1 = above(a.adj + o1, a.lo_off, v1, (int32_t)v0);
                at = o1 + s1;
                return d1 - s1;
            };
            // wedges of this root: sum over upper neighbours of |N(v1) above v0|
            int32_t wl = 0, len = 0;
            int64_t at = 0;
            for (int i0 = lo0; i0 < d0; i0 += 32) {
                len = segment(i0 + lane, at);
                wl += len;
            }
            const int32_t W = __reduce_add_sync(0xffffffffu, wl);
            if (W > a.most) {
                if (lane == 0) {
                    const unsigned long long slot = atomicAdd(&a.aux->deferred_count, 1ull);
                    a.deferred[slot] = (int32_t)v0;
                }
                continue;
            }
            if (W < 2) continue;
            // A table of four slots a wedge and more where the warp's room has
            // them: it is read out whole.
            const int bits = min(kWarpBits, max(5, 32 - __clz(4 * W - 1)));
            for (int i0 = lo0; i0 < d0; i0 += 32) {
                if (d0 - lo0 > 32) len = segment(i0 + lane, at);  // else known from above
                constexpr int kAhead = 4;
                // The group's entries laid end to end, the lanes on consecutive
                // ones: entry j belongs to the last lane whose exclusive prefix is
                // at most j.  (A lane walking its own list takes as long as the
                // longest: 34 us for 1,500 roots with a hub's list among theirs,
                // 24 so; on a uniform G(30,000, 20) 146 us a count against 126.)
                int32_t pre = len;
    #pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int32_t y = __shfl_up_sync(0xffffffffu, pre, o);
                    if (lane >= o) pre += y;
                }
                const int32_t total = __shfl_sync(0xffffffffu, pre, 31);
                pre -= len;
                for (int32_t j0 = 0; j0 < total; j0 += 32 * kAhead) {
                    int32_t xs[kAhead];
    #pragma unroll
                    for (int u = 0; u < kAhead; u++) {
                        const int32_t j = j0 + 32 * u + lane;
                        int own = 0;
    #pragma unroll
                        for (int o = 16; o > 0; o >>= 1)
                            if (__shfl_sync(0xffffffffu, pre, own + o) <= j) own += o;
                        const int64_t from = __shfl_sync(0xffffffffu, at, own);
                        const int32_t first = __shfl_sync(0xffffffffu, pre, own);
                        xs[u] = j < total ? __ldg(a.adj + from + (j - first)) : 0;
                    }
    #pragma unroll
                    for (int u = 0; u < kAhead; u++)
                        if (xs[u] > 0) table_add(key, cnt, bits, xs[u], &a.ctr->error);
                }
                if (STATS && i0 + lane < d0) bytes += 20;
            }
            if (STATS) bytes += 4ull * (unsigned)wl;
            __syncwarp();
            for (int i = lane; i < (1 << bits); i += 32) {
                if (key[i] != kEmpty) {
                    part += pairs_of(cnt[i]);
                    key[i] = kEmpty;
                    cnt[i] = 0;
                }
            }
            __syncwarp();
        }
    }
    for (int o = 16; o > 0; o >>= 1) {
        part += __shfl_xor_sync(0xffffffffu, part, o);
        if (STATS) bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
    }
    if (lane == 0) {
        atomicAdd(&a.ctr->result, part);
        if (STATS) atomicAdd(&a.ctr->bytes, bytes);
    }
}

struct RootArgs {
    Degrees deg;
    int32_t mark[kMarks];
    const int32_t *marks;
    const int64_t *off;
    const int32_t *adj;
    const int64_t *lo_off;
    int32_t V;
    int64_t heavy_begin, heavy_end;  // roots taken directly, in id order
    DevCounters *ctr;
    C4Aux *aux;
    const int32_t *deferred;         // then these (count in aux)
    int32_t *cursors;                // per CTA: max_degree list positions
    int64_t cursor_stride;
};

template <int BLOCK>
struct RootSmem {
    typedef cub::BlockReduce<long long, BLOCK> Reduce;
    // the group's segments, those of at least kLongSegment entries first,
    // then the other non-empty ones, each kind in order:
    int64_t seg_base[BLOCK];  // absolute index of the first entry
    int32_t pref[BLOCK + 2];  // exclusive prefix of the lengths of its kind,
                              // each kind followed by its total
    int32_t warp_len[2][BLOCK / 32], warp_num[2][BLOCK / 32];
    unsigned next[2];          // next entry to take (of this group and the next)
    typename Reduce::TempStorage reduce;
    int64_t root;
    long long total;
    unsigned long long in_window;
};

// Shared memory the root kernel needs: the counter region plus its state.
template <int BLOCK>
constexpr size_t root_smem_bytes() {
    return size_t(RootShape<BLOCK>::kRegionBytes) + sizeof(RootSmem<BLOCK>);
}

// Calls f(x) for every entry of this group's segments (thread t: base, len).
// Nearly all wedges lie in long segments (R-MAT 2^20: 94% in segments of 128
// entries and more), and a warp that streams one segment needs a load and an
// update per 32 entries and no search for the segment an entry belongs to
// (64 warp instructions per 32 entries when every lane looked its entry's
// segment up).  So the long segments are laid end to end and the warps take
// equal pieces of them, walking the segments of a piece with eight loads a
// lane in flight; taking whole segments left the CTA waiting at the barrier
// for its longest one.  Short segments are flattened over the whole CTA: left
// to the warps that hold them, they were a chain of dependent loads that all
// others waited for (27.9 ms).
// `parity` alternates between the calls that have long segments.
constexpr int kLongSegment = 64;
constexpr int kPieces = 4;  // pieces a warp takes of a group, about

template <int BLOCK, class F>
__device__ __forceinline__ void each_entry(RootSmem<BLOCK> &S, const int32_t *__restrict__ adj,
                                           int64_t base, int32_t len, int &parity, F &&f) {
    constexpr int kWarps = BLOCK / 32;
    static_assert(kWarps <= 32, "one lane per warp");
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int b = parity;
    __syncthreads();  // the previous group is consumed
    const bool is_long = len >= kLongSegment, is_short = len > 0 && !is_long;
    const unsigned lm = __ballot_sync(0xffffffffu, is_long);
    const unsigned sm = __ballot_sync(0xffffffffu, is_short);
    // prefixes within the warp: of the long segments, of the short
    int32_t lp = is_long ? len : 0, sp = is_short ? len : 0;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int32_t x = __shfl_up_sync(0xffffffffu, lp, o);
        const int32_t y = __shfl_up_sync(0xffffffffu, sp, o);
        if (lane >= o) {
            lp += x;
            sp += y;
        }
    }
    if (lane == 31) {
        S.warp_len[0][wid] = lp;
        S.warp_len[1][wid] = sp;
        S.warp_num[0][wid] = __popc(lm);
        S.warp_num[1][wid] = __popc(sm);
    }
    __syncthreads();
    const int32_t wl = lane < kWarps ? S.warp_len[0][lane] : 0;
    const int32_t ws = lane < kWarps ? S.warp_len[1][lane] : 0;
    const int32_t wnl = lane < kWarps ? S.warp_num[0][lane] : 0;
    const int32_t wns = lane < kWarps ? S.warp_num[1][lane] : 0;
    const int32_t total = __reduce_add_sync(0xffffffffu, wl);
    const int32_t short_total = __reduce_add_sync(0xffffffffu, ws);
    const int nlong = __reduce_add_sync(0xffffffffu, wnl);
    const int nshort = __reduce_add_sync(0xffffffffu, wns);
    if (nlong + nshort == 0) return;
    {
        const bool before = lane < wid;
        const int32_t bl = __reduce_add_sync(0xffffffffu, before ? wl : 0);
        const int32_t bs = __reduce_add_sync(0xffffffffu, before ? ws : 0);
        const int fl = __reduce_add_sync(0xffffffffu, before ? wnl : 0);
        const int fs = __reduce_add_sync(0xffffffffu, before ? wns : 0);
        const unsigned below = (1u << lane) - 1u;
        if (is_long) {
            const int at = fl + __popc(lm & below);
            S.seg_base[at] = base;
            S.pref[at] = bl + lp - len;
        } else if (is_short) {
            const int at = fs + __popc(sm & below);
            S.seg_base[nlong + at] = base;
            S.pref[nlong + 1 + at] = bs + sp - len;
        }
        if (threadIdx.x == 0) {
            S.pref[nlong] = total;
            S.pref[nlong + 1 + nshort] = short_total;
            if (nlong > 0) S.next[b ^ 1] = 0;
        }
        if (nlong > 0) parity ^= 1;
        __syncthreads();
    }
    // Short segments: each warp takes an equal block of their entries, its
    // lanes on consecutive ones.  The segment holding entry j is the last s
    // with pref[s] <= j; it only moves forward, so a lane gallops from its
    // previous one.  Four entries a lane in flight.
    if (nshort > 0) {
        const int32_t *pref = S.pref + nlong + 1;
        const int64_t *first = S.seg_base + nlong;
        const int32_t per = (short_total + kWarps - 1) / kWarps;
        const int32_t jb = wid * per, je = min(short_total, jb + per);
        int32_t lo = 0;
        constexpr int kUnroll = 4;
        for (int32_t j0 = jb + lane; j0 < je; j0 += 32 * kUnroll) {
            int32_t xs[kUnroll];
#pragma unroll
            for (int u = 0; u < kUnroll; u++) {
                const int32_t j = j0 + 32 * u;
                xs[u] = 0;
                if (j >= je) continue;
                int32_t step = 1;
                while (lo + step < nshort && pref[lo + step] <= j) {
                    lo += step;
                    step <<= 1;
                }
                int32_t n = min(lo + step, nshort) - lo;
                while (n > 1) {
                    const int32_t h = n >> 1;
                    if (pref[lo + h] <= j) {
                        lo += h;
                        n -= h;
                    } else {
                        n = h;
                    }
                }
                xs[u] = __ldg(adj + first[lo] + (j - pref[lo]));
            }
#pragma unroll
            for (int u = 0; u < kUnroll; u++)
                if (j0 + 32 * u < je) f(xs[u]);
        }
    }
    if (nlong == 0) return;
    // long segments, a piece at a time
    const int32_t piece = max(512, total / (kWarps * kPieces));
    // every warp takes one piece past the end
    static_assert(INT32_MAX + uint64_t(kWarps) * (INT32_MAX / (kWarps * kPieces)) <=
                      std::numeric_limits<std::remove_reference_t<decltype(S.next[0])>>::max(),
                  "the counter does not wrap");
    for (;;) {
        unsigned taken = 0;
        if (lane == 0) taken = atomicAdd(&S.next[b], (unsigned)piece);
        taken = __shfl_sync(0xffffffffu, taken, 0);
        if (taken >= (unsigned)total) break;
        int32_t j = (int32_t)taken;
        const int32_t je = total - j < piece ? total : j + piece;
        // the segment holding entry j: 32-ary search of the prefixes
        const bool in0 = lane * 32 < nlong && S.pref[lane * 32] <= j;
        int s = (__popc(__ballot_sync(0xffffffffu, in0)) - 1) * 32;
        const bool in1 = s + lane < nlong && S.pref[s + lane] <= j;
        s += __popc(__ballot_sync(0xffffffffu, in1)) - 1;
        while (j < je) {
            const int32_t *seg = adj + S.seg_base[s] + (j - S.pref[s]);
            const int32_t end = min(S.pref[s + 1], je), n = end - j;
            j = end;
            s++;
            constexpr int kAhead = 8;
            int32_t i = lane;
            for (; i + 32 * (kAhead - 1) < n; i += 32 * kAhead) {
                int32_t xs[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; u++) xs[u] = __ldg(seg + i + 32 * u);
#pragma unroll
                for (int u = 0; u < kAhead; u++) f(xs[u]);
            }
            for (; i - lane < n; i += 128) {
                int32_t xs[4];
#pragma unroll
                for (int u = 0; u < 4; u++) xs[u] = i + 32 * u < n ? __ldg(seg + i + 32 * u) : 0;
#pragma unroll
                for (int u = 0; u < 4; u++)
                    if (i + 32 * u < n) f(xs[u]);
            }
        }
    }
}

// sum of C(c, 2) over a word's counters of 1 << shift bits.
__device__ __forceinline__ unsigned bytes_pairs(uint32_t c) {  // (sum c^2 - sum c) / 2
    return (__dp4a(c, c, 0u) - __dp4a(c, 0x01010101u, 0u)) >> 1;
}
__device__ __forceinline__ unsigned long long pairs_in_word(uint32_t c, int shift) {
    if (shift == 3) return bytes_pairs(c);
    if (shift == 4) {
        const uint32_t x = c & 0xFFFFu, y = c >> 16;  // each below 2^31 pairs
        return (unsigned long long)(x * (x - 1u) >> 1) + (y * (y - 1u) >> 1);
    }
    if (shift == 2)
        return bytes_pairs(c & 0x0F0F0F0Fu) + bytes_pairs((c >> 4) & 0x0F0F0F0Fu);
    if (shift == 1) {
        const uint32_t hi = (c >> 1) & 0x55555555u;  // 2 -> 1 pair, 3 -> 3
        return (unsigned)(__popc(hi) + 2 * __popc(hi & c));
    }
    return pairs_of(c);
}

// Adds up C(c, 2) over a table of 2^bits slots and empties it.
template <int BLOCK>
__device__ __forceinline__ unsigned long long drain_table(int32_t *key, uint32_t *cnt, int bits) {
    unsigned long long part = 0;
    for (int s = threadIdx.x; s < (1 << bits); s += BLOCK) {
        if (key[s] != kEmpty) {
            part += pairs_of(cnt[s]);
            key[s] = kEmpty;
            cnt[s] = 0;
        }
    }
    return part;
}

// Table bits for W wedges: at most an eighth full where the region has the
// slots (a warp repeats a probe for its slowest lane), never over half.
template <int BLOCK>
__device__ __forceinline__ int table_bits(long long W) {
    constexpr int kMost = 31 - __builtin_clz(RootShape<BLOCK>::kSlots);
    return min(kMost, max(8, 32 - __clz((int)(8 * W - 1))));
}

// Graphs of fewer directed entries and at least this many heavy roots take
// the CTAs of 1,024 threads (R-MAT 2^15: 193 us a count against 236;
// Barabasi-Albert 20,000 x 9, 25 heavy roots and thousands of small ones, 164
// against 142), and so do larger ones with a dense core (R-MAT 2^17 with 15
// entries a vertex: 629 us against 728; with 7.6: 360 against 343;
// Barabasi-Albert 65,000 x 9, 88 heavy roots: 338 against 251; R-MAT 2^18 with
// 11: 1,008 either way).
constexpr int64_t kSmallEntries = 1 << 19, kMiddleEntries = 1 << 21;
constexpr int64_t kFewHeavy = 64, kCoreHeavy = 512;
constexpr int64_t kCoreDensity = 10;  // entries a vertex

// A CTA per root: heavy roots [heavy_begin, heavy_end) first, then the
// deferred ones.
template <int BLOCK, bool STATS>
__global__ void __launch_bounds__(BLOCK, RootShape<BLOCK>::kCtas)
    c4_root_kernel(const RootArgs a) {
    constexpr int kCtaSlots = RootShape<BLOCK>::kSlots, kCtaWedges = RootShape<BLOCK>::kWedges;
    constexpr int kRegionBytes = RootShape<BLOCK>::kRegionBytes;
    constexpr int kRegionWords = RootShape<BLOCK>::kRegionWords;
    extern __shared__ __align__(16) unsigned char smem[];
    uint32_t *region = reinterpret_cast<uint32_t *>(smem);
    RootSmem<BLOCK> &S = *reinterpret_cast<RootSmem<BLOCK> *>(smem + kRegionBytes);
    int32_t *tkey = reinterpret_cast<int32_t *>(smem);
    uint32_t *tcnt = region + kCtaSlots;
    int parity = 0;
    bool clear = false;  // the region has been cleared
    int32_t *cur = a.cursors + (int64_t)blockIdx.x * a.cursor_stride;
    const int64_t nheavy = a.heavy_end - a.heavy_begin;
    unsigned long long part = 0, bytes = 0;
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const int64_t i = (int64_t)atomicAdd(&a.aux->root_cursor, 1ull);
            const int64_t nd = (int64_t)*reinterpret_cast<volatile unsigned long long *>(
                &a.aux->deferred_count);
            S.root = i < nheavy ? a.heavy_begin + i : (i - nheavy < nd ? a.deferred[i - nheavy] : -1);
        }
        __syncthreads();
        const int64_t v0 = S.root;
        if (v0 < 0) break;
        const int64_t o0 = a.off[v0];
        const int32_t d0 = (int32_t)(a.off[v0 + 1] - o0);
        const int32_t lo0 = (int32_t)(a.lo_off[v0 + 1] - a.lo_off[v0]);
        const int32_t dp = d0 - lo0;
        if (dp < 2) continue;
        if (!clear) {
            // The region is all zero between roots: an empty table and
            // cleared counters alike.  (A CTA that gets no root leaves it.)
            for (int i = threadIdx.x; i < kRegionWords / 4; i += BLOCK)
                reinterpret_cast<uint4 *>(region)[i] = make_uint4(0u, 0u, 0u, 0u);
            if (threadIdx.x == 0) S.next[0] = S.next[1] = 0;
            clear = true;
        }
        const int32_t *U = a.adj + o0 + lo0;
        const int ngroups = (dp + BLOCK - 1) / BLOCK;
        // Segment starts; one group's positions stay in registers, more go
        // to the CTA's cursor array.
        int64_t my_o1 = 0;
        int32_t my_pos = 0, my_end = 0;
        long long wl = 0;
        for (int g = 0; g < ngroups; g++) {
            const int i = g * BLOCK + threadIdx.x;
            if (i < dp) {
                const int32_t v1 = U[i];
                const int64_t o1 = a.off[v1];
                const int32_t d1 = (int32_t)(a.off[v1 + 1] - o1);
                const int32_t s1 = above(a.adj + o1, a.lo_off, v1, (int32_t)v0);
                wl += d1 - s1;
                if (ngroups == 1) {
                    my_o1 = o1;
                    my_pos = s1;
                    my_end = d1;
                } else {
                    cur[i] = s1;
                }
            }
        }
        const long long W = typename RootSmem<BLOCK>::Reduce(S.reduce).Sum(wl);
        if (threadIdx.x == 0) S.total = W;
        __syncthreads();
        const long long Wall = S.total;
        if (Wall < 2) continue;
        if (STATS && threadIdx.x == 0) bytes += 4ull * (unsigned long long)Wall + 20ull * dp;
        // This thread's segment of group g from its cursor up to x_end (the
        // list's end where x_end is not below V); advances the cursor.
        auto take = [&](int g, int64_t x_end, int64_t &base) -> int32_t {
            const int i = g * BLOCK + threadIdx.x;
            if (i >= dp) return 0;
            int64_t o1 = my_o1;
            int32_t p = my_pos, d1 = my_end;
            if (ngroups > 1) {
                const int32_t v1 = U[i];
                o1 = a.off[v1];
                d1 = (int32_t)(a.off[v1 + 1] - o1);
                p = cur[i];
            }
            int32_t e = d1;
            if (x_end < a.V) {
                int m = 0;
                while (m < kMarks && x_end != a.mark[m]) m++;
                if (m < kMarks)
                    e = max(p, a.marks[(int64_t)m * a.V + U[i]]);
                else if (p < d1 && a.adj[o1 + d1 - 1] >= (int32_t)x_end)
                    e = p + upper_index(a.adj + o1 + p, d1 - p, (int32_t)x_end - 1);
                if (ngroups > 1)
                    cur[i] = e;
                else
                    my_pos = e;
            }
            base = o1 + p;
            return e - p;
        };
        // Everything from the cursors on through the CTA table.
        auto rest_by_table = [&](long long wedges) {
            const int bits = table_bits<BLOCK>(wedges);
            for (int g = 0; g < ngroups; g++) {
                int64_t base = 0;
                const int32_t len = take(g, a.V, base);
                each_entry<BLOCK>(S, a.adj, base, len, parity, [&](int32_t x) {
                    table_add(tkey, tcnt, bits, x, &a.ctr->error);
                });
            }
            __syncthreads();
            part += drain_table<BLOCK>(tkey, tcnt, bits);
        };
        long long left = Wall;
        // Windows of consecutive ids above v0, until the rest fits the CTA
        // table (wedge endpoints crowd the low, high-degree ids).
        int64_t xlo = v0 + 1 < a.mark[0] ? 0 : v0 + 1;
        while (xlo < a.deg.limit && left > kCtaWedges) {
            const Window w = window_from<BLOCK>(a.deg, (int32_t)xlo);
            if (threadIdx.x == 0) S.in_window = 0;
            long long counted = 0;
            for (int g = 0; g < ngroups; g++) {
                int64_t base = 0;
                const int32_t len = take(g, w.hi, base);
                counted += len;
                each_entry<BLOCK>(S, a.adj, base, len, parity, [&](int32_t x) {
                    const bool second = x >= w.split;
                    const unsigned bit = ((unsigned)x << (second ? w.shift2 : w.shift1)) +
                                         (second ? w.add2 : w.add1);
                    atomicAdd(&region[bit >> 5], 1u << (bit & 31u));
                });
            }
            for (int o = 16; o > 0; o >>= 1)
                counted += __shfl_xor_sync(0xffffffffu, counted, o);
            if ((threadIdx.x & 31) == 0 && counted)
                atomicAdd(&S.in_window, (unsigned long long)counted);
            __syncthreads();
            const long long in_window = (long long)S.in_window;
            if (in_window > 0) {
                uint4 *quads = reinterpret_cast<uint4 *>(region);
                for (int i = threadIdx.x; i < (w.words + 3) / 4; i += BLOCK) {
                    const uint4 q = quads[i];
                    if ((q.x | q.y | q.z | q.w) == 0u) continue;
                    quads[i] = make_uint4(0u, 0u, 0u, 0u);
                    const uint32_t c[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
                    for (int u = 0; u < 4; u++)
                        if (c[u]) part += pairs_in_word(c[u], 4 * i + u < w.words1 ? w.shift1 : w.shift2);
                }
            }
            left -= in_window;
            xlo = w.hi;
            __syncthreads();  // in_window is read, the counters are clear
        }
        if (left > 0 && xlo < a.deg.limit) rest_by_table(left);
    }
    typedef cub::BlockReduce<unsigned long long, BLOCK> R2;
    __syncthreads();
    const unsigned long long tot =
        R2(*reinterpret_cast<typename R2::TempStorage *>(&S.reduce)).Sum(part);
    if (threadIdx.x == 0) {
        atomicAdd(&a.ctr->result, tot);
        if (STATS) atomicAdd(&a.ctr->bytes, bytes);
    }
}

template <int BLOCK, bool STATS>
cudaError_t root_attr() {
    return cudaFuncSetAttribute(c4_root_kernel<BLOCK, STATS>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)root_smem_bytes<BLOCK>());
}

template <int BLOCK, bool STATS>
cudaError_t launch_root(const RootArgs &a, int grid, cudaStream_t st) {
    const cudaError_t e = root_attr<BLOCK, STATS>();
    if (e != cudaSuccess) return e;
    c4_root_kernel<BLOCK, STATS><<<grid, BLOCK, root_smem_bytes<BLOCK>(), st>>>(a);
    return cudaGetLastError();
}

template <int BLOCK, bool STATS>
int root_occupancy() {
    int n = 0;
    if (root_attr<BLOCK, STATS>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, c4_root_kernel<BLOCK, STATS>, BLOCK,
                                                      root_smem_bytes<BLOCK>()) != cudaSuccess)
        return 0;
    return n;
}

template <bool STATS>
cudaError_t light_attr() {
    return cudaFuncSetAttribute(c4_light_kernel<STATS>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLightSmem);
}

template <bool STATS>
int light_occupancy() {
    int n = 0;
    if (light_attr<STATS>() != cudaSuccess ||
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, c4_light_kernel<STATS>, kLightBlock,
                                                      kLightSmem) != cudaSuccess)
        return 0;
    return n;
}

}  // namespace

int c4_light_blocks_per_sm(bool stats) {
    return stats ? light_occupancy<true>() : light_occupancy<false>();
}

int c4_root_threads(int32_t V, int64_t E, int64_t heavy_rows) {
    const bool small = E < kSmallEntries && heavy_rows >= kFewHeavy;
    const bool core =
        E < kMiddleEntries && heavy_rows >= kCoreHeavy && E >= kCoreDensity * V;
    return small || core ? 1024 : 512;
}

int c4_root_blocks_per_sm(int threads, bool stats) {
    if (threads == 1024)
        return stats ? root_occupancy<1024, true>() : root_occupancy<1024, false>();
    return stats ? root_occupancy<512, true>() : root_occupancy<512, false>();
}

cudaError_t launch_c4(const C4Launch &L, cudaStream_t st) {
    const DevGraphView &g = L.g;
    cudaError_t e;
    if ((e = cudaMemsetAsync(L.ctr, 0, sizeof(DevCounters), st)) != cudaSuccess ||
        (e = cudaMemsetAsync(L.aux, 0, sizeof(C4Aux), st)) != cudaSuccess)
        return e;
    Degrees deg{{L.bound[0], L.bound[1], L.bound[2], L.bound[3]}, L.x_limit};
    const bool wide_cta = L.root_threads == 1024;
    int32_t mark[kMarks];
    int32_t at = 0;
    bool marked = false;
    for (int m = 0; m < kMarks; m++) {
        mark[m] = at >= deg.limit ? g.V
                                  : wide_cta ? window_from<1024>(deg, at).hi
                                             : window_from<512>(deg, at).hi;
        at = mark[m];
        marked |= at < g.V;
    }
    const int64_t lb = std::max(L.v_begin, L.heavy_end), le = L.v_end;
    const bool roots = L.v_begin < L.v_end;
    if (lb < le || (roots && marked)) {
        LightArgs la{g.off, g.adj, g.lo_off, lb, le, L.ctr, L.aux, L.deferred, g.V, {}, L.marks,
                     warp_wedges(g.V), 1};
        const int64_t share = (le - lb) / (int64_t(L.light_grid) * (kLightBlock / 32) * kRootShare);
        la.chunk = (int32_t)std::min(std::max<int64_t>(share, 1), kMostRoots);
        for (int m = 0; m < kMarks; m++) la.mark[m] = mark[m];
        if ((e = L.stats ? light_attr<true>() : light_attr<false>()) != cudaSuccess) return e;
        if (L.stats)
            c4_light_kernel<true><<<L.light_grid, kLightBlock, kLightSmem, st>>>(la);
        else
            c4_light_kernel<false><<<L.light_grid, kLightBlock, kLightSmem, st>>>(la);
        if ((e = cudaGetLastError()) != cudaSuccess) return e;
    }
    RootArgs ra{deg, {}, L.marks, g.off, g.adj, g.lo_off, g.V, L.v_begin,
                std::min(L.v_end, L.heavy_end), L.ctr, L.aux, L.deferred, L.cursors,
                L.cursor_stride};
    for (int m = 0; m < kMarks; m++) ra.mark[m] = mark[m];
    if (ra.heavy_end < ra.heavy_begin) ra.heavy_end = ra.heavy_begin;
    if (wide_cta)
        return L.stats ? launch_root<1024, true>(ra, L.root_grid, st)
                       : launch_root<1024, false>(ra, L.root_grid, st);
    return L.stats ? launch_root<512, true>(ra, L.root_grid, st)
                   : launch_root<512, false>(ra, L.root_grid, st);
}

int64_t c4_mark_ints(int32_t V) { return int64_t(kMarks) * V; }

}  // namespace gat
