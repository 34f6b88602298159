// Exact 5-cycle count by path counts at the cycle's largest vertex (sm_100a).
//
// Every 5-cycle v0 - a - x - y - b is counted at its largest id v0; the other
// four lie in G' = the graph on the ids below v0.  With L = N<(v0) and
// P[x] = |N(x) n L| (the 2-paths v0 - a - x), the closed walks
// v0 - a - x - y - b - v0 with x ~ y number sum over ordered edges (x, y) of
// G' of P[x] P[y], and a walk is no cycle exactly when
//   a = b:  x, y are two adjacent neighbours of a;
//   a = y:  x is any neighbour of a and b any neighbour of a in L;
//   b = x:  the same mirrored;   a = y and b = x together: a ~ b in L.
// So, each cycle being two walks,
//   C5(v0) =   sum_{x < v0} P[x] sum_{y in N<(x)} P[y]
//            - sum_{a in L} t'(a) - sum_{a in L} d'(a) P[a]
//            + (1/2) sum_{a in L} P[a],
// d' and t' the degree and the triangles of a in G'.  The triangle term needs
// no roots: summed over all v0, a triangle a, x < y (y the larger of the other
// two) is met once for every neighbour v0 of a above both a and y, that is
//   sum over entries y = N(a)[i] of |N(a) n N<(y)| (deg(a) - max(i+1, lo(a))).
//
// This is one pass over the edges per root (a sum of P over lower neighbours),
// where the schedule plan enumerates (v0, v1, v2, v3) and intersects two lists
// for each: 13 million intersections on a Barabasi-Albert graph of 20,011
// vertices, with fewer than two candidates for the last level's 32 lanes.
//
//  * c5_edge_kernel: a thread per entry (a, i) for the triangle term;
//  * c5_root_kernel: a CTA per root, largest id first.  P is an array of
//    16-bit counters for all ids in shared memory (so the graph has at most
//    about 98,000 vertices, and small graphs run several CTAs per SM): the
//    warps stream N(a) up to v0 for a in L with shared atomics, then scan the
//    counters 256 at a time, queue the ids with P > 0, and eight lanes each
//    sum P over an id's lower neighbours.
//
// Neither kernel waits on another CTA.  Bound: shared-memory reads of P at
// random ids and, on sparse graphs, the scan of the counters.  Barabasi-Albert
// 20,011 x 9: 11.0 ms by the plan, 0.80 by path counts.
#include <algorithm>

#include "engine.hpp"

namespace gat {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kThreads = 256;
constexpr int kWarps = kThreads / 32;

struct C5Args {
    const int64_t *off;
    const int32_t *adj;
    const int64_t *lo_off;
    const int32_t *hub_slot;  // null: no bitmaps
    const uint32_t *bitmaps;
    int64_t bitmap_words;
    int32_t V;
    int64_t E;
    DevCounters *ctr;
    int32_t max_lower;
};

__device__ __forceinline__ int32_t lower_degree(const C5Args &a, int32_t v) {
    return (int32_t)(a.lo_off[v + 1] - a.lo_off[v]);
}

// First index i of the sorted a[0, n) with a[i] >= x (one thread alone).
__device__ __forceinline__ int32_t lower_index(const int32_t *a, int32_t n, int32_t x) {
    int32_t lo = 0;
    while (n > 0) {
        const int32_t h = n >> 1;
        const bool right = a[lo + h] < x;
        lo = right ? lo + h + 1 : lo;
        n = right ? n - h - 1 : h;
    }
    return lo;
}

__device__ __forceinline__ bool in_list(const int32_t *a, int32_t n, int32_t x) {
    const int32_t i = lower_index(a, n, x);
    return i < n && a[i] == x;
}

__device__ __forceinline__ void add_total(unsigned long long v, DevCounters *ctr) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(kFull, v, o);
    if ((threadIdx.x & 31) == 0 && v) atomicAdd(&ctr->result, v);
}

// The triangle term, subtracted from the total.  Entry e of row a holds y;
// |N(a)[0, i) n N<(y)|: the shorter list's elements are looked up in the other
// vertex's bitmap row or list.
__global__ void __launch_bounds__(kThreads) c5_edge_kernel(const C5Args a) {
    unsigned long long sum = 0;
    for (int64_t e = (int64_t)blockIdx.x * kThreads + threadIdx.x; e < a.E;
         e += (int64_t)gridDim.x * kThreads) {
        // the row holding entry e
        int32_t lo = 0, n = a.V;
        while (n > 1) {
            const int32_t h = n >> 1;
            if (a.off[lo + h] <= e) {
                lo += h;
                n -= h;
            } else {
                n = h;
            }
        }
        const int32_t v = lo;
        const int64_t o = a.off[v];
        const int32_t d = (int32_t)(a.off[v + 1] - o), i = (int32_t)(e - o);
        const int32_t y = a.adj[e];
        const int32_t roots = d - max(i + 1, lower_degree(a, v));
        if (roots <= 0) continue;
        const int32_t ly = lower_degree(a, y);
        const bool mine = i <= ly;  // probe N(v)[0, i) in y's row, else N<(y) in v's
        const int32_t *probe = a.adj + (mine ? o : a.off[y]);
        const int32_t np = mine ? i : ly;
        const int32_t other = mine ? y : v;
        const int slot = a.hub_slot != nullptr ? a.hub_slot[other] : -1;
        int c = 0;
        if (slot >= 0) {
            const uint32_t *row = a.bitmaps + (int64_t)slot * a.bitmap_words;
            for (int32_t k = 0; k < np; k++) {
                const int32_t x = probe[k];
                c += (__ldg(row + (x >> 5)) >> (x & 31)) & 1u;
            }
        } else {
            const int32_t *list = a.adj + (mine ? a.off[y] : o);
            const int32_t nl = mine ? ly : i;
            for (int32_t k = 0; k < np; k++) c += in_list(list, nl, probe[k]) ? 1 : 0;
        }
        sum += (unsigned long long)c * (unsigned)roots;
    }
    add_total(0ull - sum, a.ctr);
}

struct alignas(16) C5Smem {  // the counters behind it are read 16 bytes at a time
    int32_t queue[kWarps][256];  // ids with P > 0 of a warp's 256 counters
    int32_t root;
};

__global__ void __launch_bounds__(kThreads) c5_root_kernel(const C5Args a) {
    extern __shared__ __align__(16) unsigned char smem[];
    C5Smem &S = *reinterpret_cast<C5Smem *>(smem);
    int32_t *below = reinterpret_cast<int32_t *>(smem + sizeof(C5Smem));  // d'(a), a in L
    uint32_t *words = reinterpret_cast<uint32_t *>(below + (a.max_lower + 3) / 4 * 4);
    const uint16_t *P = reinterpret_cast<const uint16_t *>(words);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int quads = (a.V + 7) / 8;  // of eight counters
    uint4 *P4 = reinterpret_cast<uint4 *>(words);
    for (int q = threadIdx.x; q < quads; q += kThreads) P4[q] = make_uint4(0u, 0u, 0u, 0u);
    unsigned long long sum = 0, inside = 0;  // inside: sum of P over L, twice its edges
    for (;;) {
        __syncthreads();
        if (threadIdx.x == 0) {
            const int64_t i = (int64_t)atomicAdd(&a.ctr->cursor, 1ull);
            S.root = i < a.V ? (int32_t)(a.V - 1 - i) : -1;
        }
        __syncthreads();
        const int32_t v0 = S.root;
        if (v0 < 0) break;
        const int32_t nL = lower_degree(a, v0);
        if (nL == 0) continue;
        const int32_t *L = a.adj + a.off[v0];
        for (int t = threadIdx.x; t < nL; t += kThreads) {
            const int32_t v = L[t], lo = lower_degree(a, v);
            const int64_t o = a.off[v];
            // v0 lies among v's upper neighbours
            below[t] = lo + lower_index(a.adj + o + lo, (int32_t)(a.off[v + 1] - o) - lo, v0);
        }
        __syncthreads();
        for (int t = wid; t < nL; t += kWarps) {
            const int32_t *nb = a.adj + a.off[L[t]];
            const int32_t n = below[t];
            constexpr int kAhead = 4;
            for (int32_t i = lane; i - lane < n; i += 32 * kAhead) {
                int32_t xs[kAhead];
#pragma unroll
                for (int u = 0; u < kAhead; u++) xs[u] = i + 32 * u < n ? __ldg(nb + i + 32 * u) : -1;
#pragma unroll
                for (int u = 0; u < kAhead; u++)
                    if (xs[u] >= 0) atomicAdd(&words[xs[u] >> 1], 1u << ((xs[u] & 1) << 4));
            }
        }
        __syncthreads();
        for (int t = threadIdx.x; t < nL; t += kThreads) {
            const unsigned p = P[L[t]];
            sum -= (unsigned long long)p * (unsigned)below[t];
            inside += p;
        }
        // sum over x < v0 of P[x] sum over y in N<(x) of P[y]
        const int used = (v0 + 7) / 8;
        for (int q0 = wid * 32; q0 < used; q0 += kWarps * 32) {
            const int q = q0 + lane;
            const uint4 c = q < used ? P4[q] : make_uint4(0u, 0u, 0u, 0u);
            const uint32_t w[4] = {c.x, c.y, c.z, c.w};
            unsigned set = 0;
#pragma unroll
            for (int u = 0; u < 4; u++)
                set |= ((w[u] & 0xFFFFu) ? 1u : 0u) << (2 * u) | ((w[u] >> 16) ? 2u : 0u) << (2 * u);
            int at = __popc(set);
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, at, o);
                if (lane >= o) at += y;
            }
            const int total = __shfl_sync(kFull, at, 31);
            if (total == 0) continue;
            at -= __popc(set);
            while (set) {
                S.queue[wid][at++] = 8 * q + __ffs(set) - 1;
                set &= set - 1;
            }
            __syncwarp();
            // eight lanes an id
            for (int t = lane >> 3; t < total; t += 4) {
                const int32_t x = S.queue[wid][t];
                const int32_t *nb = a.adj + a.off[x];
                const int32_t n = lower_degree(a, x);
                unsigned s = 0;  // at most |L| per neighbour
                unsigned long long s64 = 0;
                for (int32_t i0 = 0; i0 < n; i0 += 4096) {
                    const int32_t end = min(n, i0 + 4096);
#pragma unroll 4
                    for (int32_t i = i0 + (lane & 7); i < end; i += 8) s += P[__ldg(nb + i)];
                    s64 += s;
                    s = 0;
                }
                sum += s64 * P[x];
            }
            __syncwarp();
        }
        __syncthreads();
        for (int q = threadIdx.x; q < used; q += kThreads) P4[q] = make_uint4(0u, 0u, 0u, 0u);
    }
    // half of `inside`, a whole number over all of a root's threads: kept
    // apart (ctr->bytes) until the host halves the sum
    add_total(sum, a.ctr);
    for (int o = 16; o > 0; o >>= 1) inside += __shfl_xor_sync(kFull, inside, o);
    if (lane == 0 && inside) atomicAdd(&a.ctr->bytes, inside);
}

// The total of a job in a batch: one word.
__global__ void c5_finish_kernel(DevCounters *ctr, unsigned long long *result) {
    *result = ctr->result + ctr->bytes / 2;
}

static_assert(sizeof(C5Smem) % 16 == 0, "counters start on 16 bytes");

size_t root_smem(const DevGraphView &g) {
    return sizeof(C5Smem) + (size_t(g.max_lower) + 3) / 4 * 16 + (size_t(g.V) + 7) / 8 * 16;
}

}  // namespace

// Graphs that the path counts take: the counters fit in shared memory, and
// scanning V counters per root is no more than the plan's walk.  The scan does
// not fall with the density, the walk does: with 2 entries a vertex G(40,000)
// takes 0.51 ms by paths and 0.10 by the plan.  Measured (path / plan, ms; d
// entries a vertex):
//   G(n, d)            d = 2          4           8            12
//     n = 4,000     .027 / .074  .031 / .10   .037 / .22   .045 / .51
//        16,000     .085 / .089  .12 / .19    .15 / .60    .18 / 1.6
//        24,000     .16 / .10    .21 / .23    .29 / .87    .36 / 2.4
//        40,000     .51 / .10    .74 / .36    1.0 / 1.5    1.3 / 4.1
//        64,000     1.9 / .15    2.7 / .57    3.7 / 2.6    4.7 / 7.2
//        95,000     3.5 / .22    5.0 / .82    6.6 / 4.0    8.3 / 11
//   Barabasi-Albert 40,000  .77 / .53    1.0 / 1.6    1.5 / 4.0    2.1 / 8.2
//                   64,000  2.8 / .76    3.6 / 2.3    5.4 / 5.9    7.3 / 13
//   R-MAT of 2^15, 2^16 vertices, d = 2: .41 / 2.3, 2.5 / 6.2
// Up to 2^14 vertices, and from 12 entries a vertex on, the paths were ahead on
// every graph tried.  In between, a walk grows with the density and the longest
// rows and lower lists, the scan with V^2 over the CTAs an SM holds; of 260
// graphs of 12,000 to 95,000 vertices the line below sends none to the paths
// that lose more than 1.37 times there, and none to the plan that lose more
// than 1.56 (both a tenth of a ms to a few ms long).
bool c5_fits(const DevGraphView &g) {
    constexpr size_t kSmBytes = 227 * 1024, kCtaBytes = 1024;  // CTA: reserved by the system
    const size_t smem = root_smem(g);
    if (g.V <= 0 || g.lo_off == nullptr || g.max_lower >= 65536 || smem > 200 * 1024) return false;
    if (g.V <= 16384 || g.E >= int64_t(12) * g.V) return true;
    const double v = g.V, d = double(g.E) / v, lower = g.max_lower;
    const double ctas = double(std::min<size_t>(2048 / kThreads, kSmBytes / (smem + kCtaBytes)));
    return d * d * d * lower * lower * g.max_degree * ctas * ctas >= 2.5e-13 * v * v * v * v;
}

cudaError_t c5_blocks_per_sm(const DevGraphView &g, int *blocks) {
    const size_t smem = root_smem(g);
    *blocks = 0;
    const cudaError_t e = cudaFuncSetAttribute(
        c5_root_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, 200 * 1024);
    if (e != cudaSuccess) return e;
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(blocks, c5_root_kernel, kThreads, smem);
}

cudaError_t launch_c5(const DevGraphView &g, int sms, int grid, DevCounters *ctr,
                      unsigned long long *result, cudaStream_t st) {
    cudaError_t e = cudaMemsetAsync(ctr, 0, sizeof(DevCounters), st);
    if (e != cudaSuccess) return e;
    C5Args a{g.off, g.adj, g.lo_off, g.bitmaps ? g.hub_slot : nullptr, g.bitmaps, g.bitmap_words,
             g.V,   g.E,   ctr,      g.max_lower};
    const int64_t need = (g.E + kThreads - 1) / kThreads;
    if (need > 0)
        c5_edge_kernel<<<(unsigned)std::min<int64_t>(need, int64_t(sms) * 32), kThreads, 0, st>>>(a);
    c5_root_kernel<<<grid, kThreads, root_smem(g), st>>>(a);
    if (result) c5_finish_kernel<<<1, 1, 0, st>>>(ctr, result);
    return cudaGetLastError();
}

}  // namespace gat
