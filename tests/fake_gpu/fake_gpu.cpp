// The CUDA runtime calls and the device functions that capi.cpp and
// devmem.cpp use, on the host: device memory is host memory in a table of live
// blocks, streams run at once, kernels that prepare a graph are loops, and
// kernels that count check the arrays they are given and add nothing.  Tests
// make calls fail here that a GPU would need a fault or a full memory for.
#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <new>
#include <numeric>

#include "engine.hpp"
#include "graph.hpp"

using namespace gat;

// What tests set and read (fake.py names the slots).
enum {
    kRefuse,      // set: device allocations of this many bytes and more fail
    kThrow,       // set: host allocations of this many bytes and more throw
    kMisuse,      // dead or half-built arrays, dead pools and streams used
    kLive,        // live device blocks
    kPending,     // copies issued since the last synchronisation
    kC5Launches,
    kC5Grid,
    kC5Bitmaps,   // 1: the last 5-cycle launch was given bitmaps
    kSearches,
    kCliques,
    kDeepRows,    // the last search's DevGraphView::deep_rows
    kSlots
};
extern "C" {
int64_t fake_state[kSlots] = {INT64_MAX, INT64_MAX};
void (*fake_during)() = nullptr;  // called while a counting kernel runs
void fake_reset();
int fake_from_csr_device(int32_t V, int64_t E, const int64_t *off, const int32_t *adj);
}

namespace {

struct Block {
    size_t bytes;
    unsigned long long id;
};
std::map<const char *, Block> g_blocks;
std::multimap<size_t, char *> g_dead;  // addresses a reset has left to use again
unsigned long long g_next_id = 1;
int64_t g_context = 1;  // a pool, stream or event of another one is dead

struct Owned {
    int64_t context;
};
bool alive(const void *p) {
    const bool ok = p == nullptr || static_cast<const Owned *>(p)->context == g_context;
    if (!ok) fake_state[kMisuse]++;
    return ok;
}

const Block *block_of(const void *p, size_t bytes) {
    auto it = g_blocks.upper_bound(static_cast<const char *>(p));
    if (it == g_blocks.begin()) return nullptr;
    --it;
    const char *q = static_cast<const char *>(p);
    return q + bytes <= it->first + it->second.bytes ? &it->second : nullptr;
}

void need(const void *p, size_t bytes) {
    if (!block_of(p, bytes)) fake_state[kMisuse]++;
}

cudaError_t take(void **p, size_t bytes) {
    *p = nullptr;
    if ((int64_t)bytes >= fake_state[kRefuse]) return cudaErrorMemoryAllocation;
    auto again = g_dead.find(bytes);
    char *q = again != g_dead.end() ? again->second : static_cast<char *>(std::malloc(bytes + 64));
    if (again != g_dead.end()) g_dead.erase(again);
    std::memset(q, 0x5A, bytes + 64);
    g_blocks[q] = {bytes, g_next_id++};
    fake_state[kLive]++;
    *p = q;
    return cudaSuccess;
}

cudaError_t give(void *p) {
    if (!p) return cudaSuccess;
    auto it = g_blocks.find(static_cast<char *>(p));
    if (it == g_blocks.end()) return cudaErrorInvalidValue;
    g_blocks.erase(it);
    fake_state[kLive]--;
    std::free(p);
    return cudaSuccess;
}

// Every array of a graph that a counting kernel is handed.
void check(const DevGraphView &g, bool bitmaps) {
    if (fake_during) fake_during();
    need(g.off, 8 * (size_t(g.V) + 1));
    need(g.lo_off, 8 * (size_t(g.V) + 1));
    need(g.adj, 4 * size_t(g.E));
    if (!bitmaps || !g.hub_slot) return;
    need(g.hub_slot, 4 * size_t(g.V));
    if (!block_of(g.hub_slot, 4 * size_t(g.V))) return;
    for (int32_t v = 0; v < g.V; v++)
        if (g.hub_slot[v] >= 0)
            need(g.bitmaps + int64_t(g.hub_slot[v]) * g.bitmap_words, 4 * size_t(g.bitmap_words));
        else if (g.hub_slot[v] != -1)
            fake_state[kMisuse]++;
}

struct FakeJob {
    DevGraphView g;
    bool bitmaps;
    int result;
};

HostGraph host_view(const int64_t *off, const int32_t *adj, int32_t V) {
    HostGraph h;
    h.V = V;
    h.E = off[V];
    h.off.assign(off, off + V + 1);
    h.adj.assign(adj, adj + off[V]);
    return h;
}

CUresult buffer_id(void *out, CUpointer_attribute what, CUdeviceptr p) {
    const Block *b = block_of(reinterpret_cast<void *>(p), 1);
    if (what != CU_POINTER_ATTRIBUTE_BUFFER_ID || !b) return CUDA_ERROR_INVALID_VALUE;
    *static_cast<unsigned long long *>(out) = b->id;
    return CUDA_SUCCESS;
}

}  // namespace

// Host allocations of the library under test.
void *operator new(size_t n) {
    if ((int64_t)n >= fake_state[kThrow]) throw std::bad_alloc();
    if (void *p = std::malloc(n ? n : 1)) return p;
    throw std::bad_alloc();
}
void operator delete(void *p) noexcept { std::free(p); }
void operator delete(void *p, size_t) noexcept { std::free(p); }

extern "C" {

// cudaDeviceReset: every block, pool, stream and event of the context is gone.
void fake_reset() {
    for (auto &b : g_blocks) g_dead.insert({b.second.bytes, const_cast<char *>(b.first)});
    g_blocks.clear();
    fake_state[kLive] = 0;
    g_context++;
}

// gat_graph_from_csr_device for callers that cannot catch: -1 for a host
// allocation that failed.
int gat_graph_from_csr_device(int32_t, int64_t, const int64_t *, const int32_t *, void *,
                              struct gat_graph **);
int fake_from_csr_device(int32_t V, int64_t E, const int64_t *off, const int32_t *adj) {
    struct gat_graph *g = nullptr;
    try {
        return gat_graph_from_csr_device(V, E, off, adj, nullptr, &g);
    } catch (const std::bad_alloc &) {
        return -1;
    }
}

cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "success" : "refused"; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 100, cudaSuccess; }
cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return *p = std::malloc(n), cudaSuccess; }
cudaError_t cudaFreeHost(void *p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t pool, cudaStream_t) {
    return alive(pool) ? take(p, n) : cudaErrorInvalidValue;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t st) { return alive(st) ? give(p) : cudaErrorInvalidValue; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) {
    return *p = reinterpret_cast<cudaMemPool_t>(new Owned{g_context}), cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) { return alive(p) ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t p, cudaMemPoolAttr, void *) {
    return alive(p) ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t p, size_t) { return alive(p) ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(new Owned{g_context}), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { return alive(s) ? cudaSuccess : cudaErrorInvalidValue; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    fake_state[kPending] = 0;
    return alive(s) ? cudaSuccess : cudaErrorInvalidValue;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    *a = {};
    a->type = block_of(p, 1) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    a->device = block_of(p, 1) ? 0 : -2;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char *name, void **fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *r) {
    *fn = std::strcmp(name, "cuPointerGetAttribute") == 0 ? reinterpret_cast<void *>(&buffer_id) : nullptr;
    if (r) *r = *fn ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
cudaError_t cudaGetDriverEntryPoint(const char *name, void **fn, unsigned long long f,
                                    cudaDriverEntryPointQueryResult *r) {
    return cudaGetDriverEntryPointByVersion(name, fn, 0, f, r);
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) {
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    fake_state[kPending]++;
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
    return std::memset(p, v, n), cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }
// (captured launches are not replayed: tests prepare without a graph)
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    return *e = nullptr, cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

}  // extern "C"

namespace gat {

// ------------------------------------------------ kernels that prepare graphs

cudaError_t build_hub_bitmaps(const int64_t *off, const int32_t *adj, const int32_t *hubs,
                              int32_t n, int64_t words, uint32_t *bitmaps, cudaStream_t) {
    for (int32_t h = 0; h < n; h++)
        for (int64_t i = off[hubs[h]]; i < off[hubs[h] + 1]; i++)
            bitmaps[h * words + (adj[i] >> 5)] |= 1u << (adj[i] & 31);
    return cudaSuccess;
}

cudaError_t lower_offsets_device(const int64_t *off, const int32_t *adj, int32_t V,
                                 int64_t *lo_off, cudaStream_t) {
    lo_off[0] = 0;
    for (int32_t v = 0; v < V; v++) {
        lo_off[v + 1] = lo_off[v];
        for (int64_t i = off[v]; i < off[v + 1]; i++) lo_off[v + 1] += adj[i] < v;
    }
    return cudaSuccess;
}

cudaError_t csr_extremes_device(const int64_t *off, const int64_t *lo_off, int32_t V,
                                int64_t light_below, bool ordered, CsrExtremes *out,
                                cudaStream_t) {
    *out = CsrExtremes{lo_off[V], 0, 0, V, {V, V, V, V, V}};
    for (int32_t v = V - 1; v >= 0; v--) {
        const int64_t d = off[v + 1] - off[v];
        out->max_degree = std::max(out->max_degree, (int32_t)d);
        out->max_lower = std::max(out->max_lower, (int32_t)(lo_off[v + 1] - lo_off[v]));
        if (d < light_below) out->first_light = v;
        for (int i = 0; i < 5 && ordered; i++)
            if (d < (i < 4 ? 1 << (16 >> i) : 2)) out->below[i] = v;
    }
    return cudaSuccess;
}

cudaError_t leading_rows_device(const int64_t *off, int32_t V, int64_t d0, int64_t d1,
                                int64_t *out, cudaStream_t) {
    const int64_t want[2] = {d0, d1};
    for (int i = 0; i < 2; i++) {
        out[2 * i] = 0;
        for (int32_t v = 0; v < V; v++) out[2 * i] += off[v + 1] - off[v] >= want[i];
        out[2 * i + 1] = off[out[2 * i]];
    }
    return cudaSuccess;
}

cudaError_t hub_slots_device(int32_t *hubs, int32_t n, int32_t V, bool ordered, int32_t *slot,
                             cudaStream_t) {
    if (ordered) std::iota(hubs, hubs + n, 0);
    for (int32_t v = 0; v < V; v++) slot[v] = -1;
    for (int32_t h = 0; h < n; h++) slot[hubs[h]] = h;
    return cudaSuccess;
}

bool relabel_fits_device(int32_t V, int64_t) { return V > 0; }
cudaError_t relabel_by_degree_device(const int64_t *off, const int32_t *adj, int32_t V, int64_t,
                                     int32_t, int64_t *new_off, int32_t *new_adj, cudaStream_t) {
    HostGraph r;
    relabel_by_degree(host_view(off, adj, V), r, nullptr);
    std::copy(r.off.begin(), r.off.end(), new_off);
    std::copy(r.adj.begin(), r.adj.end(), new_adj);
    return cudaSuccess;
}

cudaError_t csr_check_device(const int64_t *, const int32_t *, int32_t, int64_t,
                             unsigned long long *flag, cudaStream_t) {
    return *flag = ~0ull, cudaSuccess;
}
cudaError_t rmat_csr_device(int, int64_t, double, double, double, uint64_t, int64_t *, int32_t **,
                            int64_t, int64_t *, cudaStream_t) {
    return cudaErrorNotSupported;
}
cudaError_t pairs_csr_device(const int32_t *, int64_t, int32_t, int64_t *, int32_t **, int64_t,
                             int64_t *, cudaStream_t) {
    return cudaErrorNotSupported;
}

// --------------------------------------------------------- kernels that count

int blocks_per_sm(const GatPlan &, const DevGraphView &, const LaunchShape &, bool) { return 4; }
int batch_blocks_per_sm(int, int) { return 4; }
int64_t tile_scratch_ints(const GatPlan &plan, int32_t max_degree) {
    return int64_t(plan.num_store) * max_degree;
}
cudaError_t launch_search(const GatPlan *, const GatPlan &, const DevGraphView &g,
                          const LaunchShape &shape, int32_t *, int64_t, DevCounters *ctr, bool,
                          cudaStream_t) {
    check(g, shape.use_bitmaps && g.bitmaps && g.hub_slot);
    fake_state[kSearches]++;
    fake_state[kDeepRows] = g.deep_rows;
    return *ctr = DevCounters{}, cudaSuccess;
}
int count_noalloc(const GatPlan &, const int64_t *, const int32_t *, int32_t, int64_t, int32_t,
                  const LaunchShape &, long long *, cudaStream_t, std::string *) {
    return 4;
}

bool c5_fits(const DevGraphView &g) { return g.V > 0; }
cudaError_t c5_blocks_per_sm(const DevGraphView &, int *blocks) { return *blocks = 2, cudaSuccess; }
cudaError_t launch_c5(const DevGraphView &g, int, int grid, DevCounters *ctr,
                      unsigned long long *result, cudaStream_t) {
    check(g, true);
    fake_state[kC5Launches]++;
    fake_state[kC5Grid] = grid;
    fake_state[kC5Bitmaps] = g.hub_slot != nullptr;
    *ctr = DevCounters{};
    if (result) *result = 0;
    return cudaSuccess;
}

int64_t clique_rows_words(int, int32_t) { return 0; }
int64_t clique_list_ints(int64_t) { return 4; }
void clique_blocks_per_sm(int, bool, int *w, int *c) { *w = *c = 2; }
cudaError_t launch_clique(const CliqueLaunch &l, cudaStream_t) {
    check(l.g, true);
    fake_state[kCliques]++;
    return *l.ctr = DevCounters{}, cudaSuccess;
}

int64_t c4_mark_ints(int32_t V) { return 2 * int64_t(V); }
int c4_light_blocks_per_sm(bool) { return 2; }
int c4_root_threads(int32_t, int64_t, int64_t) { return 512; }
int c4_root_blocks_per_sm(int, bool) { return 2; }
cudaError_t launch_c4(const C4Launch &l, cudaStream_t) {
    check(l.g, false);
    return *l.ctr = DevCounters{}, cudaSuccess;
}

size_t batch_job_bytes() { return sizeof(FakeJob); }
void batch_fill_job(void *dst, const GatPlan *, const GatPlan &, const DevGraphView &g, int,
                    bool bitmaps, int result, int, int) {
    *static_cast<FakeJob *>(dst) = {g, bitmaps && g.bitmaps && g.hub_slot, result};
}
int64_t batch_job_tasks(const void *job) { return static_cast<const FakeJob *>(job)->g.lo_total; }
int64_t batch_job_grabs(void *job, const GatPlan &, int64_t, int64_t, int, int) { return batch_job_tasks(job); }
cudaError_t launch_batch(const void *jobs, const int64_t *, int32_t n, int64_t, int, int, int,
                         unsigned long long *, unsigned long long *, int32_t *, int64_t,
                         cudaStream_t) {
    for (int32_t j = 0; j < n; j++) {
        const FakeJob &job = static_cast<const FakeJob *>(jobs)[j];
        check(job.g, job.bitmaps);
    }
    return cudaSuccess;
}

}  // namespace gat
