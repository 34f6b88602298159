// Device memory of graphs and of the temporaries of their uploads.
//
// cudaMalloc and cudaFree synchronise the device and map or unmap the pages,
// and a default pool gives its pages back at every synchronisation: an upload
// of a graph of 4M edges (R-MAT 2^18, 130 MB of bitmaps) spent 20 to 50 ms on
// that and its release 2 to 140 ms, next to 8 ms of counting.  One pool per
// device keeps up to kPoolKeepBytes mapped while the process holds a handle.
// Blocks move between streams in the pool's own stream order (its reuse
// attributes are the defaults: a block freed on one stream is handed to
// another only with the dependency in place), and the tables are locked, so
// threads may upload and free graphs at the same time.  A device reset takes
// the pool with it: each pool has a small allocation whose buffer id (unique in
// the process, so that the address may be used again) tells whether the
// context that made both is still there, and a new pool is made if not.
#include "devmem.hpp"

#include <cuda.h>

#include <cstdint>
#include <mutex>

namespace gat {
namespace {

constexpr int kMaxDevices = 64;

struct Pool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t frees = nullptr;  // orders the frees that name no stream
    void *mark = nullptr;          // what shows that the two still exist
    unsigned long long mark_id = 0;
};

std::mutex g_mu;
Pool g_pools[kMaxDevices];
int64_t g_users = 0;

// The buffer id of a device allocation, 0 if it is none.
unsigned long long buffer_id(const void *p) {
    using Get = CUresult (*)(void *, CUpointer_attribute, CUdeviceptr);
    static const Get get = [] {
        void *fn = nullptr;
        cudaDriverEntryPointQueryResult found{};
        return cudaGetDriverEntryPoint("cuPointerGetAttribute", &fn, cudaEnableDefault, &found) ==
                           cudaSuccess &&
                       found == cudaDriverEntryPointSuccess
                   ? reinterpret_cast<Get>(fn)
                   : nullptr;
    }();
    unsigned long long id = 0;
    if (!get || get(&id, CU_POINTER_ATTRIBUTE_BUFFER_ID, reinterpret_cast<CUdeviceptr>(p)) !=
                    CUDA_SUCCESS)
        return 0;
    return id;
}

// Whether the pool's context is still there.  Locked.
bool alive(const Pool &p) {
    cudaPointerAttributes at{};
    if (!p.pool || cudaPointerGetAttributes(&at, p.mark) != cudaSuccess ||
        at.type != cudaMemoryTypeDevice)
        return false;
    const unsigned long long id = buffer_id(p.mark);
    return id == 0 || id == p.mark_id;
}

// The pool of the current device, made on first use.  Locked.
cudaError_t pool_of(int dev, Pool **out) {
    if (dev < 0 || dev >= kMaxDevices) return cudaErrorInvalidDevice;
    Pool &p = g_pools[dev];
    if (!alive(p)) {
        p = Pool{};
        Pool q;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.handleTypes = cudaMemHandleTypeNone;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        uint64_t keep = kPoolKeepBytes;
        cudaError_t e;
        if ((e = cudaMemPoolCreate(&q.pool, &props)) != cudaSuccess) return e;
        if ((e = cudaMemPoolSetAttribute(q.pool, cudaMemPoolAttrReleaseThreshold, &keep)) !=
                cudaSuccess ||
            (e = cudaMalloc(&q.mark, 1)) != cudaSuccess ||
            (e = cudaStreamCreateWithFlags(&q.frees, cudaStreamNonBlocking)) != cudaSuccess) {
            cudaFree(q.mark);
            cudaMemPoolDestroy(q.pool);
            return e;
        }
        q.mark_id = buffer_id(q.mark);
        p = q;
    }
    *out = &p;
    return cudaSuccess;
}

// Gives back every pool's unused pages.
void trim_locked() {
    for (Pool &p : g_pools)
        if (alive(p)) {
            cudaStreamSynchronize(p.frees);
            cudaMemPoolTrimTo(p.pool, 0);
        }
}

void trim_pools() {
    std::lock_guard<std::mutex> lk(g_mu);
    trim_locked();
}

}  // namespace

cudaError_t dev_alloc(void **p, size_t bytes, cudaStream_t st) {
    *p = nullptr;
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    cudaMemPool_t pool = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        Pool *q = nullptr;
        if ((e = pool_of(dev, &q)) != cudaSuccess) return e;
        pool = q->pool;
    }
    e = cudaMallocFromPoolAsync(p, bytes ? bytes : 1, pool, st);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();  // blocks of another size may hold the room
    if ((e = cudaStreamSynchronize(st)) != cudaSuccess) return e;
    trim_pools();
    return cudaMallocFromPoolAsync(p, bytes ? bytes : 1, pool, st);
}

cudaError_t plain_alloc(void **p, size_t bytes) {
    const cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaErrorMemoryAllocation) return e;
    cudaGetLastError();
    trim_pools();
    return cudaMalloc(p, bytes);
}

cudaError_t dev_free(void *p, cudaStream_t st) { return p ? cudaFreeAsync(p, st) : cudaSuccess; }

void dev_free(void *p) {
    if (!p) return;
    // the memory may belong to another device than the current one, or have
    // gone with a reset
    cudaPointerAttributes at{};
    int cur = 0;
    if (cudaGetDevice(&cur) != cudaSuccess || cudaPointerGetAttributes(&at, p) != cudaSuccess ||
        at.type != cudaMemoryTypeDevice || at.device < 0 || at.device >= kMaxDevices)
        return;
    cudaStream_t frees = nullptr;
    {
        std::lock_guard<std::mutex> lk(g_mu);
        const Pool &q = g_pools[at.device];
        if (!alive(q)) return;
        frees = q.frees;
    }
    if (at.device != cur) cudaSetDevice(at.device);
    cudaFreeAsync(p, frees);
    if (at.device != cur) cudaSetDevice(cur);
}

PoolUser::PoolUser() {
    std::lock_guard<std::mutex> lk(g_mu);
    g_users++;
}

PoolUser::~PoolUser() {
    std::lock_guard<std::mutex> lk(g_mu);
    if (--g_users == 0) trim_locked();
}

}  // namespace gat
