// Device memory of plans, from one stream-ordered pool per device and context.
//
// A plan's creation and its destruction make about fifty-five allocations and
// as many frees. cudaMalloc took 0.35 ms and cudaFree 0.30 ms each on a B200
// (whatever the size, 4 kB to 256 MB), which was 20 of the 25 ms of a new
// Pilatus-1M geometry and its first frame; the pool serves an allocation it
// holds in a few microseconds. The pool keeps at most kPoolKeep bytes that no
// array uses: the driver gives memory above that back at the next
// synchronisation, and all of it when an allocation fails (torch's and other
// libraries' allocations do not see the pool).
//
// Ordering. Inside an AllocScope an array is allocated and freed in the order
// of the scope's stream, for the builders, which use their arrays on that
// stream alone and synchronise it before any other stream sees what they leave.
// Outside a scope an allocation is complete when the call returns, and a free
// waits for the device first, as cudaFree does: arrays of a living plan may be
// in use on any of the callers' streams. The wait is a cudaFree (device_wait):
// cudaDeviceSynchronize would end every stream capture in the process, of other
// threads and of relaxed mode too, and then not have waited.
#include <cuda.h>

#include <map>
#include <mutex>
#include <vector>

#include "dg_internal.h"

namespace dg {
namespace {

constexpr uint64_t kPoolKeep = uint64_t(1) << 30;

struct Pool {
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;  // order of allocations outside a scope
    std::mutex mu;
    std::vector<void *> pending;    // to be freed after the next wait for the device
};

// Number of the current CUDA context, which no later one of the process has: a
// pool and its stream end with their context (cudaDeviceReset), and a new context
// gets new ones. 0 where the driver does not tell.
uint64_t context_number() {
    using Current = CUresult (*)(CUcontext *);
    using Id = CUresult (*)(CUcontext, unsigned long long *);
    static const std::pair<Current, Id> entry = [] {
        void *current = nullptr, *id = nullptr;
        cudaDriverEntryPointQueryResult found;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &current, cudaEnableDefault, &found) != cudaSuccess ||
            cudaGetDriverEntryPoint("cuCtxGetId", &id, cudaEnableDefault, &found) != cudaSuccess)
            current = id = nullptr;
        (void)cudaGetLastError();
        return std::make_pair(reinterpret_cast<Current>(current), reinterpret_cast<Id>(id));
    }();
    CUcontext context = nullptr;
    unsigned long long number = 0;
    if (!entry.first || !entry.second || entry.first(&context) != CUDA_SUCCESS) return 0;
    if (!context) {  // the runtime makes the device's context with its first use
        (void)cudaFree(nullptr);
        if (entry.first(&context) != CUDA_SUCCESS || !context) return 0;
    }
    return entry.second(context, &number) == CUDA_SUCCESS ? number : 0;
}

// The pool of the current device and context, made on first use (and tried again
// after a failure); nullptr and the error where it cannot be.
Pool *pool_of(int device, uint64_t context, cudaError_t *error) {
    // not destroyed: arrays may outlive statics
    static auto *const mu = new std::mutex;
    static auto *const pools = new std::map<std::pair<int, uint64_t>, Pool>;
    std::lock_guard<std::mutex> lock(*mu);
    Pool &p = (*pools)[{device, context}];
    *error = cudaSuccess;
    if (p.stream) return &p;
    cudaMemPoolProps props = {};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    void *small = nullptr;  // kept for device_wait
    uint64_t keep = kPoolKeep;
    *error = cudaMemPoolCreate(&pool, &props);
    if (*error == cudaSuccess)
        *error = cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep);
    if (*error == cudaSuccess) *error = cudaMalloc(&small, 256);
    if (*error == cudaSuccess) *error = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking);
    if (*error != cudaSuccess) {
        (void)cudaFree(small);
        if (pool) (void)cudaMemPoolDestroy(pool);
        (void)cudaGetLastError();
        return nullptr;
    }
    p.pool = pool;
    p.stream = stream;
    return &p;
}
Pool &pool_of(int device, uint64_t context) {
    cudaError_t e;
    Pool *p = pool_of(device, context, &e);
    DG_CUDA(e);
    return *p;
}

thread_local const AllocScope *t_scope = nullptr;

cudaError_t take(Pool &p, void **out, size_t bytes) {
    if (t_scope) return cudaMallocFromPoolAsync(out, bytes, p.pool, t_scope->stream);
    const cudaError_t e = cudaMallocFromPoolAsync(out, bytes, p.pool, p.stream);
    return e == cudaSuccess ? cudaStreamSynchronize(p.stream) : e;
}

// Frees what earlier frees could not (a capture forbade the wait); after a wait.
void free_pending(Pool &p) {
    std::vector<void *> list;
    {
        std::lock_guard<std::mutex> lock(p.mu);
        list.swap(p.pending);
    }
    for (void *ptr : list) (void)cudaFreeAsync(ptr, p.stream);
}

}  // namespace

// 256 bytes of their own: cudaFree waits for all of the device's work, and both
// calls take 2 to 4 us as long as another small block (pool_of's) keeps the
// driver's chunk of them alive.
bool device_wait() noexcept {
    void *block = nullptr;
    cudaError_t e = cudaMalloc(&block, 256);
    if (e == cudaErrorMemoryAllocation) e = cudaDeviceSynchronize();
    else if (e == cudaSuccess) e = cudaFree(block);
    (void)cudaGetLastError();
    return e == cudaSuccess;
}

AllocScope::AllocScope(cudaStream_t s) : stream(s), outer(t_scope) { t_scope = this; }
AllocScope::~AllocScope() { t_scope = static_cast<const AllocScope *>(outer); }

cudaStream_t idle_stream() {
    int device = 0;
    DG_CUDA(cudaGetDevice(&device));
    return pool_of(device, context_number()).stream;
}

void *device_alloc(size_t bytes, int *device, uint64_t *context) {
    DG_CUDA(cudaGetDevice(device));
    *context = context_number();
    Pool &p = pool_of(*device, *context);
    void *ptr = nullptr;
    cudaError_t e = take(p, &ptr, bytes);
    if (e == cudaErrorMemoryAllocation) {  // give back what the pool holds and try again
        (void)cudaGetLastError();
        if (device_wait()) free_pending(p);
        (void)cudaStreamSynchronize(p.stream);
        (void)cudaMemPoolTrimTo(p.pool, 0);
        e = take(p, &ptr, bytes);
    }
    if (e != cudaSuccess) {
        (void)cudaGetLastError();
        fail(DG_DEVICE, "device allocation of " + std::to_string(bytes) +
                            " bytes failed: " + cudaGetErrorString(e));
    }
    return ptr;
}

void device_free(void *ptr, int device, uint64_t context) noexcept {
    if (!ptr) return;
    int previous = device;
    (void)cudaGetDevice(&previous);
    if (previous != device) (void)cudaSetDevice(device);
    cudaError_t e;
    // memory of a context that was reset is gone with it
    Pool *p = context_number() == context ? pool_of(device, context, &e) : nullptr;
    if (p) {
        bool freed = false;
        if (t_scope) {
            freed = cudaFreeAsync(ptr, t_scope->stream) == cudaSuccess;
        } else if (device_wait()) {
            free_pending(*p);
            freed = cudaFreeAsync(ptr, p->stream) == cudaSuccess;
        }
        if (!freed) {  // a capture of this thread, or a global one, forbids it: later
            try {
                std::lock_guard<std::mutex> lock(p->mu);
                p->pending.push_back(ptr);
            } catch (...) {
            }
        }
    }
    if (previous != device) (void)cudaSetDevice(previous);
    (void)cudaGetLastError();
}

}  // namespace dg
