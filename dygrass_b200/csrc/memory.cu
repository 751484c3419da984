// memory.cu -- device memory of the graph handles.
//
// A handle owns some forty arrays that grow with the calls made on it, and a
// cudaMalloc or cudaFree of a megabyte takes 0.3 to 0.7 ms (each maps or
// unmaps pages and waits for the device): building two 110,592-vertex graphs,
// one insertion and one deletion stream and closing them spent 12 of 27 ms
// there.  Memory comes from one CUDA memory pool per device instead, which
// keeps up to kPoolKeep bytes that no handle uses and gives what is above
// back to the device at the next synchronize.  The pool is the driver's:
// calls from any thread are safe.  Blocks are allocated and freed on a stream
// of the pool's own; an allocation is complete when dev_alloc returns, and a
// block is freed only when the device has finished with it, so blocks move
// freely between handles, streams and threads.  Pinned host blocks (a handle's
// scalar mirror and its packed arrays, in powers of two) are kept the same
// way, at most 8 MB of them.
#include <cuda.h>

#include <mutex>
#include <vector>

#include "dyg_internal.cuh"
#include "pinned_cache.h"

namespace dyg {

namespace {

constexpr unsigned long long kPoolKeep = 256ull << 20;
// Kept scratch of a device: all that one call may borrow while the device has
// handles (the row index is up to 2.3 GB, and allocating and freeing 0.3 GB in
// each call took 5 to 15 ms of a weighted file on an R-MAT graph of scale 18,
// of which the rest took 1), a little of it when the last is closed.
constexpr unsigned long long kScratchKeep = 3ull << 30;
constexpr unsigned long long kScratchIdle = 256ull << 20;
constexpr int kMaxDevices = 64;

struct DevicePool {
    cudaMemPool_t pool = nullptr;   // null: the device has no pools
    cudaStream_t st = nullptr;
    bool tried = false;
    unsigned long long ctx = 0;
};
std::mutex g_pool_mu;
DevicePool g_pools[kMaxDevices];

// The pool of the current device, made on first use and again when the
// device's context was replaced (cudaDeviceReset takes the pool with it).
DevicePool current_pool() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return DevicePool{};
    std::lock_guard<std::mutex> lk(g_pool_mu);
    DevicePool &p = g_pools[dev];
    const unsigned long long ctx = current_context_id();
    if (p.tried && ctx == p.ctx) return p;
    p = DevicePool{};
    p.tried = true;
    p.ctx = ctx;
    cudaMemPoolProps props{};
    props.allocType = cudaMemAllocationTypePinned;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = dev;
    unsigned long long keep = kPoolKeep;
    if (cudaMemPoolCreate(&p.pool, &props) != cudaSuccess) p.pool = nullptr;
    if (p.pool && (cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
                   cudaStreamCreateWithFlags(&p.st, cudaStreamNonBlocking) != cudaSuccess)) {
        cudaMemPoolDestroy(p.pool);
        p.pool = nullptr;
    }
    cudaGetLastError();
    // the context may have been created by the calls above
    p.ctx = current_context_id();
    return p;
}

}  // namespace

unsigned long long current_context_id() {
    typedef CUresult (*GetCurrent)(CUcontext *);
    typedef CUresult (*GetId)(CUcontext, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *f = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_current = reinterpret_cast<GetCurrent>(f);
        f = nullptr;
        if (cudaGetDriverEntryPoint("cuCtxGetId", &f, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            get_id = reinterpret_cast<GetId>(f);
        cudaGetLastError();
    });
    if (!get_current || !get_id) return 0ull;
    CUcontext c = nullptr;
    unsigned long long id = 0ull;
    if (get_current(&c) != CUDA_SUCCESS || !c || get_id(c, &id) != CUDA_SUCCESS) return 0ull;
    return id;
}

namespace {
// Allocations of this thread that are still to succeed, and to fail after
// them (dyg_testing_fail_allocations).
thread_local uint32_t t_pass = 0, t_fail = 0;

cudaError_t alloc_once(const DevicePool &p, void **out, size_t bytes) {
    *out = nullptr;
    if (t_fail) {
        if (t_pass == 0) {
            --t_fail;
            return cudaErrorMemoryAllocation;
        }
        --t_pass;
    }
    if (!p.pool) return cudaMalloc(out, bytes);
    cudaError_t e = cudaMallocFromPoolAsync(out, bytes, p.pool, p.st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(p.st);   // usable on any stream from here on
    if (e != cudaSuccess) *out = nullptr;
    return e;
}
}  // namespace

void fail_allocations(uint32_t pass, uint32_t fail) {
    scratch_drop();   // what is kept would be handed out without an allocation
    t_pass = pass;
    t_fail = fail;
}

cudaError_t dev_alloc(void **out, size_t bytes) {
    const DevicePool p = current_pool();
    cudaError_t e = alloc_once(p, out, bytes);
    if (e == cudaErrorMemoryAllocation) {
        // the kept scratch and what the pool holds in other sizes go back first
        cudaGetLastError();
        scratch_drop();
        if (p.pool) {
            cudaStreamSynchronize(p.st);
            cudaMemPoolTrimTo(p.pool, 0);
        }
        e = alloc_once(p, out, bytes);
    }
    return e;
}

void dev_free(void *ptr) {
    if (!ptr) return;
    const DevicePool p = current_pool();
    if (!p.pool || cudaFreeAsync(ptr, p.st) != cudaSuccess) {
        cudaGetLastError();
        cudaFree(ptr);
    }
    cudaGetLastError();
}

namespace {
// Scratch blocks of each device, kept between the calls that borrow them.
struct Scratch {
    std::vector<Buf> blocks;
    size_t total = 0;
    unsigned long long ctx = 0;
    int handles = 0;
};
std::mutex g_scratch_mu;
Scratch g_scratch[kMaxDevices];

// The current device's, as of its present context (g_scratch_mu held).
Scratch *current_scratch() {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kMaxDevices) return nullptr;
    const unsigned long long ctx = current_context_id();
    if (!ctx) return nullptr;
    Scratch &s = g_scratch[dev];
    if (s.ctx != ctx) {   // the blocks went with their context
        s.blocks.clear();
        s.total = 0;
        s.ctx = ctx;
    }
    return &s;
}

Buf take_scratch(Scratch &s, size_t i) {
    const Buf b = s.blocks[i];
    s.total -= b.bytes;
    s.blocks[i] = s.blocks.back();
    s.blocks.pop_back();
    return b;
}
// Frees the smallest kept blocks (any borrower can use the larger) until at
// most `keep` bytes are left.
void shrink_scratch(size_t keep) {
    std::vector<Buf> drop;
    {
        std::lock_guard<std::mutex> lk(g_scratch_mu);
        Scratch *s = current_scratch();
        while (s && s->total > keep) {
            size_t k = 0;
            for (size_t i = 1; i < s->blocks.size(); ++i)
                if (s->blocks[i].bytes < s->blocks[k].bytes) k = i;
            drop.push_back(take_scratch(*s, k));
        }
    }
    for (Buf &b : drop) dev_free(b.p);
}
}  // namespace

void scratch_handles(int dev, int change) {
    int left = 1;
    if (dev >= 0 && dev < kMaxDevices) {
        std::lock_guard<std::mutex> lk(g_scratch_mu);
        left = g_scratch[dev].handles += change;
    }
    if (left == 0) shrink_scratch(kScratchIdle);
}

void scratch_drop() { shrink_scratch(0); }

cudaError_t scratch_borrow(Buf *b, size_t bytes) {
    *b = Buf{};
    {
        std::lock_guard<std::mutex> lk(g_scratch_mu);
        Scratch *s = current_scratch();
        size_t best = s ? s->blocks.size() : 0;   // the smallest that is large enough
        for (size_t i = 0; s && i < s->blocks.size(); ++i)
            if (s->blocks[i].bytes >= bytes && (best == s->blocks.size() || s->blocks[i].bytes < s->blocks[best].bytes))
                best = i;
        if (s && best < s->blocks.size()) {
            *b = take_scratch(*s, best);
            return cudaSuccess;
        }
    }
    const size_t want = (bytes + bytes / 8 + 0xFFFF) & ~(size_t)0xFFFF;
    const DevicePool p = current_pool();
    cudaError_t e = alloc_once(p, &b->p, want);
    if (e == cudaErrorMemoryAllocation) {
        // the kept blocks, all too small, go first; the pool stays as it is:
        // the caller can do without
        cudaGetLastError();
        scratch_drop();
        e = alloc_once(p, &b->p, want);
    }
    b->bytes = e == cudaSuccess ? want : 0;
    return e;
}

void scratch_return(Buf *b) {
    if (!b->p) return;
    bool kept = false;
    size_t keep = 0;
    {
        std::lock_guard<std::mutex> lk(g_scratch_mu);
        Scratch *s = current_scratch();
        if (s) {
            keep = s->handles > 0 ? kScratchKeep : kScratchIdle;
            if (b->bytes <= keep) {
                s->blocks.push_back(*b);
                s->total += b->bytes;
                kept = true;
                if (s->total <= keep) keep = 0;
            }
        }
    }
    if (!kept) dev_free(b->p);
    else if (keep) shrink_scratch(keep);
    *b = Buf{};
}

namespace {
constexpr size_t kPinnedKeep = 8u << 20;
std::mutex g_pinned_mu;
PinnedCache g_pinned(kPinnedKeep);

// The current device, if its context can be told from one that replaced it.
bool current_place(int *dev, unsigned long long *ctx) {
    *ctx = current_context_id();
    return *ctx && cudaGetDevice(dev) == cudaSuccess;
}
}  // namespace

cudaError_t host_alloc(void **out, size_t bytes) {
    int dev = 0;
    unsigned long long ctx = 0;
    *out = nullptr;
    if (current_place(&dev, &ctx)) {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        *out = g_pinned.take(dev, ctx, bytes);
    }
    return *out ? cudaSuccess : cudaMallocHost(out, bytes);
}

void host_free(void *p, size_t bytes) {
    int dev = 0;
    unsigned long long ctx = 0;
    if (!p) return;
    if (current_place(&dev, &ctx)) {
        std::lock_guard<std::mutex> lk(g_pinned_mu);
        if (g_pinned.keep(dev, ctx, p, bytes)) return;
    }
    cudaFreeHost(p);
}

}  // namespace dyg
