// Device memory and copies to pageable host memory.
//
// A call such as calculate_vext makes a system, runs one field and drops the
// system again: about twenty cudaMalloc and cudaFree, 4 ms of its 5.5 ms for
// a small framework.  Device memory therefore comes from a stream-ordered pool
// per device, used on a stream of its own that every allocation waits for, so
// the memory may be used on any stream and by any thread.  What is freed beyond
// kPoolKeep bytes goes back to the device at once (not by the pool's own
// threshold, which every synchronisation of the process would look at), all of
// it when an allocation fails; the pool belongs to the context it was made in.
// A freed block goes to the pool only after a wait for its users has succeeded:
// one that is refused (a stream is being captured) leaves it for the next free.
//
// Large results go to pageable memory through page-locked buffers: a few
// threads each copy their chunks from the device and on to the destination
// (whose first touch, page by page, is most of the cost), with the next chunk
// in flight meanwhile.  cudaMemcpy alone took 13 ms for a 55 MB field.
#include <cuda.h>

#include <algorithm>
#include <atomic>
#include <cstring>
#include <set>
#include <thread>
#include <utility>
#include <vector>

#include "internal.cuh"

namespace vext {

constexpr size_t kPoolKeep = 1536ull << 20;   // a 60^3 x 64 field's lists and buffers: 1.0 GB
// Larger arrays than this would hardly stay in the pool, and it maps memory
// more slowly than cudaMalloc does: the 27 GB of pose lists of 24 systems took
// 0.4-0.8 s from it, 0.2 s by cudaMalloc.
constexpr size_t kPoolLargest = 512ull << 20;

unsigned long long current_context_id() {
    using GetCurrentFn = CUresult (*)(CUcontext *);
    using GetIdFn = CUresult (*)(CUcontext, unsigned long long *);
    static const std::pair<GetCurrentFn, GetIdFn> fns = [] {
        void *a = nullptr, *b = nullptr;
        cudaDriverEntryPointQueryResult qa = cudaDriverEntryPointSymbolNotFound, qb = qa;
        const bool ok =
            cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault, &qa) ==
                cudaSuccess &&
            qa == cudaDriverEntryPointSuccess &&
            cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault, &qb) == cudaSuccess &&
            qb == cudaDriverEntryPointSuccess;
        if (!ok) {
            cudaGetLastError();
            return std::pair<GetCurrentFn, GetIdFn>(nullptr, nullptr);
        }
        return std::pair<GetCurrentFn, GetIdFn>(reinterpret_cast<GetCurrentFn>(a),
                                                reinterpret_cast<GetIdFn>(b));
    }();
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (!fns.first || fns.first(&ctx) != CUDA_SUCCESS || !ctx ||
        fns.second(ctx, &id) != CUDA_SUCCESS)
        return 0;
    return id;
}

namespace {

struct DevicePool {
    std::mutex lock;
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    unsigned long long ctx_id = 0;
    bool plain = false;   // no pool on this device: cudaMalloc and cudaFree
    std::set<void *> direct;   // allocations beyond kPoolLargest, by cudaMalloc
    std::vector<void *> freed; // blocks that something may still use
    void *mark = nullptr;      // device_idle's block
    void *anchor = nullptr;    // and its neighbour
};

DevicePool &device_pool(int device) {
    static DevicePool pools[64];
    return pools[device & 63];
}

// The pool of the current device, made (or made anew after a device reset) on
// first use; the caller holds its lock.
void open_pool(DevicePool &p, int device) {
    cudaFree(nullptr);   // a context, when the thread has none yet
    const unsigned long long ctx = current_context_id();
    if (p.pool && ctx != 0 && ctx != p.ctx_id) {
        p.pool = nullptr;   // went with its context
        p.stream = nullptr;
        p.direct.clear();
        p.freed.clear();
        p.mark = nullptr;
    }
    if (p.pool || p.plain) return;
    int supported = 0;
    cudaMemPoolProps props;
    std::memset(&props, 0, sizeof props);
    props.allocType = cudaMemAllocationTypePinned;
    props.handleTypes = cudaMemHandleTypeNone;
    props.location.type = cudaMemLocationTypeDevice;
    props.location.id = device;
    unsigned long long keep = ~0ull;   // device_free trims
    if (ctx == 0 ||
        cudaDeviceGetAttribute(&supported, cudaDevAttrMemoryPoolsSupported, device) !=
            cudaSuccess ||
        !supported || cudaMemPoolCreate(&p.pool, &props) != cudaSuccess ||
        cudaMemPoolSetAttribute(p.pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess ||
        cudaStreamCreateWithFlags(&p.stream, cudaStreamNonBlocking) != cudaSuccess) {
        cudaGetLastError();
        if (p.pool) cudaMemPoolDestroy(p.pool);
        p.pool = nullptr;
        p.stream = nullptr;
        p.plain = true;
    }
    if (cudaMalloc(&p.anchor, 256) != cudaSuccess) {
        cudaGetLastError();
        p.anchor = nullptr;
    }
    p.ctx_id = ctx;
}

// Wait for all work queued on the device; false when that is refused.  By
// freeing a small block, as cudaFree waits for every stream, and a thread-local
// capture of another thread goes on meanwhile; cudaDeviceSynchronize would be
// refused during such a capture, and ends it.  The block lies in a 2 MB page
// that `anchor` keeps mapped: cudaMalloc and cudaFree take 1.1 and 2.5 us then,
// 720 and 610 us on average where the page comes and goes
// (cudaDeviceSynchronize: 1.5 us).
bool device_idle(DevicePool &p) {
    cudaError_t e = cudaSuccess;
    if (!p.mark) e = cudaMalloc(&p.mark, 256);
    if (e == cudaErrorMemoryAllocation && p.pool) {
        cudaGetLastError();
        cudaMemPoolTrimTo(p.pool, 0);   // (blocks given back before)
        e = cudaMalloc(&p.mark, 256);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        p.mark = nullptr;
        return false;
    }
    if (cudaFree(p.mark) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    p.mark = nullptr;
    return true;
}

// Give back the freed blocks, once nothing uses them any more.
void settle(DevicePool &p) {
    if (p.freed.empty() || !device_idle(p)) return;
    std::vector<void *> left;
    for (void *ptr : p.freed) {
        const bool pooled = !p.plain && p.pool && !p.direct.count(ptr);
        if ((pooled ? cudaFreeAsync(ptr, p.stream) : cudaFree(ptr)) != cudaSuccess) {
            cudaGetLastError();
            left.push_back(ptr);
        } else if (!pooled) {
            p.direct.erase(ptr);
        }
    }
    p.freed.swap(left);
}

// settle, and no more than kPoolKeep bytes stay in the pool.
void give_back(DevicePool &p) {
    settle(p);
    unsigned long long held = 0;
    if (p.pool &&
        cudaMemPoolGetAttribute(p.pool, cudaMemPoolAttrReservedMemCurrent, &held) == cudaSuccess &&
        held > kPoolKeep) {
        cudaStreamSynchronize(p.stream);
        cudaMemPoolTrimTo(p.pool, kPoolKeep);
    }
}

thread_local int frees_together = 0;
thread_local unsigned long long frees_devices = 0;   // with blocks to give back

}  // namespace

FreeTogether::FreeTogether() { ++frees_together; }

FreeTogether::~FreeTogether() {
    if (--frees_together > 0) return;
    int current = 0;
    if (cudaGetDevice(&current) != cudaSuccess) {
        cudaGetLastError();
        return;
    }
    for (int d = 0; frees_devices; ++d, frees_devices >>= 1) {
        if (!(frees_devices & 1)) continue;
        if (d != current) cudaSetDevice(d);
        DevicePool &p = device_pool(d);
        std::lock_guard<std::mutex> guard(p.lock);
        give_back(p);
        if (d != current) cudaSetDevice(current);
    }
}

cudaError_t device_malloc_bytes(void **out, size_t bytes) {
    *out = nullptr;
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    DevicePool &p = device_pool(device);
    std::lock_guard<std::mutex> guard(p.lock);
    open_pool(p, device);
    if (p.plain) return cudaMalloc(out, bytes);
    if (bytes > kPoolLargest) {
        e = cudaMalloc(out, bytes);
        if (e == cudaErrorMemoryAllocation) {
            cudaGetLastError();
            settle(p);
            cudaStreamSynchronize(p.stream);
            cudaMemPoolTrimTo(p.pool, 0);
            e = cudaMalloc(out, bytes);
        }
        if (e == cudaSuccess) {
            p.direct.insert(*out);
        } else {
            cudaGetLastError();
            *out = nullptr;
        }
        return e;
    }
    e = cudaMallocFromPoolAsync(out, bytes, p.pool, p.stream);
    if (e == cudaErrorMemoryAllocation) {
        cudaGetLastError();
        settle(p);
        cudaStreamSynchronize(p.stream);
        cudaMemPoolTrimTo(p.pool, 0);
        e = cudaMallocFromPoolAsync(out, bytes, p.pool, p.stream);
    }
    if (e != cudaSuccess) {
        cudaGetLastError();
        *out = nullptr;
        return e;
    }
    return cudaStreamSynchronize(p.stream);   // from here on for every stream
}

void device_free(void *ptr) {
    if (!ptr) return;
    cudaPointerAttributes at;
    int current = 0;
    if (cudaGetDevice(&current) != cudaSuccess ||
        cudaPointerGetAttributes(&at, ptr) != cudaSuccess || at.type != cudaMemoryTypeDevice) {
        cudaGetLastError();   // allocated in a context that has gone
        return;
    }
    if (at.device != current) cudaSetDevice(at.device);
    DevicePool &p = device_pool(at.device);
    {
        std::lock_guard<std::mutex> guard(p.lock);
        p.freed.push_back(ptr);
        if (frees_together > 0) frees_devices |= 1ull << (at.device & 63);
        else give_back(p);
    }
    if (at.device != current) cudaSetDevice(current);
}

// ---------------------------------------------------------------- host copies

namespace {

constexpr int kCopyThreads = 8;
constexpr size_t kCopyChunk = 1u << 20;          // page-locked buffer: two per thread
constexpr size_t kCopyDirect = 4u << 20;         // smaller copies: one cudaMemcpy

struct CopyLanes {
    std::mutex lock;
    char *pinned = nullptr;                      // [kCopyThreads][2][kCopyChunk]
    cudaStream_t stream[kCopyThreads] = {};
    int device = 0;
    unsigned long long ctx_id = 0;
};

CopyLanes &copy_lanes(int device) {
    static CopyLanes lanes[64];
    return lanes[device & 63];
}

bool all_finite(const char *bytes, size_t n) {
    const uint32_t *w = reinterpret_cast<const uint32_t *>(bytes);
    uint32_t bad = 0;
    for (size_t i = 0; i < n / 4; ++i) bad |= (w[i] & 0x7f800000u) == 0x7f800000u;
    return bad == 0;
}

// Buffers and streams for `device`, the current one; false when there are none.
bool open_lanes(CopyLanes &l, int device) {
    const unsigned long long ctx = current_context_id();
    if (l.pinned && ctx == l.ctx_id && device == l.device) return true;
    l.pinned = nullptr;   // (went with its context)
    void *p = nullptr;
    if (cudaHostAlloc(&p, 2 * kCopyThreads * kCopyChunk, cudaHostAllocDefault) != cudaSuccess) {
        cudaGetLastError();
        return false;
    }
    for (int t = 0; t < kCopyThreads; ++t)
        if (cudaStreamCreateWithFlags(&l.stream[t], cudaStreamNonBlocking) != cudaSuccess) {
            cudaGetLastError();
            while (t > 0) cudaStreamDestroy(l.stream[--t]);
            cudaFreeHost(p);
            return false;
        }
    l.pinned = static_cast<char *>(p);
    l.device = device;
    l.ctx_id = ctx;
    return true;
}

// Thread t's chunks t, t + threads, ...: the next one in flight while this one
// moves on to the destination.
cudaError_t copy_lane(CopyLanes &l, int t, int threads, char *dst, const char *src, size_t bytes,
                      std::atomic<bool> *finite) {
    cudaError_t e = cudaSetDevice(l.device);
    if (e != cudaSuccess) return e;
    char *buf[2] = {l.pinned + 2 * t * kCopyChunk, l.pinned + (2 * t + 1) * kCopyChunk};
    const size_t chunks = (bytes + kCopyChunk - 1) / kCopyChunk;
    auto size_of = [&](size_t c) { return std::min(kCopyChunk, bytes - c * kCopyChunk); };
    auto fetch = [&](size_t c, int b) {
        return cudaMemcpyAsync(buf[b], src + c * kCopyChunk, size_of(c), cudaMemcpyDeviceToHost,
                               l.stream[t]);
    };
    int b = 0;
    if ((size_t)t < chunks) e = fetch(t, 0);
    for (size_t c = t; c < chunks && e == cudaSuccess; c += threads, b ^= 1) {
        e = cudaStreamSynchronize(l.stream[t]);
        if (e != cudaSuccess) break;
        if (c + threads < chunks) e = fetch(c + threads, b ^ 1);
        if (finite && !all_finite(buf[b], size_of(c))) *finite = false;
        std::memcpy(dst + c * kCopyChunk, buf[b], size_of(c));
    }
    const cudaError_t last = cudaStreamSynchronize(l.stream[t]);
    return e != cudaSuccess ? e : last;
}

}  // namespace

int copy_to_host(void *dst, const void *src, size_t bytes, bool *finite) {
    if (bytes == 0) return 0;
    cudaPointerAttributes at;
    bool pageable = true;
    if (cudaPointerGetAttributes(&at, dst) == cudaSuccess)
        pageable = at.type == cudaMemoryTypeUnregistered;
    else
        cudaGetLastError();
    int device = 0;
    VEXT_CUDA(cudaGetDevice(&device));
    CopyLanes &l = copy_lanes(device);
    std::unique_lock<std::mutex> guard(l.lock, std::defer_lock);
    if (pageable && bytes >= kCopyDirect) guard.lock();
    if (!guard.owns_lock() || !open_lanes(l, device)) {
        VEXT_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyDeviceToHost));
        if (finite && !all_finite(static_cast<const char *>(dst), bytes)) *finite = false;
        return 0;
    }
    const int threads = (int)std::min<size_t>(
        kCopyThreads, std::max(1u, std::thread::hardware_concurrency() / 2));
    std::atomic<bool> fine{true};
    cudaError_t errors[kCopyThreads] = {};
    std::thread pool[kCopyThreads];
    char *to = static_cast<char *>(dst);
    const char *from = static_cast<const char *>(src);
    auto lane = [&](int t) {
        errors[t] = copy_lane(l, t, threads, to, from, bytes, finite ? &fine : nullptr);
    };
    int started = 1;
    try {
        for (; started < threads; ++started) pool[started] = std::thread(lane, started);
    } catch (...) {   // no more threads: their shares follow below
    }
    lane(0);
    for (int t = 1; t < started; ++t) pool[t].join();
    for (int t = started; t < threads; ++t) lane(t);
    for (int t = 0; t < threads; ++t) VEXT_CUDA(errors[t]);
    if (finite && !fine) *finite = false;
    return 0;
}

}  // namespace vext

using namespace vext;

extern "C" int vext_release_memory(void) {
    int device = 0;
    VEXT_CUDA(cudaGetDevice(&device));
    release_build_scratch(device);
    DevicePool &p = device_pool(device);
    std::lock_guard<std::mutex> guard(p.lock);
    open_pool(p, device);
    settle(p);
    if (p.pool) {
        VEXT_CUDA(cudaStreamSynchronize(p.stream));
        VEXT_CUDA(cudaMemPoolTrimTo(p.pool, 0));
    }
    if (!p.freed.empty())
        return fail(VEXT_ERR_CUDA, "%zu blocks may still be in use (a stream capture?)",
                    p.freed.size());
    return 0;
}
