// A CUDA runtime of host memory for string_vext_b200/csrc/memory.cu, and the
// scenarios that tests/test_memory.py runs on it: what the allocator does when
// a call is refused, which a test cannot bring about on a GPU without risk to
// whoever else uses the device.  Built with nvcc, linked without cudart.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace vext {   // as in string_vext_b200/csrc/internal.cuh
cudaError_t device_malloc_bytes(void **p, size_t bytes);
void device_free(void *p);
int fail(int code, const char *, ...) { return code; }
struct FreeTogether {
    FreeTogether();
    ~FreeTogether();
};
void release_build_scratch(int) {}
int copy_to_host(void *dst, const void *src, size_t bytes, bool *finite = nullptr);
}  // namespace vext
extern "C" int vext_release_memory(void);

// ---------------------------------------------------------------- the runtime

namespace {

struct Block {
    size_t bytes;
    bool pool;
    int device;
};
std::recursive_mutex lock;
std::map<void *, Block> blocks;          // allocated
std::map<void *, Block> queued;          // freed in pool-stream order, still mapped
thread_local int device = 0;
bool refuse_waits = false;               // as while another stream is being captured
bool captures_ended = false;             // a wait for the whole device ends such captures
size_t limit = ~(size_t)0;               // device memory in all
int waits = 0;
int host_allocs = 0, host_frees = 0;

size_t mapped() {
    size_t n = 0;
    for (auto &b : blocks) n += b.second.bytes;
    for (auto &b : queued) n += b.second.bytes;
    return n;
}
cudaError_t allocate(void **p, size_t bytes, bool pool) {
    std::lock_guard<std::recursive_mutex> g(lock);
    if (pool)
        for (auto it = queued.begin(); it != queued.end(); ++it)
            if (it->second.bytes == bytes && it->second.device == device) {   // reused
                *p = it->first;
                blocks[it->first] = it->second;
                queued.erase(it);
                return cudaSuccess;
            }
    if (mapped() + bytes > limit) return cudaErrorMemoryAllocation;
    *p = std::malloc(bytes < (1u << 20) ? bytes : 1u << 20);   // (never written to)
    blocks[*p] = {bytes, pool, device};
    return cudaSuccess;
}

CUresult get_current(CUcontext *c) {
    *c = reinterpret_cast<CUcontext>((uintptr_t)(16 + device));
    return CUDA_SUCCESS;
}
CUresult get_id(CUcontext c, unsigned long long *id) {
    *id = (unsigned long long)(uintptr_t)c;
    return CUDA_SUCCESS;
}

}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int *d) { return *d = device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return device = d, cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 1, cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char *name, void **f, unsigned long long,
                                    cudaDriverEntryPointQueryResult *q) {
    *q = cudaDriverEntryPointSuccess;
    *f = std::string(name) == "cuCtxGetId" ? (void *)get_id : (void *)get_current;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void **p, size_t n) { return allocate(p, n, false); }
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::recursive_mutex> g(lock);
    if (!p) return cudaSuccess;
    if (refuse_waits) return cudaErrorStreamCaptureUnsupported;
    ++waits;
    if (!blocks.count(p)) std::abort();
    blocks.erase(p);
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    if (!refuse_waits) return cudaSuccess;
    captures_ended = true;
    return cudaErrorStreamCaptureUnsupported;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) {
    return *p = reinterpret_cast<cudaMemPool_t>(8), cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *v) {
    std::lock_guard<std::recursive_mutex> g(lock);
    unsigned long long n = 0;
    for (auto &b : blocks) n += b.second.pool ? b.second.bytes : 0;
    for (auto &b : queued) n += b.second.bytes;
    return *static_cast<unsigned long long *>(v) = n, cudaSuccess;
}
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t keep) {
    std::lock_guard<std::recursive_mutex> g(lock);
    unsigned long long held = 0;
    cudaMemPoolGetAttribute(nullptr, cudaMemPoolAttrReservedMemCurrent, &held);
    while (held > keep && !queued.empty()) {
        held -= queued.begin()->second.bytes;
        queued.erase(queued.begin());
    }
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) {
    return allocate(p, n, true);
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
    std::lock_guard<std::recursive_mutex> g(lock);
    if (!blocks.count(p)) std::abort();
    queued[p] = blocks[p];
    blocks.erase(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::lock_guard<std::recursive_mutex> g(lock);
    std::memset(a, 0, sizeof *a);
    auto it = blocks.find(const_cast<void *>(p));
    if (it == blocks.end()) return a->type = cudaMemoryTypeUnregistered, cudaSuccess;
    a->type = cudaMemoryTypeDevice;
    a->device = it->second.device;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    return *s = reinterpret_cast<cudaStream_t>(24), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) {
    ++host_allocs;
    return *p = std::malloc(n), cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    ++host_frees;
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *, const void *, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memset(d, 0, n), cudaSuccess;
}
// what nvcc's registration code refers to
void **__cudaRegisterFatBinary(void *) { return nullptr; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
char __cudaInitModule(void **) { return 0; }
}

// ---------------------------------------------------------------- scenarios

using namespace vext;

#define CHECK(c)                                                 \
    do {                                                         \
        if (!(c)) {                                              \
            std::printf("line %d: %s\n", __LINE__, #c);          \
            return 1;                                            \
        }                                                        \
    } while (0)

static void *take(size_t bytes) {
    void *p = nullptr;
    return device_malloc_bytes(&p, bytes) == cudaSuccess ? p : nullptr;
}

// A block freed while the wait for its users is refused is not given out again
// before a later wait succeeds, and the wait ends nobody's capture.
static int refused_wait(size_t bytes) {
    void *a = take(bytes);
    CHECK(a);
    refuse_waits = true;
    device_free(a);
    CHECK(blocks.count(a) && !queued.count(a) && !captures_ended);
    void *b = take(bytes);
    CHECK(b && b != a);
    refuse_waits = false;
    device_free(b);
    CHECK(!blocks.count(a) && !blocks.count(b) && !captures_ended);
    // and it serves an allocation that would not fit without it
    a = take(bytes);
    refuse_waits = true;
    device_free(a);
    refuse_waits = false;
    limit = mapped() + 8192;
    b = take(bytes + 4096);
    CHECK(b && b != a && !blocks.count(a) && !captures_ended);
    limit = ~(size_t)0;
    return 0;
}

// What was freed goes back to the device on request, all of it or with an error.
static int released() {
    void *a = take((size_t)300 << 20), *b = take((size_t)300 << 20);
    const size_t others = mapped() - ((size_t)600 << 20);
    device_free(a);
    CHECK(mapped() > others + ((size_t)500 << 20));
    CHECK(vext_release_memory() == 0);
    CHECK(mapped() == others + ((size_t)300 << 20) && blocks.count(b));
    refuse_waits = true;
    device_free(b);
    CHECK(vext_release_memory() != 0 && blocks.count(b) && !captures_ended);
    refuse_waits = false;
    CHECK(vext_release_memory() == 0 && mapped() == others);
    return 0;
}

// Large copies from two devices in turn keep their staging buffers.
static int two_devices() {
    const size_t bytes = (size_t)6 << 20;
    char *to = static_cast<char *>(std::malloc(bytes));
    for (int i = 0; i < 8; ++i) {
        device = i & 1;
        std::memset(to, 1, bytes);
        CHECK(copy_to_host(to, to, bytes) == 0 && to[0] == 0 && to[bytes - 1] == 0);
    }
    CHECK(host_allocs - host_frees <= 2);
    return 0;
}

// Blocks freed together are waited for once, whichever device they are on.
static int together() {
    void *p[6];
    for (int i = 0; i < 6; ++i) {
        device = i & 1;
        CHECK(p[i] = take((size_t)(i + 1) << 20));
    }
    device = 0;
    waits = 0;
    {
        FreeTogether outer;
        {
            FreeTogether inner;
            for (int i = 0; i < 3; ++i) device_free(p[i]);
        }
        for (int i = 0; i < 3; ++i) CHECK(blocks.count(p[i]));
        for (int i = 3; i < 6; ++i) device_free(p[i]);
        CHECK(waits == 0);
    }
    for (int i = 0; i < 6; ++i) CHECK(!blocks.count(p[i]));
    CHECK(waits == 2 && device == 0);
    return 0;
}

int main(int argc, char **argv) {
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "refused_wait") return refused_wait(1 << 20);
    if (what == "refused_wait_large") return refused_wait((size_t)600 << 20);
    if (what == "released") return released();
    if (what == "two_devices") return two_devices();
    if (what == "together") return together();
    std::printf("unknown scenario\n");
    return 2;
}
