// A CUDA runtime without a device, preloaded under libso_tracer.so (tests/test_host_pools.py) so that the host code
// of frames and batches runs on the CPU: kernels do nothing, device memory is lazily mapped host memory out
// of a budget, events are always complete.  The fake_* functions set the budget, make an allocation fail,
// give the record pools' counters, and read what the library did.
#include <sys/mman.h>

#include <cstddef>
#include <cstdint>
#include <cstring>
#include <map>

namespace {
enum { Ok = 0, ErrMemory = 2, ErrHandle = 400 };
std::map<void*, size_t> blocks;
size_t total = size_t(64) << 30, held = 0;
long long fail_in = -1;  // allocations until the one that fails
unsigned long long pool_counts[3];  // what a pool's three counters read back as
size_t counts_given = 0;            // (device to host copies of this size)
int last_error = Ok;
long long n_malloc = 0, n_graphs = 0, n_launch = 0;
uintptr_t serial = 0x1000;

int note(int e) {
    if (e != Ok) last_error = e;
    return e;
}
int take(void** p, size_t n) {
    ++n_malloc;
    *p = nullptr;
    if (fail_in >= 0 && fail_in-- == 0) return note(ErrMemory);
    if (n > total - held) return note(ErrMemory);
    void* m = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED) return note(ErrMemory);
    blocks[m] = n;
    held += n;
    *p = m;
    return Ok;
}
int give(void* p) {
    auto it = blocks.find(p);
    if (it != blocks.end()) {
        munmap(p, it->second);
        held -= it->second;
        blocks.erase(it);
    }
    return Ok;
}
int handle(void** p) {
    *p = reinterpret_cast<void*>(serial += 16);
    return Ok;
}
int copy(void* d, const void* s, size_t n, int kind) {
    if (kind == 2 && n == counts_given) std::memcpy(d, pool_counts, n);
    else std::memcpy(d, s, n);
    return Ok;
}
}  // namespace

extern "C" {
void fake_memory(size_t bytes) { total = bytes; }
size_t fake_held() { return held; }
void fake_fail_in(long long n) { fail_in = n; }
void fake_counts(size_t bytes, unsigned long long segments, unsigned long long short_samples, unsigned long long records) {
    counts_given = bytes;  // 24: the pools of the FP64 passes, 16: that of the FP32 rays
    pool_counts[0] = segments;
    pool_counts[1] = short_samples;
    pool_counts[2] = records;
}
long long fake_mallocs() { return n_malloc; }
long long fake_graphs() { return n_graphs; }
long long fake_launches() { return n_launch; }
size_t fake_largest() {
    size_t v = 0;
    for (auto& b : blocks) v = b.second > v ? b.second : v;
    return v;
}

void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(...) {}
void __cudaRegisterVar(...) {}
unsigned __cudaPushCallConfiguration(...) { return 0; }
int __cudaPopCallConfiguration(...) { return Ok; }
int cudaLaunchKernel(...) {
    ++n_launch;
    return Ok;
}
int cudaFuncSetAttribute(...) { return Ok; }
int cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 4;
    return Ok;
}
int cudaGetDeviceCount(int* n) {
    *n = 1;
    return Ok;
}
int cudaGetDevice(int* n) {
    *n = 0;
    return Ok;
}
int cudaSetDevice(int) { return Ok; }
int cudaDeviceGetAttribute(int* v, int, int) {
    *v = 148;
    return Ok;
}
int cudaDeviceSynchronize() { return Ok; }
int cudaGetLastError() {
    const int e = last_error;
    last_error = Ok;
    return e;
}
const char* cudaGetErrorString(int e) { return e == ErrMemory ? "out of memory" : "no error"; }

int cudaMalloc(void** p, size_t n) { return take(p, n); }
int cudaMallocHost(void** p, size_t n) { return take(p, n); }
int cudaFree(void* p) { return give(p); }
int cudaFreeHost(void* p) { return give(p); }
int cudaMemGetInfo(size_t* f, size_t* t) {
    *f = total - held;
    *t = total;
    return Ok;
}
int cudaMemcpy(void* d, const void* s, size_t n, int kind) { return copy(d, s, n, kind); }
int cudaMemcpyAsync(void* d, const void* s, size_t n, int kind, void*) { return copy(d, s, n, kind); }
int cudaMemset(void* d, int v, size_t n) {
    std::memset(d, v, n);
    return Ok;
}
int cudaMemsetAsync(void* d, int v, size_t n, void*) { return cudaMemset(d, v, n); }
int cudaMemcpy2DToArray(...) { return Ok; }
int cudaGetSymbolAddress(void** p, const void*) { return handle(p); }

int cudaMalloc3DArray(void** a, ...) { return handle(a); }
int cudaMallocMipmappedArray(void** a, ...) { return handle(a); }
int cudaGetMipmappedArrayLevel(void** a, ...) { return handle(a); }
int cudaFreeArray(void*) { return Ok; }
int cudaFreeMipmappedArray(void*) { return Ok; }
struct FakeChannel {
    int x, y, z, w, f;
};
FakeChannel cudaCreateChannelDesc(int x, int y, int z, int w, int f) { return {x, y, z, w, f}; }
int cudaCreateTextureObject(unsigned long long* o, ...) {
    *o = 1;
    return Ok;
}
int cudaCreateSurfaceObject(unsigned long long* o, ...) {
    *o = 1;
    return Ok;
}
int cudaDestroyTextureObject(unsigned long long) { return Ok; }
int cudaDestroySurfaceObject(unsigned long long) { return Ok; }

int cudaStreamCreate(void** s) { return handle(s); }
int cudaStreamCreateWithFlags(void** s, unsigned) { return handle(s); }
int cudaStreamDestroy(void*) { return Ok; }
int cudaStreamSynchronize(void*) { return Ok; }
int cudaStreamWaitEvent(void* s, void* e, unsigned) { return note(s && e ? Ok : ErrHandle); }
int cudaEventCreate(void** e) { return handle(e); }
int cudaEventCreateWithFlags(void** e, unsigned) { return handle(e); }
int cudaEventDestroy(void*) { return Ok; }
int cudaEventQuery(void*) { return Ok; }
int cudaEventRecord(void* e, void*) { return note(e ? Ok : ErrHandle); }
int cudaEventSynchronize(void*) { return Ok; }
int cudaEventElapsedTime(float* ms, void*, void*) {
    *ms = 0.f;
    return Ok;
}
int cudaStreamBeginCapture(void*, int) { return Ok; }
int cudaStreamEndCapture(void*, void** g) { return handle(g); }
int cudaGraphInstantiate(void** e, void*, unsigned long long) {
    ++n_graphs;
    return handle(e);
}
int cudaGraphLaunch(void*, void*) { return Ok; }
int cudaGraphDestroy(void*) { return Ok; }
int cudaGraphExecDestroy(void*) { return Ok; }
}
