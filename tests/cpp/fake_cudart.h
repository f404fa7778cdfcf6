// fake_cudart.h -- a CUDA runtime without a GPU, for tests of the library's host
// code: the test is linked with the library's object files and these definitions
// in place of libcudart.  Device memory is host memory.  Streams are queues whose
// copies and kernels run when the host waits for them, no earlier, so what a call
// leaves in flight is still there to be seen; kernels do nothing unless the test
// gives them a body; and any call can be made to fail.
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <deque>
#include <functional>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

namespace fake {

struct Op {
    std::function<void()> run;
    cudaEvent_t record = nullptr;  // event that is reached here
};
struct Stream {
    std::deque<Op> ops;
};
struct Event {
    Stream *stream = nullptr;  // where it is recorded but not reached yet
};

inline std::recursive_mutex mu;
inline int device = 0;                           // of 64
inline int host_page_tables = 1;                 // cudaDevAttrPageableMemoryAccessUsesHostPageTables
inline cudaError_t launch_error = cudaSuccess;   // cudaGetLastError after a launch
inline std::map<std::string, int> fail_after;    // name of a call -> calls that still succeed
inline std::map<std::string, int> calls;         // name of a call -> how often it was made
inline std::vector<std::string> prepared;        // kernels whose attributes were set or asked for
inline std::vector<std::string> launched;        // kernels, in launch order
// Body of a launched kernel (arguments as the launch got them; called at launch).
inline std::function<std::function<void()>(const std::string &, dim3, void **)> kernel_body;

inline std::map<const void *, std::string> &functions() { static std::map<const void *, std::string> m; return m; }
inline std::map<const void *, std::vector<uint8_t>> &variables() { static std::map<const void *, std::vector<uint8_t>> m; return m; }
inline std::vector<Stream *> &streams() { static std::vector<Stream *> v{new Stream}; return v; }

inline Stream *get(cudaStream_t s) { return s ? reinterpret_cast<Stream *>(s) : streams()[0]; }
inline Event *get(cudaEvent_t e) { return reinterpret_cast<Event *>(e); }

inline bool fails(const char *name) {
    ++calls[name];
    auto it = fail_after.find(name);
    return it != fail_after.end() && it->second-- <= 0;
}
// Run a stream up to the point where event e is reached (null: to its end).
inline void drain(Stream *s, cudaEvent_t e = nullptr) {
    while (!s->ops.empty()) {
        Op op = std::move(s->ops.front());
        s->ops.pop_front();
        if (op.run) op.run();
        if (op.record && get(op.record)->stream == s) get(op.record)->stream = nullptr;
        if (e && op.record == e) return;
    }
}
inline void reach(cudaEvent_t e) { if (get(e)->stream) drain(get(e)->stream, e); }
inline size_t in_flight() {
    size_t n = 0;
    for (Stream *s : streams()) n += s->ops.size();
    return n;
}
template <class F> cudaError_t call(const char *name, F f) {
    std::lock_guard<std::recursive_mutex> lk(mu);
    if (fails(name)) return strstr(name, "Malloc") ? cudaErrorMemoryAllocation : cudaErrorUnknown;
    f();
    return cudaSuccess;
}

}  // namespace fake

#define FAKE(...) return fake::call(__func__, [&] { __VA_ARGS__; })

extern "C" {

void **__cudaRegisterFatBinary(void *) { static void *h; return &h; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
    fake::functions()[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t size, int, int) {
    fake::variables()[host].resize(size);
}
struct FakeLaunch { dim3 grid, block; size_t smem; void *stream; };
static thread_local FakeLaunch fake_launch;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) { fake_launch = {g, b, smem, st}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *st) {
    *g = fake_launch.grid; *b = fake_launch.block; *smem = fake_launch.smem;
    *static_cast<void **>(st) = fake_launch.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *f) { *k = (cudaKernel_t)f; return cudaSuccess; }
static cudaError_t fake_launch_kernel(cudaKernel_t k, dim3 g, void **args, cudaStream_t st) {
    return fake::call("launch", [&] { const std::string &name = fake::functions()[(const void *)k];
         fake::launched.push_back(name);
         fake::get(st)->ops.push_back({fake::kernel_body ? fake::kernel_body(name, g, args) : nullptr, nullptr}); });
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void **args, size_t, cudaStream_t st) {
    return fake::launch_error = fake_launch_kernel(k, g, args, st);
}

cudaError_t cudaGetDevice(int *d) { *d = fake::device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { fake::device = d; return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { *n = 64; return cudaSuccess; }
cudaError_t cudaGetLastError(void) { return std::exchange(fake::launch_error, cudaSuccess); }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? fake::host_page_tables : 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) { *n = 3; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int) { FAKE(fake::prepared.push_back(fake::functions()[f])); }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *, const void *f) { FAKE(fake::prepared.push_back(fake::functions()[f])); }

cudaError_t cudaMalloc(void **p, size_t n) { FAKE(*p = memset(aligned_alloc(256, (n + 255) & ~(size_t)255), 0, n)); }
cudaError_t cudaFree(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { FAKE(*p = aligned_alloc(256, (n + 255) & ~(size_t)255)); }
cudaError_t cudaFreeHost(void *p) { free(p); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void **p, size_t n, cudaMemPool_t, cudaStream_t) { FAKE(*p = aligned_alloc(256, (n + 255) & ~(size_t)255)); }
cudaError_t cudaFreeAsync(void *p, cudaStream_t st) { FAKE(fake::get(st)->ops.push_back({[=] { free(p); }, nullptr})); }
cudaError_t cudaMemGetInfo(size_t *f, size_t *t) { *f = *t = (size_t)64 << 30; return cudaSuccess; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t *p, const cudaMemPoolProps *) { *p = nullptr; return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { return cudaSuccess; }
cudaError_t cudaMemPoolGetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *v) { *static_cast<uint64_t *>(v) = 0; return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaMemPoolTrimTo(cudaMemPool_t, size_t) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *) { *a = {}; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *sym) { *p = fake::variables()[sym].data(); return cudaSuccess; }
cudaError_t cudaMemcpyToSymbol(const void *, const void *, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { FAKE(memcpy(d, s, n)); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    FAKE(fake::get(st)->ops.push_back({[=] { memcpy(d, s, n); }, nullptr}));
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t st) {
    FAKE(fake::get(st)->ops.push_back({[=] { memset(d, v, n); }, nullptr}));
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    FAKE(fake::streams().push_back(new fake::Stream); *s = reinterpret_cast<cudaStream_t>(fake::streams().back()));
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { FAKE(fake::drain(fake::get(s))); }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    FAKE(if (fake::get(e)->stream) fake::get(s)->ops.push_back({[=] { fake::reach(e); }, nullptr}));
}
cudaError_t cudaDeviceSynchronize(void) { FAKE(for (fake::Stream *s : fake::streams()) fake::drain(s)); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { FAKE(*e = reinterpret_cast<cudaEvent_t>(new fake::Event)); }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t st) {
    FAKE(fake::get(e)->stream = fake::get(st); fake::get(st)->ops.push_back({nullptr, e}));
}
cudaError_t cudaEventQuery(cudaEvent_t e) { FAKE(fake::reach(e)); }
cudaError_t cudaEventSynchronize(cudaEvent_t e) { FAKE(fake::reach(e)); }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { *ms = 0.0f; return cudaSuccess; }

}  // extern "C"

#undef FAKE

#define CHECK(cond)                                                        \
    do {                                                                   \
        if (!(cond)) {                                                     \
            fprintf(stderr, "%s:%d: %s\n", __FILE__, __LINE__, #cond);     \
            exit(1);                                                       \
        }                                                                  \
    } while (0)
