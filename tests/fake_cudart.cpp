// fake_cudart.cpp -- a CUDA runtime for tests of the library's host side on
// machines without a GPU: linked with the library's object files in place of
// the real one.  Device memory is host memory, copies and memsets are done at
// once, kernels are noted and not run.
//
// Besides, it keeps the rules of order that a caller on a stream of its own
// depends on: copies from pageable memory and memsets on the null stream may
// return before they are done, and neither they nor the work on a non-blocking
// stream wait for one another.  fake_unordered() counts the kernels and graphs
// launched on another stream with such work outstanding, and the copies and
// memsets on the null stream with such kernels or graphs outstanding.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <string>

namespace {

size_t g_room = ~(size_t)0;  // bytes of device memory
size_t g_used = 0;
std::map<void*, size_t> g_size;
cudaError_t g_error = cudaSuccess;
bool g_pending = false;      // null-stream work that nothing has waited for
bool g_busy = false;         // kernels or graphs on another stream, likewise
int g_unordered = 0;
std::map<const void*, std::string> g_name;  // mangled, by host stub
std::string g_launched;                     // names, a line each
std::set<cudaStream_t> g_capturing;
float (*g_elapsed)(int) = nullptr;  // time of that many graphs in a row
int g_graphs = 0;                   // launched since the last event
int g_between = 0;                  // between the last two events
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} g_config;

cudaError_t result(cudaError_t e) {
    if (e != cudaSuccess) g_error = e;
    return e;
}

cudaError_t issued(cudaStream_t st) {
    if (!st) g_pending = true;
    return cudaSuccess;
}

cudaError_t copied(cudaStream_t st) {
    if (!st && g_busy) ++g_unordered;
    return issued(st);
}

cudaError_t ran(cudaStream_t st) {
    if (st && g_pending) ++g_unordered;
    if (st) g_busy = true;
    return issued(st);
}

cudaError_t launched(const void* f, cudaStream_t st) {
    g_launched += g_name[f] + "\n";
    return g_capturing.count(st) ? cudaSuccess : ran(st);
}

template <class T>
cudaError_t made(T* handle) {
    *handle = reinterpret_cast<T>(std::malloc(1));
    return cudaSuccess;
}

template <class T>
cudaError_t gone(T handle) {
    std::free(reinterpret_cast<void*>(handle));
    return cudaSuccess;
}

}  // namespace

extern "C" {

void fake_reset(size_t room) {
    g_room = room;
    g_error = cudaSuccess;
    g_pending = g_busy = false;
    g_unordered = 0;
    g_launched.clear();
    g_elapsed = nullptr;
}
void fake_elapsed(float (*ms)(int)) { g_elapsed = ms; }
void fake_room(size_t room) { g_room = room; }
int fake_unordered() { return g_unordered; }
size_t fake_used() { return g_used; }
const char* fake_launched() { return g_launched.c_str(); }

void** __cudaRegisterFatBinary(void*) { return reinterpret_cast<void**>(&g_config); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
    g_name[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    g_config = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = g_config.grid;
    *block = g_config.block;
    *smem = g_config.smem;
    *static_cast<cudaStream_t*>(stream) = g_config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(f));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t st) {
    return launched(k, st);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return launched(f, c->stream);
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
    *p = nullptr;
    if (bytes > g_room || g_used > g_room - bytes) return result(cudaErrorMemoryAllocation);
    *p = std::calloc(bytes ? bytes : 1, 1);  // pages that nothing touches take no room
    if (!*p) return result(cudaErrorMemoryAllocation);
    g_used += bytes;
    g_size[*p] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    g_used -= g_size[p];
    g_size.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t bytes, cudaStream_t) { return cudaMalloc(p, bytes); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return cudaFree(p); }

cudaError_t cudaMemcpy(void* to, const void* from, size_t bytes, cudaMemcpyKind kind) {
    std::memmove(to, from, bytes);
    copied(nullptr);
    if (kind == cudaMemcpyDeviceToHost) g_pending = false;  // returns when it is done
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind, cudaStream_t st) {
    std::memmove(to, from, bytes);
    return copied(st);
}
cudaError_t cudaMemset(void* p, int v, size_t bytes) {
    std::memset(p, v, bytes);
    return copied(nullptr);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t bytes, cudaStream_t st) {
    std::memset(p, v, bytes);
    return copied(st);
}
cudaError_t cudaDeviceSynchronize() { g_pending = g_busy = false; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) {
    (st ? g_busy : g_pending) = false;
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return made(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return gone(s); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    g_capturing.insert(s);
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* status) {
    *status = g_capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    g_capturing.erase(s);
    return made(g);
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { return made(e); }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return gone(g); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return gone(e); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) {
    ++g_graphs;
    return g_capturing.count(st) ? cudaSuccess : ran(st);
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return made(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return made(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return gone(e); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) {
    g_between = g_graphs;
    g_graphs = 0;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = g_elapsed ? g_elapsed(g_between) : 1.0f;
    return cudaSuccess;
}

cudaError_t cudaGetLastError() {
    const cudaError_t e = g_error;
    g_error = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = &g_config; return cudaSuccess; }

}  // extern "C"
