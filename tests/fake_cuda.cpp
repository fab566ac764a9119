// A CUDA runtime of host memory: the runtime calls that the library's host code makes, linked
// with its compiled units in place of the real one, so the host code's order of calls and its
// handling of failed calls can be tested without a GPU. Device memory is host memory; kernels
// do not run; every call is reported to a hook, which may fill a copy's destination and may
// fail the call with an error code.
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {

// (call, kernel, stream, pointer, bytes or value, grid) -> error code
using Hook = int (*)(const char*, const char*, uint64_t, void*, uint64_t, uint64_t);
Hook g_hook = nullptr;
cudaError_t g_last = cudaSuccess;
std::map<const void*, std::string>& kernels() {
    static std::map<const void*, std::string> names;
    return names;
}

cudaError_t emit(const char* call, const char* kernel, const void* stream, const void* pointer, uint64_t bytes,
                 uint64_t grid = 0) {
    const int e = g_hook ? g_hook(call, kernel, reinterpret_cast<uint64_t>(stream), const_cast<void*>(pointer), bytes, grid) : 0;
    if (e) g_last = cudaError_t(e);
    return cudaError_t(e);
}

const char* name_of(const void* fn) {
    auto it = kernels().find(fn);
    return it == kernels().end() ? "" : it->second.c_str();
}

struct Node {
    const void* fn;  // kernel, or null for a copy
    uint64_t grid, shared;
    void* dst;
    const void* src;
    size_t bytes;
};
struct Graph { std::vector<Node> nodes; };

cudaError_t copy(const char* call, void* dst, const void* src, size_t bytes, const void* stream) {
    std::memcpy(dst, src, bytes);
    return emit(call, "", stream, dst, bytes);
}

struct { dim3 grid, block; size_t shared; cudaStream_t stream; } g_call;

}  // namespace

extern "C" {

void fake_hook(Hook hook) {
    g_hook = hook;
    g_last = cudaSuccess;
}

// Registration of the compiled units' kernels and the launch syntax.
void** __cudaRegisterFatBinary(void*) { static void* handle = nullptr; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 0; }
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
    g_call = {grid, block, shared, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* stream) {
    *grid = g_call.grid; *block = g_call.block; *shared = g_call.shared;
    *static_cast<cudaStream_t*>(stream) = g_call.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* kernel, const void* fn) {
    *kernel = reinterpret_cast<cudaKernel_t>(const_cast<void*>(fn));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3 grid, dim3, void**, size_t shared, cudaStream_t stream) {
    return emit("launch", name_of(reinterpret_cast<const void*>(kernel)), stream, nullptr, shared, grid.x);
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 grid, dim3, void**, size_t shared, cudaStream_t stream) {
    return emit("launch", name_of(fn), stream, nullptr, shared, grid.x);
}

// Device.
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    *p = cudaDeviceProp{};
    std::strcpy(p->name, "host memory");
    p->major = 10; p->minor = 3; p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr, int) { *value = 152; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute, int value) {
    return emit("attribute", name_of(fn), nullptr, nullptr, uint64_t(value));
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* blocks, const void*, int, size_t) {
    *blocks = 2;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { const cudaError_t e = g_last; g_last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "failed by the test"; }

// Memory.
cudaError_t cudaMalloc(void** p, size_t n) { *p = std::calloc(n ? n : 1, 1); return emit("malloc", "", nullptr, *p, n); }
cudaError_t cudaFree(void* p) { const cudaError_t e = emit("free", "", nullptr, p, 0); std::free(p); return e; }
cudaError_t cudaMallocHost(void** p, size_t n) { *p = std::calloc(n ? n : 1, 1); return emit("malloc host", "", nullptr, *p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) { const cudaError_t e = emit("free host", "", nullptr, p, 0); std::free(p); return e; }
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    return copy("copy", dst, src, n, s);
}
cudaError_t cudaMemsetAsync(void* p, int value, size_t n, cudaStream_t s) {
    std::memset(p, value, n);
    return emit("memset", "", s, p, n);
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind) { return copy("copy", dst, src, n, nullptr); }
cudaError_t cudaMemset(void* p, int value, size_t n) { return cudaMemsetAsync(p, value, n, nullptr); }
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) { *p = const_cast<void*>(symbol); return cudaSuccess; }
cudaError_t cudaMemset2DAsync(void* p, size_t, int, size_t width, size_t height, cudaStream_t s) {
    return emit("memset", "", s, p, width * height);
}

// Streams, events.
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    static uint64_t next = 1;
    *s = reinterpret_cast<cudaStream_t>(next++);
    return emit("stream", "", *s, nullptr, 0);
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) { return emit("synchronize", "", s, nullptr, 0); }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return emit("stream destroy", "", s, nullptr, 0); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = reinterpret_cast<cudaEvent_t>(uint64_t(1)); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }

// Graphs: their kernels are reported when the graph is launched.
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) { *g = reinterpret_cast<cudaGraph_t>(new Graph); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete reinterpret_cast<Graph*>(g); return cudaSuccess; }
cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t* node, cudaGraph_t g, const cudaGraphNode_t*, size_t,
                                   const cudaKernelNodeParams* p) {
    reinterpret_cast<Graph*>(g)->nodes.push_back({p->func, p->gridDim.x, p->sharedMemBytes, nullptr, nullptr, 0});
    *node = reinterpret_cast<cudaGraphNode_t>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphAddMemsetNode(cudaGraphNode_t* node, cudaGraph_t g, const cudaGraphNode_t*, size_t, const cudaMemsetParams*) {
    *node = reinterpret_cast<cudaGraphNode_t>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphAddMemcpyNode1D(cudaGraphNode_t* node, cudaGraph_t g, const cudaGraphNode_t*, size_t, void* dst,
                                     const void* src, size_t n, cudaMemcpyKind) {
    reinterpret_cast<Graph*>(g)->nodes.push_back({nullptr, 0, 0, dst, src, n});
    *node = reinterpret_cast<cudaGraphNode_t>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t g, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph*>(g)));
    return emit("graph instantiate", "", nullptr, nullptr, 0);
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { delete reinterpret_cast<Graph*>(e); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t e, cudaStream_t s) {
    if (const cudaError_t failed = emit("graph launch", "", s, nullptr, 0)) return failed;
    for (const Node& n : reinterpret_cast<Graph*>(e)->nodes) {
        const cudaError_t failed = n.fn ? emit("graph kernel", name_of(n.fn), s, nullptr, n.shared, n.grid)
                                        : copy("copy", n.dst, n.src, n.bytes, s);
        if (failed) return failed;
    }
    return cudaSuccess;
}

}  // extern "C"
