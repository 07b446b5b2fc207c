// A CUDA runtime without a GPU for tests of the library's host code: device
// memory is host memory, copies happen at once, kernels are only written
// down, and a call can be told to fail.  It is linked with the library's
// object files in place of libcudart (tests/test_host_cpu.py).
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {

struct Node {
    std::string kernel;
    std::vector<int> deps;
};
struct Graph {
    std::vector<Node> nodes;
};
struct Stream {
    bool capturing = false;
    std::vector<int> deps;  // of the next captured node
    std::vector<cudaGraphNode_t> handles;
};
struct Event {
    bool captured = false;
    std::vector<int> deps;
};

std::vector<std::string> g_log;
std::string g_line;
std::map<std::string, int> g_fail;  // calls of a name until one fails
Graph* g_capture = nullptr;  // the capture in progress
std::vector<Stream*> g_captured_streams;
std::vector<Node> g_last_graph;
int g_sms = 152;
cudaError_t g_error = cudaSuccess;

// Filled while the library's objects are initialised, in whatever order.
std::map<const void*, std::string>& kernels() {
    static std::map<const void*, std::string> k;
    return k;
}

void note(const std::string& s) { g_log.push_back(s); }
std::string num(const void* p) { return std::to_string((unsigned long long)p); }

bool fails(const char* name) {
    auto it = g_fail.find(name);
    if (it == g_fail.end() || --it->second > 0) return false;
    g_fail.erase(it);
    note(std::string("failed ") + name);
    return true;
}
#define MAY_FAIL(name) \
    if (fails(name)) return g_error = cudaErrorUnknown

// One node of the capture behind the stream's dependencies.
void captured(Stream* s, const std::string& kernel) {
    g_capture->nodes.push_back({kernel, s->deps});
    s->deps = {(int)g_capture->nodes.size() - 1};
}

cudaError_t launch(const void* fn, cudaStream_t stream) {
    MAY_FAIL("launch");
    Stream* s = (Stream*)stream;
    const std::string& k = kernels()[fn];
    if (s && s->capturing) captured(s, k);
    else note("launch " + k);
    return cudaSuccess;
}

struct Call {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
std::vector<Call> g_calls;

}  // namespace

extern "C" {

// -- what the tests ask ------------------------------------------------------
void fake_clear(void) { g_log.clear(); g_fail.clear(); g_error = cudaSuccess; }
int fake_log_size(void) { return (int)g_log.size(); }
const char* fake_log(int i) { return g_log[i].c_str(); }
void fake_fail(const char* name, int nth) { g_fail[name] = nth; }  // the nth next call (once)
void fake_set_sms(int n) { g_sms = n; }
int fake_graph_size(void) { return (int)g_last_graph.size(); }
const char* fake_graph_node(int i) {  // "kernel: dep dep"
    g_line = g_last_graph[i].kernel + ":";
    for (int d : g_last_graph[i].deps) g_line += " " + std::to_string(d);
    return g_line.c_str();
}

// -- registration and launches -------------------------------------------------
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
    kernels()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    g_calls.push_back({grid, block, smem, stream});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    const Call c = g_calls.back();
    g_calls.pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *(cudaStream_t*)stream = c.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) {
    *k = (cudaKernel_t)host;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void**, size_t, cudaStream_t s) {
    return launch((const void*)k, s);
}
cudaError_t cudaLaunchCooperativeKernel(const void* fn, dim3, dim3, void**, size_t, cudaStream_t s) {
    return launch(fn, s);
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t,
                                                                   unsigned) {
    *n = 4;
    return cudaSuccess;
}

// -- device, memory ------------------------------------------------------------
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? g_sms : 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) { const cudaError_t e = g_error; g_error = cudaSuccess; return e; }
cudaError_t cudaPeekAtLastError(void) { return g_error; }
const char* cudaGetErrorString(cudaError_t) { return "an error of the fake runtime"; }
cudaError_t cudaMalloc(void** p, size_t n) {
    MAY_FAIL("cudaMalloc");
    *p = nullptr;
    return posix_memalign(p, 256, n ? n : 1) ? cudaErrorMemoryAllocation : cudaSuccess;
}
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
    note("page-locked");
    *p = malloc(n);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    note("blocking copy");
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    MAY_FAIL("cudaMemcpyAsync");
    note("copy " + num(d) + " " + num(s) + " " + std::to_string(n));
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    note("blocking set");
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorUnknown; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult*) {
    *f = nullptr;
    return cudaErrorUnknown;
}

// -- streams, events, capture --------------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    note("stream created");
    *s = (cudaStream_t) new Stream();
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete (Stream*)s; return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { note("synchronised"); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    note("event created");
    *e = (cudaEvent_t) new Event();
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete (Event*)e; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    Stream* st = (Stream*)s;
    Event* ev = (Event*)e;
    ev->captured = st && st->capturing;
    if (ev->captured) ev->deps = st->deps;
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    Stream* st = (Stream*)s;
    Event* ev = (Event*)e;
    if (!ev->captured || !g_capture) return cudaSuccess;
    if (!st->capturing) {
        st->capturing = true;
        st->deps.clear();
        g_captured_streams.push_back(st);
    }
    for (int d : ev->deps) st->deps.push_back(d);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    g_capture = new Graph();
    ((Stream*)s)->capturing = true;
    ((Stream*)s)->deps.clear();
    g_captured_streams = {(Stream*)s};
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    for (Stream* s : g_captured_streams) s->capturing = false;
    g_last_graph = g_capture->nodes;
    *g = (cudaGraph_t)g_capture;
    g_capture = nullptr;
    return cudaSuccess;
}
// Nodes are handed out as their index + 1.
cudaError_t cudaStreamGetCaptureInfo(cudaStream_t s, cudaStreamCaptureStatus* status,
                                     unsigned long long*, cudaGraph_t*, const cudaGraphNode_t** deps,
                                     const cudaGraphEdgeData** edges, size_t* n) {
    MAY_FAIL("cudaStreamGetCaptureInfo");
    Stream* st = (Stream*)s;
    *status = st->capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    st->handles.clear();
    for (int d : st->deps) st->handles.push_back((cudaGraphNode_t)(size_t)(d + 1));
    if (deps) *deps = st->handles.data();
    if (edges) *edges = nullptr;
    if (n) *n = st->handles.size();
    return cudaSuccess;
}
cudaError_t cudaStreamUpdateCaptureDependencies(cudaStream_t s, cudaGraphNode_t* deps,
                                                const cudaGraphEdgeData*, size_t n, unsigned flags) {
    MAY_FAIL("cudaStreamUpdateCaptureDependencies");
    Stream* st = (Stream*)s;
    if (flags == cudaStreamSetCaptureDependencies) st->deps.clear();
    for (size_t k = 0; k < n; ++k) st->deps.push_back((int)(size_t)deps[k] - 1);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
    *x = (cudaGraphExec_t) new Graph(*(Graph*)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) { delete (Graph*)g; return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { delete (Graph*)x; return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    MAY_FAIL("cudaGraphLaunch");
    for (const Node& n : ((Graph*)x)->nodes) note("launch " + n.kernel);
    return cudaSuccess;
}

}  // extern "C"
