#include "fake_cudart.h"

#include <cstdlib>
#include <cstring>
#include <memory>
#include <set>

namespace fake {

std::vector<Op> ops;
std::vector<std::string> faults;
std::function<void(Op&)> on_kernel;
std::function<void(void*, size_t)> on_d2h;
std::function<cudaError_t(const std::string&)> launch_error;
std::function<float()> elapsed;
std::vector<std::vector<Node>> graphs;
long long allocations = 0, fail_from = 1, fail_to = 0;
size_t free_bytes = (size_t)64 << 30;

namespace {
struct Stream {
    Clock clock;
    bool capturing = false;
};
struct Event {
    Clock clock;
    bool capturing = false;
};
std::map<const char*, size_t> device;  // live allocations
std::map<const void*, std::string> kernels;
std::set<void*> streams;
std::vector<std::pair<cudaStream_t, unsigned>> copies;  // host copies and their ticks
Clock host;
std::vector<std::tuple<dim3, dim3, size_t, cudaStream_t>> configs;

Stream& of(cudaStream_t s) {
    static Stream legacy;
    return s ? *reinterpret_cast<Stream*>(s) : legacy;
}
void join(Clock& a, const Clock& b) {
    for (const auto& t : b) a[t.first] = std::max(a[t.first], t.second);
}
Op& record(Op::Kind kind, cudaStream_t s) {
    Stream& st = of(s);
    join(st.clock, host);
    Op o{};
    o.kind = kind;
    o.stream = s;
    o.at = ++st.clock[&st];
    o.clock = st.clock;
    o.captured = st.capturing;
    ops.push_back(o);
    return ops.back();
}
void synced(const Clock& c) {
    join(host, c);
    std::vector<std::pair<cudaStream_t, unsigned>> left;
    for (const auto& p : copies)
        if (host[&of(p.first)] < p.second) left.push_back(p);
    copies.swap(left);
}
void sync_all() {
    for (void* s : streams) synced(of((cudaStream_t)s).clock);
    synced(of(nullptr).clock);
}
bool is_device(const void* p) { return room(p) != 0; }
void check(const void* p, size_t n, const char* what) {
    auto it = device.upper_bound((const char*)p);
    if (it == device.begin()) return;
    --it;
    const size_t off = (const char*)p - it->first;
    if (off < it->second && off + n > it->second)
        fault(std::string(what) + " of " + std::to_string(n) + " bytes past an allocation of " + std::to_string(it->second));
}
cudaError_t alloc(void** p, size_t n) {
    *p = nullptr;
    const long long k = allocations++;
    if (k >= fail_from && k <= fail_to) return cudaErrorMemoryAllocation;
    *p = std::calloc(1, n);
    device[(const char*)*p] = n;
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
void release(void* p) {
    if (!p) return;
    if (!device.erase((const char*)p)) fault("free of memory that is not allocated");
    std::free(p);
}
cudaError_t copy(void* dst, const void* src, size_t n) {
    check(dst, n, "copy to");
    check(src, n, "copy from");
    std::memcpy(dst, src, n);
    if (on_d2h && is_device(src) && !is_device(dst)) on_d2h(dst, n);
    return cudaSuccess;
}
cudaError_t launch(const void* f, dim3 grid, void** args, cudaStream_t s) {
    const std::string& name = kernels[f];
    if (launch_error) {
        const cudaError_t e = launch_error(name);
        if (e != cudaSuccess) return e;
    }
    Op& o = record(Op::KERNEL, s);
    o.name = name;
    o.grid = grid;
    o.args = args;
    if (on_kernel) on_kernel(o);
    o.args = nullptr;
    return cudaSuccess;
}
cudaError_t last = cudaSuccess;
cudaError_t keep(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
}  // namespace

bool before(const Op& a, const Op& b) {
    const auto it = b.clock.find(&of(a.stream));
    return it != b.clock.end() && it->second >= a.at && &a != &b;
}
size_t allocated() {
    size_t n = 0;
    for (const auto& d : device) n += d.second;
    return n;
}
size_t room(const void* p) {
    auto it = device.upper_bound((const char*)p);
    if (it == device.begin()) return 0;
    --it;
    const size_t off = (const char*)p - it->first;
    return off < it->second ? it->second - off : 0;
}
void fault(const std::string& what) { faults.push_back(what); }
int copies_in_flight() { return (int)copies.size(); }

}  // namespace fake

using namespace fake;

extern "C" {

// ---- kernels: registration by name, launches ----
void** CUDARTAPI __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void CUDARTAPI __cudaRegisterFatBinaryEnd(void**) {}
void CUDARTAPI __cudaUnregisterFatBinary(void**) {}
void CUDARTAPI __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels[f] = name;
}
void CUDARTAPI __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned CUDARTAPI __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* s) {
    configs.emplace_back(g, b, smem, s);
    return 0;
}
cudaError_t CUDARTAPI __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    std::tie(*g, *b, *smem, *static_cast<cudaStream_t*>(s)) = configs.back();
    configs.pop_back();
    return cudaSuccess;
}
cudaError_t CUDARTAPI __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t CUDARTAPI __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3, void** args, size_t, cudaStream_t s) {
    return keep(launch((const void*)k, g, args, s));
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return keep(launch(f, c->gridDim, args, c->stream));
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3, void** args, size_t, cudaStream_t s) {
    return keep(launch(f, g, args, s));
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}

// ---- device ----
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* lo, int* hi) {
    *lo = 0;
    *hi = -5;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize(void) {
    sync_all();
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) {
    *f = free_bytes;
    *t = free_bytes;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    *p = nullptr;
    return cudaErrorInvalidSymbol;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes*, const void*) { return cudaErrorInvalidValue; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long, cudaDriverEntryPointQueryResult*) {
    return cudaErrorNotSupported;
}

// ---- memory ----
cudaError_t cudaMalloc(void** p, size_t n) { return keep(alloc(p, n)); }
cudaError_t cudaFree(void* p) {
    sync_all();
    release(p);
    return cudaSuccess;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t n, cudaMemPool_t, cudaStream_t) { return keep(alloc(p, n)); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return keep(alloc(p, n)); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) {
    release(p);
    return cudaSuccess;
}
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) {
    *p = (cudaMemPool_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaMemPoolDestroy(cudaMemPool_t p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) {
    *p = std::calloc(1, n);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return copy(d, s, n); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    Op& o = record(Op::COPY, st);
    o.dst = (const char*)d;
    o.bytes = n;
    if (!is_device(d) || !is_device(s)) copies.push_back({st, o.at});
    return copy(d, s, n);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t st) {
    Op& o = record(Op::MEMSET, st);
    o.dst = (const char*)p;
    o.bytes = n;
    check(p, n, "fill");
    std::memset(p, v, n);
    return cudaSuccess;
}

// ---- streams and events ----
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    Stream* p = new Stream();
    streams.insert(p);
    *s = (cudaStream_t)p;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned f, int) { return cudaStreamCreateWithFlags(s, f); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    streams.erase((void*)s);  // its clock outlives it: operations refer to it
    return cudaSuccess;
}
cudaError_t cudaStreamGetPriority(cudaStream_t, int* p) {
    *p = 0;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (of(s).capturing) return keep(cudaErrorStreamCaptureUnsupported);
    synced(of(s).clock);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    Event& ev = *reinterpret_cast<Event*>(e);
    join(of(s).clock, ev.clock);
    if (ev.capturing) of(s).capturing = true;
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) {
    *e = (cudaEvent_t) new Event();
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    delete reinterpret_cast<Event*>(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    Event& ev = *reinterpret_cast<Event*>(e);
    join(of(s).clock, host);
    ev.clock = of(s).clock;
    ev.capturing = of(s).capturing;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t e) {
    synced(reinterpret_cast<Event*>(e)->clock);
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t e) { return cudaEventSynchronize(e); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = elapsed ? elapsed() : 1.f;
    return cudaSuccess;
}

// ---- graphs ----
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    record(Op::CAPTURE, s);
    of(s).capturing = true;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    for (void* s : streams) of((cudaStream_t)s).capturing = false;
    *g = (cudaGraph_t)std::malloc(1);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) {
    *x = (cudaGraphExec_t)std::malloc(1);
    return cudaSuccess;
}
// a graph is its index in graphs, plus one; a node its index in its graph, plus one
cudaError_t cudaGraphCreate(cudaGraph_t* g, unsigned) {
    graphs.emplace_back();
    *g = (cudaGraph_t)graphs.size();
    return cudaSuccess;
}
cudaError_t cudaGraphAddKernelNode(cudaGraphNode_t* node, cudaGraph_t g, const cudaGraphNode_t* deps, size_t n,
                                   const cudaKernelNodeParams* p) {
    std::vector<Node>& nodes = graphs[(size_t)g - 1];
    Node k{kernels[p->func], {}};
    std::set<size_t> after;
    for (size_t i = 0; i < n; ++i) {
        const size_t d = (size_t)deps[i] - 1;
        after.insert(d);
        after.insert(nodes[d].after.begin(), nodes[d].after.end());
    }
    k.after.assign(after.begin(), after.end());
    nodes.push_back(k);
    *node = (cudaGraphNode_t)nodes.size();
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    if ((size_t)g > graphs.size()) std::free(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    std::free(x);
    return cudaSuccess;
}
cudaError_t cudaGraphUpload(cudaGraphExec_t, cudaStream_t s) {
    record(Op::GRAPH_UPLOAD, s);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) {
    record(Op::GRAPH_LAUNCH, s);
    return cudaSuccess;
}

}  // extern "C"
