// A CUDA runtime without a device, for tests of the engine's host code on the CPU.
//
// The engine's objects link against fake_cudart.cpp instead of libcudart.  "Device" memory is host memory, so
// copies and fills really happen and are checked against the allocations they touch; kernels do nothing but
// leave a record.  Every record carries a vector clock over the streams and the host (stream order, events,
// synchronising calls), so a test can ask whether one operation is ordered before another.  What kernels would
// have written for the host to read is supplied by a hook on device-to-host copies.
#pragma once
#include <cstddef>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include <cuda_runtime.h>

namespace fake {

using Clock = std::map<const void*, unsigned>;  // by stream; the host under nullptr

struct Op {
    enum Kind { KERNEL, MEMSET, COPY, GRAPH_LAUNCH, GRAPH_UPLOAD, CAPTURE } kind;
    std::string name;      // kernel: its (mangled) name
    cudaStream_t stream;
    Clock clock;
    unsigned at;           // this operation's own tick on its stream
    bool captured;         // recorded into a graph, not executed
    dim3 grid;
    void** args;           // kernel: pointers to its arguments, valid during on_kernel only
    const char* dst;       // fill or copy
    size_t bytes;
};
bool before(const Op& a, const Op& b);  // a is ordered before b
struct Node {              // a kernel node of a graph built by hand
    std::string name;
    std::vector<size_t> after;  // indices of the nodes it depends on, directly or not
};
extern std::vector<std::vector<Node>> graphs;  // every graph created

extern std::vector<Op> ops;
extern std::vector<std::string> faults;                              // accesses outside an allocation
extern std::function<void(Op&)> on_kernel;                           // sees every launch, with its arguments
extern std::function<void(void* dst, size_t bytes)> on_d2h;          // after a device-to-host copy
extern long long allocations;                                        // device allocations so far
extern long long fail_from, fail_to;                                 // those with these indices fail
extern std::function<float()> elapsed;                               // milliseconds between two events
extern size_t free_bytes;                                            // what cudaMemGetInfo reports
extern std::function<cudaError_t(const std::string& kernel)> launch_error;  // result of a launch
size_t allocated();  // device bytes allocated now
// the allocation that holds p: bytes from p to its end (0: none)
size_t room(const void* p);
void fault(const std::string& what);
// copies queued to or from host memory whose stream the host has not waited for since
int copies_in_flight();

}  // namespace fake
