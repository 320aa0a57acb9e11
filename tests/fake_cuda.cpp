// A fake CUDA runtime for the host code's fault tests (test_host_faults.py):
// the library's objects are linked against it instead of the real one. Memory
// is host memory and copies are done at once; kernels do not run, except that
// a run's first kernel copies the run's cell and its last one writes counters
// that the test gives. Every call that a test looks at goes to a log, and a
// test can have the n-th call of any of them return an error.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <atomic>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <thread>
#include <vector>

namespace {

std::recursive_mutex mu;
std::vector<std::string> calls;
std::map<void*, size_t> device, pinned;
std::map<std::string, std::pair<int, int>> failures;  // call: how many from now, the error
std::vector<std::pair<uint32_t, uint32_t>> counters;  // words of a run's counters
bool capturing = false;
int host_tables = 0;  // whether the device uses the host's page tables
thread_local cudaError_t last = cudaSuccess;

struct Launch {
    std::string name;
    std::vector<void*> args;  // its first three, where the fake acts on them
};
std::vector<Launch>* graph_of_capture = nullptr;

// (the objects' static constructors fill it in, before or after this file's)
std::map<const void*, std::string>& kernels() {
    static auto* m = new std::map<const void*, std::string>;
    return *m;
}

using Lock = std::lock_guard<std::recursive_mutex>;

cudaError_t call(const char* api, const std::string& what = "") {
    Lock g(mu);
    auto it = failures.find(api);
    if (it != failures.end() && --it->second.first == 0) {
        last = (cudaError_t)it->second.second;
        failures.erase(it);
        calls.push_back(std::string("failed ") + api);
        return last;
    }
    calls.push_back(std::string(api) + (what.empty() ? "" : " " + what));
    return cudaSuccess;
}

// What the run's first and last kernel leave: the cell's copy, and the counters.
void act(const Launch& l) {
    if (l.name.find("k_begin") != std::string::npos) {
        std::memcpy(l.args[1], l.args[0], 48);  // RunCell
    } else {  // k_export: the cell's counters; k_batch_export: its own argument's
        uint32_t* ctr = static_cast<uint32_t*>(l.args[0]);
        if (l.name.find("k_batch") == std::string::npos) ctr = *reinterpret_cast<uint32_t**>(static_cast<char*>(l.args[2]) + 16);
        for (auto& c : counters) ctr[c.first] = c.second;
    }
}

cudaError_t launch(const void* func, dim3 grid, void** args) {
    Lock g(mu);
    Launch l{kernels()[func], {}};
    if (cudaError_t e = call("launch", l.name + " " + std::to_string(grid.x) + "x" + std::to_string(grid.y) +
                                           (capturing ? " captured" : "")))
        return e;
    if (l.name.find("k_begin") != std::string::npos || l.name.find("k_export") != std::string::npos)
        for (int i = 0; i < 3; ++i) l.args.push_back(*static_cast<void**>(args[i]));
    else if (l.name.find("k_batch_export") != std::string::npos)
        l.args.push_back(*static_cast<void**>(args[10]));
    if (capturing)
        graph_of_capture->push_back(l);
    else if (!l.args.empty())
        act(l);
    return cudaSuccess;
}

template <class P>
cudaError_t handle(P* out) {
    *out = reinterpret_cast<P>(std::malloc(1));
    return cudaSuccess;
}

// cuTensorMapEncodeTiled: a driver call, which leaves no runtime error
CUresult encode(...) {
    const cudaError_t before = last, e = call("encode");
    last = before;
    return e == cudaSuccess ? CUDA_SUCCESS : CUDA_ERROR_INVALID_VALUE;
}

void rows(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h) {
    for (size_t y = 0; y < h; ++y) std::memcpy((char*)d + y * dp, (const char*)s + y * sp, w);
}

}  // namespace

extern "C" {

// ---- the tests' side ----
void fake_reset() {
    Lock g(mu);
    calls.clear();
    failures.clear();
    counters.clear();
}
void fake_fail(const char* api, int nth, int error) {
    Lock g(mu);
    failures[api] = {nth, error};
}
void fake_counter(uint32_t word, uint32_t value) {
    Lock g(mu);
    counters.emplace_back(word, value);
}
// the log since the last call, a line for each entry
size_t fake_log(char* out, size_t cap) {
    Lock g(mu);
    std::string s;
    for (auto& c : calls) s += c + "\n";
    calls.clear();
    const size_t n = s.size() < cap ? s.size() : cap - 1;
    std::memcpy(out, s.data(), n);
    out[n] = 0;
    return s.size();
}
void fake_host_tables(int on) { host_tables = on; }
// threads that free results of their own (malloc'd ones) until told to stop
void fake_free_results(void (*free_result)(void*), int threads) {
    static std::atomic<bool> stop;
    static std::vector<std::thread> running;
    stop = true;
    for (auto& t : running) t.join();
    running.clear();
    stop = false;
    for (int i = 0; i < threads; ++i)
        running.emplace_back([free_result] {
            while (!stop) {
                struct { uint32_t n; void *kps, *desc; } r{1, std::malloc(64), nullptr};
                free_result(&r);
            }
        });
}
int fake_live_device() {
    Lock g(mu);
    return (int)device.size();
}

// ---- the runtime's ----
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st*) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) {
    *g = *b = dim3(1, 1, 1);
    *s = 0;
    *static_cast<cudaStream_t*>(st) = nullptr;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* func) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(func));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3, void** args, size_t, cudaStream_t) {
    return launch(k, grid, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* func, void** args) {
    return launch(func, c->gridDim, args);
}

cudaError_t cudaMalloc(void** p, size_t n) {
    Lock g(mu);
    *p = nullptr;
    if (cudaError_t e = call("cudaMalloc")) return e;
    *p = std::calloc(n ? n : 1, 1);
    device[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    Lock g(mu);
    device.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    Lock g(mu);
    *p = nullptr;
    if (cudaError_t e = call("cudaHostAlloc")) return e;
    *p = std::calloc(n ? n : 1, 1);
    pinned[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    Lock g(mu);
    call("cudaFreeHost");
    pinned.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
    *d = h;
    return call("cudaHostGetDevicePointer");
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    Lock g(mu);
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    for (auto& m : pinned)
        if (p >= m.first && p < (char*)m.first + m.second) {
            a->type = cudaMemoryTypeHost;
            a->devicePointer = const_cast<void*>(p);
        }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    if (cudaError_t e = call("cudaMemcpy")) return e;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (cudaError_t e = call("cudaMemcpyAsync")) return e;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2D(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind) {
    rows(d, dp, s, sp, w, h);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    if (cudaError_t e = call("cudaMemcpy2DAsync")) return e;
    rows(d, dp, s, sp, w, h);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    if (cudaError_t e = call("cudaMemsetAsync")) return e;
    std::memset(p, v, n);
    return cudaSuccess;
}

cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    Lock g(mu);
    if (cudaError_t e = call("cudaStreamBeginCapture")) return e;
    capturing = true;
    graph_of_capture = new std::vector<Launch>;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* out) {
    Lock g(mu);
    capturing = false;
    *out = reinterpret_cast<cudaGraph_t>(graph_of_capture);
    return call("cudaStreamEndCapture");
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t graph, unsigned long long) {
    if (cudaError_t e = call("cudaGraphInstantiate")) return e;
    *x = reinterpret_cast<cudaGraphExec_t>(new std::vector<Launch>(*reinterpret_cast<std::vector<Launch>*>(graph)));
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    Lock g(mu);
    if (cudaError_t e = call("cudaGraphLaunch")) return e;
    for (auto& l : *reinterpret_cast<std::vector<Launch>*>(x))
        if (!l.args.empty()) act(l);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    delete reinterpret_cast<std::vector<Launch>*>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    delete reinterpret_cast<std::vector<Launch>*>(x);
    return cudaSuccess;
}

cudaError_t cudaStreamSynchronize(cudaStream_t) { return call("cudaStreamSynchronize"); }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return handle(s); }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t* s, unsigned, int) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    std::free(s);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    std::free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return call("cudaEventRecord"); }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrPageableMemoryAccess                    ? 1
         : a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? host_tables
                                                                  : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) {
    *least = 0;
    *greatest = -5;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return call("cudaFuncSetAttribute"); }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    *p = nullptr;
    return cudaErrorInvalidValue;
}
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult* q) {
    *f = reinterpret_cast<void*>(&encode);
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
const char* cudaGetErrorName(cudaError_t) { return "fake"; }

}  // extern "C"
