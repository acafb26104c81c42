// A stand-in for the CUDA runtime, for tests of the engine's host code without a GPU: the .cu files under test are linked
// with this file instead of the runtime.
//
// Memory is the host's.  Work on a stream is queued and runs as late as a caller may count on: when the stream is
// waited for, or when a copy on it that blocks for pageable memory is queued.  The kernels the tests need are restated as simple
// functions of the same arguments (fake_kernel below); the rest do nothing.  fake_fail makes a coming call fail.
#include <cuda_runtime_api.h>
#include <sys/mman.h>
#include <unistd.h>

#include <cstdint>
#include <cstring>
#include <cstdlib>
#include <deque>
#include <functional>
#include <map>
#include <string>
#include <vector>

#include "../../auto_gb300/csrc/engine.cuh"

namespace {

struct Stream {
    std::deque<std::function<void()>> queue;
};
struct Range {
    size_t bytes;
    cudaMemoryType type;
};
std::map<const void*, std::string> names;      // kernels by their host stub
std::map<const void*, int> smem_limit;         // cudaFuncAttributeMaxDynamicSharedMemorySize
std::map<uintptr_t, Range> ranges;             // cudaMalloc and cudaHostAlloc
std::vector<Stream*> streams;
cudaError_t last = cudaSuccess;
int reads_host = 1;
std::string fail_what;
int fail_skip = 0;
void (*on_attribute)() = nullptr;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t s;
} config;

cudaError_t report(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
// whether this call of `what` is the one to fail
bool fails(const char* what) {
    if (fail_what.empty() || std::string(what).find(fail_what) == std::string::npos || fail_skip-- > 0) return false;
    fail_what.clear();
    return true;
}
const Range* find(const void* p) {
    auto it = ranges.upper_bound((uintptr_t)p);
    if (it == ranges.begin()) return nullptr;
    --it;
    return (uintptr_t)p < it->first + it->second.bytes ? &it->second : nullptr;
}
void drain(Stream* s) {
    while (!s->queue.empty()) {
        auto f = s->queue.front();
        s->queue.pop_front();
        f();
    }
}
Stream* of(cudaStream_t s) { return reinterpret_cast<Stream*>(s); }

// pages of the caller's pageable memory that a kernel was launched on and that the host had not touched
int absent = 0;
void expect_present(const void* p, size_t bytes) {
    if (find(p)) return;
    const uintptr_t page = (uintptr_t)sysconf(_SC_PAGESIZE), a = (uintptr_t)p / page * page, n = ((uintptr_t)p + bytes - a + page - 1) / page;
    std::vector<unsigned char> v(n);
    if (mincore((void*)a, n * page, v.data())) return;
    for (unsigned char c : v) absent += !(c & 1);
}

template <class T>
T arg(void** a, int i) { return *static_cast<T*>(a[i]); }

constexpr int IN = 16, OUT = 3, NPARAM = 70915;

// The kernel's effect, with its arguments taken now.
std::function<void()> fake_kernel(const std::string& name, void** a) {
    if (name.find("mlp_rank") != std::string::npos) {  // a probability is its row's sum plus its index
        const float* x = arg<const float*>(a, 0);
        const int n = arg<int>(a, 1);
        float* p = arg<float*>(a, 4);
        expect_present(x, (size_t)n * IN * 4);
        expect_present(p, (size_t)n * OUT * 4);
        return [=] {
            std::vector<float> r((size_t)n * OUT);
            for (int b = 0; b < n; b++) {
                float s = 0;
                for (int i = 0; i < IN; i++) s += x[(size_t)b * IN + i];
                for (int o = 0; o < OUT; o++) r[(size_t)b * OUT + o] = s + o;
            }
            memcpy(p, r.data(), r.size() * 4);
        };
    }
    if (name.find("mlp_tile") != std::string::npos) {  // every gradient: the sum of all inputs and labels; a loss: its row's first input
        const float *x = arg<const float*>(a, 0), *y = arg<const float*>(a, 1);
        const int n = arg<int>(a, 2);
        float *g = arg<float*>(a, 5), *loss = arg<float*>(a, 6);
        expect_present(x, (size_t)n * IN * 4);
        expect_present(y, (size_t)n * OUT * 4);
        return [=] {
            double s = 0;
            for (size_t i = 0; i < (size_t)n * IN; i++) s += x[i];
            for (size_t i = 0; i < (size_t)n * OUT; i++) s += y[i];
            for (int i = 0; i < NPARAM; i++) g[i] = (float)s;
            for (int b = 0; b < n; b++) loss[b] = x[(size_t)b * IN];
        };
    }
    if (name.find("copy_out") != std::string::npos) {
        const float* x = arg<const float*>(a, 0);
        float* y = arg<float*>(a, 1);
        const int n = arg<int>(a, 2);
        expect_present(y, (size_t)n * 4);
        return [=] { memcpy(y, x, (size_t)n * 4); };
    }
    if (name.find("copy_words") != std::string::npos) {
        float* d = arg<float*>(a, 0);
        const float* s = arg<const float*>(a, 1);
        const unsigned n = arg<unsigned>(a, 2);
        expect_present(d, (size_t)n * 16);
        expect_present(s, (size_t)n * 16);
        return [=] { memcpy(d, s, (size_t)n * 16); };
    }
    return [] {};
}

cudaError_t launch(const void* f, void** args, size_t smem, cudaStream_t s) {
    const std::string& name = names[f];
    const int limit = smem_limit.count(f) ? smem_limit[f] : 48 << 10;
    if (fails(name.c_str()) || smem > (size_t)limit) return report(cudaErrorInvalidValue);
    of(s)->queue.push_back(fake_kernel(name, args));
    return cudaSuccess;
}

}  // namespace

extern "C" {

// -------------------------------------------------------------- controls
// The call of `what` (part of a kernel's name, or cudaMemcpyAsync:up / :down) after `skip` others fails.
void fake_fail(const char* what, int skip) { fail_what = what, fail_skip = skip; }
int fake_failed() { return fail_what.empty(); }
// queued work that nobody has waited for
int fake_pending() {
    int n = 0;
    for (Stream* s : streams) n += (int)s->queue.size();
    return n;
}
// a range of the caller's as page-locked memory
void fake_lock(void* p, size_t n) { ranges[(uintptr_t)p] = {n, cudaMemoryTypeHost}; }
void fake_unlock(void* p) { ranges.erase((uintptr_t)p); }
void fake_leave_error() { last = cudaErrorInvalidValue; }  // an error that nobody has asked for
int fake_absent() {
    const int n = absent;
    absent = 0;
    return n;
}
void fake_reads_host(int on) { reads_host = on; }
void fake_on_attribute(void (*f)()) { on_attribute = f; }
// entries of the engine's that are not exported
int fake_world_stats(int sides) {
    static cudaStream_t s = nullptr;
    if (!s) cudaStreamCreateWithFlags(&s, 0);
    const bool ok = lenia::launch_world_stats(nullptr, 1, sides, nullptr, s) && cudaGetLastError() == cudaSuccess;
    drain(of(s));
    return ok;
}

// -------------------------------------------------------------- the runtime
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) {
    config = {g, b, smem, s};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = config.grid, *b = config.block, *smem = config.smem, *static_cast<cudaStream_t*>(s) = config.s;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t)const_cast<void*>(f);
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** args, size_t smem, cudaStream_t s) {
    return launch((const void*)k, args, smem, s);
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void** args, size_t smem, cudaStream_t s) {
    return launch(f, args, smem, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return launch(f, args, c->dynamicSmemBytes, c->stream);
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrPageableMemoryAccessUsesHostPageTables ? reads_host : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
    smem_limit[f] = v;
    if (auto g = on_attribute) {
        on_attribute = nullptr;
        g();
    }
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = calloc(n ? n : 1, 1);
    ranges[(uintptr_t)*p] = {n, cudaMemoryTypeDevice};
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) {
    *p = calloc(n ? n : 1, 1);
    ranges[(uintptr_t)*p] = {n, cudaMemoryTypeHost};
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    ranges.erase((uintptr_t)p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    memset(a, 0, sizeof(*a));
    const Range* r = find(p);
    a->type = r ? r->type : cudaMemoryTypeUnregistered;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t st) {
    if (fails(kind == cudaMemcpyHostToDevice ? "cudaMemcpyAsync:up" : "cudaMemcpyAsync:down")) return report(cudaErrorInvalidValue);
    of(st)->queue.push_back([=] { memcpy(d, s, n); });
    if (!find(kind == cudaMemcpyHostToDevice ? s : d)) drain(of(st));  // pageable memory: blocks
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) {
    of(s)->queue.push_back([=] { cudaFree(p); });
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    of(st)->queue.push_back([=] { memset(d, v, n); });
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    streams.push_back(new Stream);
    *s = reinterpret_cast<cudaStream_t>(streams.back());
    return cudaSuccess;
}
// events and graphs: every queue is drained where an order is asked for
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(&last);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) {
    drain(of(s));
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    *e = reinterpret_cast<cudaGraphExec_t>(&last);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "refused"; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof(*p));
    p->major = 10, p->minor = 3, p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    drain(of(s));
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    drain(of(s));
    return cudaSuccess;
}

}  // extern "C"
