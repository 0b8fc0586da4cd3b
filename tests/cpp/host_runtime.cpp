// host_runtime.cpp -- a CUDA runtime without a device, for tests of the
// engine's host code.  Linked with the engine's sources in place of libcudart:
// device memory is host memory, copies and clears are done, kernel launches
// are not.  It keeps a log of what the engine asked for (host_log) and fails
// what a test tells it to fail (host_set).  A launch whose dynamic shared memory exceeds the
// kernel's limit at that moment is refused, as the real runtime does.
#include <cuda_runtime_api.h>
#include <cxxabi.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>

namespace {

std::mutex g_mu;
std::map<const void*, std::string> g_names;
std::map<const void*, size_t> g_limit;   // dynamic shared memory a kernel may be launched with
std::map<std::string, int> g_set;
std::string g_log;
thread_local cudaError_t t_last = cudaSuccess;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local Config t_config;

cudaError_t done(cudaError_t e) {
    if (e != cudaSuccess) t_last = e;
    return e;
}
std::string name_of(const void* f) {
    auto it = g_names.find(f);
    return it == g_names.end() ? "?" : it->second;
}
void note(const std::string& s) { g_log += s + "\n"; }
int setting(const char* name, int other) {
    auto it = g_set.find(name);
    return it == g_set.end() ? other : it->second;
}
cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t smem, const char* verb) {
    std::lock_guard<std::mutex> l(g_mu);
    const size_t limit = g_limit.count(f) ? g_limit[f] : 48 * 1024;
    const std::string what = name_of(f) + " grid " + std::to_string(grid.x) + " block " + std::to_string(block.x) +
                             " smem " + std::to_string(smem);
    const bool ok = smem <= limit && !(std::strcmp(verb, "cluster") == 0 && setting("refuse_clusters", 0));
    note(std::string(ok ? verb : "refused") + " " + what);
    return done(ok ? cudaSuccess : cudaErrorInvalidValue);
}

}  // namespace

extern "C" {

__attribute__((visibility("default"))) const char* host_log() {
    static std::string copy;
    std::lock_guard<std::mutex> l(g_mu);
    copy = g_log;
    g_log.clear();
    return copy.c_str();
}
__attribute__((visibility("default"))) void host_set(const char* name, int value) {
    std::lock_guard<std::mutex> l(g_mu);
    g_set[name] = value;
}

// what compiled .cu files call
void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 0; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* fun, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    int status = 0;
    char* plain = abi::__cxa_demangle(name, nullptr, nullptr, &status);
    std::string s = status == 0 ? plain : name;
    std::free(plain);
    // "void pm::(anonymous namespace)::k_name<...>(...)" -> "k_name<...>"
    const size_t k = s.find("k_");
    std::lock_guard<std::mutex> l(g_mu);
    g_names[fun] = k == std::string::npos ? s : s.substr(k, s.find('(', k) - k);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, void* stream) {
    t_config = {grid, block, smem, static_cast<cudaStream_t>(stream)};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = t_config.grid;
    *block = t_config.block;
    *smem = t_config.smem;
    *static_cast<cudaStream_t*>(stream) = t_config.stream;
    return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
    return launch(f, grid, block, smem, "launch");
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, "cluster");
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute attr, int value) {
    std::lock_guard<std::mutex> l(g_mu);
    if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (value > 227 * 1024) return done(cudaErrorInvalidValue);
        if (g_limit.count(f) && g_limit[f] > (size_t)value) note("lowered " + name_of(f));
        g_limit[f] = (size_t)value;
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* blocks, const void* f, int threads, size_t smem,
                                                                   unsigned) {
    std::lock_guard<std::mutex> l(g_mu);
    note("occupancy " + name_of(f));
    const int by_smem = (int)(228 * 1024 / (smem + 1024)), by_threads = 1024 / threads;
    *blocks = by_smem < by_threads ? by_smem : by_threads;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* clusters, const void* f, const cudaLaunchConfig_t*) {
    std::lock_guard<std::mutex> l(g_mu);
    note("clusters " + name_of(f));
    *clusters = setting("clusters", 8);
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
    std::lock_guard<std::mutex> l(g_mu);
    note("malloc " + std::to_string(bytes));
    *p = std::aligned_alloc(256, (bytes + 255) / 256 * 256);
    return done(*p ? cudaSuccess : cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    for (size_t i = 0; i < h; ++i) std::memcpy(static_cast<char*>(d) + i * dp, static_cast<const char*>(s) + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static void* symbol = std::aligned_alloc(256, 8 << 20);
    *p = symbol;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = t_last;
    t_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "the host runtime's error"; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(16);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return done(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return done(cudaErrorNotSupported); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return done(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return done(cudaErrorNotSupported); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }

}  // extern "C"
