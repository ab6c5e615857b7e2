// fake_cudart.cpp -- TEST INFRASTRUCTURE: the CUDA runtime calls of
// libcortrace on the host, without a GPU, so that the host side of the C ABI
// (what it launches, copies, frees and reports) can be tested for the cases
// that no test can bring about on a device: a launch or a copy that fails, a
// copy that is still pending when its source is freed, another thread's call
// at a given point.  tests/test_host_runtime.py links it with the library's
// own objects in place of the runtime.
//
// Device memory is host memory.  A kernel does nothing; its launch is recorded,
// and fails as on a device if it asks for more dynamic shared memory than the
// function's limit.  A copy to or from the device is queued and made when its
// stream is waited for, as late as the runtime allows; a free of memory that a
// queued copy still reads or writes is counted (--wrap=free).
#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <vector>

extern "C" void __real_free(void*);

namespace {

struct Copy {
    void* dst;
    const void* src;
    size_t n;
    cudaStream_t stream;
};
struct Launch {
    std::string name;
    unsigned grid, block;
    size_t smem;
};

// never destroyed: the library's own exit handlers run after this file's
std::recursive_mutex& mu = *new std::recursive_mutex;
std::vector<Copy>& pending = *new std::vector<Copy>;
std::map<std::string, int>& loaded = *new std::map<std::string, int>;   // kernels used so far, launched or not
std::vector<Launch>& launches = *new std::vector<Launch>;
std::map<const void*, std::string>& names = *new std::map<const void*, std::string>;
std::map<const void*, size_t>& limits = *new std::map<const void*, size_t>;
std::map<std::string, std::vector<size_t>>& limits_set = *new std::map<std::string, std::vector<size_t>>;
std::string& fail_launch = *new std::string;
std::map<std::string, int>& fail_call = *new std::map<std::string, int>;   // calls until the one that fails
std::map<void*, size_t>& allocated = *new std::map<void*, size_t>;
size_t in_use = 0, memory = ~(size_t)0;
int freed_pending = 0;
void (*after_attribute)(const char*) = nullptr;
void (*during_wait)() = nullptr;
thread_local cudaError_t last = cudaSuccess;

using Lock = std::lock_guard<std::recursive_mutex>;

cudaError_t set(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}

bool fails(const char* call) {
    Lock l(mu);
    auto it = fail_call.find(call);
    if (it == fail_call.end() || --it->second > 0) return false;
    fail_call.erase(it);
    return true;
}

void finish(bool all, cudaStream_t s) {
    Lock l(mu);
    std::vector<Copy> rest;
    for (const Copy& c : pending) {
        if (all || c.stream == s) memcpy(c.dst, c.src, c.n);
        else rest.push_back(c);
    }
    pending.swap(rest);
}

struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local std::vector<Config>* configs = nullptr;

}  // namespace

extern "C" {

// ---- what the tests ask for ------------------------------------------------
void fake_reset(void) {
    finish(true, nullptr);
    Lock l(mu);
    launches.clear();
    limits_set.clear();
    fail_launch.clear();
    fail_call.clear();
    freed_pending = 0;
    after_attribute = nullptr;
    during_wait = nullptr;
    last = cudaSuccess;
    loaded.clear();
    memory = ~(size_t)0;
}
// Device memory in all, and how much of it is allocated.
void fake_memory(uint64_t bytes) { memory = bytes; }
uint64_t fake_in_use(void) { return in_use; }
void fake_fail_launch(const char* part) { fail_launch = part; }
void fake_fail_call(const char* call, int nth) { fail_call[call] = nth; }
int fake_freed_pending(void) { return freed_pending; }
int fake_pending(void) { return (int)pending.size(); }
void fake_after_attribute(void (*f)(const char*)) { after_attribute = f; }
void fake_during_wait(void (*f)()) { during_wait = f; }
int fake_launch_count(void) { return (int)launches.size(); }
int fake_launch(int i, char* name, int cap, unsigned* grid, unsigned* block, uint64_t* smem) {
    if (i < 0 || i >= (int)launches.size()) return -1;
    snprintf(name, (size_t)cap, "%s", launches[i].name.c_str());
    *grid = launches[i].grid;
    *block = launches[i].block;
    *smem = launches[i].smem;
    return 0;
}
// Kernels with `part` in their names that were used for the first time by their launch.
int fake_loaded_by_launch(const char* part) {
    int n = 0;
    for (const auto& k : loaded)
        if (k.first.find(part) != std::string::npos) n += k.second;
    return n;
}
// The number of different limits set for the functions whose name has `part`.
int fake_limits_set(const char* part) {
    int most = 0;
    for (const auto& f : limits_set) {
        if (f.first.find(part) == std::string::npos) continue;
        std::map<size_t, int> seen;
        for (size_t v : f.second) seen[v] = 1;
        if ((int)seen.size() > most) most = (int)seen.size();
    }
    return most;
}

void __wrap_free(void* p) {
    {
        Lock l(mu);
        for (const Copy& c : pending)
            if (p && (p == c.src || p == c.dst)) {
                freed_pending++;
                finish(true, nullptr);   // so that the test itself reads nothing freed
                break;
            }
    }
    __real_free(p);
}

// ---- the runtime -----------------------------------------------------------
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names[(const void*)host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* stream) {
    if (!configs) configs = new std::vector<Config>;
    configs->push_back({grid, block, smem, stream});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    const Config c = configs->back();
    configs->pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *(cudaStream_t*)stream = c.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
    Lock l(mu);
    const std::string& name = names[(const void*)k];
    const auto lim = limits.find((const void*)k);
    if (smem > (lim == limits.end() ? 48 * 1024 : lim->second)) return set(cudaErrorInvalidValue);
    if (!fail_launch.empty() && name.find(fail_launch) != std::string::npos) return set(cudaErrorLaunchOutOfResources);
    loaded.emplace(name, 1);
    launches.push_back({name, grid.x, block.x, smem});
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    std::string name;
    {
        Lock l(mu);
        name = names[f];
        loaded.emplace(name, 0);
        if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
            limits[f] = (size_t)v;
            limits_set[name].push_back((size_t)v);
        }
    }
    if (fails("cudaFuncSetAttribute")) return set(cudaErrorInvalidValue);
    if (after_attribute) after_attribute(name.c_str());
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void* f) {
    Lock l(mu);
    *a = cudaFuncAttributes{};
    loaded.emplace(names[f], 0);
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return fails("cudaOccupancy") ? set(cudaErrorInvalidValue) : cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
    *n = fails("cudaOccupancyMaxActiveClusters") ? 0 : 38;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 152;
    return cudaSuccess;
}
cudaError_t cudaGetLastError(void) {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "an error"; }
cudaError_t cudaMalloc(void** p, size_t n) {
    Lock l(mu);
    if (fails("cudaMalloc") || n > memory || in_use > memory - n) return set(cudaErrorMemoryAllocation);
    *p = calloc(1, n ? n : 1);
    allocated[*p] = n;
    in_use += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    finish(true, nullptr);   // waits for the device
    Lock l(mu);
    const auto a = allocated.find(p);
    if (a != allocated.end()) {
        in_use -= a->second;
        allocated.erase(a);
    }
    __real_free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static char scratch[2 * 1048576];
    *p = scratch;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind, cudaStream_t s) {
    if (fails("cudaMemcpyAsync")) return set(cudaErrorInvalidValue);
    Lock l(mu);
    pending.push_back({dst, src, n, s});
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind) {
    finish(true, nullptr);
    memcpy(dst, src, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) { return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) {
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    __real_free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (during_wait) during_wait();
    if (fails("cudaStreamSynchronize")) return set(cudaErrorUnknown);
    finish(false, s);
    return cudaSuccess;
}
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaErrorNotReady; }
cudaError_t cudaDeviceSynchronize(void) {
    finish(true, nullptr);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    __real_free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.f;
    return cudaSuccess;
}

}  // extern "C"
