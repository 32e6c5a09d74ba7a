// A CUDA runtime of host memory, linked with the library's objects in place of the real one:
// allocations are host memory, copies run at once, kernels are recorded and not run. For the host
// logic that a GPU run cannot show: the order of copies and launches, allocations that
// fail, the sizes of workspaces and grids.
//
// Order: a copy or a memset on the legacy stream may return before the device has it, and the
// library's streams are non-blocking, so it counts as pending until the legacy stream, or the
// device, is waited for; a launch or an asynchronous copy on another stream before that is a
// violation.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Launch {
    std::string name;
    dim3 grid, block;
};
struct State {
    std::map<const void*, std::string> kernels;
    std::map<void*, size_t> live;
    std::vector<Launch> launches;
    std::string violations;
    std::string pending;
    long mallocs = 0, fail_at = -1;  // allocation (from 0) that fails
    size_t live_bytes = 0, peak = 0, largest = 0;
    dim3 grid, block;
    size_t smem = 0;
    cudaStream_t stream = nullptr;
};
State& st() {
    static State s;
    return s;
}

bool legacy(cudaStream_t s) { return s == nullptr || s == cudaStreamLegacy; }

void use(cudaStream_t s, const std::string& what) {
    if (!legacy(s) && !st().pending.empty()) st().violations += what + " after " + st().pending + "; ";
}

cudaError_t allocate(void** p, size_t n) {
    *p = nullptr;
    if (st().mallocs++ == st().fail_at) return cudaErrorMemoryAllocation;
    if (posix_memalign(p, 256, std::max<size_t>(n, 1))) return cudaErrorMemoryAllocation;
    std::memset(*p, 0xff, n);
    st().live[*p] = n;
    st().live_bytes += n;
    st().peak = std::max(st().peak, st().live_bytes);
    st().largest = std::max(st().largest, n);
    return cudaSuccess;
}

cudaError_t release(void* p) {
    if (!p) return cudaSuccess;
    const auto it = st().live.find(p);
    if (it == st().live.end()) {
        st().violations += "free of an address that was not allocated; ";
        return cudaErrorInvalidValue;
    }
    st().live_bytes -= it->second;
    st().live.erase(it);
    std::free(p);
    return cudaSuccess;
}

void launch(const void* fn, dim3 grid, dim3 block, cudaStream_t s) {
    const std::string& name = st().kernels[fn];
    use(s, "launch of " + name);
    st().launches.push_back({name, grid, block});
}
}  // namespace

extern "C" {

// what the tests read and set
void fake_reset() {
    st().launches.clear();
    st().violations.clear();
    st().pending.clear();
    st().mallocs = 0;
    st().fail_at = -1;
    st().peak = st().live_bytes;
    st().largest = 0;
}
void fake_fail_at(long k) {
    st().mallocs = 0;
    st().fail_at = k;
}
long fake_mallocs() { return st().mallocs; }
size_t fake_peak() { return st().peak; }
size_t fake_largest() { return st().largest; }
const char* fake_violations() { return st().violations.c_str(); }
int fake_n_launches() { return static_cast<int>(st().launches.size()); }
const char* fake_launch(int k, unsigned* grid) {
    const Launch& l = st().launches[k];
    grid[0] = l.grid.x;
    grid[1] = l.grid.y;
    grid[2] = l.grid.z;
    return l.name.c_str();
}

// registration and launches
void** __cudaRegisterFatBinary(void*) {
    static void* handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    st().kernels[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* s) {
    st().grid = grid;
    st().block = block;
    st().smem = smem;
    st().stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
    *grid = st().grid;
    *block = st().block;
    *smem = st().smem;
    *static_cast<cudaStream_t*>(s) = st().stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* fn) {
    *k = reinterpret_cast<cudaKernel_t>(const_cast<void*>(fn));
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void**, size_t, cudaStream_t s) {
    launch(k, grid, block, s);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 grid, dim3 block, void**, size_t, cudaStream_t s) {
    launch(fn, grid, block, s);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
    launch(fn, c->gridDim, c->blockDim, c->stream);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }

// memory
cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaFree(void* p) { return release(p); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return allocate(p, n); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return release(p); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind kind) {
    std::memcpy(d, s, n);
    if (kind == cudaMemcpyHostToDevice) st().pending = "a copy on the legacy stream";
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    std::memset(d, v, n);
    st().pending = "a memset on the legacy stream";
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t q) {
    use(q, "copy");
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t q) {
    use(q, "copy");
    for (size_t r = 0; r < h; ++r) std::memcpy(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t q) {
    use(q, "memset");
    std::memset(d, v, n);
    return cudaSuccess;
}

// streams, events, the device
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    static long n = 0x1000;
    *s = reinterpret_cast<cudaStream_t>(n += 16);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (legacy(s)) st().pending.clear();
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() {
    st().pending.clear();
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = reinterpret_cast<cudaEvent_t>(0x10);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.f;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount                   ? 152
         : a == cudaDevAttrMaxSharedMemoryPerBlockOptin       ? 232448
         : a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472
                                                            : 1 << 26;
    return cudaSuccess;
}
cudaError_t cudaDeviceSetLimit(cudaLimit, size_t) { return cudaSuccess; }
cudaError_t cudaDeviceGetLimit(size_t* v, cudaLimit) {
    *v = 0;
    return cudaSuccess;
}
cudaError_t cudaCtxResetPersistingL2Cache() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static char array[1 << 20];
    *p = array;
    return cudaSuccess;
}

}  // extern "C"
