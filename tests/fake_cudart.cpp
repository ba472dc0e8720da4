// A CUDA runtime without a GPU, for tests of the library's host code: linked with the library's objects
// in place of cudart.  Device memory is zeroed host memory, copies are immediate, kernels do not run but
// are recorded (name, device, grid, threads, dynamic shared memory), and the rules that the host code
// has to keep are enforced: a launch with more than 48 KB of dynamic shared memory fails unless the
// attribute of that function was set on the current device.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>
#include <vector>

namespace {

constexpr int kDevices = 8;
struct Launch {
    std::string name;
    int device;
    unsigned gx, gy, gz, threads;
    size_t smem;
    bool captured;
};
struct Block {
    void* p;
    size_t bytes;
    bool host;
};

std::mutex mu;
thread_local int device = 0;
thread_local bool capturing = false;
std::map<const void*, std::string> names;                 // host stub -> kernel name
std::map<std::pair<int, const void*>, size_t> smem_limit;  // (device, kernel) -> dynamic shared memory
std::vector<Launch> launches;
std::vector<Block> blocks;
std::map<const void*, Block> symbols;
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local std::vector<Config> configs;

void* map(size_t n, bool host) {
    n = (n + 4095) / 4096 * 4096;
    void* p = mmap(nullptr, n, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (p == MAP_FAILED) return nullptr;
    std::lock_guard<std::mutex> g(mu);
    blocks.push_back({p, n, host});
    return p;
}
cudaError_t unmap(void* p) {
    std::lock_guard<std::mutex> g(mu);
    for (size_t i = 0; i < blocks.size(); ++i)
        if (blocks[i].p == p) {
            munmap(p, blocks[i].bytes);
            blocks.erase(blocks.begin() + i);
            return cudaSuccess;
        }
    return p ? cudaErrorInvalidValue : cudaSuccess;
}
cudaError_t launch(const void* fn, dim3 grid, dim3 block, size_t smem) {
    std::lock_guard<std::mutex> g(mu);
    auto it = smem_limit.find({device, fn});
    if (smem > 48 * 1024 && (it == smem_limit.end() || it->second < smem)) return cudaErrorInvalidValue;
    if (!grid.x || !grid.y || !grid.z || grid.y > 65535) return cudaErrorInvalidConfiguration;
    launches.push_back({names[fn], device, grid.x, grid.y, grid.z, block.x * block.y * block.z, smem, capturing});
    return cudaSuccess;
}
template <class T>
T handle() {
    return reinterpret_cast<T>(new char[8]);
}

}  // namespace

extern "C" {

// ---- what a test asks
int fake_launch_count() { return (int)launches.size(); }
void fake_clear_launches() { launches.clear(); }
const char* fake_launch_name(int i) { return launches[i].name.c_str(); }
// device, grid x y z, threads, dynamic shared memory
void fake_launch_shape(int i, long long out[6]) {
    const Launch& l = launches[i];
    const long long v[6] = {l.device, l.gx, l.gy, l.gz, l.threads, (long long)l.smem};
    std::memcpy(out, v, sizeof v);
}
int fake_alloc_count(int host) {
    int n = 0;
    for (const Block& b : blocks) n += b.host == (host != 0);
    return n;
}
// The k-th live allocation of host (1) or device (0) memory.
void* fake_alloc(int host, int k) {
    for (const Block& b : blocks)
        if (b.host == (host != 0) && k-- == 0) return b.p;
    return nullptr;
}

// ---- registration (called by the objects' static initialisers)
void** __cudaRegisterFatBinary(void*) { return new void*(nullptr); }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names[host] = name;
}
void __cudaRegisterVar(void**, char* host, char*, const char*, int, size_t size, int, int) {
    symbols[host] = {nullptr, size, false};
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st* st) {
    configs.push_back({grid, block, smem, st});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
    const Config c = configs.back();
    configs.pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *static_cast<cudaStream_t*>(st) = c.stream;
    return cudaSuccess;
}

// ---- devices, errors
cudaError_t cudaGetDeviceCount(int* n) { return *n = kDevices, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d >= kDevices) return cudaErrorInvalidDevice;
    return device = d, cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : (a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 232448 : 1);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "error of the stand-in runtime"; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }

// ---- kernels
cudaError_t cudaFuncSetAttribute(const void* fn, cudaFuncAttribute a, int v) {
    std::lock_guard<std::mutex> g(mu);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) smem_limit[{device, fn}] = (size_t)v;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* fn, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
    return launch(fn, grid, block, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* fn, void**) {
    return launch(fn, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { return *n = 2, cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* sym) {
    Block& b = symbols[sym];
    if (!b.p) b.p = map(b.bytes ? b.bytes : 8, false);
    return *p = b.p, cudaSuccess;
}

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) { return (*p = map(n, false)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return cudaMalloc(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return (*p = map(n, true)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { return unmap(p); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { return unmap(p); }
cudaError_t cudaFreeHost(void* p) { return unmap(p); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    for (size_t r = 0; r < h; ++r) std::memcpy(static_cast<char*>(d) + r * dp, static_cast<const char*>(s) + r * sp, w);
    return cudaSuccess;
}
// fresh memory is zero: clearing large buffers would only touch their pages
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
    if (v || n < (1u << 16)) std::memset(p, v, n);
    return cudaSuccess;
}

// ---- streams, events, graphs
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = handle<cudaStream_t>(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { return delete[] reinterpret_cast<char*>(s), cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return capturing = true, cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    capturing = false;
    return *g = handle<cudaGraph_t>(), cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = handle<cudaEvent_t>(), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { return delete[] reinterpret_cast<char*>(e), cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { return delete[] reinterpret_cast<char*>(g), cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    return *e = handle<cudaGraphExec_t>(), cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { return delete[] reinterpret_cast<char*>(e), cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

}  // extern "C"
