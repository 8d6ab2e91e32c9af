// A stand-in for the CUDA runtime, preloaded under libcuco_gb300.so by the
// host-side tests: two devices whose memory is host memory, kernels that do
// nothing.  It keeps what a real runtime keeps per device (a kernel's dynamic
// shared-memory limit, an allocation's device) and counts and logs what the
// library asks for.
#include <cuda_runtime_api.h>

#include <algorithm>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <string>
#include <utility>

namespace {
constexpr int kDevices = 2;
constexpr size_t kDefaultSmem = 48 * 1024;
std::recursive_mutex g_mu;
int g_device = 0;
cudaError_t g_last = cudaSuccess;
size_t g_live = 0, g_peak = 0;
std::map<const void *, std::string> g_names;
std::map<std::pair<int, const void *>, size_t> g_smem;
struct Block {
    size_t size;
    int device;
};
std::map<uintptr_t, Block> g_blocks;
std::string g_log;
int g_failures = 0;  // cudaFuncSetAttribute calls still to fail

cudaError_t done(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}

const Block *find(const void *p) {
    auto it = g_blocks.upper_bound((uintptr_t)p);
    if (it == g_blocks.begin()) return nullptr;
    --it;
    return (uintptr_t)p < it->first + it->second.size ? &it->second : nullptr;
}

void *take(size_t size) {
    void *p = calloc(1, size ? size : 1);
    g_blocks[(uintptr_t)p] = Block{size, g_device};
    g_live += size;
    g_peak = std::max(g_peak, g_live);
    return p;
}

void give(void *p) {
    auto it = g_blocks.find((uintptr_t)p);
    if (it == g_blocks.end()) return;
    g_live -= it->second.size;
    g_blocks.erase(it);
    free(p);
}

void note(const std::string &what, const void *p) {
    char at[32];
    snprintf(at, sizeof at, " %llx\n", (unsigned long long)(uintptr_t)p);
    g_log += what + at;
}

cudaError_t launch(const void *func, size_t smem, void **args) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    void *first = nullptr;
    memcpy(&first, args[0], sizeof first);
    note("launch " + g_names[func], first);
    auto it = g_smem.find({g_device, func});
    if (smem > (it == g_smem.end() ? kDefaultSmem : it->second)) return done(cudaErrorInvalidValue);
    return cudaSuccess;
}

cudaError_t copy(const char *what, void *dst, const void *src, size_t n) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    note(std::string(what) + " from", src);
    note(std::string(what) + " to", dst);
    memmove(dst, src, n);
    return cudaSuccess;
}

template <typename T>
cudaError_t handle(T *h) {
    *h = (T)malloc(16);
    return cudaSuccess;
}

struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} g_config;
}  // namespace

extern "C" {
// ---- the tests' side
void fake_reset() {
    g_log.clear();
    g_peak = g_live;
}
const char *fake_log() { return g_log.c_str(); }
unsigned long long fake_live() { return g_live; }
unsigned long long fake_peak() { return g_peak; }
void fake_fail_attributes(int n) { g_failures = n; }
void *fake_alloc(size_t size, int device) {
    const int old = g_device;
    g_device = device;
    void *p = take(size);
    g_device = old;
    return p;
}

// ---- what nvcc's host code calls
void **__cudaRegisterFatBinary(void *) { return (void **)malloc(16); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    g_names[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    g_config = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = g_config.grid, *block = g_config.block, *smem = g_config.smem;
    *(cudaStream_t *)stream = g_config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *kernel, const void *func) {
    *kernel = (cudaKernel_t)func;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3, dim3, void **args, size_t smem, cudaStream_t) {
    return launch((const void *)kernel, smem, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *func, void **args) {
    return launch(func, c->dynamicSmemBytes, args);
}

// ---- the runtime
cudaError_t cudaFuncSetAttribute(const void *func, enum cudaFuncAttribute attr, int value) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (g_failures > 0) {
        --g_failures;
        return done(cudaErrorUnknown);
    }
    if (attr == cudaFuncAttributeMaxDynamicSharedMemorySize) g_smem[{g_device, func}] = (size_t)value;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = g_device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d >= kDevices) return done(cudaErrorInvalidDevice);
    g_device = d;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, enum cudaDeviceAttr attr, int) {
    *v = attr == cudaDevAttrMultiProcessorCount ? 152 : 0;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(struct cudaDeviceProp *p, int) {
    memset(p, 0, sizeof *p);
    p->multiProcessorCount = 152;
    p->major = 10, p->minor = 3;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetDefaultMemPool(cudaMemPool_t *pool, int) { return handle(pool); }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, enum cudaMemPoolAttr, void *) { return cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) {
    *lo = *hi = 0;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 4;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "an error of the stand-in runtime"; }

cudaError_t cudaMalloc(void **p, size_t size) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    *p = take(size);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t size, cudaStream_t) { return cudaMalloc(p, size); }
cudaError_t cudaFree(void *p) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    if (p) give(p);
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) { return cudaFree(p); }
cudaError_t cudaHostAlloc(void **p, size_t size, unsigned) {
    *p = calloc(1, size ? size : 1);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t size) { return cudaHostAlloc(p, size, 0); }
cudaError_t cudaFreeHost(void *p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *symbol) {
    static std::map<std::pair<int, const void *>, void *> at;
    void *&a = at[{g_device, symbol}];
    if (!a) a = calloc(1, 16 << 20);
    *p = a;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(struct cudaPointerAttributes *a, const void *p) {
    std::lock_guard<std::recursive_mutex> lk(g_mu);
    memset(a, 0, sizeof *a);
    const Block *b = find(p);
    a->type = b ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    a->device = b ? b->device : -2;
    a->devicePointer = b ? (void *)p : nullptr;
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *dst, const void *src, size_t n, enum cudaMemcpyKind) { return copy("copy", dst, src, n); }
cudaError_t cudaMemcpyAsync(void *dst, const void *src, size_t n, enum cudaMemcpyKind, cudaStream_t) {
    return copy("copy", dst, src, n);
}
cudaError_t cudaMemcpy2D(void *dst, size_t dp, const void *src, size_t sp, size_t w, size_t h, enum cudaMemcpyKind) {
    for (size_t i = 0; i < h; ++i) memmove((char *)dst + i * dp, (const char *)src + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return cudaMemset(p, v, n); }

cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
// (shorter at each call: a tuner's last candidate wins)
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    static int calls = 0;
    *ms = 1.f / (float)++calls;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) { return handle(x); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    free(x);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    free(g);
    return cudaSuccess;
}
}
