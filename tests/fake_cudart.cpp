// A CUDA runtime without a device, for host tests: the library's objects linked with this file instead of
// the CUDA runtime. Device memory is host memory (more than 1 GB of it is only address space), launches are
// recorded with the kernel's name, grid and block, and the occupancy query can be made to fail.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Launch {
    std::string kernel;
    unsigned grid, block;
};
std::map<const void *, std::string> &names()
{
    static std::map<const void *, std::string> m;
    return m;
}
std::map<void *, size_t> sizes;
std::vector<Launch> launches;
int failing_queries = 0, failing_mallocs = 0;
cudaError_t last = cudaSuccess;
struct {
    dim3 grid, block;
    size_t shared;
    void *stream;
} pushed;

cudaError_t record(const void *f, dim3 grid, dim3 block)
{
    launches.push_back({ names()[f], grid.x, block.x });
    return cudaSuccess;
}
cudaError_t occupancy(int *blocks, const void *f)
{
    if (failing_queries > 0) {
        --failing_queries;
        return last = cudaErrorUnknown;
    }
    // the k17_pool_kernel instances with 32-bit slot offsets end in a true template argument
    *blocks = names()[f].find("Lb1EEEv") != std::string::npos ? 5 : 3;
    return cudaSuccess;
}
} // namespace

extern "C" {

void fake_fail_occupancy(int times) { failing_queries = times; }
void fake_fail_malloc(int times) { failing_mallocs = times; }
int fake_launches() { return (int)launches.size(); }
const char *fake_launch(int i, unsigned *grid, unsigned *block)
{
    const Launch &l = launches.at((size_t)i);
    *grid = l.grid;
    *block = l.block;
    return l.kernel.c_str();
}

void **__cudaRegisterFatBinary(void *) { static void *handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *, int *)
{
    names()[host] = name;
}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, void *stream)
{
    pushed = { grid, block, shared, stream };
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *shared, void *stream)
{
    *grid = pushed.grid;
    *block = pushed.block;
    *shared = pushed.shared;
    *static_cast<void **>(stream) = pushed.stream;
    return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void *f, dim3 grid, dim3 block, void **, size_t, cudaStream_t) { return record(f, grid, block); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t *c, const void *f, void **) { return record(f, c->gridDim, c->blockDim); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int *n, const void *f, int, size_t) { return occupancy(n, f); }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *f, int, size_t, unsigned) { return occupancy(n, f); }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n)
{
    if (failing_mallocs > 0) {
        --failing_mallocs;
        *p = nullptr;
        return last = cudaErrorMemoryAllocation;
    }
    const int access = n > (1ull << 30) ? PROT_NONE : PROT_READ | PROT_WRITE;
    *p = mmap(nullptr, n, access, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (*p == MAP_FAILED)
        return last = cudaErrorMemoryAllocation;
    sizes[*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p)
{
    if (p) {
        munmap(p, sizes[p]);
        sizes.erase(p);
    }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void *d, int v, size_t n) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }

cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char *cudaGetErrorString(cudaError_t) { return "an error of the fake runtime"; }
cudaError_t cudaGetDevice(int *d) { *d = 0; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) { *v = a == cudaDevAttrMultiProcessorCount ? 148 : 0; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *s) { *s = cudaStreamCaptureStatusNone; return cudaSuccess; }

// not used by these tests
cudaError_t cudaMemcpy2DAsync(void *, size_t, const void *, size_t, size_t, size_t, cudaMemcpyKind, cudaStream_t) { return last = cudaErrorNotSupported; }
cudaError_t cudaEventCreate(cudaEvent_t *) { return last = cudaErrorNotSupported; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *, cudaEvent_t, cudaEvent_t) { return last = cudaErrorNotSupported; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return last = cudaErrorNotSupported; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return last = cudaErrorNotSupported; }
cudaError_t cudaGetSymbolAddress(void **, const void *) { return last = cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *, cudaGraph_t, unsigned long long) { return last = cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return last = cudaErrorNotSupported; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return last = cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *) { return last = cudaErrorNotSupported; }
cudaError_t cudaIpcCloseMemHandle(void *) { return last = cudaErrorNotSupported; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t *, void *) { return last = cudaErrorNotSupported; }
cudaError_t cudaIpcOpenMemHandle(void **, cudaIpcMemHandle_t, unsigned) { return last = cudaErrorNotSupported; }

} // extern "C"
