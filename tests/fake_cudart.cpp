// A CUDA runtime for host tests of the C-ABI's control flow: memory is host memory,
// launches are recorded and run nothing. Linked with the library's own objects in place
// of cudart (fake_cuda.py), it shows without a GPU what a call launches, what it
// allocates and what it leaves behind when an allocation fails.
#include <cuda_runtime_api.h>
#include <sys/mman.h>

#include <cstdint>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Launch {
    std::string name;
    unsigned grid[3], block[3];
};
std::vector<Launch> launches;
std::map<const void *, std::string> kernels;
std::map<void *, size_t> blocks;
int allocs_left = -1;      // allocations that still succeed (-1: all)
int64_t readback = -1;     // the value of 8-byte device-to-host copies (-1: memory's)
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
} config;
int dummy;

cudaError_t take(void **p, size_t n) {
    *p = nullptr;
    if (allocs_left == 0) return cudaErrorMemoryAllocation;
    if (allocs_left > 0) allocs_left--;
    void *m = mmap(nullptr, n ? n : 1, PROT_READ | PROT_WRITE, MAP_PRIVATE | MAP_ANONYMOUS | MAP_NORESERVE, -1, 0);
    if (m == MAP_FAILED) return cudaErrorMemoryAllocation;
    blocks[m] = n ? n : 1;
    *p = m;
    return cudaSuccess;
}
cudaError_t give(void *p) {
    auto it = blocks.find(p);
    if (it == blocks.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    munmap(p, it->second);
    blocks.erase(it);
    return cudaSuccess;
}
}  // namespace

extern "C" {
// the tests' controls
void fake_allocs_left(int n) { allocs_left = n; }
void fake_readback(int64_t v) { readback = v; }
void fake_clear_launches() { launches.clear(); }
int fake_launches() { return (int)launches.size(); }
const char *fake_launch(int i, unsigned *grid_x, unsigned *grid_y, unsigned *block_x) {
    *grid_x = launches[i].grid[0];
    *grid_y = launches[i].grid[1];
    *block_x = launches[i].block[0];
    return launches[i].name.c_str();
}

void **__cudaRegisterFatBinary(void *) { return reinterpret_cast<void **>(&dummy); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    kernels[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    config = Config{grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = config.grid;
    *block = config.block;
    *smem = config.smem;
    *static_cast<cudaStream_t *>(stream) = config.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3 g, dim3 b, void **, size_t, cudaStream_t) {
    launches.push_back(Launch{kernels[f], {g.x, g.y, g.z}, {b.x, b.y, b.z}});
    return cudaSuccess;
}

cudaError_t cudaMalloc(void **p, size_t n) { return take(p, n); }
cudaError_t cudaMallocHost(void **p, size_t n) { return take(p, n); }
cudaError_t cudaHostAlloc(void **p, size_t n, unsigned) { return take(p, n); }
cudaError_t cudaMallocManaged(void **p, size_t n, unsigned) { return take(p, n); }
cudaError_t cudaFree(void *p) { return give(p); }
cudaError_t cudaFreeHost(void *p) { return give(p); }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    if (kind == cudaMemcpyDeviceToHost && n == sizeof readback && readback >= 0) std::memcpy(d, &readback, n);
    else std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }

cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    return *n = 4, cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) { return *p = &dummy, cudaSuccess; }
const char *cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaPeekAtLastError() { return cudaSuccess; }

cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = reinterpret_cast<cudaEvent_t>(&dummy), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.f, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    return *g = reinterpret_cast<cudaGraph_t>(&dummy), cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    return *e = reinterpret_cast<cudaGraphExec_t>(&dummy), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
}
