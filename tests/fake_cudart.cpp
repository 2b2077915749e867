// A CUDA runtime without a device, for tests of the host code: linked with the library's own
// objects instead of libcudart.  Memory is host memory, kernels do not run; every launch is
// recorded, and a test can have a call fail, set the devices' memory or add a device.
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Launch {
    std::string name;
    unsigned grid, block;
    size_t smem;
    int device;
};
struct Kernel {
    std::string name;
    size_t opted[8];  // dynamic shared memory a device was opted in for
};
std::map<const void*, Kernel> kernels;
std::map<void*, size_t> blocks;
std::vector<Launch> launches;
size_t total_memory = 280ull << 30, used_memory = 0;
int device = 0, attribute_calls = 0;
std::string fail_name;  // the call, or part of a kernel's name, that fails, fail_count times
int fail_count = 0;
cudaError_t last_error = cudaSuccess;
dim3 pushed_grid, pushed_block;
size_t pushed_smem;
cudaStream_t pushed_stream;

cudaError_t result(cudaError_t e) {
    if (e != cudaSuccess) last_error = e;
    return e;
}
bool failing(const char* what) {
    if (fail_count <= 0 || !strstr(what, fail_name.c_str())) return false;
    fail_count--;
    return true;
}
cudaError_t launch(const void* f, dim3 grid, dim3 block, size_t smem) {
    Kernel& k = kernels[f];
    if (failing(k.name.c_str())) return result(cudaErrorLaunchFailure);
    if (smem > 48u * 1024u && smem > k.opted[device]) return result(cudaErrorInvalidValue);
    launches.push_back({k.name, grid.x * grid.y * grid.z, block.x * block.y * block.z, smem, device});
    return cudaSuccess;
}
}  // namespace

extern "C" {
// what a test sets and reads
void fake_fail(const char* call, int times) { fail_name = call; fail_count = times; }
void fake_memory(size_t total) { total_memory = total; }
size_t fake_used() { return used_memory; }
int fake_attribute_calls() { return attribute_calls; }
void fake_clear() { launches.clear(); }
int fake_launches() { return (int)launches.size(); }
const char* fake_launch(int i, unsigned* grid, unsigned* block, size_t* smem, int* dev) {
    const Launch& l = launches[i];
    *grid = l.grid; *block = l.block; *smem = l.smem; *dev = l.device;
    return l.name.c_str();
}

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels[f] = Kernel{name, {}};
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t s) {
    pushed_grid = grid; pushed_block = block; pushed_smem = smem; pushed_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* s) {
    *grid = pushed_grid; *block = pushed_block; *smem = pushed_smem; *(cudaStream_t*)s = pushed_stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void**, size_t smem, cudaStream_t) {
    return launch((const void*)k, grid, block, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return launch(f, c->gridDim, c->blockDim, c->dynamicSmemBytes);
}

cudaError_t cudaGetLastError() { const cudaError_t e = last_error; last_error = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int* d) { *d = device; return cudaSuccess; }
cudaError_t cudaSetDevice(int d) { device = d; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) {
    attribute_calls++;
    if (failing("cudaFuncSetAttribute")) return result(cudaErrorUnknown);
    kernels[f].opted[device] = (size_t)v;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int threads, size_t smem, unsigned) {
    if (failing("cudaOccupancy")) return result(cudaErrorUnknown);
    const int by_smem = (int)((227u * 1024u) / (smem + 1024u)), by_regs = 65536 / (64 * threads);
    *n = by_smem < by_regs ? by_smem : by_regs;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int threads, size_t smem) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, threads, smem, 0);
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
    *p = nullptr;
    if (failing("cudaMalloc") || used_memory + bytes > total_memory || !(*p = calloc(bytes ? bytes : 1, 1)))
        return result(cudaErrorMemoryAllocation);
    blocks[*p] = bytes;
    used_memory += bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p) { used_memory -= blocks[p]; blocks.erase(p); free(p); }
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) { *p = calloc(bytes, 1); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { *t = total_memory; *f = total_memory - used_memory; return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemset(void* d, int v, size_t n) { memset(d, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    if (n > 65536 && v == 0) return cudaSuccess;  // (cudaMalloc's memory is zero, and stays untouched)
    memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static char buf[1 << 16]; *p = buf; return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return result(cudaErrorNotSupported); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return result(cudaErrorNotSupported); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return result(cudaErrorNotSupported); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return result(cudaErrorNotSupported); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }
}
