// A CUDA runtime without a GPU: two devices that run nothing.  It keeps what a
// launch is judged by (the device, the kernel's shared-memory attribute there, the
// arguments) so that tests can look at how the library launches its kernels.
#include <map>
#include <string>
#include <utility>
#include <cstring>
#include <cuda_runtime_api.h>

namespace {
int device = 0;
cudaError_t last = cudaSuccess;
std::map<const void*, std::string> names;
std::map<std::pair<int, const void*>, int> shared;
struct Config { dim3 grid, block; size_t smem; cudaStream_t stream; };
Config pushed;
using Hook = void (*)(const char* name, int device, unsigned blocks, size_t smem, void** args);
Hook hook = nullptr;

cudaError_t done(cudaError_t e) { return e == cudaSuccess ? e : last = e; }

cudaError_t launch(const void* f, dim3 grid, size_t smem, void** args) {
    const auto it = shared.find({device, f});
    if (smem > size_t(it == shared.end() ? 48 * 1024 : it->second)) return done(cudaErrorInvalidValue);
    if (hook) hook(names[f].c_str(), device, grid.x * grid.y * grid.z, smem, args);
    return cudaSuccess;
}
}  // namespace

extern "C" {
void fake_hook(Hook h) { hook = h; }

void** __cudaRegisterFatBinary(void*) { static void* handle; return &handle; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t stream) {
    pushed = {grid, block, smem, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = pushed.grid, *block = pushed.block, *smem = pushed.smem;
    *static_cast<cudaStream_t*>(stream) = pushed.stream;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { return *d = device, cudaSuccess; }
cudaError_t cudaSetDevice(int d) { return d < 0 || d > 1 ? done(cudaErrorInvalidDevice) : (device = d, cudaSuccess); }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 2, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : a == cudaDevAttrComputeCapabilityMajor ? 10
         : a == cudaDevAttrMaxGridDimX ? 0x7fffffff : 0;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof(*a));
    a->binaryVersion = a->ptxVersion = 100;
    a->maxThreadsPerBlock = 1024;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (v > 227 * 1024) return done(cudaErrorInvalidValue);
        shared[{device, f}] = v;
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    return *n = 1, cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { return *n = 1, cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void** args, size_t smem, cudaStream_t) {
    return launch(f, grid, smem, args);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return launch(f, c->gridDim, c->dynamicSmemBytes, args);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3, void** args, size_t smem, cudaStream_t) {
    return launch(f, grid, smem, args);
}
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; return last = cudaSuccess, e; }
cudaError_t cudaPeekAtLastError() { return last; }
const char* cudaGetErrorString(cudaError_t) { return "refused by the test's runtime"; }
}
