// fake_cudart.cpp — see fake_cudart.hpp.
#include "fake_cudart.hpp"

#include <cstdlib>
#include <cstring>

namespace fake {

static thread_local Launch pushed;

static cudaError_t done(cudaError_t e) {
    if (e != cudaSuccess) last_error = e;
    return e;
}
static cudaError_t launch(const void* f, dim3 g, dim3 b, void** args, size_t smem) {
    Launch l{names()[f], g, b, smem, args};
    return done(on_launch ? on_launch(l) : cudaSuccess);
}

}  // namespace fake

extern "C" {
void** __cudaRegisterFatBinary(void*) {
    static void* h = nullptr;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
    fake::names()[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st*) {
    fake::pushed.grid = g;
    fake::pushed.block = b;
    fake::pushed.smem = smem;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* stream) {
    *g = fake::pushed.grid;
    *b = fake::pushed.block;
    *smem = fake::pushed.smem;
    *static_cast<void**>(stream) = nullptr;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t smem,
                             cudaStream_t) {
    return fake::launch(f, g, b, args, smem);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return fake::launch(f, c->gridDim, c->blockDim, args, c->dynamicSmemBytes);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    const std::string& k = fake::names()[f];
    if (fake::on_attribute && fake::on_attribute(k) != cudaSuccess)
        return fake::done(cudaErrorInvalidValue);
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) fake::smem_limit[k].insert(v);
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::last_error;
    fake::last_error = cudaSuccess;
    return e;
}
cudaError_t cudaPeekAtLastError() { return fake::last_error; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "ok" : "refused"; }

cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t,
                                                                   unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
    *n = 15;
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    std::memset(a, 0, sizeof *a);
    a->ptxVersion = a->binaryVersion = 100;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static char scratch[16 << 20];
    *p = scratch;
    return cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = std::calloc(n ? n : 1, 1);
    return *p ? cudaSuccess : fake::done(cudaErrorMemoryAllocation);
}
cudaError_t cudaFree(void* p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMalloc(p, n); }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned) {
    *d = h;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    std::memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamQuery(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = nullptr;
    return cudaErrorNotSupported;
}
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaErrorNotSupported; }
}
