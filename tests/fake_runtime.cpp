// A CUDA runtime of two devices that runs nothing: what the one-token launches ask of it (linked with csrc/qgemv.cu's object, no GPU).
#include <cuda_runtime.h>

#include <cstring>
#include <map>
#include <utility>

#include "qgemm.cuh"

static int g_dev = 0, g_queries = 0, g_blocks = 0;
static size_t g_smem = 0;
static std::map<std::pair<int, const void*>, int> g_attr;      // (device, kernel) -> dynamic shared memory allowed there

extern "C" {
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char*, char*, const char*, int, uint3*, uint3*, dim3*, dim3*, int*) {}
unsigned __cudaPopCallConfiguration(dim3*, dim3*, size_t*, void*) { return 0; }

cudaError_t cudaGetDevice(int* d) { *d = g_dev; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int d) { g_queries++; *v = d ? 2 : 148; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute, int v) { g_attr[{g_dev, f}] = v; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    auto it = g_attr.find({g_dev, f});
    g_smem = c->dynamicSmemBytes;
    g_blocks = (int)c->gridDim.x;
    return c->dynamicSmemBytes <= (it == g_attr.end() ? 48u * 1024u : (size_t)it->second) ? cudaSuccess : cudaErrorInvalidValue;
}

void fake_device(int d) { g_dev = d; }
int fake_queries() { return g_queries; }
size_t fake_smem() { return g_smem; }
int fake_blocks() { return g_blocks; }
int fake_gemv(int format, unsigned K, unsigned N) {
    qg::GemmArgs a;
    memset(&a, 0, sizeof(a));
    a.format = format; a.X = a.W0 = (const void*)256; a.Y = (void*)256; a.M = 1; a.N = N; a.K = K;
    return (int)qg::launch_gemv(a, nullptr);
}
}
