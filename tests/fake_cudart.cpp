// The library on a CUDA runtime that runs nothing: device memory is host memory, and launches are logged by name.  For checks
// of what a call launches, on machines without a GPU.
#include "kernels.h"

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

static std::map<const void*, std::string> names;
static std::string log_text;

static cudaError_t launch(const void* f, dim3 grid, void** args) {
    const std::string& n = names[f];
    char line[96];
    std::snprintf(line, sizeof line, " %u %u %u", grid.x, grid.y, grid.z);
    log_text += n + line;
    if (n.find("lut_sparse_kernel") != std::string::npos) {   // split and early_trigger of SparseParams, behind its LutArgs
        const uint32_t* p = reinterpret_cast<const uint32_t*>(static_cast<const char*>(args[3]) + sizeof(lutamm::LutArgs));
        std::snprintf(line, sizeof line, " split=%u early=%u", p[1], p[8]);
        log_text += line;
    }
    log_text += "\n";
    return cudaSuccess;
}
static CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                       CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }
static CUresult attributes(unsigned int, CUpointer_attribute*, void** data, CUdeviceptr) {   // memory type, managed, ordinal
    *static_cast<unsigned int*>(data[0]) = CU_MEMORYTYPE_DEVICE;
    return CUDA_SUCCESS;
}

extern "C" {
const char* fake_log() { static std::string out; out.swap(log_text); log_text.clear(); return out.c_str(); }

cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void** args, size_t, cudaStream_t) { return launch(f, grid, args); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) { return launch(f, c->gridDim, args); }
static dim3 call_grid, call_block;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t, void*) { call_grid = g; call_block = b; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* s, void* st) { *g = call_grid; *b = call_block; *s = 0; *static_cast<void**>(st) = nullptr; return cudaSuccess; }
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, void*, void*, void*, void*, int*) { names[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) { std::memset(p, 0, sizeof *p); p->major = 10; p->multiProcessorCount = 148; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 148; return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned int) { *n = 8; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *f = std::strcmp(name, "cuTensorMapEncodeTiled") == 0 ? reinterpret_cast<void*>(encode) : std::strcmp(name, "cuPointerGetAttributes") == 0 ? reinterpret_cast<void*>(attributes) : nullptr;
    if (q) *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { std::memset(a, 0, sizeof *a); a->type = cudaMemoryTypeDevice; return cudaSuccess; }

cudaError_t cudaMalloc(void** p, size_t n) { *p = std::aligned_alloc(256, (n + 255) / 256 * 256); return *p ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFree(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) { *p = std::calloc(1, n); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { std::free(p); return cudaSuccess; }
cudaError_t cudaHostRegister(void*, size_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaHostGetDevicePointer(void** d, void* h, unsigned int) { *d = h; return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { static void* scratch = std::aligned_alloc(256, 16 << 20); *p = scratch; return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { std::memset(d, v, n); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) { *s = nullptr; return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.f; return cudaSuccess; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaErrorNotSupported; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned int) { return cudaErrorNotSupported; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaErrorNotSupported; }
}
