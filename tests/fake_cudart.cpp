// A CUDA runtime for the library's host code on a machine without a GPU:
// device memory is host memory, copies are made at once, a kernel launch is a
// line in a log (k_sample_voxels and k_dm_count, whose output the host reads, are
// made here).  Allocations and device-to-host copies can be made to fail.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::map<const void*, std::string>& names()
{
    static std::map<const void*, std::string> n;
    return n;
}
std::string text;
int no_memory = 0;
size_t largest = ~(size_t)0;
unsigned jobs_each = 0;
size_t bad_read = 0;

void log(const char* what, const void* a, const std::string& b = "")
{
    char p[32];
    snprintf(p, sizeof(p), " %llx ", (unsigned long long)(uintptr_t)a);
    text += what + std::string(p) + b + "\n";
}

cudaError_t allocate(void** p, size_t n)
{
    if (no_memory || n > largest) return cudaErrorMemoryAllocation;
    *p = calloc(n ? n : 1, 1);
    return cudaSuccess;
}

cudaError_t copy(void* d, const void* s, size_t n, cudaMemcpyKind k)
{
    if (k == cudaMemcpyDeviceToHost && n == bad_read) return cudaErrorUnknown;
    memmove(d, s, n);
    return cudaSuccess;
}
}  // namespace

extern "C" {
const char* fake_log() { return text.c_str(); }
void fake_clear() { text.clear(); }
void fake_no_memory(int on) { no_memory = on; }
void fake_bad_read(size_t bytes) { bad_read = bytes; }
void fake_largest_allocation(size_t bytes) { largest = bytes; }
void fake_jobs_each(unsigned n) { jobs_each = n; }

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) { names()[host] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}

static dim3 call_grid, call_block;
static size_t call_shared;
static cudaStream_t call_stream;
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t sh, cudaStream_t s)
{
    call_grid = g; call_block = b; call_shared = sh; call_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* sh, void* s)
{
    *g = call_grid; *b = call_block; *sh = call_shared; *(cudaStream_t*)s = call_stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* host) { *k = (cudaKernel_t)host; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** a, size_t, cudaStream_t s)
{
    const std::string& name = names()[(const void*)k];
    log("launch", s, name);
    if (name.find("k_sample_voxels") != std::string::npos) {
        const uint16_t* vox = *(const uint16_t**)a[0];
        const size_t n = *(size_t*)a[1];
        const int step = *(int*)a[2];
        uint16_t* out = *(uint16_t**)a[3];
        for (size_t i = 0; i * step < n; i++) out[i] = vox[i * step];
    }
    /* (parameters, medium, window: (pixels, row, items, ..), jobs: seven arrays, total, ..) */
    if (name.find("k_dm_count") != std::string::npos) *((uint32_t**)a[3])[7] = jobs_each * ((uint32_t*)a[2])[2];
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** a, size_t sh, cudaStream_t s) { return __cudaLaunchKernel((cudaKernel_t)f, g, b, a, sh, s); }

cudaError_t cudaMalloc(void** p, size_t n) { return allocate(p, n); }
cudaError_t cudaMallocAsync(void** p, size_t n, cudaStream_t) { return allocate(p, n); }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { *p = calloc(n ? n : 1, 1); return cudaSuccess; }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaHostAlloc(p, n, 0); }
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind k) { return copy(d, s, n, k); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind k, cudaStream_t st) { log("copy", st); return copy(d, s, n, k); }
cudaError_t cudaMemcpy3DAsync(const cudaMemcpy3DParms* q, cudaStream_t st)
{
    log("copy", st);
    for (size_t z = 0; z < q->extent.depth; z++)
        for (size_t y = 0; y < q->extent.height; y++)
            memmove((char*)q->dstPtr.ptr + ((z + q->dstPos.z) * q->dstPtr.ysize + y + q->dstPos.y) * q->dstPtr.pitch + q->dstPos.x,
                    (const char*)q->srcPtr.ptr + (z * q->srcPtr.ysize + y) * q->srcPtr.pitch, q->extent.width);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) { log("set", s); memset(p, v, n); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorInvalidSymbol; }

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* p, int)
{
    memset(p, 0, sizeof(*p));
    strcpy(p->name, "no GPU");
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long, cudaDriverEntryPointQueryResult*) { return cudaErrorUnknown; }

cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)calloc(1, 1); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { log("record", s, std::to_string((uintptr_t)e)); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1.0f; return cudaSuccess; }

cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)calloc(1, 1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { log("synchronize", s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { log("wait", s, std::to_string((uintptr_t)e)); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)calloc(1, 1); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) { *e = (cudaGraphExec_t)calloc(1, 1); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t s) { log("graph", s); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) { free(e); return cudaSuccess; }
}
