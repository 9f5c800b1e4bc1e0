// The CUDA runtime calls that the library makes, on the host: memory is host memory, kernels do nothing, and what a
// device would refuse a launch for (more dynamic shared memory than the kernel has been allowed on THAT device) is
// refused.  Linked with the library's objects in place of the runtime, it shows what the host code asks for.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <utility>
#include <vector>

namespace {

constexpr int kDevices = 4, kSms = 148, kSmemOptin = 227 * 1024, kSmemDefault = 48 * 1024;

struct Launch {
    std::string kernel;
    int device;
    size_t smem;
    int ctas;
    bool programmatic;
};

// Kernels are registered by the constructors of other units: made when first used.
struct State {
    int device = 0;
    std::map<const void*, std::string> names;
    std::map<std::pair<const void*, int>, size_t> allowed;      // dynamic shared memory per kernel and device
    std::vector<Launch> launches;
    std::map<void*, size_t> blocks;
    size_t in_use = 0, memory = (size_t)8 << 30;
    size_t pushed = 0;                  // dynamic shared memory and grid of the launch in the making
    dim3 pushed_grid{1, 1, 1};
    int refused = 0;
};
State& S() {
    static State* s = new State;
    return *s;
}

cudaError_t launched(const void* f, dim3 grid, size_t smem, bool programmatic) {
    const auto a = S().allowed.find({f, S().device});
    if (smem > (a == S().allowed.end() ? (size_t)kSmemDefault : a->second)) {
        S().refused++;
        return cudaErrorInvalidValue;
    }
    S().launches.push_back({S().names[f], S().device, smem, (int)(grid.x * grid.y * grid.z), programmatic});
    return cudaSuccess;
}

CUresult encode_tiled(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                      CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    return CUDA_SUCCESS;
}

}  // namespace

extern "C" {

// ---- what tests ask --------------------------------------------------------------------------------
// Launches of kernels whose (mangled) name contains `part`; programmatic: 1 with the attribute, 0 without, -1 either.
int fake_launches(const char* part, int programmatic) {
    int n = 0;
    for (const Launch& l : S().launches)
        n += l.kernel.find(part) != std::string::npos && (programmatic < 0 || l.programmatic == (programmatic == 1));
    return n;
}
// Dynamic shared memory and CTAs of the last launch.
size_t fake_smem() { return S().launches.empty() ? 0 : S().launches.back().smem; }
int fake_ctas() { return S().launches.empty() ? 0 : S().launches.back().ctas; }
int fake_refused() { return S().refused; }
void fake_forget() { S().launches.clear(); S().refused = 0; }
size_t fake_in_use() { return S().in_use; }
void fake_memory(size_t bytes) { S().memory = bytes; }

// ---- registration ----------------------------------------------------------------------------------
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, void*, void*, void*, void*, int*) { S().names[f] = name; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3, size_t smem, struct CUstream_st*) { S().pushed_grid = grid; S().pushed = smem; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* stream) {
    *grid = S().pushed_grid;
    *block = dim3{1, 1, 1};
    *smem = S().pushed;
    *(void**)stream = nullptr;
    return cudaSuccess;
}

// ---- devices ---------------------------------------------------------------------------------------
cudaError_t cudaSetDevice(int d) {
    if (d < 0 || d >= kDevices) return cudaErrorInvalidDevice;
    S().device = d;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = S().device; return cudaSuccess; }
cudaError_t cudaGetDeviceProperties_v2(cudaDeviceProp* p, int) {
    memset(p, 0, sizeof *p);
    p->major = 10;
    p->multiProcessorCount = kSms;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? kSms : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? kSmemOptin : a == cudaDevAttrCooperativeLaunch;
    return cudaSuccess;
}
cudaError_t cudaDeviceCanAccessPeer(int* can, int, int) { *can = 0; return cudaSuccess; }
cudaError_t cudaDeviceEnablePeerAccess(int, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorInvalidValue ? "invalid argument" : e == cudaErrorMemoryAllocation ? "out of S().memory" : "error"; }
cudaError_t cudaGetDriverEntryPoint(const char* name, void** f, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *f = strcmp(name, "cuTensorMapEncodeTiled") ? nullptr : (void*)encode_tiled;
    if (q) *q = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}

// ---- S().memory ----------------------------------------------------------------------------------------
cudaError_t cudaMalloc(void** p, size_t n) {
    if (S().in_use + n > S().memory) return cudaErrorMemoryAllocation;
    *p = aligned_alloc(256, (n + 255) & ~(size_t)255);
    memset(*p, 0, n);
    S().blocks[*p] = n;
    S().in_use += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    const auto b = S().blocks.find(p);
    if (b == S().blocks.end()) return cudaErrorInvalidValue;
    S().in_use -= b->second;
    S().blocks.erase(b);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return (*p = calloc(1, n ? n : 1)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaMemcpy(void* to, const void* from, size_t n, cudaMemcpyKind) { memmove(to, from, n); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t n, cudaMemcpyKind, cudaStream_t) { memmove(to, from, n); return cudaSuccess; }
cudaError_t cudaMemcpyPeerAsync(void* to, int, const void* from, int, size_t n, cudaStream_t) { memmove(to, from, n); return cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { memset(p, v, n); return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) { memset(a, 0, sizeof *a); return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* s) { *p = const_cast<void*>(s); return cudaSuccess; }
cudaError_t cudaIpcGetMemHandle(cudaIpcMemHandle_t*, void*) { return cudaErrorNotSupported; }
cudaError_t cudaIpcOpenMemHandle(void**, cudaIpcMemHandle_t, unsigned) { return cudaErrorNotSupported; }
cudaError_t cudaIpcCloseMemHandle(void*) { return cudaErrorNotSupported; }

// ---- streams, events, graphs -----------------------------------------------------------------------
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)malloc(1); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { free(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)malloc(1); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t e) { free(e); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = (cudaGraph_t)malloc(1); return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { *x = (cudaGraphExec_t)malloc(1); return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) { free(g); return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) { free(x); return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

// ---- kernels ---------------------------------------------------------------------------------------
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
        if (v > kSmemOptin) return cudaErrorInvalidValue;
        S().allowed[{f, S().device}] = v;
    }
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void*, int, size_t) { *n = 1; return cudaSuccess; }
cudaError_t cudaLaunchKernel(const void* f, dim3 grid, dim3, void**, size_t smem, cudaStream_t) { return launched(f, grid, smem, false); }
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 grid, dim3, void**, size_t smem, cudaStream_t) { return launched(f, grid, smem, false); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    bool programmatic = false;
    for (unsigned i = 0; i < c->numAttrs; i++)
        programmatic |= c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization && c->attrs[i].val.programmaticStreamSerializationAllowed;
    return launched(f, c->gridDim, c->dynamicSmemBytes, programmatic);
}

}  // extern "C"
