// A stand-in for the CUDA runtime, linked with the library's objects in place of libcudart, so that
// the host side of every entry point (order of calls, streams, error paths, allocation limits)
// runs on a machine without a GPU. Device memory is address space only: nothing reads or
// writes it, and kernels do not run. Calls are written to a log; a rule can refuse an allocation or
// a launch.
#include <cstdio>
#include <cstring>
#include <map>
#include <string>
#include <vector>

#include <cuda_runtime.h>
#undef cudaGetDriverEntryPointByVersion

namespace {
std::map<const void*, std::string> kernels;  // host stub -> device name
std::string text;
size_t limit = ~(size_t)0, held = 0;
std::map<void*, size_t> blocks;
std::string refuse_kernel;
int refuse_status = 0;
cudaError_t last = cudaSuccess;
dim3 cfg_grid, cfg_block;
size_t cfg_smem;
cudaStream_t cfg_stream;

cudaError_t answer(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
void note(const char* what, const void* a, size_t n, const void* stream) {
    char s[256];
    std::snprintf(s, sizeof s, "%s %llx %zu %llx\n", what, (unsigned long long)a, n, (unsigned long long)stream);
    text += s;
}
cudaError_t launch(const void* f, cudaStream_t st, void** args) {
    const std::string name = kernels.count(f) ? kernels[f] : "?";
    // the list counts: what the sensor clears (its last argument, unsigned*), what the lists are made with
    if (name.find("k_sensorILb0E") != std::string::npos && name.substr(name.size() - 2) == "Pj")
        note("clears", *(void**)args[4], 0, st);
    if (name.find("k_weno_list") != std::string::npos) note("counts", ((void**)args[2])[1], 0, st);
    const bool no = !refuse_kernel.empty() && name.find(refuse_kernel) != std::string::npos;
    note((std::string(no ? "refused:" : "launch:") + name).c_str(), nullptr, 0, st);
    return answer(no ? (cudaError_t)refuse_status : cudaSuccess);
}
}  // namespace

extern "C" {
// ---- the test's side
void fake_reset() { text.clear(); limit = ~(size_t)0; refuse_kernel.clear(); last = cudaSuccess; }
void fake_limit(size_t bytes) { limit = bytes; }  // device memory in all
void fake_refuse(const char* kernel, int status) { refuse_kernel = kernel; refuse_status = status; }
const char* fake_log() { return text.c_str(); }
size_t fake_held() { return held; }

// ---- what the compiler's host stubs call
void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    kernels[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t st) {
    cfg_grid = g; cfg_block = b; cfg_smem = smem; cfg_stream = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    *g = cfg_grid; *b = cfg_block; *smem = cfg_smem; *(cudaStream_t*)st = cfg_stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3, dim3, void** a, size_t, cudaStream_t st) { return launch((const void*)k, st, a); }

// ---- the runtime
cudaError_t cudaMalloc(void** p, size_t n) {
    static unsigned long long next = 0x700000000000ull;
    if (n > limit || held > limit - n) {
        note("refused:malloc", nullptr, n, nullptr);
        *p = nullptr;
        return answer(cudaErrorMemoryAllocation);
    }
    *p = (void*)next;
    next += (n + 0xfffff) & ~0xfffffull;
    blocks[*p] = n;
    held += n;
    note("malloc", *p, n, nullptr);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (p) { held -= blocks[p]; blocks.erase(p); note("free", p, 0, nullptr); }
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int, size_t n) { note("memset", p, n, nullptr); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int, size_t n, cudaStream_t st) { note("memset", p, n, st); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void* d, const void*, size_t n, cudaMemcpyKind, cudaStream_t st) { note("memcpy", d, n, st); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t st) { note("sync", nullptr, 0, st); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { note("sync-device", nullptr, 0, nullptr); return cudaSuccess; }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) { return launch(f, c->stream, a); }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t) { return "stand-in error"; }
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) { *n = 4; return cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void** f, unsigned, unsigned long long, cudaDriverEntryPointQueryResult*) {
    *f = nullptr;
    return cudaErrorNotSupported;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = (void*)0x600000000000ull; return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = nullptr; return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { *g = nullptr; return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t, unsigned long long) { *x = (cudaGraphExec_t)1; return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t st) { note("graph", nullptr, 0, st); return cudaSuccess; }
}
