// A libcudart.so.12 for host-side tests: it launches nothing and records what libdiffsoup_b200.so asks of the
// runtime, one line per call, with the checks that the real one makes of a launch's dynamic shared memory.
//   launch <stream> <chained> <smem> <kernel>   wait|record|memset|memcpy <stream>   limit <bytes> <kernel>
#include <cuda_runtime_api.h>

#include <cstdio>
#include <map>
#include <mutex>
#include <string>

namespace {

std::recursive_mutex mu;
std::string text;
std::map<const void*, std::string> names;
std::map<const void*, size_t> limits;
cudaError_t last = cudaSuccess;
size_t handles = 0x1000;
void (*before_launch)() = nullptr;

struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};
thread_local Config pushed;

void line(const char* what, cudaStream_t st) {
    std::lock_guard<std::recursive_mutex> l(mu);
    text += std::string(what) + " " + std::to_string((size_t)st) + "\n";
}

cudaError_t launch(const void* f, size_t smem, cudaStream_t st, bool chained) {
    if (auto call = before_launch) {  // what another thread might do between a call's set-up and its launch
        before_launch = nullptr;
        call();
    }
    std::lock_guard<std::recursive_mutex> l(mu);
    const auto at = limits.find(f);
    if (smem > (at == limits.end() ? 48 * 1024 : at->second)) return last = cudaErrorInvalidValue;
    text += "launch " + std::to_string((size_t)st) + (chained ? " 1 " : " 0 ") + std::to_string(smem) + " " + names[f] + "\n";
    return cudaSuccess;
}

}  // namespace

extern "C" {

// For the tests: the lines so far (cleared by the call), and a function called once before the next launch.
const char* fake_take() {
    static std::string out;
    std::lock_guard<std::recursive_mutex> l(mu);
    out.swap(text);
    text.clear();
    return out.c_str();
}
void fake_before_launch(void (*f)()) { before_launch = f; }

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* f, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names[f] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, struct CUstream_st* st) {
    pushed = Config{g, b, smem, st};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    *g = pushed.grid; *b = pushed.block; *smem = pushed.smem;
    *static_cast<cudaStream_t*>(st) = pushed.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3, dim3, void**, size_t smem, cudaStream_t st) {
    return launch(f, smem, st, false);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    bool chained = false;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        chained = chained || c->attrs[i].id == cudaLaunchAttributeProgrammaticStreamSerialization;
    return launch(f, c->dynamicSmemBytes, c->stream, chained);
}
cudaError_t cudaFuncSetAttribute(const void* f, cudaFuncAttribute a, int v) {
    std::lock_guard<std::recursive_mutex> l(mu);
    if (a != cudaFuncAttributeMaxDynamicSharedMemorySize) return cudaSuccess;
    if (v > 232448) return last = cudaErrorInvalidValue;
    limits[f] = (size_t)v;
    text += "limit " + std::to_string(v) + " " + names[f] + "\n";
    return cudaSuccess;
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes* a, const void*) {
    *a = cudaFuncAttributes{};
    a->numRegs = 64;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t smem, unsigned) {
    *n = smem > 0 ? (int)(232448 / smem) : 8;
    if (*n > 8) *n = 8;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* n, const void* f, int t, size_t smem) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(n, f, t, smem, 0);
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 148 : (a == cudaDevAttrMaxSharedMemoryPerMultiprocessor ? 233472 : 1024);
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaGetLastError() { const cudaError_t e = last; last = cudaSuccess; return e; }
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "invalid argument"; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) { *p = (void*)0x100000; return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)(handles += 16); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)(handles += 16); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t st) { line("record", st); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t st, cudaEvent_t, unsigned) { line("wait", st); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t st) { line("synchronize", st); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void*, int, size_t, cudaStream_t st) { line("memset", st); return cudaSuccess; }
cudaError_t cudaMemcpyAsync(void*, const void*, size_t, cudaMemcpyKind, cudaStream_t st) {
    line("memcpy", st);
    return cudaSuccess;
}

}  // extern "C"
