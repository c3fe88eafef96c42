// Stand-in for the CUDA runtime (LD_PRELOAD): no device, every call succeeds and is logged, copies and
// sets act on host memory at once.  Lets a test read the order of a plan's copies, launches, events and
// waits on any host.  The calls are those that libpysit_gb300.so imports.
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::string log_;
std::map<const void*, std::string> names_;
struct Config { dim3 grid, block; size_t smem; cudaStream_t stream; } cfg_;
long next_ = 1;
cudaError_t last_ = cudaSuccess;

template <typename... A>
void say(const char* f, A... a) {
    char line[512];
    snprintf(line, sizeof line, f, a...);
    log_ += line;
    log_ += '\n';
}
const char* name(const void* f) {
    auto it = names_.find(f);
    return it == names_.end() ? "?" : it->second.c_str();
}
void launched(const void* f, dim3 g, dim3 b, size_t smem, cudaStream_t s, unsigned cluster) {
    say("launch %ld %s grid %u %u %u block %u smem %zu cluster %u", (long)s, name(f), g.x, g.y, g.z, b.x, smem, cluster);
}
}  // namespace

extern "C" {
const char* fake_log() { return log_.c_str(); }
void fake_clear() { log_.clear(); }

void** __cudaRegisterFatBinary(void*) { static void* h; return &h; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* dev, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names_[host] = dev;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) { *k = (cudaKernel_t)f; return cudaSuccess; }
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, cudaStream_t s) { cfg_ = {g, b, smem, s}; return 0; }
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* s) {
    *g = cfg_.grid; *b = cfg_.block; *smem = cfg_.smem; *(cudaStream_t*)s = cfg_.stream;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t smem, cudaStream_t s) {
    launched((const void*)k, g, b, smem, s, 0);
    return cudaSuccess;
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    unsigned cluster = 0;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
    launched(f, c->gridDim, c->blockDim, c->dynamicSmemBytes, c->stream, cluster);
    return cudaSuccess;
}
// FAKE_MAX_CLUSTER: the largest cluster that the stand-in device places (default 16)
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t* c) {
    const char* e = getenv("FAKE_MAX_CLUSTER");
    unsigned cluster = 1;
    for (unsigned i = 0; i < c->numAttrs; ++i)
        if (c->attrs[i].id == cudaLaunchAttributeClusterDimension) cluster = c->attrs[i].val.clusterDim.x;
    *n = (int)cluster <= (e ? atoi(e) : 16);
    say("query cluster %u", cluster);
    return cudaSuccess;
}
// FAKE_PORTABLE: the device takes no clusters of more than eight blocks
cudaError_t cudaFuncSetAttribute(const void*, enum cudaFuncAttribute a, int) {
    return a == cudaFuncAttributeNonPortableClusterSizeAllowed && getenv("FAKE_PORTABLE") ? last_ = cudaErrorInvalidValue
                                                                                         : cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)(1000 + next_++); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) { say("sync %ld", (long)s); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { say("wait %ld %ld", (long)s, (long)e); return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, enum cudaStreamCaptureMode) { return cudaErrorNotSupported; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaErrorNotSupported; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaErrorNotSupported; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaErrorNotSupported; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)(5000 + next_++); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { say("record %ld %ld", (long)s, (long)e); return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
// FAKE_MS: comma-separated times that consecutive calls report, the last one repeated (default 1)
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    static const char* at = getenv("FAKE_MS");
    *ms = at ? strtof(at, nullptr) : 1.0f;
    if (const char* c = at ? strchr(at, ',') : nullptr) at = c + 1;
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, enum cudaMemcpyKind, cudaStream_t st) {
    memmove(d, s, n);
    say("memcpy %ld %zu", (long)st, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t st) {
    memset(d, v, n);
    say("memset %ld %zu", (long)st, n);
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = last_;
    last_ = cudaSuccess;
    return e;
}
const char* cudaGetErrorName(cudaError_t) { return "fake"; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetSymbolAddress(void**, const void*) { return cudaErrorNotSupported; }
cudaError_t cudaGetDriverEntryPointByVersion(const char*, void**, unsigned, unsigned long long,
                                             enum cudaDriverEntryPointQueryResult*) { return cudaErrorNotSupported; }
}
