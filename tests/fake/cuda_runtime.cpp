// The CUDA runtime calls of the module's host code, without a GPU: device memory is host memory, streams
// and events do nothing, kernels are not run but listed (which one, its grid, its DevArgs). Linked with the module's own
// objects in place of libcudart, so that a test can let a call fail and see what the host code then
// launches, allocates and answers.
#include <cuda_runtime_api.h>
#include <cxxabi.h>
#include <stdint.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>
#include <vector>

extern "C" {
size_t fake_args_size();
void fake_args_read(const void *args, uint64_t *out6);
uint32_t *fake_args_suspend_count(const void *args);
}

namespace {

struct Launch {
    std::string name;
    dim3 grid, block;
    std::vector<unsigned char> args;   // DevArgs, if the kernel takes one
};
std::map<const void *, std::string> names;   // host stub -> kernel
std::vector<Launch> launches;
std::map<void *, size_t> blocks, stream_blocks;
size_t stream_bytes = 0, stream_peak = 0;
std::map<std::string, std::pair<int, int>> failing;   // call -> (calls that still succeed, error)
cudaError_t last = cudaSuccess;
dim3 cfg_grid, cfg_block;
size_t cfg_smem = 0;
cudaStream_t cfg_stream = nullptr;
size_t stack_limit = 1024;

cudaError_t answer(const char *call) {
    auto it = failing.find(call);
    if (it == failing.end() || it->second.first-- > 0) return cudaSuccess;
    last = (cudaError_t)it->second.second;
    failing.erase(it);
    return last;
}
template <class T> cudaError_t handle(T *out) {
    *out = (T)malloc(8);
    return cudaSuccess;
}

}   // namespace

extern "C" {

// ---- for the tests ----
void fake_reset_launches() { launches.clear(); }
void fake_reset_errors() {
    failing.clear();
    last = cudaSuccess;
}
uint32_t fake_launch_count() { return (uint32_t)launches.size(); }
const char *fake_launch_name(uint32_t i) { return launches[i].name.c_str(); }
// grid, block, lanes, resume, budget, drain, wait_polls of launch i, and its tables
void fake_launch_info(uint32_t i, uint64_t *out8) {
    const Launch &l = launches[i];
    memset(out8, 0, 8 * sizeof(uint64_t));
    out8[0] = l.grid.x;
    out8[1] = l.block.x;
    if (!l.args.empty()) fake_args_read(l.args.data(), out8 + 2);
}
// What the kernels would have parked: the next launch that is not a resume leaves `count` in its suspension list.
static uint32_t parked_by_next = 0;
void fake_park(uint32_t count) { parked_by_next = count; }
// The call after `after` more that succeed answers `error`, once.
void fake_fail(const char *call, int after, int error) { failing[call] = {after, error}; }
void fake_stream_bytes(uint64_t *now, uint64_t *peak) {
    *now = stream_bytes;
    *peak = stream_peak;
}

// ---- kernels ----
void **__cudaRegisterFatBinary(void *) { return (void **)malloc(8); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {
    int bad = 0;
    char *plain = abi::__cxa_demangle(name, nullptr, nullptr, &bad);
    names[host] = bad ? name : plain;
    free(plain);
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *stream) {
    cfg_grid = grid;
    cfg_block = block;
    cfg_smem = smem;
    cfg_stream = stream;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = cfg_grid;
    *block = cfg_block;
    *smem = cfg_smem;
    *(cudaStream_t *)stream = cfg_stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *host) {
    *k = (cudaKernel_t)host;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3 block, void **args, size_t, cudaStream_t) {
    Launch l;
    l.name = names[(const void *)k];
    l.grid = grid;
    l.block = block;
    if (l.name.find("DevArgs") != std::string::npos) {
        const unsigned char *a = (const unsigned char *)args[0];
        l.args.assign(a, a + fake_args_size());
        uint64_t v[6];
        fake_args_read(a, v);
        if (parked_by_next && !v[1] && fake_args_suspend_count(a)) {
            *fake_args_suspend_count(a) = parked_by_next;
            parked_by_next = 0;
        }
    }
    launches.push_back(l);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return answer("cudaFuncSetAttribute"); }
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    memset(a, 0, sizeof(*a));
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}

// ---- memory ----
cudaError_t cudaMalloc(void **p, size_t bytes) {
    *p = nullptr;
    if (cudaError_t e = answer("cudaMalloc")) return e;
    *p = aligned_alloc(256, (bytes + 255) / 256 * 256);
    blocks[*p] = bytes;
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    if (p && !blocks.erase(p)) abort();   // not an allocation of this runtime, or freed twice
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocAsync(void **p, size_t bytes, cudaStream_t) {
    *p = nullptr;
    if (cudaError_t e = answer("cudaMallocAsync")) return e;
    *p = aligned_alloc(256, (bytes + 255) / 256 * 256);
    stream_blocks[*p] = bytes;
    stream_bytes += bytes;
    if (stream_bytes > stream_peak) stream_peak = stream_bytes;
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void *p, cudaStream_t) {
    auto it = stream_blocks.find(p);
    if (it == stream_blocks.end()) abort();
    stream_bytes -= it->second;
    stream_blocks.erase(it);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void *to, const void *from, size_t n, cudaMemcpyKind) {
    if (cudaError_t e = answer("cudaMemcpy")) return e;
    memcpy(to, from, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *to, const void *from, size_t n, cudaMemcpyKind, cudaStream_t) {
    memcpy(to, from, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void *to, size_t tp, const void *from, size_t fp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    for (size_t r = 0; r < h; ++r) memcpy((char *)to + r * tp, (const char *)from + r * fp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void *p, int v, size_t n) {
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) {
    memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *free_b, size_t *total) {
    *free_b = *total = (size_t)280 << 30;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void *, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void *) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    *p = nullptr;
    return cudaErrorInvalidSymbol;
}

// ---- device, streams, events, graphs ----
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) {
    memset(p, 0, sizeof(*p));
    strcpy(p->name, "none");
    p->major = 10;
    p->minor = 3;
    p->multiProcessorCount = 152;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? 152 : a == cudaDevAttrMaxSharedMemoryPerBlockOptin ? 227 * 1024 : 0;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetLimit(size_t *v, cudaLimit) {
    *v = stack_limit;
    return cudaSuccess;
}
cudaError_t cudaDeviceSetLimit(cudaLimit, size_t v) {
    stack_limit = v;
    return cudaSuccess;
}
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return handle(s); }
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return handle(g); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) { return handle(e); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    free(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t e) {
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) { return handle(e); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return handle(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "error"; }

}   // extern "C"
