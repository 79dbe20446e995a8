// A CUDA runtime on the CPU for tests of the library's host code: device memory is host memory, kernels are not
// run but recorded (name, grid, block), streams and events do nothing.  Linked with the library's own object files
// in place of the CUDA runtime (tests/_fake_gpu.py).  What a test sets: which host memory is page-locked, how much
// device memory there is, whether cooperative launches are refused.
#include <cuda_runtime_api.h>
#include <driver_types.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <string>
#include <vector>

namespace {
struct Rec {
    std::string name;
    unsigned grid, block;
};
std::map<const void*, std::string>& names() {
    static std::map<const void*, std::string> m;
    return m;
}
std::vector<Rec> recs;
std::map<char*, size_t> pinned;          // page-locked ranges
std::map<void*, size_t> device;          // device allocations
size_t used = 0, room = (size_t)1 << 40;  // bytes of device memory
cudaError_t last = cudaSuccess, refuse_coop = cudaSuccess;
int sms = 152;
bool clearing = false;   // a memset on the null stream that nothing has waited for
bool marked = false;     // ... with an event behind it
int early = 0;           // launches while it may still run
std::vector<cudaLaunchConfig_t> configs;

cudaError_t ret(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
cudaError_t record(const void* f, dim3 g, dim3 b) {
    auto it = names().find(f);
    early += clearing;
    recs.push_back({it == names().end() ? "?" : it->second, g.x * g.y * g.z, b.x * b.y * b.z});
    return cudaSuccess;
}
int token;   // every handle
}  // namespace

extern "C" {
// ---- the test's side
void fake_clear() { recs.clear(); }
int fake_launches() { return (int)recs.size(); }
const char* fake_launch(int i, unsigned* grid, unsigned* block) {
    *grid = recs[i].grid;
    *block = recs[i].block;
    return recs[i].name.c_str();
}
void fake_pin(void* p, size_t n) { pinned[(char*)p] = n; }
void fake_unpin(void* p) { pinned.erase((char*)p); }
void fake_room(size_t bytes) { room = used + bytes; }
void fake_refuse_cooperative(int e) { refuse_coop = (cudaError_t)e; }
int fake_pending_error() { return (int)last; }
int fake_early_launches() { return early; }

// ---- module registration and launches
void** __cudaRegisterFatBinary(void*) { return (void**)&token; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    names()[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t smem, void* st) {
    cudaLaunchConfig_t c = {};
    c.gridDim = g;
    c.blockDim = b;
    c.dynamicSmemBytes = smem;
    c.stream = (cudaStream_t)st;
    configs.push_back(c);
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* smem, void* st) {
    const cudaLaunchConfig_t c = configs.back();
    configs.pop_back();
    *g = c.gridDim;
    *b = c.blockDim;
    *smem = c.dynamicSmemBytes;
    *(cudaStream_t*)st = c.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* k, const void* f) {
    *k = (cudaKernel_t)f;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 g, dim3 b, void**, size_t, cudaStream_t) { return record(k, g, b); }
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void**, size_t, cudaStream_t) { return record(f, g, b); }
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void**) {
    return record(f, c->gridDim, c->blockDim);
}
cudaError_t cudaLaunchCooperativeKernel(const void* f, dim3 g, dim3 b, void**, size_t, cudaStream_t) {
    return refuse_coop != cudaSuccess ? ret(refuse_coop) : record(f, g, b);
}

// ---- device
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr a, int) {
    *v = a == cudaDevAttrMultiProcessorCount ? sms : 1;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t smem, unsigned) {
    return *n = smem > 113 * 1024 ? 1 : 2, cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static void* scratch = calloc(1, 8 << 20);
    return *p = scratch, cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake"; }

// ---- memory
cudaError_t cudaMalloc(void** p, size_t n) {
    if (used + n > room) return ret(cudaErrorMemoryAllocation);
    *p = calloc(n ? n : 1, 1);
    device[*p] = n;
    used += n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    auto it = device.find(p);
    if (it == device.end()) return p ? ret(cudaErrorInvalidValue) : cudaSuccess;
    used -= it->second;
    device.erase(it);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) {
    *p = calloc(n + 64, 1);   // (room for a test that reaches beyond)
    pinned[(char*)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return cudaMallocHost(p, n); }
cudaError_t cudaFreeHost(void* p) {
    if (!pinned.erase((char*)p)) return ret(cudaErrorInvalidValue);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    std::memset(a, 0, sizeof(*a));
    a->type = cudaMemoryTypeUnregistered;
    for (auto& q : pinned)
        if ((char*)p >= q.first && (char*)p < q.first + q.second) {
            a->type = cudaMemoryTypeHost;
            a->devicePointer = a->hostPointer = (void*)p;
        }
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    clearing = false;
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpy2DAsync(void* d, size_t dp, const void* s, size_t sp, size_t w, size_t h, cudaMemcpyKind,
                              cudaStream_t) {
    for (size_t r = 0; r < h; ++r) std::memcpy((char*)d + r * dp, (const char*)s + r * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* d, int v, size_t n) {
    clearing = true;
    marked = false;
    return std::memset(d, v, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) { return std::memset(d, v, n), cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t* f, size_t* t) { return *f = room - used, *t = room, cudaSuccess; }

// ---- streams, events, graphs (what is captured is recorded once, at the capture; no conditional nodes)
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = (cudaStream_t)&token, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (!s) clearing = false;   // (the library's own streams do not wait for the null stream)
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) {
    if (marked) clearing = false;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)&token, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t s) {
    marked |= !s;
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) { return *g = (cudaGraph_t)&token, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    return *e = (cudaGraphExec_t)&token, cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t fake_unsupported() { return ret(cudaErrorNotSupported); }
}
#define UNSUPPORTED(name) asm(".globl " #name "\n.set " #name ", fake_unsupported")
UNSUPPORTED(cudaGraphAddNode);
UNSUPPORTED(cudaGraphConditionalHandleCreate);
UNSUPPORTED(cudaStreamBeginCaptureToGraph);
UNSUPPORTED(cudaStreamGetCaptureInfo);
UNSUPPORTED(cudaStreamUpdateCaptureDependencies);
