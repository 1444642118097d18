// A CUDA runtime without a GPU: the library's objects are linked against it, so
// that the host side (allocations, lists, graphs, error paths) runs on the CPU.
// Device memory is host memory, kernels are recorded and not run.  A call can
// be made to fail (fake_fail), and a launch that names memory which is not
// allocated, or a work list with an instance that is not there, counts as a
// violation.
#include <cuda_runtime_api.h>

#include <cstring>
#include <cstdlib>
#include <map>
#include <string>
#include <vector>

#include "sfg_internal.h"

namespace {

std::map<const char*, size_t> g_live;           // allocations by address
std::map<const char*, int> g_device;            // allocations of another device
std::map<const void*, std::string> g_names;     // host stub -> device name
struct Fail {
    int skip, times;
};
std::map<std::string, Fail> g_fail;             // call -> calls to let pass, then to fail
const double* g_residual = nullptr;             // StageView::r of the last tile or sweep
int g_violations = 0, g_capturing = 0, g_tiles = 0;
std::string g_violation;
cudaError_t g_last = cudaSuccess;
dim3 g_grid, g_block;
size_t g_smem;
cudaStream_t g_stream;

struct Launch {
    std::string name;
    std::vector<const char*> p;  // the leading pointer arguments of a batch kernel
};
struct Graph {
    std::vector<Launch> launches;
};
Graph* g_graph = nullptr;

cudaError_t failing(const char* call) {
    auto it = g_fail.find(call);
    if (it == g_fail.end() || it->second.times == 0) return cudaSuccess;
    if (it->second.skip-- > 0) return cudaSuccess;
    --it->second.times;
    g_last = cudaErrorMemoryAllocation;
    return g_last;
}

bool live(const void* p, size_t bytes) {
    auto it = g_live.upper_bound((const char*)p);
    if (it == g_live.begin()) return false;
    --it;
    return (const char*)p + bytes <= it->first + it->second;
}

void violation(const std::string& what) {
    ++g_violations;
    if (g_violation.empty()) g_violation = what;
}

// batch_*_kernel(inst, items, ctl, ...): the list must be there and name
// instances that are.
void check(const Launch& l) {
    if (l.p.empty()) return;
    const int* ctl = (const int*)l.p[2];
    if (!live(ctl, 2 * sizeof(int))) return violation(l.name + ": control block not allocated");
    const bool laws = l.name.find("batch_law") != std::string::npos;
    const int n = laws ? ctl[4] : ctl[0], n_inst = ctl[1];
    if (!laws) g_tiles = n;
    if (n == 0) return;
    const int* items = (const int*)l.p[1];
    if (!live(items, 16 * (size_t)n)) return violation(l.name + ": list not allocated");
    for (int i = 0; i < n; ++i)
        if (items[4 * i] < 0 || items[4 * i] >= n_inst) return violation(l.name + ": list names no instance");
}

}  // namespace

#define API extern "C" __attribute__((visibility("default")))

API void fake_fail(const char* call, int skip, int times) { g_fail[call] = {skip, times}; }
API void* fake_alloc(size_t bytes, int device) {
    void* p = nullptr;
    cudaMalloc(&p, bytes);
    if (device) g_device[(char*)p] = device;
    return p;
}
API const void* fake_residual() { return g_residual; }
API int fake_violations() { return g_violations; }
API const char* fake_violation() { return g_violation.c_str(); }
API int fake_tiles() { return g_tiles; }  // of the last batch stage launched
API void fake_reset() {
    g_fail.clear();
    g_violations = g_tiles = 0;
    g_violation.clear();
    g_last = cudaSuccess;
}

extern "C" {

void** __cudaRegisterFatBinary(void*) {
    static void* handle;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    g_names[host] = name;
}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, cudaStream_t st) {
    g_grid = grid, g_block = block, g_smem = smem, g_stream = st;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* smem, void* st) {
    *grid = g_grid, *block = g_block, *smem = g_smem, *(cudaStream_t*)st = g_stream;
    return cudaSuccess;
}

cudaError_t cudaLaunchKernel(const void* func, dim3, dim3, void** args, size_t, cudaStream_t) {
    if (cudaError_t e = failing("cudaLaunchKernel")) return e;
    Launch l{g_names[func], {}};
    for (const char* k : {"tile1d_kernel", "tile2d_kernel", "sweep_x", "sweep_yz"})
        if (l.name.find(k) != std::string::npos) g_residual = ((const sfg::StageView*)args[1])->r;
    for (const char* k : {"batch_stage_kernel", "batch_copy_kernel", "batch_law_kernel"})
        if (l.name.find(k) != std::string::npos)
            for (int i = 0; i < 3; ++i) l.p.push_back(*(const char**)args[i]);
    if (g_capturing) g_graph->launches.push_back(l);
    else check(l);
    return cudaSuccess;
}

cudaError_t cudaMalloc(void** p, size_t n) {
    *p = nullptr;
    if (cudaError_t e = failing("cudaMalloc")) return e;
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    memset(*p, 0xa5, n);
    g_live[(char*)*p] = n;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    if (!p) return cudaSuccess;
    if (!g_live.erase((char*)p)) violation("cudaFree of memory that is not allocated");
    else free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void** p, size_t n) { return (*p = calloc(1, n)) ? cudaSuccess : cudaErrorMemoryAllocation; }
cudaError_t cudaFreeHost(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind kind) {
    if (cudaError_t e = failing("cudaMemcpy")) return e;
    if (((kind == cudaMemcpyHostToDevice || kind == cudaMemcpyDeviceToDevice) && !live(d, n)) ||
        ((kind == cudaMemcpyDeviceToHost || kind == cudaMemcpyDeviceToDevice) && !live(s, n)))
        return g_last = cudaErrorInvalidValue;
    memmove(d, s, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind kind, cudaStream_t) {
    return g_capturing ? cudaSuccess : cudaMemcpy(d, s, n, kind);
}
cudaError_t cudaMemsetAsync(void* d, int v, size_t n, cudaStream_t) {
    if (!live(d, n)) violation("memset of memory that is not allocated");
    else memset(d, v, n);
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static void* image = nullptr;
    if (!image) cudaMalloc(&image, 16 << 20), memset(image, 0, 16 << 20);
    *p = image;
    return cudaSuccess;
}

cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
    *a = {};
    a->type = live(p, 1) ? cudaMemoryTypeDevice : cudaMemoryTypeUnregistered;
    if (live(p, 1)) {
        auto it = g_device.find((--g_live.upper_bound((const char*)p))->first);
        a->device = it == g_device.end() ? 0 : it->second;
    }
    return cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    if (cudaError_t e = failing("cudaStreamBeginCapture")) return e;
    g_capturing = 1;
    g_graph = new Graph;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* g) {
    g_capturing = 0;
    *g = (cudaGraph_t)g_graph;
    return failing("cudaStreamEndCapture");
}
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
    *s = cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* x, cudaGraph_t g, unsigned long long) {
    if (cudaError_t e = failing("cudaGraphInstantiate")) return e;
    *x = (cudaGraphExec_t) new Graph(*(Graph*)g);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    delete (Graph*)g;
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    delete (Graph*)x;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    for (const Launch& l : ((Graph*)x)->launches) check(l);
    return cudaSuccess;
}

__attribute__((visibility("default"))) cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaGetDevice(int* d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    *s = (cudaStream_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
    free(s);
    return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
    *e = (cudaEvent_t)malloc(1);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t e) {
    free(e);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
    *ms = 0.f;
    return cudaSuccess;
}

}  // extern "C"
