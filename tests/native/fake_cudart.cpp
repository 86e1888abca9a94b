// A CUDA runtime without a device, for host-side tests: linked with the
// library's own objects in place of the CUDA runtime, it keeps "device" memory
// on the heap, runs copies and memsets where they are issued (or, captured, when
// their graph is launched), launches no kernel, and logs every operation with its stream.
// A test can have it refuse cooperative launches and place a pointer on another
// device.  One host thread; a capture takes the operations of every stream.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <string>
#include <vector>

namespace {

struct Op {
    std::string text;
    std::function<void()> run;
    bool cooperative;
};
struct Graph {
    std::vector<Op> ops;
};
struct Config {
    dim3 grid, block;
    size_t smem;
    cudaStream_t stream;
};

std::string g_log;
std::map<const void *, std::string> g_kernels;          // host stub -> kernel name
std::map<const void *, std::pair<size_t, int>> g_memory;  // device range -> bytes, device
std::vector<Config> g_configs;
Graph *g_capture = nullptr;
cudaError_t g_last = cudaSuccess;
// cooperative launches: 0 accepted, 1 refused when issued, 2 refused when their
// graph is launched, 3 refused when issued, which also invalidates the capture
int g_refuse = 0;
bool g_invalidated = false;

cudaError_t set(cudaError_t e) {
    if (e != cudaSuccess) g_last = e;
    return e;
}

cudaError_t issue(const std::string &text, cudaStream_t s, std::function<void()> run = {}, bool cooperative = false) {
    char line[64];
    std::snprintf(line, sizeof line, " stream=%p", static_cast<void *>(s));
    Op op{text + line, run, cooperative};
    if (g_capture) {
        g_capture->ops.push_back(op);
        return cudaSuccess;
    }
    g_log += op.text + "\n";
    if (op.run) op.run();
    return cudaSuccess;
}

std::string hex(const void *p) {
    char b[32];
    std::snprintf(b, sizeof b, "%p", p);
    return b;
}

void *handle() { return std::malloc(1); }

}  // namespace

extern "C" {

const char *fake_log() { return g_log.c_str(); }
void fake_clear_log() { g_log.clear(); }
void fake_refuse_cooperative(int how) { g_refuse = how; }
// The range becomes memory of `device`, as a caller's own buffer there.
void fake_memory(const void *p, size_t bytes, int device) { g_memory[p] = {bytes, device}; }

// ------------------------------------------------------------ kernels
void **__cudaRegisterFatBinary(void *) {
    static void *h = nullptr;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, void *, void *, void *, void *,
                            int *) {
    g_kernels[host] = name;
}
void __cudaRegisterVar(void **, char *host, char *, const char *, int, size_t size, int, int) {
    g_memory[std::calloc(1, size)] = {size, 0};
    g_kernels[host] = "symbol";
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t smem, struct CUstream_st *stream) {
    g_configs.push_back({grid, block, smem, stream});
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    const Config c = g_configs.back();
    g_configs.pop_back();
    *grid = c.grid;
    *block = c.block;
    *smem = c.smem;
    *static_cast<cudaStream_t *>(stream) = c.stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *f, dim3, dim3, void **, size_t, cudaStream_t s) {
    return issue("kernel " + g_kernels[f], s);
}
cudaError_t cudaLaunchCooperativeKernel(const void *f, dim3, dim3, void **, size_t, cudaStream_t s) {
    if (g_refuse == 3) g_invalidated = g_capture != nullptr;
    if (g_refuse == 1 || g_refuse == 3) return set(cudaErrorCooperativeLaunchTooLarge);
    return issue("cooperative " + g_kernels[f], s, {}, true);
}
cudaError_t cudaFuncGetAttributes(cudaFuncAttributes *a, const void *) {
    std::memset(a, 0, sizeof *a);
    return cudaSuccess;
}
cudaError_t cudaFuncSetAttribute(const void *, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    *n = 2;
    return cudaSuccess;
}

// ------------------------------------------------------------ memory
cudaError_t cudaMalloc(void **p, size_t bytes) {
    *p = std::calloc(1, bytes);
    g_memory[*p] = {bytes, 0};
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    g_memory.erase(p);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) {
    *p = std::calloc(1, bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) {
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    std::memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeUnregistered;
    auto it = g_memory.upper_bound(p);
    if (it != g_memory.begin()) {
        --it;
        if (static_cast<const char *>(p) < static_cast<const char *>(it->first) + it->second.first) {
            a->type = cudaMemoryTypeDevice;
            a->device = it->second.second;
        }
    }
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    for (const auto &m : g_memory)
        if (m.second.first >= (1u << 22)) {  // the one large symbol
            *p = const_cast<void *>(m.first);
            return cudaSuccess;
        }
    return set(cudaErrorInvalidSymbol);
}
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind kind, cudaStream_t stream) {
    return issue("copy kind=" + std::to_string(kind) + " dst=" + hex(d) + " bytes=" + std::to_string(n), stream,
                 [=]() { std::memmove(d, s, n); });
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind kind) { return cudaMemcpyAsync(d, s, n, kind, nullptr); }
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t rows, cudaMemcpyKind kind,
                              cudaStream_t stream) {
    return issue("copy kind=" + std::to_string(kind) + " dst=" + hex(d) + " bytes=" + std::to_string(w * rows), stream, [=]() {
        for (size_t r = 0; r < rows; ++r) std::memmove(static_cast<char *>(d) + r * dp, static_cast<const char *>(s) + r * sp, w);
    });
}
cudaError_t cudaMemsetAsync(void *d, int v, size_t n, cudaStream_t stream) {
    return issue("set dst=" + hex(d) + " bytes=" + std::to_string(n), stream, [=]() { std::memset(d, v, n); });
}

// ------------------------------------------------------------ device, streams, events
cudaError_t cudaGetDevice(int *d) {
    *d = 0;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) {
    *v = 148;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int *lo, int *hi) {
    *lo = *hi = 0;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t) { return "error of the fake runtime"; }
cudaError_t cudaGetDriverEntryPointByVersion(const char *, void **fn, unsigned, unsigned long long,
                                             cudaDriverEntryPointQueryResult *r) {
    *fn = nullptr;
    if (r) *r = cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = static_cast<cudaStream_t>(handle());
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned flags, int) { return cudaStreamCreateWithFlags(s, flags); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
    *st = g_capture ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = static_cast<cudaEvent_t>(handle());
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }

// ------------------------------------------------------------ graphs
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    if (g_capture) return set(cudaErrorIllegalState);
    g_capture = new Graph;
    g_invalidated = false;
    return cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    *g = g_invalidated ? nullptr : reinterpret_cast<cudaGraph_t>(g_capture);
    g_capture = nullptr;
    return g_invalidated ? set(cudaErrorStreamCaptureInvalidated) : cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t g, unsigned long long) {
    *x = reinterpret_cast<cudaGraphExec_t>(new Graph(*reinterpret_cast<Graph *>(g)));
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t g) {
    delete reinterpret_cast<Graph *>(g);
    return cudaSuccess;
}
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t x) {
    delete reinterpret_cast<Graph *>(x);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t x, cudaStream_t) {
    const Graph *g = reinterpret_cast<Graph *>(x);
    for (const Op &op : g->ops)
        if (op.cooperative && g_refuse == 2) return set(cudaErrorCooperativeLaunchTooLarge);
    for (const Op &op : g->ops) {
        g_log += op.text + "\n";
        if (op.run) op.run();
    }
    return cudaSuccess;
}

}  // extern "C"
