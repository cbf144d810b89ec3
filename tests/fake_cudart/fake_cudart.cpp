// A CUDA runtime without a device, for tests of the library's host code: it
// is loaded in front of libcudart (LD_PRELOAD), keeps "device" memory on the
// host, runs no kernel, and notes every call that orders work as a line of
// text (fake_log).  Kernels therefore find and leave nothing; a test that
// needs a result puts it there in its callback (fake_on_event), which sees
// each line as it is written.
#include <cuda_runtime.h>

#include <cstdarg>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

namespace {
std::string g_log;
std::map<const void*, std::string> g_kernels;
void (*g_on_event)(const char*) = nullptr;
char g_fail[128];         // kernels whose name holds this fail to launch ("cudaMalloc": that call)
int g_device = 0;
cudaError_t g_last = cudaSuccess;
uintptr_t g_next = 1;
struct Config {
    dim3 grid, block;
    size_t shared;
    cudaStream_t stream;
} g_config;

void note(const char* format, ...) {
    char line[1024];
    va_list args;
    va_start(args, format);
    vsnprintf(line, sizeof(line), format, args);
    va_end(args);
    g_log += line;
    g_log += '\n';
    if (g_on_event) g_on_event(line);
}

const char* name_of(const void* kernel) {
    auto it = g_kernels.find(kernel);
    return it == g_kernels.end() ? "?" : it->second.c_str();
}

cudaError_t launch(const void* kernel, dim3 grid, dim3 block, cudaStream_t stream) {
    const char* name = name_of(kernel);
    if (g_fail[0] && strstr(name, g_fail)) return g_last = cudaErrorLaunchFailure;
    note("launch %p %s %u %u", (void*)stream, name, grid.x * grid.y * grid.z, block.x);
    return cudaSuccess;
}

const char* kind_of(cudaMemcpyKind kind) {
    return kind == cudaMemcpyHostToDevice ? "h2d" : kind == cudaMemcpyDeviceToHost ? "d2h" : "d2d";
}
}  // namespace

extern "C" {
const char* fake_log() { return g_log.c_str(); }
void fake_clear() { g_log.clear(); }
void fake_on_event(void (*f)(const char*)) { g_on_event = f; }
void fake_fail(const char* kernel) { snprintf(g_fail, sizeof(g_fail), "%s", kernel); }
void fake_set_device(int device) { g_device = device; }

void** __cudaRegisterFatBinary(void*) { return (void**)&g_log; }
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*, dim3*, dim3*, int*) {
    g_kernels[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t shared, cudaStream_t stream) {
    g_config = Config{grid, block, shared, stream};
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* grid, dim3* block, size_t* shared, void* stream) {
    *grid = g_config.grid;
    *block = g_config.block;
    *shared = g_config.shared;
    *(cudaStream_t*)stream = g_config.stream;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t* kernel, const void* host) {
    *kernel = (cudaKernel_t)host;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t kernel, dim3 grid, dim3 block, void**, size_t, cudaStream_t stream) {
    return launch((const void*)kernel, grid, block, stream);
}
cudaError_t cudaLaunchKernel(const void* kernel, dim3 grid, dim3 block, void**, size_t, cudaStream_t stream) {
    return launch(kernel, grid, block, stream);
}
cudaError_t cudaLaunchCooperativeKernel(const void* kernel, dim3 grid, dim3 block, void**, size_t, cudaStream_t stream) {
    return launch(kernel, grid, block, stream);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* config, const void* kernel, void**) {
    return launch(kernel, config->gridDim, config->blockDim, config->stream);
}

cudaError_t cudaMalloc(void** p, size_t bytes) {
    if (!strcmp(g_fail, "cudaMalloc")) {
        *p = nullptr;
        return g_last = cudaErrorMemoryAllocation;
    }
    *p = calloc(bytes ? bytes : 1, 1);
    note("malloc %p %zu", *p, bytes);
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    note("free %p", p);
    free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned) {
    *p = calloc(bytes, 1);
    note("host %p %zu", *p, bytes);
    return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
    free(p);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* to, const void* from, size_t bytes, cudaMemcpyKind kind) {
    note("copy %p %s %p %p %zu", (void*)nullptr, kind_of(kind), to, from, bytes);
    memcpy(to, from, bytes);
    if (kind == cudaMemcpyDeviceToHost) note("sync %p", (void*)nullptr);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* to, const void* from, size_t bytes, cudaMemcpyKind kind, cudaStream_t stream) {
    note("copy %p %s %p %p %zu", (void*)stream, kind_of(kind), to, from, bytes);
    memmove(to, from, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int value, size_t bytes) {
    note("set %p %p %zu", (void*)nullptr, p, bytes);
    memset(p, value, bytes);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int value, size_t bytes, cudaStream_t stream) {
    note("set %p %p %zu", (void*)stream, p, bytes);
    memset(p, value, bytes);
    return cudaSuccess;
}

cudaError_t cudaStreamCreateWithPriority(cudaStream_t* stream, unsigned, int) {
    *stream = (cudaStream_t)(g_next++ << 8);
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* stream, unsigned flags) {
    return cudaStreamCreateWithPriority(stream, flags, 0);
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t stream) {
    note("sync %p", (void*)stream);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t stream, cudaEvent_t event, unsigned) {
    note("wait %p %p", (void*)stream, (void*)event);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* event, unsigned) {
    *event = (cudaEvent_t)(g_next++ << 8);
    note("event %p", (void*)*event);
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* event) { return cudaEventCreateWithFlags(event, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t event) {
    note("unevent %p", (void*)event);
    return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t event, cudaStream_t stream) {
    note("record %p %p", (void*)event, (void*)stream);
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t event) {
    note("esync %p", (void*)event);
    return cudaSuccess;
}
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t from, cudaEvent_t to) {
    note("elapsed %p %p", (void*)from, (void*)to);
    *ms = 0.01f;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t* graph) {
    *graph = (cudaGraph_t)(g_next++ << 8);
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* exec, cudaGraph_t, unsigned long long) {
    *exec = (cudaGraphExec_t)(g_next++ << 8);
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t stream) {
    note("launch %p graph 1 1", (void*)stream);
    return cudaSuccess;
}
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

cudaError_t cudaGetDevice(int* device) {
    *device = g_device;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int device) {
    g_device = device;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceCount(int* count) {
    *count = 2;
    return cudaSuccess;
}
cudaError_t cudaGetDeviceProperties(cudaDeviceProp* prop, int) {
    memset(prop, 0, sizeof(*prop));
    snprintf(prop->name, sizeof(prop->name), "no device");
    return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* value, cudaDeviceAttr attr, int) {
    *value = attr == cudaDevAttrMultiProcessorCount ? 152 : 1;
    return cudaSuccess;
}
cudaError_t cudaDeviceGetStreamPriorityRange(int* least, int* greatest) {
    *least = *greatest = 0;
    return cudaSuccess;
}
// resident blocks by kernel and device
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* blocks, const void* kernel, int, size_t, unsigned) {
    int sum = 0;
    for (const char* c = name_of(kernel); *c; ++c) sum += *c;
    *blocks = 1 + sum % 3 + 3 * g_device;
    return cudaSuccess;
}
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessor(int* blocks, const void* kernel, int threads, size_t shared) {
    return cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(blocks, kernel, threads, shared, 0);
}
cudaError_t cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void*) {
    memset(a, 0, sizeof(*a));
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void** p, const void*) {
    static char room[1 << 16];
    *p = room;
    return cudaSuccess;
}
cudaError_t cudaHostRegister(void*, size_t, unsigned) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
// (no compiled programs: the interpreter's kernels are launched)
cudaError_t cudaLibraryLoadData(cudaLibrary_t*, const void*, cudaJitOption*, void**, unsigned, cudaLibraryOption*, void**, unsigned) {
    return cudaErrorNotSupported;
}
cudaError_t cudaLibraryUnload(cudaLibrary_t) { return cudaSuccess; }
cudaError_t cudaLibraryGetKernel(cudaKernel_t*, cudaLibrary_t, const char*) { return cudaErrorNotSupported; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = g_last;
    g_last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaSuccess ? "no error" : "injected failure"; }
}
