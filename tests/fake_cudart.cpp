// fake_cudart.cpp -- a stand-in for the CUDA runtime, linked with the library's
// own object files, so that its host side runs without a device: memory is
// host memory, copies and memsets happen at once, kernels are recorded by name
// and not run (fake_kernels.cu acts out what a test needs of them).  Failures
// are made here, on the host: a launch that is refused, a context that is reset.
#include <cuda.h>
#include <cuda_runtime_api.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

void act_out(const std::string& name, void** args, std::string& faults);  // fake_kernels.cu
bool pinned_word(const void* p, size_t n);

namespace {
std::map<const void*, std::string> names;    // host stub -> kernel name
std::map<char*, size_t> device, pinned;      // live allocations
std::map<cudaStream_t, bool> capturing;
std::string launched, refuse, faults;
unsigned long long context = 1;
cudaError_t last = cudaSuccess;
dim3 call_grid, call_block;
cudaStream_t call_stream;

cudaError_t note(cudaError_t e) {
    if (e != cudaSuccess) last = e;
    return e;
}
bool inside(const std::map<char*, size_t>& m, const void* p, size_t n) {
    for (auto& a : m)
        if ((const char*)p >= a.first && (const char*)p + n <= a.first + a.second) return true;
    return false;
}
void release(std::map<char*, size_t>& m) {
    for (auto& a : m) free(a.first);
    m.clear();
}
cudaError_t take(std::map<char*, size_t>& m, void** p, size_t n) {
    char* q = (char*)calloc(1, n ? n : 1);
    m[q] = n;
    *p = q;
    return cudaSuccess;
}

cudaError_t launch(const void* f, dim3 grid, dim3 block, void** args, cudaStream_t s) {
    const std::string& name = names[f];
    if (!refuse.empty() && name.find(refuse) != std::string::npos)
        return note(cudaErrorLaunchOutOfResources);
    if (grid.x == 0 || grid.y == 0 || grid.z == 0 || grid.y > 65535 || grid.z > 65535 ||
        block.x * block.y * block.z > 1024)
        return note(cudaErrorInvalidConfiguration);
    char at[96];
    snprintf(at, sizeof at, " %u %u %u;", grid.x, grid.y, grid.z);
    launched += name + at;
    if (!capturing[s]) act_out(name, args, faults);
    return cudaSuccess;
}

CUresult ctx_current(CUcontext* c) {
    *c = (CUcontext)(uintptr_t)(0x1000 + context);
    return CUDA_SUCCESS;
}
CUresult ctx_id(CUcontext c, unsigned long long* id) {
    *id = c ? (unsigned long long)(uintptr_t)c - 0x1000 : context;
    return CUDA_SUCCESS;
}
}  // namespace

// Whether [p, p + n) is pinned memory that has not been given back.
bool pinned_word(const void* p, size_t n) { return inside(pinned, p, n); }

extern "C" {
// ------------------------------------------------------------ for the tests
// Kernels launched since the last call: "name gx gy gz;" each.
const char* fake_launched() {
    static std::string out;
    out.swap(launched);
    launched.clear();
    return out.c_str();
}
// What was done to memory that is not there, since the last call.
const char* fake_faults() {
    static std::string out;
    out.swap(faults);
    faults.clear();
    return out.c_str();
}
void fake_refuse(const char* part_of_name) { refuse = part_of_name; }
int fake_pages() { return (int)pinned.size(); }  // pinned allocations
// cudaDeviceReset: the context and all of its memory go.
void fake_reset() {
    release(device);
    release(pinned);
    context++;
}

// ------------------------------------------------------- registration, launch
void** __cudaRegisterFatBinary(void*) {
    static void* h;
    return &h;
}
void __cudaRegisterFatBinaryEnd(void**) {}
void __cudaUnregisterFatBinary(void**) {}
char __cudaInitModule(void**) { return 1; }
void __cudaRegisterVar(void**, char*, char*, const char*, int, size_t, int, int) {}
void __cudaRegisterFunction(void**, const char* host, char*, const char* name, int, uint3*, uint3*,
                            dim3*, dim3*, int*) {
    names[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 g, dim3 b, size_t, cudaStream_t s) {
    call_grid = g;
    call_block = b;
    call_stream = s;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3* g, dim3* b, size_t* m, void* s) {
    *g = call_grid;
    *b = call_block;
    *m = 0;
    *(cudaStream_t*)s = call_stream;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void* f, dim3 g, dim3 b, void** args, size_t, cudaStream_t s) {
    return launch(f, g, b, args, s);
}
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** args) {
    return launch(f, c->gridDim, c->blockDim, args, c->stream);
}

// ------------------------------------------------------------ the runtime's calls
cudaError_t cudaGetLastError() {
    const cudaError_t e = last;
    last = cudaSuccess;
    return e;
}
const char* cudaGetErrorString(cudaError_t e) { return e ? "refused" : "no error"; }
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { return *v = 148, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t,
                                                                   unsigned) {
    return *n = 8, cudaSuccess;
}
cudaError_t cudaMalloc(void** p, size_t n) { return take(device, p, n); }
cudaError_t cudaFree(void* p) {
    if (device.erase((char*)p)) free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return take(pinned, p, n); }
cudaError_t cudaFreeHost(void* p) {
    if (pinned.erase((char*)p)) free(p);
    return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
    if (!capturing[s]) memset(p, v, n);
    return cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    return memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    return memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpyToSymbol(const void*, const void*, size_t, size_t, cudaMemcpyKind) {
    return cudaSuccess;
}
cudaError_t cudaMemcpyFromSymbol(void* d, const void*, size_t n, size_t, cudaMemcpyKind) {
    return memset(d, 0, n), cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void**, const void*) { return note(cudaErrorInvalidSymbol); }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes*, const void*) {
    return note(cudaErrorInvalidValue);
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) {
    static char tokens[1 << 16], *next = tokens + 1;
    return *s = (cudaStream_t)next++, cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    *st = capturing[s] ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t s, cudaStreamCaptureMode) {
    return capturing[s] = true, cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t s, cudaGraph_t* g) {
    capturing[s] = false;
    return *g = (cudaGraph_t)1, cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* e, cudaGraph_t, unsigned long long) {
    return *e = (cudaGraphExec_t)1, cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = (cudaEvent_t)1, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 0, cudaSuccess; }
cudaError_t cudaGetDriverEntryPointByVersion(const char* name, void** f, unsigned,
                                             unsigned long long,
                                             cudaDriverEntryPointQueryResult* r) {
    *f = strcmp(name, "cuCtxGetId") == 0        ? (void*)ctx_id
         : strcmp(name, "cuCtxGetCurrent") == 0 ? (void*)ctx_current
                                                : nullptr;
    if (r) *r = *f ? cudaDriverEntryPointSuccess : cudaDriverEntryPointSymbolNotFound;
    return cudaSuccess;
}
}  // extern "C"
