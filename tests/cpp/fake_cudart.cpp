// A CUDA runtime without a GPU, for tests of the library's host code: linked
// with the library's objects in place of libcudart. Device memory is host
// memory, copies and fills happen at the call, kernels do not run. Calls that
// matter to the tests are counted or logged, and one can be made to fail.
#include <cuda_runtime_api.h>
#include <stdint.h>
#include <stdio.h>
#include <stdlib.h>
#include <string.h>

#include <map>
#include <string>
#include <utility>
#include <vector>

namespace {
std::string log_text;
// host stub -> mangled name (made at its first use: the objects register
// their kernels while the library is loaded)
std::map<const void *, std::string> &kernels() {
    static auto *m = new std::map<const void *, std::string>;
    return *m;
}
int streams = 0, events = 0;
std::string fail_fn;
int fail_after = 0;  // calls of fail_fn to let through first
unsigned false_bits = 0;   // what a sample of the state finds
unsigned kept_pairs = 0;   // what filtered passes keep
uintptr_t far_begin = 0, far_end = 0;  // memory of device 1
dim3 cfg_grid, cfg_block;

void note(const char *fmt, unsigned long long a, unsigned long long b, unsigned long long c) {
    char s[160];
    snprintf(s, sizeof s, fmt, a, b, c);
    log_text += s;
}

bool fails(const char *fn) { return fail_fn == fn && fail_after-- == 0; }

template <typename T>
T handle() {
    static uintptr_t next = 0x1000;
    return (T) (next += 16);
}
}  // namespace

extern "C" {

const char *fake_log() { return log_text.c_str(); }
int fake_streams() { return streams; }
int fake_events() { return events; }
void fake_reset() {
    log_text.clear();
    fail_fn.clear();
    false_bits = kept_pairs = 0;
    far_begin = far_end = 0;
}
void fake_fail(const char *fn, int after) {
    fail_fn = fn;
    fail_after = after;
}
void fake_filter(unsigned n_false, unsigned kept) {
    false_bits = n_false;
    kept_pairs = kept;
}
void fake_far(void *p, size_t bytes) {
    far_begin = (uintptr_t) p;
    far_end = far_begin + bytes;
}

void **__cudaRegisterFatBinary(void *) { return handle<void **>(); }
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
void __cudaRegisterVar(void **, char *, char *, const char *, int, size_t, int, int) {}
void __cudaRegisterFunction(void **, const char *host, char *, const char *name, int, uint3 *, uint3 *, dim3 *, dim3 *,
                            int *) {
    kernels()[host] = name;
}
unsigned __cudaPushCallConfiguration(dim3 grid, dim3 block, size_t, struct CUstream_st *) {
    cfg_grid = grid, cfg_block = block;
    return 0;
}
cudaError_t __cudaPopCallConfiguration(dim3 *grid, dim3 *block, size_t *smem, void *stream) {
    *grid = cfg_grid, *block = cfg_block, *smem = 0, *(void **) stream = nullptr;
    return cudaSuccess;
}
cudaError_t __cudaGetKernel(cudaKernel_t *k, const void *host) {
    *k = (cudaKernel_t) host;
    return cudaSuccess;
}
cudaError_t __cudaLaunchKernel(cudaKernel_t k, dim3 grid, dim3, void **args, size_t, cudaStream_t) {
    const std::string &name = kernels()[(const void *) k];
    log_text += "launch " + name;
    // the buffers these read
    const bool masks = name.find("load_masks_kernel") != std::string::npos;
    if (masks || name.find("load_state_kernel") != std::string::npos)
        for (int i : {0, masks ? 1 : 0, masks ? 6 : 0}) note(" %llx", *(unsigned long long *) args[i], 0, 0);
    if (!masks && name.find("load_state_kernel") != std::string::npos && *(void **) args[2]) log_text += " table";
    note(" grid %llu\n", grid.x, 0, 0);
    if (masks && *(void **) args[6]) **(unsigned **) args[9] = false_bits;  // (.., state, pairs, samples, count)
    if (name.find("deliver_kernel") != std::string::npos)  // (.., n_parts, cap, host: counters, error flag, kept)
        (*(unsigned **) args[5])[*(unsigned *) args[3] + 1] = kept_pairs;
    return cudaSuccess;
}

cudaError_t cudaGetLastError() { return cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceSynchronize() { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int *v, cudaDeviceAttr, int) { return *v = 152, cudaSuccess; }
cudaError_t cudaDeviceGetStreamPriorityRange(int *a, int *b) { return *a = 0, *b = -5, cudaSuccess; }
cudaError_t cudaMemGetInfo(size_t *a, size_t *b) { return *a = *b = 1ull << 38, cudaSuccess; }
cudaError_t cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int *n, const void *, int, size_t, unsigned) {
    log_text += "occupancy\n";
    if (fails("occupancy")) return cudaErrorUnknown;
    return *n = 4, cudaSuccess;
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return streams++, *s = handle<cudaStream_t>(), cudaSuccess; }
cudaError_t cudaStreamCreateWithPriority(cudaStream_t *s, unsigned, int) {
    return streams++, *s = handle<cudaStream_t>(), cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return streams--, cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return log_text += "wait\n", cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return events++, *e = handle<cudaEvent_t>(), cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return events--, cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }

cudaError_t cudaMalloc(void **p, size_t n) {
    if (fails("malloc")) return cudaErrorMemoryAllocation;
    return *p = aligned_alloc(256, (n + 255) / 256 * 256), memset(*p, 0, n), cudaSuccess;
}
cudaError_t cudaFree(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaMallocHost(void **p, size_t n) {
    if (fails("malloc_host")) return cudaErrorMemoryAllocation;
    return *p = calloc(1, n), cudaSuccess;
}
cudaError_t cudaFreeHost(void *p) { return free(p), cudaSuccess; }
cudaError_t cudaMemcpyAsync(void *d, const void *s, size_t n, cudaMemcpyKind, cudaStream_t) {
    note("copy %llx %llx %llu\n", (unsigned long long) d, (unsigned long long) s, n);
    return memmove(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpy(void *d, const void *s, size_t n, cudaMemcpyKind k) { return cudaMemcpyAsync(d, s, n, k, nullptr); }
cudaError_t cudaMemcpy2DAsync(void *d, size_t dp, const void *s, size_t sp, size_t w, size_t h, cudaMemcpyKind, cudaStream_t) {
    note("copy2d %llx %llx %llu\n", (unsigned long long) d, (unsigned long long) s, w * h);
    for (size_t i = 0; i < h; i++) memmove((char *) d + i * dp, (const char *) s + i * sp, w);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *p, int v, size_t n, cudaStream_t) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaMemset(void *p, int v, size_t n) { return memset(p, v, n), cudaSuccess; }
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes *a, const void *p) {
    memset(a, 0, sizeof *a);
    a->type = cudaMemoryTypeDevice;
    a->device = (uintptr_t) p >= far_begin && (uintptr_t) p < far_end ? 1 : 0;
    a->devicePointer = (void *) p;
    return cudaSuccess;
}
cudaError_t cudaGetSymbolAddress(void **p, const void *) {
    static char room[1 << 20];
    return *p = room, cudaSuccess;
}

cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return log_text += "capture\n", cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = handle<cudaGraph_t>(), cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
    return *e = handle<cudaGraphExec_t>(), cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return log_text += "graph\n", cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

}  // extern "C"
