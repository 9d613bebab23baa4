// A CUDA runtime without a device: md_b200.cu linked against this file runs its
// host side on the CPU.  Device memory is a ledger of unique addresses under a
// budget, copies out of it give zeros, launches do nothing.  The fake_* calls
// let a test set the budget, open a caller's stream capture and read the ledger.
#include <cuda_runtime_api.h>

#include <cstdint>
#include <cstring>
#include <map>
#include <set>
#include <utility>

namespace {

std::map<uintptr_t, size_t> blocks;   // live device blocks: address -> bytes
uintptr_t next_addr = uintptr_t(1) << 40;
size_t budget = ~size_t(0), used = 0;
int refused = 0, mallocs = 0, device = 0, graphs = 0, attr_calls = 0;
bool caller_capturing = false;
cudaError_t last_error = cudaSuccess;
std::map<int, std::set<const void *>> attrs;   // device -> kernels given their attributes

}  // namespace

extern "C" {

void fake_budget(size_t bytes) { budget = bytes; }
size_t fake_used() { return used; }
int fake_refused() { return refused; }
int fake_mallocs() { return mallocs; }
void fake_capture(int on) { caller_capturing = on != 0; }
int fake_graphs() { return graphs; }
// Attribute calls since the counter was last cleared.
int fake_attr_calls(int clear) {
    if (clear) attr_calls = 0;
    return attr_calls;
}
int fake_attrs(int dev) { return (int)attrs[dev].size(); }
// Bytes of the live block that starts at `addr`; 0 when there is none.
size_t fake_block(uintptr_t addr) {
    auto it = blocks.find(addr);
    return it == blocks.end() ? 0 : it->second;
}

cudaError_t cudaMalloc(void **p, size_t n) {
    ++mallocs;
    if (used + n > budget) {
        ++refused;
        return last_error = cudaErrorMemoryAllocation;
    }
    *p = reinterpret_cast<void *>(next_addr);
    blocks[next_addr] = n;
    used += n;
    next_addr += (n + 4096) & ~uintptr_t(255);
    return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
    auto it = blocks.find(reinterpret_cast<uintptr_t>(p));
    if (it == blocks.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    used -= it->second;
    blocks.erase(it);
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *dst, const void *, size_t n, cudaMemcpyKind k, cudaStream_t) {
    if (k == cudaMemcpyDeviceToHost) std::memset(dst, 0, n);
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaFuncSetAttribute(const void *f, cudaFuncAttribute, int) {
    attrs[device].insert(f);
    ++attr_calls;
    return cudaSuccess;
}
cudaError_t cudaLaunchKernel(const void *, dim3, dim3, void **, size_t, cudaStream_t) { return cudaSuccess; }

cudaError_t cudaGetDeviceCount(int *n) {
    *n = 2;
    return cudaSuccess;
}
cudaError_t cudaSetDevice(int d) {
    device = d;
    return cudaSuccess;
}
cudaError_t cudaGetDevice(int *d) {
    *d = device;
    return cudaSuccess;
}
cudaError_t cudaGetLastError() {
    const cudaError_t e = last_error;
    last_error = cudaSuccess;
    return e;
}
const char *cudaGetErrorString(cudaError_t e) {
    return e == cudaErrorMemoryAllocation ? "out of memory" : e == cudaSuccess ? "no error" : "error";
}

cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) {
    *s = reinterpret_cast<cudaStream_t>(next_addr++);
    return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus *st) {
    *st = caller_capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) {
    return caller_capturing ? cudaErrorIllegalState : cudaSuccess;
}
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) {
    *g = nullptr;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t *e) {
    *e = reinterpret_cast<cudaEvent_t>(next_addr++);
    return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) {
    *ms = 1.0f;
    return cudaSuccess;
}
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *x, cudaGraph_t, unsigned long long) {
    *x = reinterpret_cast<cudaGraphExec_t>(next_addr++);
    ++graphs;
    return cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }

// what the compiler's kernel registration and launch stubs call
unsigned __cudaPushCallConfiguration(dim3, dim3, size_t, struct CUstream_st *) { return 0; }
cudaError_t __cudaPopCallConfiguration(dim3 *g, dim3 *b, size_t *smem, void *stream) {
    *g = *b = dim3(1, 1, 1);
    *smem = 0;
    *static_cast<void **>(stream) = nullptr;
    return cudaSuccess;
}
void **__cudaRegisterFatBinary(void *) {
    static void *handle = nullptr;
    return &handle;
}
void __cudaRegisterFatBinaryEnd(void **) {}
void __cudaUnregisterFatBinary(void **) {}
char __cudaInitModule(void **) { return 1; }
void __cudaRegisterFunction(void **, const char *, char *, const char *, int, uint3 *, uint3 *, dim3 *, dim3 *, int *) {}

}  // extern "C"
