// A CUDA runtime on host memory for the library's host code (csrc/fz_api.cu): copies with a stream
// run when the stream is waited for, a chosen call fails, and every call is written down.  Compiled
// as C++ it is that runtime (nvcc would take some of its names for the device runtime's), as CUDA the
// stubs of the kernel launchers.
#include <cuda_runtime.h>

cudaError_t fake_call(const char* name);

#ifndef __CUDACC__
#include <cstdlib>
#include <cstring>
#include <functional>
#include <string>
#include <vector>

namespace {
std::vector<std::function<void()>> queue;
std::string                        text, fail_name;
int                                fail_nth = 0, fail_err = 0;

void drain()
{
    for (auto& f : queue) f();
    queue.clear();
}
}  // namespace

cudaError_t fake_call(const char* name)
{
    text += std::string(name) + " ";
    if (fail_name == name && --fail_nth == 0) return static_cast<cudaError_t>(fail_err);
    return cudaSuccess;
}

extern "C" {
void        fake_fail(const char* name, int nth, int err) { fail_name = name, fail_nth = nth, fail_err = err; }
const char* fake_calls() { return text.c_str(); }
int         fake_pending() { return (int)queue.size(); }
void        fake_reset() { text.clear(), fail_name.clear(), drain(); }

cudaError_t cudaMalloc(void** p, size_t n) { return *p = calloc(1, n), fake_call("cudaMalloc"); }
cudaError_t cudaMallocHost(void** p, size_t n) { return *p = calloc(1, n), fake_call("cudaMallocHost"); }
cudaError_t cudaFree(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return free(p), cudaSuccess; }
cudaError_t cudaGetDevice(int* d) { return *d = 0, cudaSuccess; }
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) { return memcpy(d, s, n), fake_call("cudaMemcpy"); }
cudaError_t cudaMemset(void* p, int v, size_t n) { return memset(p, v, n), fake_call("cudaMemset"); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) { return memset(p, v, n), fake_call("cudaMemsetAsync"); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t)
{
    const cudaError_t e = fake_call("cudaMemcpyAsync");
    if (e == cudaSuccess) queue.push_back([=] { memcpy(d, s, n); });
    return e;
}
cudaError_t cudaStreamSynchronize(cudaStream_t)
{
    const cudaError_t e = fake_call("cudaStreamSynchronize");
    if (e == cudaSuccess) drain();
    return e;
}
cudaError_t cudaEventCreate(cudaEvent_t*) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float*, cudaEvent_t, cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t*, cudaGraph_t, unsigned long long) { return cudaSuccess; }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t*, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
void**      __cudaRegisterFatBinary(void*) { return nullptr; }
void        __cudaRegisterFatBinaryEnd(void**) {}
void        __cudaUnregisterFatBinary(void**) {}
}

#else
#include "../fz-gpu_gb300/csrc/fz_internal.h"

namespace fz {
void field_items(uint32_t n, uint32_t nb, uint32_t ntiles, bool rel, uint32_t& nr, uint32_t& ne, uint32_t& nc)
{
    nr = rel ? (uint32_t)cdiv(n, 1024) : 0u, ne = (uint32_t)cdiv(ntiles, 8), nc = (uint32_t)cdiv(nb, 32);
}
uint32_t    fake_cluster = 16;
uint32_t    small_items(int, bool) { return fake_cluster; }
bool        whole_field_fits(int, bool, uint32_t, bool) { return false; }
cudaError_t launch_fields(FieldPhase p, int, bool, const FieldJob*, const Segment*, uint32_t, uint32_t, const FieldJob&, cudaStream_t, uint32_t)
{
    return fake_call(p == FieldPhase::Range ? "range" : p == FieldPhase::Encode ? "encode" : "compact");
}
cudaError_t launch_whole_field(int, const FieldJob&, cudaStream_t) { return fake_call("whole"); }
cudaError_t launch_offsets(const uint8_t*, uint64_t, uint32_t, uint32_t, uint64_t, uint32_t*, uint64_t*, uint32_t*, uint32_t*, uint32_t*, cudaStream_t) { return fake_call("offsets"); }
cudaError_t launch_zero_tail(float*, uint32_t, uint32_t, cudaStream_t) { return fake_call("zero_tail"); }
cudaError_t launch_reconstruct(const ReconArgs&, cudaStream_t) { return fake_call("reconstruct"); }
cudaError_t launch_scan_encode(const uint8_t*, const uint32_t*, uint32_t, uint32_t*, uint8_t*, uint64_t*, uint32_t*, uint32_t*, uint32_t* total, uint32_t*, cudaStream_t)
{
    *total = 7;
    return fake_call("scan_encode");
}
cudaError_t launch_wait_selftest(const uint64_t*, const uint32_t*, uint32_t*, cudaStream_t) { return fake_call("wait_selftest"); }
cudaError_t launch_bitshuffle_flag(const uint32_t*, uint32_t*, uint32_t, uint32_t*, uint32_t*, cudaStream_t) { return fake_call("bitshuffle"); }
cudaError_t launch_decompress_fused(const DecodeArgs&, cudaStream_t) { return fake_call("decompress"); }
cudaError_t launch_lorenzo_construct(const float*, uint16_t*, uint8_t*, uint32_t, uint32_t, uint32_t, float, cudaStream_t) { return fake_call("construct"); }
}  // namespace fz
extern "C" void fake_largest_cluster(uint32_t items) { fz::fake_cluster = items; }
#endif
