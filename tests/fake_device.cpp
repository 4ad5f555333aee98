// A stand-in for the CUDA runtime and for the kernels, for tests of the batch scheduler (csrc/api.cu) without a GPU: device memory is
// ordinary memory, full of 0xCC at first; copies to it are made as late as the order of their stream allows; kernels do nothing
// but what a test asks of them.  Streams know whether they are being captured, events where they were recorded.
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <vector>

#include <cuda.h>
#include <cuda_runtime.h>

#include "../datago_b200/csrc/kernels.h"

namespace {
struct Copy { void* dst; const void* src; size_t n; };
struct Stream { bool capturing = false; std::vector<Copy> late; };
struct Event { bool captured = false; Stream* of = nullptr; };
std::mutex mu;
unsigned long long to_device = 0, to_host = 0;
unsigned int timeouts_per_pass = 0;
int host_allocations = 0;
bool capturing(cudaStream_t s) { return s && reinterpret_cast<Stream*>(s)->capturing; }
void catch_up(Stream* s) {  // mu is held
    if (!s) return;
    for (const Copy& c : s->late) memcpy(c.dst, c.src, c.n);
    s->late.clear();
}
CUresult encode(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*, const cuuint32_t*,
                CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill) { return CUDA_SUCCESS; }
}  // namespace

extern "C" {
cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int* n) { *n = 1; return cudaSuccess; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "?"; }
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = aligned_alloc(256, (n + 255) / 256 * 256);
    if (*p) memset(*p, 0xCC, n < ((size_t)1 << 24) ? n : (size_t)1 << 24);
    return *p ? cudaSuccess : cudaErrorMemoryAllocation;
}
cudaError_t cudaFree(void* p) { free(p); return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned int) { ++host_allocations; return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaHostRegister(void*, size_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaHostUnregister(void*) { return cudaSuccess; }
cudaError_t cudaGetSymbolAddress(void** p, const void* symbol) { *p = const_cast<void*>(symbol); return cudaSuccess; }
cudaError_t cudaGetDriverEntryPoint(const char*, void** p, unsigned long long, cudaDriverEntryPointQueryResult* q) {
    *p = reinterpret_cast<void*>(&encode);
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) { *s = reinterpret_cast<cudaStream_t>(new Stream); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { delete reinterpret_cast<Stream*>(s); return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    if (capturing(s)) return cudaErrorStreamCaptureUnsupported;
    std::lock_guard<std::mutex> lock(mu);
    catch_up(reinterpret_cast<Stream*>(s));
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* st) {
    *st = capturing(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) { *e = reinterpret_cast<cudaEvent_t>(new Event); return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) { return cudaEventCreateWithFlags(e, 0); }
cudaError_t cudaEventDestroy(cudaEvent_t e) { delete reinterpret_cast<Event*>(e); return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 0.f; return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    reinterpret_cast<Event*>(e)->captured = capturing(s);
    reinterpret_cast<Event*>(e)->of = reinterpret_cast<Stream*>(s);
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned int) {
    std::lock_guard<std::mutex> lock(mu);
    if (capturing(s) && !reinterpret_cast<Event*>(e)->captured) return cudaErrorStreamCaptureIsolation;
    catch_up(reinterpret_cast<Event*>(e)->of);
    if (reinterpret_cast<Event*>(e)->captured) reinterpret_cast<Stream*>(s)->capturing = true;  // joins the capture
    return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu);
    Stream* const st = reinterpret_cast<Stream*>(s);
    if (kind == cudaMemcpyHostToDevice) {
        st->late.push_back({dst, src, n});
        to_device += n;
        return cudaSuccess;
    }
    catch_up(st);
    memcpy(dst, src, n);
    to_host += n;
    return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu);
    catch_up(reinterpret_cast<Stream*>(s));
    memset(p, v, n);
    return cudaSuccess;
}

void fake_capture(void* s, int on) { reinterpret_cast<Stream*>(s)->capturing = on != 0; }
void fake_timeouts(unsigned int per_pass) { timeouts_per_pass = per_pass; }
unsigned long long fake_to_device() { return to_device; }
unsigned long long fake_to_host() { return to_host; }
int fake_host_allocations() { return host_allocations; }
}

namespace dg {
void launch_unstuff(const JpegWave&, cudaStream_t) {}
void launch_huff_guess(const JpegWave&, cudaStream_t) {}
void launch_huff_chain(const JpegWave&, cudaStream_t) {}
void launch_huff_write(const JpegWave&, cudaStream_t) {}
void launch_huff_restart(const JpegWave&, cudaStream_t) {}
void launch_whole_blocks(const JpegWave&, uint32_t, cudaStream_t) {}
void launch_idct(const JpegWave&, uint32_t, uint32_t, cudaStream_t) {}
void launch_color(const JpegWave&, uint32_t, uint32_t, cudaStream_t) {}
void launch_idct_chroma(const JpegWave&, uint32_t, uint32_t, cudaStream_t) {}
void launch_luma_color(const JpegWave&, uint32_t, uint32_t, cudaStream_t) {}
static void pass(uint32_t mma_tiles, unsigned int* timeouts, cudaStream_t s) {
    std::lock_guard<std::mutex> lock(mu);
    catch_up(reinterpret_cast<Stream*>(s));
    if (mma_tiles) *timeouts += timeouts_per_pass;
}
void launch_conv_h(const ConvPass*, OwnerMap, const uint32_t*, uint32_t mma_tiles, unsigned int* timeouts, cudaStream_t s) { pass(mma_tiles, timeouts, s); }
void launch_conv_v(const ConvPass*, OwnerMap, const uint32_t*, uint32_t mma_tiles, unsigned int* timeouts, cudaStream_t s) { pass(mma_tiles, timeouts, s); }
void launch_copy(const CopyJob*, OwnerMap, cudaStream_t) {}
void launch_alpha(const AlphaJob*, OwnerMap, cudaStream_t) {}
void launch_to_rgb8(const ToRgbJob*, OwnerMap, cudaStream_t) {}
}  // namespace dg
