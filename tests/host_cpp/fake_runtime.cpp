// A CUDA runtime that only keeps a record, and launches that launch nothing: what the attention library's host side
// (goml_b200/csrc/fa_api.cu) asks for can then be read on a machine without a GPU.  A stream handle is its id.
#include <cuda_runtime.h>
#include <stdlib.h>

#include <mutex>
#include <string>

#include "../../goml_b200/csrc/fa_fwd_sm100.h"
#include "../../include/fa_sm120.h"

static std::mutex lock_;
static std::string log_;
static size_t next_ = 0x1000;
static size_t fail_allocation_ = 0;   // the n-th allocation from now on fails
static int rows_with_scratch_ = 0;    // forwards of shorter sequences take none
static void note(const std::string& s) {
    std::lock_guard<std::mutex> g(lock_);
    log_ += s + "\n";
}
static std::string n(const void* p) { return std::to_string(reinterpret_cast<size_t>(p)); }
template <typename T>
static T fresh() {
    std::lock_guard<std::mutex> g(lock_);
    return reinterpret_cast<T>(next_ += 0x1000);
}

extern "C" {
const char* fake_log(void) { return log_.c_str(); }
void fake_clear(void) { log_.clear(); }
void fake_fail_allocation(size_t nth) { fail_allocation_ = nth; }
void fake_rows_with_scratch(int rows) { rows_with_scratch_ = rows; }

cudaError_t cudaGetDevice(int* d) { *d = 0; return cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 10; return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaMemPoolCreate(cudaMemPool_t* p, const cudaMemPoolProps*) { *p = fresh<cudaMemPool_t>(); note("pool_create"); return cudaSuccess; }
cudaError_t cudaMemPoolSetAttribute(cudaMemPool_t, cudaMemPoolAttr, void*) { return cudaSuccess; }
cudaError_t cudaMemPoolDestroy(cudaMemPool_t) { note("pool_destroy"); return cudaSuccess; }
cudaError_t cudaMallocFromPoolAsync(void** p, size_t bytes, cudaMemPool_t, cudaStream_t s) {
    if (fail_allocation_ && --fail_allocation_ == 0) return cudaErrorMemoryAllocation;
    *p = fresh<void*>();
    note("alloc " + n(*p) + " stream " + n(s) + " bytes " + std::to_string(bytes));
    return cudaSuccess;
}
cudaError_t cudaFreeAsync(void* p, cudaStream_t s) { note("free " + n(p) + " stream " + n(s)); return cudaSuccess; }
cudaError_t cudaFree(void*) { note("SYNC cudaFree"); return cudaSuccess; }
cudaError_t cudaDeviceSynchronize(void) { note("SYNC cudaDeviceSynchronize"); return cudaSuccess; }
cudaError_t cudaMemsetAsync(void* p, int, size_t, cudaStream_t s) { note("memset " + n(p) + " stream " + n(s)); return cudaSuccess; }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* c) { *c = cudaStreamCaptureStatusNone; return cudaSuccess; }
cudaError_t cudaThreadExchangeStreamCaptureMode(cudaStreamCaptureMode*) { return cudaSuccess; }
cudaError_t cudaStreamGetId(cudaStream_t s, unsigned long long* id) { *id = reinterpret_cast<size_t>(s); return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = fresh<cudaStream_t>(); note("stream_create " + n(*s)); return cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t s) { note("stream_destroy " + n(s)); return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) { note("wait stream " + n(s) + " event " + n(e)); return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = fresh<cudaEvent_t>(); return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) { note("record event " + n(e) + " stream " + n(s)); return cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
}

namespace fa_sm100 {
bool needs_no_scratch(const LaunchArgs& a) { return a.sl < rows_with_scratch_; }
size_t workspace_bytes(int bh, int sl, int hd) { return (size_t)bh * sl * hd * 2; }
size_t v_flag_count(int bh, int) { return bh; }
cudaError_t launch(const LaunchArgs& a) { note("launch stream " + n(a.stream) + " scratch " + n(a.v16_workspace) + " flags " + n(a.v_flags)); return cudaSuccess; }
size_t decode_workspace_bytes(int, int, int, int, int) { return 1 << 20; }
size_t decode_arrival_count(int batch, int, int kv_heads, int, int) { return (size_t)batch * kv_heads; }
cudaError_t launch_decode(const DecodeArgs& a) {
    note("launch stream " + n(a.stream) + " scratch " + n(a.workspace) + " zeros " + n(a.arrivals));
    return cudaSuccess;
}
cudaError_t launch_clear_words(uint32_t* w, size_t, cudaStream_t s) { note("clear " + n(w) + " stream " + n(s)); return cudaSuccess; }
cudaError_t launch_wait_expiry_selftest(cudaStream_t) { return cudaSuccess; }
int device_status() { return 0; }
}  // namespace fa_sm100
