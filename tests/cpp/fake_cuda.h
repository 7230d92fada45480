// A CUDA runtime of host memory for tests of the host code behind the C ABI: "device" memory
// comes from malloc, with the bytes in use, their peak and an optional limit; copies and
// clears run at once; every operation is recorded with its stream, and streams, events and
// captures are plain values. Linked in place of the real runtime with the kernels' launch
// functions left out (those a test does not define are never called).
#pragma once
#include <cuda_runtime.h>

#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <set>
#include <vector>

namespace fake {

struct Op {
    enum Kind { kSet, kCopy, kRecord, kWait, kSync } kind;
    cudaStream_t stream;  // nullptr: the legacy default stream
    const void* what;     // the destination, or the event
    size_t bytes;
};
inline std::vector<Op> ops;
inline std::map<void*, size_t> blocks;
inline size_t inUse = 0, peak = 0, limit = 0;  // limit 0: none
inline cudaError_t lastError = cudaSuccess;
inline std::set<cudaStream_t> capturing;
inline uintptr_t handles = 0x1000;

template <class T>
T Handle() {
    return reinterpret_cast<T>(handles += 16);
}

}  // namespace fake

extern "C" {
cudaError_t cudaGetDeviceCount(int* n) { return *n = 1, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError() {
    const cudaError_t e = fake::lastError;
    return fake::lastError = cudaSuccess, e;
}
const char* cudaGetErrorString(cudaError_t e) { return e == cudaErrorMemoryAllocation ? "out of memory" : "error"; }
cudaError_t cudaMalloc(void** p, size_t n) {
    *p = nullptr;
    if (fake::limit && fake::inUse + n > fake::limit) return fake::lastError = cudaErrorMemoryAllocation;
    *p = std::memset(std::malloc(n), 0xA5, n);
    fake::blocks[*p] = n;
    fake::inUse += n;
    if (fake::inUse > fake::peak) fake::peak = fake::inUse;
    return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
    auto it = fake::blocks.find(p);
    if (it == fake::blocks.end()) return p ? cudaErrorInvalidValue : cudaSuccess;
    fake::inUse -= it->second;
    fake::blocks.erase(it);
    std::free(p);
    return cudaSuccess;
}
cudaError_t cudaHostAlloc(void** p, size_t n, unsigned) { return *p = std::calloc(1, n), cudaSuccess; }
cudaError_t cudaFreeHost(void* p) { return std::free(p), cudaSuccess; }
cudaError_t cudaMemset(void* p, int v, size_t n) {
    fake::ops.push_back({fake::Op::kSet, nullptr, p, n});
    return std::memset(p, v, n), cudaSuccess;
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t s) {
    fake::ops.push_back({fake::Op::kSet, s, p, n});
    return std::memset(p, v, n), cudaSuccess;
}
cudaError_t cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    fake::ops.push_back({fake::Op::kCopy, nullptr, d, n});
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t st) {
    fake::ops.push_back({fake::Op::kCopy, st, d, n});
    return std::memcpy(d, s, n), cudaSuccess;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { return *s = fake::Handle<cudaStream_t>(), cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t s) {
    fake::ops.push_back({fake::Op::kSync, s, nullptr, 0});
    return cudaSuccess;
}
cudaError_t cudaStreamWaitEvent(cudaStream_t s, cudaEvent_t e, unsigned) {
    fake::ops.push_back({fake::Op::kWait, s, e, 0});
    return cudaSuccess;
}
cudaError_t cudaStreamIsCapturing(cudaStream_t s, cudaStreamCaptureStatus* out) {
    *out = fake::capturing.count(s) ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
    return cudaSuccess;
}
cudaError_t cudaEventCreate(cudaEvent_t* e) { return *e = fake::Handle<cudaEvent_t>(), cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t e, cudaStream_t s) {
    fake::ops.push_back({fake::Op::kRecord, s, e, 0});
    return cudaSuccess;
}
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventQuery(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { return *ms = 1.0f, cudaSuccess; }
}
