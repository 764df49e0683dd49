// A CUDA runtime on host memory and recorders in place of the kernel launches, so that the host code of the engine
// (jne_context.h and the units built on it) runs without a GPU.  "Device" buffers are host buffers; streams and
// events do nothing; allocations and uploads fail on demand.
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <cstring>
#include <functional>
#include <vector>

#include "../../johansen-null-eigenspectra_gb300/csrc/jne_context.h"

namespace fake {

struct MixedLaunch {
  jne_accum_args a;
  int fin_model;                      // -2: accumulation only
  std::vector<jne_chunk_time> table;  // the chunk table the kernel would read
};

constexpr int kSms = 3;
inline std::function<float(const MixedLaunch&)> ms;  // what events around the last mixed launch measure (1 by default)
inline bool fail_malloc = false, fail_upload = false;
inline std::vector<MixedLaunch> mixed;
inline std::vector<std::vector<int4>> entries;  // the entry tables of the FP64 launches on explicit increments

}  // namespace fake

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaMalloc(void** p, size_t n) {
  *p = nullptr;
  if (fake::fail_malloc) return cudaErrorMemoryAllocation;
  *p = std::calloc(n ? n : 1, 1);
  return cudaSuccess;
}
cudaError_t cudaFree(void* p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t n, cudaMemcpyKind kind, cudaStream_t) {
  if (fake::fail_upload && kind == cudaMemcpyHostToDevice) return cudaErrorUnknown;
  std::memcpy(dst, src, n);
  return cudaSuccess;
}
cudaError_t cudaMemcpy(void* dst, const void* src, size_t n, cudaMemcpyKind kind) {
  return cudaMemcpyAsync(dst, src, n, kind, nullptr);
}
cudaError_t cudaMemsetAsync(void* p, int v, size_t n, cudaStream_t) {
  std::memset(p, v, n);
  return cudaSuccess;
}
cudaError_t cudaMemset(void* p, int v, size_t n) { return cudaMemsetAsync(p, v, n, nullptr); }
cudaError_t cudaMallocHost(void** p, size_t n) { return cudaMalloc(p, n); }
cudaError_t cudaFreeHost(void* p) { return cudaFree(p); }
cudaError_t cudaGetDeviceCount(int* n) {
  *n = 1;
  return cudaSuccess;
}
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) {
  *v = fake::kSms;
  return cudaSuccess;
}
cudaError_t cudaGetLastError() { return cudaSuccess; }
const char* cudaGetErrorString(cudaError_t) { return "fake error"; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) {
  *s = nullptr;
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned int) { return cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t* e) {
  *e = nullptr;
  return cudaSuccess;
}
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) { return cudaEventCreate(e); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) {
  *ms = fake::ms && !fake::mixed.empty() ? fake::ms(fake::mixed.back()) : 1.0f;
  return cudaSuccess;
}
}

cudaError_t jne_launch_accum_mixed(const jne_accum_args& a, const jne_finalize_args* fin, int, cudaStream_t) {
  const int nch = (a.steps + a.chunk - 1) / a.chunk;
  fake::MixedLaunch l{a, fin ? fin->model : -2, {}};
  if (a.chunk_tab) l.table.assign(a.chunk_tab, a.chunk_tab + nch);
  fake::mixed.push_back(l);
  return cudaSuccess;
}
cudaError_t jne_launch_accum_digits(const jne_accum_args&, const jne_finalize_args*, int, cudaStream_t) {
  return cudaSuccess;
}
cudaError_t jne_launch_accum_f64(const jne_accum_args&, const int4* ent, int nent, int, cudaStream_t) {
  fake::entries.emplace_back();
  if (ent) fake::entries.back().assign(ent, ent + nent);
  return cudaSuccess;
}
cudaError_t jne_launch_finalize(const jne_finalize_args*, int, cudaStream_t) { return cudaSuccess; }
