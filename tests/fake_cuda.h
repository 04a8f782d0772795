// fake_cuda.h -- a CUDA runtime and kernel launchers on host memory, to run the
// engine's host code (mlp_engine.cpp, mlp_capi.cpp) without a GPU: device memory
// is malloc'ed, launches are counted and do nothing, any call can be made to
// fail, and a stream can be declared capturing, which then refuses what a
// capture forbids.  Included by one translation unit.
#pragma once

#include <cuda_runtime.h>

#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <map>
#include <string>

#include "mlp_kernels.cuh"

namespace fake {
std::map<std::string, int> calls;                  // calls by name
std::map<std::string, std::pair<int, int>> fails;  // name -> (calls that still succeed, error)
bool once = false;                                 // an armed failure happens once
int held = 0;                                      // stream-ordered allocations not freed
bool capturing = false;
const void* grasp_table = nullptr;                 // the last launch_grasp's table

inline cudaError_t call(const char* name) {
  calls[name]++;
  const auto f = fails.find(name);
  if (f == fails.end() || f->second.first-- > 0) return cudaSuccess;
  const cudaError_t e = (cudaError_t)f->second.second;
  if (once) fails.erase(f);
  return e;
}
inline void fail(const char* name, cudaError_t e, int after = 0) { fails[name] = {after, (int)e}; }
inline cudaError_t no_capture(const char* name) { return capturing ? cudaErrorStreamCaptureUnsupported : call(name); }
inline cudaError_t alloc(const char* name, void** p, size_t bytes) {
  const cudaError_t e = no_capture(name);
  if (e == cudaSuccess) *p = std::calloc(1, bytes + 16);
  return e;
}
}  // namespace fake

extern "C" {
cudaError_t cudaEventCreate(cudaEvent_t* e) { *e = (cudaEvent_t)8; return fake::call(__func__); }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned) { *e = (cudaEvent_t)8; return fake::call(__func__); }
cudaError_t cudaEventDestroy(cudaEvent_t) { return fake::call(__func__); }
cudaError_t cudaEventElapsedTime(float* ms, cudaEvent_t, cudaEvent_t) { *ms = 1; return fake::call(__func__); }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return fake::call(__func__); }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return fake::no_capture(__func__); }
cudaError_t cudaFree(void* p) { std::free(p); return fake::no_capture(__func__); }
cudaError_t cudaFreeAsync(void* p, cudaStream_t) { std::free(p); fake::held -= p != nullptr; return fake::call(__func__); }
cudaError_t cudaFreeHost(void* p) { std::free(p); return fake::no_capture(__func__); }
cudaError_t cudaGetDevice(int* d) { *d = 0; return fake::call(__func__); }
cudaError_t cudaDeviceGetAttribute(int* v, cudaDeviceAttr, int) { *v = 152; return fake::call(__func__); }
cudaError_t cudaSetDevice(int) { return fake::call(__func__); }
cudaError_t cudaGetDeviceCount(int* c) { *c = 1; return fake::call(__func__); }
const char* cudaGetErrorName(cudaError_t) { return "fake"; }
const char* cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError(void) { return cudaSuccess; }
cudaError_t cudaGraphAddNode(cudaGraphNode_t*, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                             cudaGraphNodeParams*) { return fake::call(__func__); }
cudaError_t cudaGraphConditionalHandleCreate(cudaGraphConditionalHandle*, cudaGraph_t, unsigned, unsigned) { return fake::call(__func__); }
cudaError_t cudaGraphCreate(cudaGraph_t*, unsigned) { return fake::call(__func__); }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return fake::call(__func__); }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return fake::call(__func__); }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t* g, cudaGraph_t, unsigned long long) { *g = (cudaGraphExec_t)8; return fake::call(__func__); }
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return fake::call(__func__); }
cudaError_t cudaHostAlloc(void** p, size_t b, unsigned) { return fake::alloc(__func__, p, b); }
cudaError_t cudaMallocHost(void** p, size_t b) { return fake::alloc(__func__, p, b); }
cudaError_t cudaMalloc(void** p, size_t b) { return fake::alloc(__func__, p, b); }
cudaError_t cudaMallocAsync(void** p, size_t b, cudaStream_t) {
  const cudaError_t e = fake::alloc(__func__, p, b);
  fake::held += e == cudaSuccess;
  return e;
}
cudaError_t cudaMallocFromPoolAsync(void** p, size_t b, cudaMemPool_t, cudaStream_t) { return fake::alloc(__func__, p, b); }
cudaError_t cudaMemcpy(void* d, const void* s, size_t b, cudaMemcpyKind) { std::memcpy(d, s, b); return fake::no_capture(__func__); }
cudaError_t cudaMemcpyAsync(void* d, const void* s, size_t b, cudaMemcpyKind, cudaStream_t) { std::memcpy(d, s, b); return fake::call(__func__); }
cudaError_t cudaMemset(void* p, int v, size_t b) { std::memset(p, v, b); return fake::no_capture(__func__); }
cudaError_t cudaMemsetAsync(void* p, int v, size_t b, cudaStream_t) { std::memset(p, v, b); return fake::call(__func__); }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return fake::no_capture(__func__); }
cudaError_t cudaStreamBeginCaptureToGraph(cudaStream_t, cudaGraph_t, const cudaGraphNode_t*, const cudaGraphEdgeData*, size_t,
                                          cudaStreamCaptureMode) { return fake::no_capture(__func__); }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned) { *s = (cudaStream_t)8; return fake::call(__func__); }
cudaError_t cudaStreamDestroy(cudaStream_t) { return fake::call(__func__); }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t*) { return fake::call(__func__); }
cudaError_t cudaStreamIsCapturing(cudaStream_t, cudaStreamCaptureStatus* s) {
  *s = fake::capturing ? cudaStreamCaptureStatusActive : cudaStreamCaptureStatusNone;
  return fake::call(__func__);
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return fake::no_capture(__func__); }
}

namespace mlp {
// Limits of the order of the kernels' own.
size_t merge_smem_bytes(int) { return 1024; }
size_t merge_ws_bytes(int) { return 1024; }
int merge_smem_max_size() { return 2000; }
int solo_smem_max_size() { return 1500; }
size_t oropt_pass_scratch_bytes(int size, int) { return 64 * (size_t)size; }
bool small_fits(int size, int) { return size <= 385; }
bool merge_one_serves(int njobs, int max_size) { return max_size <= (njobs == 1 ? 2000 : 1000); }
cudaError_t configure_merge(size_t) { return fake::call(__func__); }
cudaError_t configure_merge_one() { return fake::call(__func__); }
cudaError_t configure_small() { return fake::call(__func__); }
cudaError_t launch_ads(const JobDev*, const int32_t*, const int32_t*, uint32_t*, int, int, cudaStream_t, uint32_t*, int) { return fake::call(__func__); }
cudaError_t launch_dist(const int32_t*, const int32_t*, int, int, int32_t*, int32_t*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_dvnd_small(const JobDev*, int, bool, int64_t, int, int, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_grasp(const GraspTask*, int, int, const uint16_t* table, int*, cudaStream_t) {
  fake::grasp_table = table;
  return fake::call(__func__);
}
cudaError_t launch_grasp_ref(const GraspTask*, int, uint32_t*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_grasp_sort(const GraspSortJob*, int, int64_t, int, uint16_t*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_loop_condition(const JobDev*, int, cudaGraphConditionalHandle, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_merge(const JobDev*, int, bool, bool, int, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_merge_one(const JobDev*, int, bool, int, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_merge_solo(const JobDev*, int, bool, bool, int, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_oropt_eval(const JobDev*, int, int, bool, uint64_t*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_oropt_pass(const JobDev*, int, bool, const uint64_t*, uint8_t*, uint32_t*, int64_t*, int*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_oropt_result(const int64_t*, const int*, const uint32_t*, const int64_t*, int, int64_t*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_pass_result(const int64_t*, const uint32_t*, const int64_t*, int, int64_t*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_prepare(const JobDev*, int, bool, bool, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_result(const int64_t*, int, int, const int32_t*, int, int64_t*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_set_fields(JobDev*, int, int, int, int, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_stats_begin(const JobDev*, int, int64_t, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_sweep(const SweepTile*, int, const JobDev*, bool, int, bool, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_sweep_collect(const SweepTile*, int, const JobDev*, bool, int, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_sweep_dvnd(const SweepTile*, int, const JobDev*, int, bool, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_sweep_dvnd_wide(const SweepTile*, int, const JobDev*, int, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_take_keys(const JobDev*, int, int, int, uint64_t*, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_total_finish(const JobDev*, int, bool, bool, int, cudaStream_t) { return fake::call(__func__); }
cudaError_t launch_total_select(const JobDev*, int, bool, cudaStream_t) { return fake::call(__func__); }
}  // namespace mlp
