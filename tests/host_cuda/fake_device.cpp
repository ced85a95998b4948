// A CUDA runtime and kernel layer without a device, for tests of what the host
// does about memory: allocations are addresses with nothing behind them, every
// call succeeds unless memory_left or fail_pinned says otherwise, kernels do
// nothing, and copies to the host are zeros.
#include "fake_device.hpp"

#include "../../include/qmetal/qmetal_kernels.h"

#include <cuda_runtime_api.h>

#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <utility>
#include <vector>

namespace fake {

std::mutex lock;
size_t total = size_t(1) << 40, used = 0;
int fail_pinned = 0, small_runs = 0, overlaps = 0;
size_t used_after_failed_pinned = 0;
bool pinned_failed = false;
std::map<uint32_t, int> permutations;

namespace {
std::map<char *, size_t> blocks;
char *next = reinterpret_cast<char *>(size_t(1) << 44);
}  // namespace

}  // namespace fake

using namespace fake;

extern "C" {

cudaError_t cudaMalloc(void **p, size_t bytes) {
  std::lock_guard<std::mutex> g(lock);
  if (pinned_failed) {
    used_after_failed_pinned = used;
    pinned_failed = false;
  }
  if (used + bytes > total) return cudaErrorMemoryAllocation;
  *p = next;
  blocks[next] = bytes;
  next += (bytes + 511) & ~size_t(255);
  used += bytes;
  return cudaSuccess;
}
cudaError_t cudaFree(void *p) {
  std::lock_guard<std::mutex> g(lock);
  const auto it = blocks.find(static_cast<char *>(p));
  if (it != blocks.end()) {
    used -= it->second;
    blocks.erase(it);
  }
  return cudaSuccess;
}
cudaError_t cudaMemGetInfo(size_t *free_bytes, size_t *all) {
  std::lock_guard<std::mutex> g(lock);
  *free_bytes = total - used;
  *all = total;
  return cudaSuccess;
}
cudaError_t cudaMallocHost(void **p, size_t bytes) {
  std::lock_guard<std::mutex> g(lock);
  if (fail_pinned > 0) {
    fail_pinned--;
    pinned_failed = true;
    return cudaErrorMemoryAllocation;
  }
  *p = std::calloc(bytes, 1);
  return cudaSuccess;
}
cudaError_t cudaHostAlloc(void **p, size_t bytes, unsigned) { return cudaMallocHost(p, bytes); }
cudaError_t cudaFreeHost(void *p) {
  std::free(p);
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void *to, const void *, size_t bytes, cudaMemcpyKind kind, cudaStream_t) {
  if (kind == cudaMemcpyDeviceToHost) std::memset(to, 0, bytes);
  return cudaSuccess;
}
cudaError_t cudaMemsetAsync(void *, int, size_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaGetDevice(int *d) { return *d = 0, cudaSuccess; }
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetDeviceCount(int *n) { return *n = 1, cudaSuccess; }
cudaError_t cudaGetDeviceProperties(cudaDeviceProp *p, int) { return *p = {}, cudaSuccess; }
const char *cudaGetErrorString(cudaError_t) { return "fake"; }
cudaError_t cudaGetLastError() { return cudaSuccess; }
cudaError_t cudaStreamCreateWithFlags(cudaStream_t *s, unsigned) { return *s = nullptr, cudaSuccess; }
cudaError_t cudaStreamDestroy(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaStreamWaitEvent(cudaStream_t, cudaEvent_t, unsigned) { return cudaSuccess; }
cudaError_t cudaStreamBeginCapture(cudaStream_t, cudaStreamCaptureMode) { return cudaSuccess; }
cudaError_t cudaStreamEndCapture(cudaStream_t, cudaGraph_t *g) { return *g = nullptr, cudaSuccess; }
cudaError_t cudaEventCreate(cudaEvent_t *e) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t *e, unsigned) { return *e = nullptr, cudaSuccess; }
cudaError_t cudaEventDestroy(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaEventElapsedTime(float *ms, cudaEvent_t, cudaEvent_t) { return *ms = 0.0f, cudaSuccess; }
cudaError_t cudaGraphDestroy(cudaGraph_t) { return cudaSuccess; }
cudaError_t cudaGraphExecDestroy(cudaGraphExec_t) { return cudaSuccess; }
cudaError_t cudaGraphGetNodes(cudaGraph_t, cudaGraphNode_t *, size_t *n) { return *n = 0, cudaSuccess; }
cudaError_t cudaGraphInstantiate(cudaGraphExec_t *e, cudaGraph_t, unsigned long long) {
  return *e = nullptr, cudaSuccess;
}
cudaError_t cudaGraphLaunch(cudaGraphExec_t, cudaStream_t) { return cudaSuccess; }

// The kernel layer, but for the calls of fake_kernels.c.
size_t qmk_workspace_bytes(uint32_t) { return 1u << 20; }
size_t qmk_sample_workspace_bytes(uint32_t) { return 1u << 20; }
size_t qmk_workspace_scratch_bytes(uint32_t) { return 1u << 18; }
// Neither grows with the width, as the real ones.
uint32_t qmk_small_saves(uint32_t n) { return n > 12 ? 0 : n == 12 ? 16 : 32; }
uint32_t qmk_small_tables(uint32_t n) { return n > 13 ? 0 : n == 13 ? 4 : 32; }
int qmk_apply_permutation(float *, const float *, uint32_t n, const uint64_t *, uint64_t, void *) {
  std::lock_guard<std::mutex> g(lock);
  permutations[n]++;
  return 0;
}
unsigned int *qmk_wait_counter(void *ws) { return static_cast<unsigned int *>(ws); }
int qmk_run_small_counted(float *state, uint32_t n, size_t, const qmk_small_op *,
                          const qmk_small_adjoint *adj, void *tables, size_t bytes, float *saves,
                          uint32_t num_saves, void *, uint32_t *launches) {
  std::lock_guard<std::mutex> g(lock);
  small_runs++;
  *launches = 1;
  const size_t amps = size_t(8) << n;
  std::vector<std::pair<const char *, size_t>> held;
  auto hold = [&](const void *p, size_t size) {
    if (p && size) held.push_back({static_cast<const char *>(p), size});
  };
  hold(state, amps);
  hold(tables, bytes);
  hold(saves, num_saves * amps);
  if (adj) {
    hold(adj->costate, amps);
    hold(adj->grad, 8 * adj->num_grad);
    hold(adj->energy, 8);
  }
  for (size_t i = 0; i < held.size(); i++)
    for (size_t j = 0; j < i; j++)
      if (held[i].first < held[j].first + held[j].second &&
          held[j].first < held[i].first + held[i].second)
        overlaps++;
  for (const auto &h : held) {   // inside one allocation
    auto it = blocks.upper_bound(const_cast<char *>(h.first));
    if (it == blocks.begin() || (--it)->first + it->second < h.first + h.second) overlaps++;
  }
  return 0;
}
}  // extern "C"
