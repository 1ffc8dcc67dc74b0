// csrc/transfer.cu on a stand-in of the CUDA runtime in host memory, for tests/test_transfer.py: the
// copies run at once, and calls fail on request.
#include <cuda_runtime.h>

#include <atomic>
#include <cstdint>
#include <cstdlib>
#include <cstring>
#include <map>
#include <mutex>
#include <random>

#include "transfer.cu"

namespace {

std::mutex g_mu;
std::map<void*, size_t> g_pinned;
std::atomic<int> g_allocs{0}, g_allowed_allocs{0}, g_streams{0}, g_allowed_streams{0}, g_pinned_copies{0},
    g_failing_copy{0}, g_pageable_copies{0};
thread_local cudaError_t t_last = cudaSuccess;

cudaError_t done(cudaError_t e) {
  if (e != cudaSuccess) t_last = e;
  return e;
}

bool pinned(const void* p) {
  std::lock_guard<std::mutex> g(g_mu);
  auto it = g_pinned.upper_bound((void*)p);
  return it != g_pinned.begin() && (const char*)p < (const char*)(--it)->first + it->second;
}

}  // namespace

extern "C" {
cudaError_t cudaSetDevice(int) { return cudaSuccess; }
cudaError_t cudaGetLastError(void) {
  const cudaError_t e = t_last;
  t_last = cudaSuccess;
  return e;
}
cudaError_t cudaStreamCreateWithFlags(cudaStream_t* s, unsigned int) {
  if (g_streams++ >= g_allowed_streams) return done(cudaErrorMemoryAllocation);
  *s = (cudaStream_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaStreamDestroy(cudaStream_t s) {
  free(s);
  return cudaSuccess;
}
cudaError_t cudaStreamSynchronize(cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventCreateWithFlags(cudaEvent_t* e, unsigned int) {
  *e = (cudaEvent_t)malloc(1);
  return cudaSuccess;
}
cudaError_t cudaEventDestroy(cudaEvent_t e) {
  free(e);
  return cudaSuccess;
}
cudaError_t cudaEventRecord(cudaEvent_t, cudaStream_t) { return cudaSuccess; }
cudaError_t cudaEventSynchronize(cudaEvent_t) { return cudaSuccess; }
cudaError_t cudaHostAlloc(void** p, size_t bytes, unsigned int) {
  if (g_allocs++ >= g_allowed_allocs) return done(cudaErrorMemoryAllocation);
  *p = malloc(bytes);
  std::lock_guard<std::mutex> g(g_mu);
  g_pinned[*p] = bytes;
  return cudaSuccess;
}
cudaError_t cudaFreeHost(void* p) {
  std::lock_guard<std::mutex> g(g_mu);
  g_pinned.erase(p);
  free(p);
  return cudaSuccess;
}
cudaError_t cudaPointerGetAttributes(cudaPointerAttributes* a, const void* p) {
  a->type = pinned(p) ? cudaMemoryTypeHost : cudaMemoryTypeUnregistered;
  return cudaSuccess;
}
cudaError_t cudaMemcpyAsync(void* dst, const void* src, size_t bytes, cudaMemcpyKind kind, cudaStream_t) {
  if (pinned(kind == cudaMemcpyHostToDevice ? src : dst)) {
    if (++g_pinned_copies == g_failing_copy) return done(cudaErrorUnknown);
  } else {
    g_pageable_copies++;
  }
  memcpy(dst, src, bytes);
  return cudaSuccess;
}
}

// Copies of n_bytes and of 1,000 bytes, the first in three pieces when it goes to the device; out: result
// of the call, bytes that differ, the thread's last error after it, pageable copies made.
extern "C" void transfer_check(int64_t n_bytes, int to_device, int allowed_allocs, int allowed_streams, int failing_copy,
                               int64_t* out) {
  g_allocs = g_streams = g_pinned_copies = g_pageable_copies = 0;
  g_allowed_allocs = allowed_allocs;
  g_allowed_streams = allowed_streams;
  g_failing_copy = failing_copy;
  const size_t sizes[2] = {(size_t)n_bytes, 1000};
  std::mt19937 rng(1);
  std::vector<std::vector<char>> host(2), dev(2);
  std::vector<nsg::TeamCopy> copies;
  for (int q = 0; q < 2; q++) {
    host[q].resize(sizes[q]);
    dev[q].resize(sizes[q]);
    for (char& c : to_device ? host[q] : dev[q]) c = (char)rng();
    nsg::TeamCopy t{dev[q].data(), sizes[q], {}};
    if (to_device && q == 0)
      for (size_t off : {(size_t)0, sizes[0] / 3, sizes[0] / 2 + 1}) t.pieces.push_back({host[q].data() + off, off});
    else
      t.pieces.push_back({host[q].data(), 0});
    copies.push_back(t);
  }
  out[0] = (int64_t)nsg::team_copy(copies, to_device != 0, 0, nullptr);
  out[1] = 0;
  for (int q = 0; q < 2; q++)
    for (size_t i = 0; i < sizes[q]; i++) out[1] += host[q][i] != dev[q][i];
  out[2] = (int64_t)cudaGetLastError();
  out[3] = g_pageable_copies;
  nsg::team_release();
  std::lock_guard<std::mutex> g(g_mu);
  if (!g_pinned.empty()) out[0] = -1;  // everything pinned is given back
}
