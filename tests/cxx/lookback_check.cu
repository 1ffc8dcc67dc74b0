// Kernels around csrc/kernels/lookback.cuh for tests/test_gpu_lookback.py.
#include <cuda_runtime.h>

#include "kernels/lookback.cuh"

namespace {

constexpr int kThreads = 256;

// Every thread brings an error word and a condition of its own; out receives every thread's decision.
__global__ void __launch_bounds__(kThreads) k_decide(unsigned long long* state, unsigned int* ticket, int32_t* err,
                                                     const int32_t* condition, int32_t* out) {
  const nsg::LookBack lb{state, ticket, err + threadIdx.x};
  unsigned int t;
  out[threadIdx.x] = nsg::take_ticket_if(lb, [&] { return condition[threadIdx.x] != 0; }, &t) ? 1 + (int)t : 0;
}

// A ticket per block; out receives every block's offset of its first warp.
__global__ void __launch_bounds__(kThreads) k_offsets(nsg::LookBack lb, unsigned int words, int64_t* out) {
  __shared__ unsigned int s_ticket;
  const unsigned int t = nsg::take_ticket(lb, &s_ticket);
  if (t >= words) return;
  const int64_t off = nsg::warp_offset<kThreads>(lb, t, 1);
  if (threadIdx.x == 0) out[t] = off;
}

}  // namespace

extern "C" int decide(unsigned long long* state, unsigned int* ticket, int32_t* err, const int32_t* condition,
                      int32_t* out) {
  k_decide<<<1, kThreads>>>(state, ticket, err, condition, out);
  return (int)cudaDeviceSynchronize();
}

extern "C" int offsets(unsigned long long* state, unsigned int* ticket, int32_t* err, unsigned int words, int blocks,
                       int64_t* out) {
  k_offsets<<<blocks, kThreads>>>(nsg::LookBack{state, ticket, err}, words, out);
  return (int)cudaDeviceSynchronize();
}
