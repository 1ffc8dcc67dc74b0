// Ordered offsets in one pass: the blocks of a kernel take tickets, publish the item count of
// their ticket and add up the counts of the tickets before it (decoupled look-back, D. Merrill and
// M. Garland, "Single-pass parallel prefix scan with decoupled look-back", 2016), so that a kernel
// counts, places and writes its items reading its input once, without a scan launch and without a
// host round trip for the total.
//
// A ticket is taken by a block that already runs, and a block publishes its count before it looks
// back, so every count that a block waits for is published by a running block.  The wait is bounded
// all the same: a block that gives up sets *err and returns -1, and its caller writes nothing.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace nsg {

// state: one word per ticket, zero at launch (flag in the top two bits: 1 the ticket's own count,
// 2 the sum up to and including it); ticket: zero at launch.
struct LookBack {
  unsigned long long* state;
  unsigned int* ticket;
  int32_t* err;
};

constexpr int kLookBackErr = 8;

// The block's next ticket (all threads of the block call it).
__device__ __forceinline__ unsigned int take_ticket(const LookBack& lb, unsigned int* s_ticket) {
  __syncthreads();
  if (threadIdx.x == 0) *s_ticket = atomicAdd(lb.ticket, 1u);
  __syncthreads();
  return *s_ticket;
}

// The block's only ticket, and whether the block goes on: its thread 0 decides for all of its threads,
// because another block of the same launch may set the error word at any moment, and threads that
// read it for themselves could part before a warp-wide exchange (all threads of the block call it).
// A block that does not go on leaves a count of 0, so that nobody waits for it.
template <class Condition>
__device__ __forceinline__ bool take_ticket_if(const LookBack& lb, Condition complete, unsigned int* ticket) {
  __shared__ unsigned int s_ticket;
  __shared__ int s_go;
  if (threadIdx.x == 0) {
    const unsigned int t = atomicAdd(lb.ticket, 1u);
    const bool go = *(volatile const int32_t*)lb.err == 0 && complete();
    if (!go) *(volatile unsigned long long*)(lb.state + t) = 1ull << 62;
    s_ticket = t;
    s_go = go;
  }
  __syncthreads();
  *ticket = s_ticket;
  return s_go != 0;
}

// Sum of the counts of the tickets before t, given this ticket's count; the whole block takes part
// and every thread gets the result (-1 when the wait ran out).  A step looks at one earlier ticket
// per thread: with a 32-ticket window the chain of sums moved 32 tickets per L2 round trip, about
// 30 ns a ticket, which was the time of the whole pass on large inputs.
template <int kThreads>
__device__ __forceinline__ int64_t look_back(const LookBack& lb, unsigned int t, int64_t count) {
  constexpr unsigned long long kOwn = 1ull << 62, kSum = 2ull << 62, kMask = kOwn - 1;
  constexpr int kWarps = kThreads / 32;
  __shared__ int s_first[kWarps];
  __shared__ int64_t s_part[kWarps];
  volatile unsigned long long* state = lb.state;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) state[t] = (t == 0 ? kSum : kOwn) | (unsigned long long)count;
  if (t == 0) return 0;
  int64_t sum = 0;
  for (int64_t end = (int64_t)t - 1;; end -= kThreads) {
    const int64_t q = end - threadIdx.x;  // thread 0 looks at the nearest ticket
    unsigned long long w = kSum;          // before ticket 0: nothing
    if (q >= 0) {
      w = state[q];
      for (int spin = 0; (w >> 62) == 0 && spin < (1 << 22); spin++) {
        __nanosleep(20);
        w = state[q];
      }
    }
    // the nearest ticket of the warp whose sum is known; 32: none, -1: a wait ran out
    const unsigned lost = __ballot_sync(0xffffffffu, (w >> 62) == 0);
    const unsigned done = __ballot_sync(0xffffffffu, (w >> 62) == 2);
    const int first = done ? __ffs(done) - 1 : 32;
    int64_t v = lane <= first ? (int64_t)(w & kMask) : 0;
#pragma unroll
    for (int o = 16; o; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if (lane == 0) {
      s_first[warp] = lost ? -1 : first;
      s_part[warp] = v;
    }
    __syncthreads();
    bool found = false, failed = false;
    int64_t part = 0;
#pragma unroll
    for (int x = 0; x < kWarps; x++) {
      if (found) continue;
      failed = failed || s_first[x] < 0;
      part += s_part[x];
      found = s_first[x] < 32;
    }
    __syncthreads();
    if (failed) {
      if (threadIdx.x == 0) atomicExch(lb.err, kLookBackErr);
      return -1;
    }
    sum += part;
    if (found) break;
  }
  if (threadIdx.x == 0) state[t] = kSum | (unsigned long long)(sum + count);
  return sum;
}

// Inclusive sum over a warp.
__device__ __forceinline__ int warp_incl(int v) {
  const int lane = threadIdx.x & 31;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int u = __shfl_up_sync(0xffffffffu, v, o);
    if (lane >= o) v += u;
  }
  return v;
}

// Smallest lane whose inclusive prefix v exceeds k (k below the warp total).
__device__ __forceinline__ int owner_lane(int v, int k) {
  int rr = 0;
#pragma unroll
  for (int step = 16; step; step >>= 1) {
    const int x = __shfl_sync(0xffffffffu, v, rr + step - 1);
    if (x <= k) rr += step;
  }
  return rr;
}

// Offsets of a ticket whose items the warps hold in warp order: every warp brings its item count and
// gets the index of its first item (negative when the wait ran out).
template <int kThreads>
__device__ __forceinline__ int64_t warp_offset(const LookBack& lb, unsigned int t, int warp_count) {
  __shared__ int s_warp[kThreads / 32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) s_warp[w] = warp_count;
  __syncthreads();
  int before = 0, all = 0;
#pragma unroll
  for (int q = 0; q < kThreads / 32; q++) {
    const int v = s_warp[q];
    if (q < w) before += v;
    all += v;
  }
  const int64_t base = look_back<kThreads>(lb, t, all);
  return base < 0 ? -1 : base + before;
}

// Sum over a warp, in every lane.
__device__ __forceinline__ int warp_total(int v) { return (int)__reduce_add_sync(0xffffffffu, (unsigned)v); }

}  // namespace nsg
