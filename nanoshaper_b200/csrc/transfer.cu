// Host thread team for pageable copies (transfer.h).
#include "transfer.h"

#include <algorithm>
#include <atomic>
#include <condition_variable>
#include <cstring>
#include <mutex>
#include <thread>

namespace nsg {

namespace {

constexpr size_t kBlock = (size_t)1 << 20;      // one of a thread's two pinned blocks
constexpr size_t kSmallest = (size_t)1 << 20;   // below, waking the team takes longer than the driver's copy
constexpr int kMostThreads = 8;                 // 8 threads copy at about the rate of the link

struct Chunk {
  int copy;
  size_t off, bytes;
};

struct Job {
  const std::vector<TeamCopy>* copies;
  std::vector<Chunk> chunks;
  bool to_device;
  int device;
  std::atomic<size_t> next{0};
  std::atomic<int> err{0};
};

// Host bytes [off, off + bytes) of a copy, to or from a pinned block.
void host_copy(const TeamCopy& c, size_t off, size_t bytes, char* block, bool to_block) {
  auto it = std::upper_bound(c.pieces.begin(), c.pieces.end(), off,
                             [](size_t o, const HostPiece& p) { return o < p.off; });
  size_t q = (size_t)(it - c.pieces.begin()) - 1;
  while (bytes) {
    const size_t end = q + 1 < c.pieces.size() ? c.pieces[q + 1].off : c.bytes;
    const size_t n = std::min(bytes, end - off);
    char* host = c.pieces[q].host + (off - c.pieces[q].off);
    if (to_block) memcpy(block, host, n);
    else memcpy(host, block, n);
    block += n;
    off += n;
    bytes -= n;
    q++;
  }
}

struct Member {
  char* block[2] = {nullptr, nullptr};
  int device = -1;
  cudaStream_t stream = nullptr;
  cudaEvent_t ev[2] = {nullptr, nullptr};

  void drop_stream() {
    if (stream) cudaStreamDestroy(stream);
    for (auto& e : ev) {
      if (e) cudaEventDestroy(e);
      e = nullptr;
    }
    stream = nullptr;
    device = -1;
  }

  cudaError_t ready(int dev) {
    cudaError_t e = cudaSetDevice(dev);
    if (e != cudaSuccess) return e;
    if (device != dev) {
      drop_stream();
      if ((e = cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking)) != cudaSuccess) {
        stream = nullptr;
        return e;
      }
      for (auto& v : ev)
        if ((e = cudaEventCreateWithFlags(&v, cudaEventDisableTiming)) != cudaSuccess) {
          v = nullptr;
          drop_stream();
          return e;
        }
      device = dev;
    }
    for (auto& b : block)
      if (!b && (e = cudaHostAlloc((void**)&b, kBlock, cudaHostAllocPortable)) != cudaSuccess) {
        b = nullptr;
        return e;
      }
    return cudaSuccess;
  }

  // This member's share of the job; without a stream or pinned blocks it leaves the chunks to the others.
  void work(Job& job) {
    cudaError_t e = ready(job.device);
    if (e != cudaSuccess) {
      cudaGetLastError();
      return;
    }
    int k = 0;
    Chunk prev{};
    while (e == cudaSuccess && job.err.load(std::memory_order_relaxed) == 0) {
      const size_t i = job.next.fetch_add(1);
      if (i >= job.chunks.size()) break;
      const Chunk ch = job.chunks[i];
      const TeamCopy& c = (*job.copies)[ch.copy];
      char* b = block[k & 1];
      if (job.to_device) {
        if (k >= 2) e = cudaEventSynchronize(ev[k & 1]);
        if (e != cudaSuccess) break;
        host_copy(c, ch.off, ch.bytes, b, true);
        e = cudaMemcpyAsync(c.dev + ch.off, b, ch.bytes, cudaMemcpyHostToDevice, stream);
        if (e == cudaSuccess) e = cudaEventRecord(ev[k & 1], stream);
      } else {
        e = cudaMemcpyAsync(b, c.dev + ch.off, ch.bytes, cudaMemcpyDeviceToHost, stream);
        if (e == cudaSuccess) e = cudaEventRecord(ev[k & 1], stream);
        if (e == cudaSuccess && k > 0) e = finish(job, prev, (k - 1) & 1);
        prev = ch;
      }
      k++;
    }
    // the last block, and whatever is still on the link before the blocks are used again
    if (!job.to_device && e == cudaSuccess && k > 0) e = finish(job, prev, (k - 1) & 1);
    const cudaError_t s = cudaStreamSynchronize(stream);
    if (e == cudaSuccess) e = s;
    if (e != cudaSuccess) {
      int none = 0;
      job.err.compare_exchange_strong(none, (int)e);
    }
  }

  cudaError_t finish(Job& job, const Chunk& ch, int b) {
    const cudaError_t e = cudaEventSynchronize(ev[b]);
    if (e == cudaSuccess) host_copy((*job.copies)[ch.copy], ch.off, ch.bytes, block[b], false);
    return e;
  }
};

// One job at a time: `use` is held by the thread whose job it is, which works as member 0.
struct Team {
  std::mutex use;
  std::mutex mu;
  std::condition_variable wake, done;
  Member member[kMostThreads];
  int threads = 0;  // of member[1..threads]
  uint64_t generation = 0;
  int working = 0;
  Job* job = nullptr;

  void start() {
    if (threads) return;
    const unsigned hw = std::thread::hardware_concurrency();
    const int want = std::max(1, std::min<int>(kMostThreads, (int)hw / 2)) - 1;
    for (int q = 1; q <= want; q++) {
      try {
        std::thread([this, q] { loop(q); }).detach();
      } catch (...) {
        break;  // fewer threads: the others, and the caller, do the work
      }
      threads = q;
    }
  }

  void loop(int q) {
    uint64_t seen = 0;
    std::unique_lock<std::mutex> l(mu);
    while (true) {
      wake.wait(l, [&] { return generation != seen; });
      seen = generation;
      Job* j = job;
      if (!j) continue;
      l.unlock();
      member[q].work(*j);
      l.lock();
      if (--working == 0) done.notify_one();
    }
  }

  void run(Job& j) {
    {
      std::lock_guard<std::mutex> l(mu);
      job = &j;
      working = threads;
      generation++;
    }
    wake.notify_all();
    member[0].work(j);
    std::unique_lock<std::mutex> l(mu);
    done.wait(l, [&] { return working == 0; });
    job = nullptr;
  }
};

Team& team() {
  static Team* t = new Team;  // its threads run to the process's end
  return *t;
}

bool is_pageable(const void* p) {
  cudaPointerAttributes a{};
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return a.type == cudaMemoryTypeUnregistered;
}

cudaError_t plain_copy(const TeamCopy& c, bool to_device, cudaStream_t stream) {
  for (size_t q = 0; q < c.pieces.size(); q++) {
    const size_t off = c.pieces[q].off;
    const size_t n = (q + 1 < c.pieces.size() ? c.pieces[q + 1].off : c.bytes) - off;
    if (!n) continue;
    const cudaError_t e = to_device
                              ? cudaMemcpyAsync(c.dev + off, c.pieces[q].host, n, cudaMemcpyHostToDevice, stream)
                              : cudaMemcpyAsync(c.pieces[q].host, c.dev + off, n, cudaMemcpyDeviceToHost, stream);
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

}  // namespace

cudaError_t team_copy(const std::vector<TeamCopy>& copies, bool to_device, int device, cudaStream_t stream) {
  // a copy goes to the team when its host side is pageable; its small companions go with it
  size_t total = 0;
  std::vector<char> paged(copies.size(), 0);
  for (size_t q = 0; q < copies.size(); q++)
    if (copies[q].bytes && !copies[q].pieces.empty() && is_pageable(copies[q].pieces[0].host)) {
      paged[q] = 1;
      total += copies[q].bytes;
    }
  Team& t = team();
  std::unique_lock<std::mutex> use(t.use, std::defer_lock);
  const bool by_team = total >= kSmallest && use.try_lock();
  cudaError_t e = cudaSuccess;
  for (size_t q = 0; q < copies.size(); q++)
    if (copies[q].bytes && !(by_team && paged[q]))
      if ((e = plain_copy(copies[q], to_device, stream)) != cudaSuccess) return e;
  if (!by_team || !to_device) {
    // downloads: what was queued has arrived; the team copies what the stream has finished
    if (!to_device && (e = cudaStreamSynchronize(stream)) != cudaSuccess) return e;
    if (!by_team) return cudaSuccess;
  } else if ((e = cudaStreamSynchronize(stream)) != cudaSuccess) {
    return e;
  }
  t.start();
  Job job;
  job.copies = &copies;
  job.to_device = to_device;
  job.device = device;
  // chunks small enough for every thread to get two
  const size_t share = total / (2 * ((size_t)t.threads + 1));
  const size_t step = std::min(kBlock, std::max<size_t>((size_t)128 << 10, (share + 65535) & ~(size_t)65535));
  for (size_t q = 0; q < copies.size(); q++)
    if (paged[q])
      for (size_t off = 0; off < copies[q].bytes; off += step)
        job.chunks.push_back(Chunk{(int)q, off, std::min(step, copies[q].bytes - off)});
  t.run(job);
  e = (cudaError_t)job.err.load();
  if (e != cudaSuccess || job.next.load() >= job.chunks.size()) return e;
  // no member could start (a limit on pinned memory, say): the runtime's copy
  for (size_t q = 0; q < copies.size(); q++)
    if (paged[q] && (e = plain_copy(copies[q], to_device, stream)) != cudaSuccess) return e;
  return to_device ? cudaSuccess : cudaStreamSynchronize(stream);
}

void team_release() {
  Team& t = team();
  std::lock_guard<std::mutex> use(t.use);
  for (Member& m : t.member) {
    m.drop_stream();
    for (auto& b : m.block) {
      if (b) cudaFreeHost(b);
      b = nullptr;
    }
  }
}

}  // namespace nsg
