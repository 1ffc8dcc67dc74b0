// Copies between ordinary (pageable) host memory and the device through pinned blocks, by several
// host threads.
//
// The driver stages a pageable copy through one thread: about 10 GB/s, less where the destination's
// pages are touched for the first time, against 55 GB/s on the link.  Here each thread of a small
// team takes chunks of the copy in turn, with two pinned blocks and a stream of its own: one block
// is on the link while the thread copies the other, and page faults are taken in parallel.
#pragma once
#include <cuda_runtime.h>
#include <stddef.h>

#include <vector>

namespace nsg {

// A run of host memory at offset `off` of a copy (host side of an upload; a download has one piece).
struct HostPiece {
  char* host;
  size_t off;
};

// `bytes` contiguous device bytes and the host pieces, ascending, that make them up.
struct TeamCopy {
  char* dev;
  size_t bytes;
  std::vector<HostPiece> pieces;
};

// Runs the copies (all to the device or all from it) and returns when the data has arrived.  Work
// already queued on `stream` (which may use the device memory) is waited for first.  Copies that are
// small or from pinned memory, and all copies while another thread uses the team or when none of its
// threads can make its stream and pinned blocks, are queued on `stream` itself: an upload may then
// still be on its way out of pinned memory when the call returns, as cudaMemcpyAsync leaves it; a
// download has arrived in every case.
cudaError_t team_copy(const std::vector<TeamCopy>& copies, bool to_device, int device, cudaStream_t stream);

// Frees the team's pinned blocks (kept from one copy to the next, at most 2 MB per thread).
void team_release();

}  // namespace nsg
