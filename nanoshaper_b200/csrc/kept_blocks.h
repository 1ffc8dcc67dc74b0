// Free blocks of memory that are kept for the next request, up to a number of bytes.
#pragma once
#include <stddef.h>

#include <utility>
#include <vector>

namespace nsg {

struct KeptBlocks {
  std::vector<std::pair<void*, size_t>> blocks;
  size_t bytes = 0;

  // The smallest block of `want` bytes and more, so that a small request does not take the block that the
  // next large one would find.
  bool take(size_t want, void** p, size_t* size) {
    size_t best = blocks.size();
    for (size_t q = 0; q < blocks.size(); q++)
      if (blocks[q].second >= want && (best == blocks.size() || blocks[q].second < blocks[best].second)) best = q;
    if (best == blocks.size()) return false;
    *p = blocks[best].first;
    *size = blocks[best].second;
    bytes -= *size;
    blocks.erase(blocks.begin() + best);
    return true;
  }
  // False when the block would exceed `most` bytes in all: the caller frees it.
  bool give(void* p, size_t size, size_t most) {
    if (bytes + size > most) return false;
    blocks.emplace_back(p, size);
    bytes += size;
    return true;
  }
};

}  // namespace nsg
