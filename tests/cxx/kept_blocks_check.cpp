// csrc/kept_blocks.h for tests/test_kept_blocks.py.
#include "kept_blocks.h"

namespace {
nsg::KeptBlocks g_kept;
}

extern "C" long give(long p, long size, long most) { return g_kept.give((void*)p, (size_t)size, (size_t)most); }
extern "C" long take(long want) {  // the block's number, 0 without one
  void* p = nullptr;
  size_t size = 0;
  return g_kept.take((size_t)want, &p, &size) && size >= (size_t)want ? (long)p : 0;
}
extern "C" long bytes() { return (long)g_kept.bytes; }
