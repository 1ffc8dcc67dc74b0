// The marching-cubes case table in device memory, laid out at compile time from mc_cases.h: the
// triangle edge lists (16 bytes per case, -1 terminated, so that a block copies the table with one
// 16-byte load per thread), the cut-edge mask and the triangle count of every case.
#pragma once
#include <stdint.h>

#include "../mc_cases.h"

namespace nsg {

struct McTables {
  alignas(16) int8_t tri[256][16];
  alignas(16) uint8_t ntri[256];
  uint16_t emask[256];
};

constexpr McTables make_mc_tables() {
  McTables T{};
  const int ec[12][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}, {4, 5}, {5, 6}, {6, 7}, {7, 4}, {0, 4}, {1, 5}, {2, 6}, {3, 7}};
  for (int c = 0; c < 256; c++) {
    const char* s = kNsMcCases[c];
    int q = 0;
    for (; s[q] && q < 16; q++) T.tri[c][q] = (int8_t)(s[q] <= '9' ? s[q] - '0' : s[q] - 'a' + 10);
    T.ntri[c] = (uint8_t)(q / 3);
    for (; q < 16; q++) T.tri[c][q] = -1;
    int m = 0;
    for (int e = 0; e < 12; e++)
      if (((c >> ec[e][0]) & 1) != ((c >> ec[e][1]) & 1)) m |= 1 << e;
    T.emask[c] = (uint16_t)m;
  }
  return T;
}

static __device__ const McTables d_mc = make_mc_tables();

}  // namespace nsg
