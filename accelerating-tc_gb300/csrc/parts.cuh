// Part tables: a sorted list's id range cut into equal parts, so that one read brackets an id to the
// few list elements of its part.  Shared by the searched counts (tc.cu) and the k-clique rows
// (kcl.cu).  Internal header.
#pragma once

#include <stdint.h>

namespace atc {

namespace {

// The part table of the sorted list T[0, d), d <= 65535, built by `threads` threads (this one `t`)
// with sync() between the steps: start[b] = the first element of part b or above, then part[].
// Returns the shift.
template <class Sync>
__device__ __forceinline__ int build_parts(const int32_t* T, int d, int max_parts, uint16_t* start, uint32_t* part, int t,
                                           int threads, Sync sync) {
  const int32_t base = T[0];
  const uint32_t range = (uint32_t)(T[d - 1] - base);
  int parts = 32;
  while (parts < 2 * d && parts < max_parts) parts <<= 1;
  int shift = 0;
  while ((range >> shift) >= (uint32_t)parts) ++shift;
  for (int j = t; j < d; j += threads) {
    const int c = (int)((uint32_t)(T[j] - base) >> shift);
    const int p = j ? (int)((uint32_t)(T[j - 1] - base) >> shift) : -1;
    for (int b = p + 1; b <= c; ++b) start[b] = (uint16_t)j;
    if (j == d - 1) start[c + 1] = (uint16_t)d;
  }
  sync();
  const int used = (int)(range >> shift) + 1;
  for (int b = t; b < used; b += threads) part[b] = (uint32_t)start[b] | (uint32_t)start[b + 1] << 16;
  sync();
  return shift;
}

}  // namespace

}  // namespace atc
