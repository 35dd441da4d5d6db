// The degree-ranked copy of a CSR's edges (csrc/ranked.cu) and its work items, shared by the
// Bisson-style count (ranked.cu) and the searched families (tc.cu).  Internal header.
#pragma once

#include "bisson.cuh"

namespace atc {

// counters of one copy; the first six are the kinds of work items
enum { kc15, kc16, kc17, kcFilter, kcWarp, kcBlock, kcNext15, kcNext16, kcNext17, kcNextFilter, kcNextWarp,
       kcNextBlock, kcMid,
       kcBig, kcNextMid, kcNextBig, kcTooLong, kcMaxRow, kcError, kcNextDense, kcCount };

// Work items (target, chunk): the kinds of ranked.cu, or, for the searches, the targets that take a
// warp or a CTA with N+(v) as a list (`list`: warp items from the front, CTA items from the back).
struct RankItemLists {
  int2 *t15, *t16, *t17, *filter, *list;
  int64_t lcap;
  int chunk;       // entries per warp item of the 15- and 16-bit kinds and the filter
  int warp_chunk;  // and of the list kinds
  int block_chunk;
  int warp_max;    // longest N+(v) of a warp's list item
  int mid_min;     // fewest entries for which a target of rank below 2^17 takes a CTA's bitmap
};

struct RankedCopy {
  DevBuf<char> mem;          // null: there was no room
  int64_t n = 0, m = 0;
  const int64_t* roff = nullptr;    // n + 1: rows by rank
  const int32_t* rcols = nullptr;   // m + 16: ids are ranks, rows ascending
  const uint4* r16 = nullptr;       // rows of 16-bit ids, starting at multiples of eight
  const int64_t* gstart = nullptr;  // n + 1: the entries of every target
  const uint2* ent = nullptr;       // (row start, prefix length)
  const int32_t* nids = nullptr;    // n: how many of them a target has; the rest of its edges are tested as words
  const uint4* dense = nullptr;     // rows of the ranks below dense_rows as bitmaps (null: none)
  int dense_rows = 0, dense_sources = 0;
  int* ctr = nullptr;               // kcCount
  RankItemLists li{};
  bool long_rows = false;           // rows above the register sorts may exist (ctr[kcTooLong])
};

// bitmaps: items of all kinds and the 16-bit rows; otherwise list items only.
atc_status build_ranked(const atc_csr* csr, bool bitmaps, RankedCopy* rc, cudaStream_t s, int* launches);

namespace {

// The list items, for the kernels of bisson.cuh and tc.cu.
struct RankedItems {
  static constexpr bool kBatch = false;
  static constexpr int kMinBlocks = 0;
  const int2* p;
  const int64_t* gstart;
  int64_t cap;
  int64_t chunk;
  bool block;
  __device__ __forceinline__ GroupItem get(const CsrView& g, int i) const {
    const int2 c = block ? p[cap - 1 - i] : p[i];
    const int64_t b = gstart[c.x] + c.y * chunk, e = min(gstart[c.x + 1], b + chunk);
    const int64_t hb = g.off[c.x], dh = g.off[c.x + 1] - hb;
    int32_t mode;
    if (!block) mode = dh <= 8 ? 0 : 1;
    else mode = dh <= kHashMax ? 0 : (g.cols[hb + dh - 1] - g.cols[hb] < kTabWords * 32 ? 1 : 2);
    return GroupItem{c.x, mode, b, e};
  }
};

}  // namespace

}  // namespace atc
