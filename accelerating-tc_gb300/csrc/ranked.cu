// Triangle counting on a degree-ranked copy of the edges: the Bisson-style count of a whole
// CSR built by preTC (Bisson/tc.cu:18-104: a bitmap of N+(u), other lists streamed through it).
//
// The count does not depend on the orientation, so this path picks its own.  Vertices are
// numbered by descending degree (rank 0 = the largest) and every edge points from its endpoint
// of higher rank to the one of lower rank; rows are sorted.  For an edge u -> v the common
// successors w all have rank(w) < rank(v), so they lie in the part of row u before v: only that
// prefix is tested against N+(v).  Over all edges these are sum_u C(d+(u), 2) tests, 0.6 of the
// sum of min(d+u, d+v) that the grouping of whole lists streams (R-MAT scales 16..20), and
// rows are short, so a row's later reads hit in L2.  And N+(v) lies in [0, rank(v)): the targets
// that take nearly all tests have small ranks, and their N+(v) is a bitmap in shared memory
// addressed by the id itself: one 4-byte shared load and a shift per test, against a hash, a
// 16-byte bucket, four compares and a queue (about 8 instructions per 32 tests against 31).
//
//   passes: degrees -> rank (radix sort on the degree bits) -> out-degrees and group sizes ->
//   scans -> rows (scatter, then sorted in registers) -> rows of the lowest ranks as bitmaps ->
//   entries (row start, prefix length) grouped by target -> work items -> count.  Nothing waits on
//   the host before the count.
//   a long prefix before a target of low rank: the source's and the target's rows as bitmaps, ANDed
//   word by word, 128 candidates per 16 bytes against eight ids; such edges need no entry.  Other
//   targets of rank below 2^16: a warp per chunk of entries, its own bitmap of 4 or 8 KB, rows
//   read as 16-bit ids; the rest (a quarter of the tests at R-MAT scale 24): a warp's bitmap that is
//   exact for low ids and a filter for the others, or, with many entries, a CTA's of 16 KB.
//
// Measured (R-MAT scale 24, A-direction + A-order; whole lists grouped at the longer endpoint ->
// this path): 117.5 -> 35.6 ms, of which the passes take 12.3 ms (entries 4.8, group sizes 2.3,
// row sorts 2.9, rows 1.4) and the count 23.3: words 4, other ranks below 2^15 5, 2^16 5.5, 2^17 3,
// the filter 6.  Without the words the ranks below 2^15 took 15.7 and the entries 5.7 (47.1 in all):
// bound by the shared and L1 pipe (two wavefronts per 32 tests, one of them bank conflicts) and by
// issue (10 warp instructions per 32 tests).  Scale 22: 8.6 -> 6.2 ms, scale 20: 1.86 ->
// 1.4 (4.45 by whole lists); Chung-Lu n = 700 001, which has few dense rows: 1.30 -> 1.09.
// Tried: 32-bit rows and one entry a warp at a time 68 ms; 32-lane scans of short prefixes
// instead of lane groups 88 ms; rows on 128-byte lines 1-4 % for twice the copy.
#include <algorithm>
#include <climits>
#include <cmath>

#include "ranked.cuh"

namespace atc {

namespace {

constexpr int kHub = 8192;              // group sizes of the lowest ranks are counted in shared memory
constexpr int kHubEntry = 1024;         // ranks whose group cursors are reserved once per tile
constexpr int kTile = 4096;             // edges per tile of the entry pass
constexpr int kRank15 = (1 << 15) - 1;  // targets below: a warp's bitmap of 4 KB
constexpr int kRank16 = (1 << 16) - 1;  // below: a warp's bitmap of 8 KB; ids in 16 bits
constexpr int kRank17 = 1 << 17;        // below, with entries, on wide graphs: a small CTA's bitmap of 16 KB
constexpr int kRankBlockChunk = 1024;   // entries per CTA item
constexpr int kRankMidMin = 96;         // fewer entries than these do not pay for a CTA's bitmap
// Lanes that read a prefix, by the mean of min(d+u, d+v).  Targets below 2^15, whose long prefixes are
// words: four, from kWideMean15 eight (R-MAT scale 20, mean 132: 1.47 and 1.51 ms; scale 22, 187: 7.1 and
// 7.0; scale 24, 270: 41.0 and 40.2; Chung-Lu 1.26 and 1.31); the filter likewise.  Targets below 2^16:
// eight, from kWideMean 16; from there too, targets below 2^17 take a CTA's bitmap (scale 24: 37.5 ms,
// 38.5 with the filter; scale 22: 6.7 and 6.5).
constexpr int64_t kWideMean15 = 160, kWideMean = 224;
constexpr int kDenseRows = 1 << 15;     // rows that may be kept as bitmaps
constexpr int kDenseSources = 4;        // times as many rows are looked at for targets among them
// Small items (filter, middle rows to sort, rows with few words) per atomic on their counter: one
// address takes about one atomic per ns, which was the whole time of the filter's 470 000 items on
// Chung-Lu n = 700 001 (303 us; 189 by fours) and of the words' 105 000 rows there (104; 80).  The larger
// items of the ranks below 2^16 lose by it (103 -> 125 us): their tail.
constexpr int kGrab = 4;
constexpr int kRankRowMax = kTabWords;  // longest row the CTA sort holds (64 KB)
constexpr int kRankWarpRow = 1024;      // longest row a warp sorts in registers

__global__ void rank_keys_kernel(const int64_t* off, const int32_t* indeg, int64_t n, int B, int db, uint64_t* keys) {
  const uint64_t top = (1ull << db) - 1;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    const uint64_t d = (uint64_t)(off[v + 1] - off[v]) + (uint64_t)indeg[v];
    keys[v] = (top - d) << B | (uint64_t)v;
  }
}

__global__ void rank_scatter_kernel(const uint64_t* sorted, int64_t n, int B, int32_t* rank) {
  const uint64_t mask = (1ull << B) - 1;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    rank[sorted[i] & mask] = (int32_t)i;
}

// Out-degrees by rank, every edge's slot in its row, and the edges per target.  Edges of one
// source are contiguous, so a warp takes each run of one row with one atomic; the targets are
// hubs, whose counters would serialise: the lowest ranks are counted per CTA.
__global__ void __launch_bounds__(512) rank_count_kernel(const int32_t* esrc, const int32_t* cols, int64_t m,
                                                         const int32_t* rank, int32_t* deg, int32_t* cnt, uint32_t* slot) {
  __shared__ int hub[kHub];
  for (int j = threadIdx.x; j < kHub; j += blockDim.x) hub[j] = 0;
  __syncthreads();
  const int lane = threadIdx.x & 31;
  const int64_t m_pad = (m + 31) & ~31ll;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m_pad; i += (int64_t)gridDim.x * blockDim.x) {
    int32_t hi = -1, lo = 0;
    if (i < m) {
      const int32_t a = __ldg(rank + esrc[i]), b = __ldg(rank + cols[i]);
      hi = max(a, b);
      lo = min(a, b);
      if (lo < kHub) atomicAdd(&hub[lo], 1);
      else atomicAdd(&cnt[lo], 1);
    }
    const unsigned same = __match_any_sync(0xffffffffu, hi);
    const int lead = __ffs(same) - 1;
    int base = 0;
    if (hi >= 0 && lane == lead) base = atomicAdd(&deg[hi], __popc(same));
    base = __shfl_sync(0xffffffffu, base, lead);
    if (hi >= 0) slot[i] = (uint32_t)(base + __popc(same & ((1u << lane) - 1)));
  }
  __syncthreads();
  for (int j = threadIdx.x; j < kHub; j += blockDim.x)
    if (hub[j]) atomicAdd(&cnt[j], hub[j]);
}

// Rows of the 16-bit copy start at multiples of eight ids: their lengths in such pieces.
__global__ void rank_pieces_kernel(const int32_t* deg, int64_t n, int32_t* pieces) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v <= n; v += (int64_t)gridDim.x * blockDim.x)
    pieces[v] = v < n ? (deg[v] + 7) >> 3 : 0;
}

__global__ void rank_rows_kernel(const int32_t* esrc, const int32_t* cols, int64_t m, const int32_t* rank,
                                 const uint32_t* slot, const int64_t* roff, int32_t* rcols) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += (int64_t)gridDim.x * blockDim.x) {
    const int32_t a = __ldg(rank + esrc[i]), b = __ldg(rank + cols[i]);
    rcols[__ldg(roff + max(a, b)) + slot[i]] = min(a, b);
  }
}

// Rows of up to 32 elements: a warp takes 32 consecutive rows, cuts them into windows of whole
// rows of at most 32 elements together and sorts each window by (row, id) across its lanes.
// Longer rows go on a list each for the warp and the CTA sort.  Key: 32 bits, five for the row of
// the window and 27 for the id, 64 for more than 2^27 vertices
// (Chung-Lu n = 700 001, 11 M edges: 80 us with 64, 64 with 32).
template <class Key>
__global__ void rank_sort_small_kernel(const int64_t* roff, int64_t n, int32_t* rcols, int32_t* mid, int32_t* big,
                                       int* ctr) {
  constexpr int kIdBits = sizeof(Key) == 4 ? 27 : 32;
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t rb = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; rb * 32 < n; rb += warps) {
    const int64_t row = min(rb * 32 + lane, n);
    const int64_t start = __ldg(roff + row), end = __ldg(roff + min(row + 1, n));
    const int len = (int)(end - start);
    const unsigned mm = __ballot_sync(0xffffffffu, len > 32 && len <= kRankWarpRow);
    const unsigned mb = __ballot_sync(0xffffffffu, len > kRankWarpRow);
    if (mm) {
      int at = 0;
      if (lane == 0) at = atomicAdd(&ctr[kcMid], __popc(mm));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (len > 32 && len <= kRankWarpRow) mid[at + __popc(mm & ((1u << lane) - 1))] = (int32_t)row;
    }
    if (mb) {
      int at = 0;
      if (lane == 0) at = atomicAdd(&ctr[kcBig], __popc(mb));
      at = __shfl_sync(0xffffffffu, at, 0);
      if (len > kRankWarpRow) big[at + __popc(mb & ((1u << lane) - 1))] = (int32_t)row;
    }
    const unsigned multi = __ballot_sync(0xffffffffu, len >= 2 && len <= 32);
    int c = 0;  // first row of the window
    while (c < 32 && (multi >> c)) {
      c += __ffs(multi >> c) - 1;  // rows of fewer than two elements need no sort
      const int64_t s0 = __shfl_sync(0xffffffffu, start, c);
      const unsigned fit = __ballot_sync(0xffffffffu, lane >= c && end - s0 <= 32);
      const int last = 31 - __clz(fit);  // rows c..last; row c fits
      const int64_t e0 = __shfl_sync(0xffffffffu, end, last);
      const bool valid = s0 + lane < e0;
      int k = 0;  // the last row that starts at or before this element
      const int rel = (int)(start - s0);  // negative for rows before the window
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, rel, k + step) <= lane) k += step;
      Key key = valid ? (Key)k << kIdBits | (uint32_t)rcols[s0 + lane] : ~(Key)0;
#pragma unroll
      for (int kk = 2; kk <= 32; kk <<= 1)
#pragma unroll
        for (int j = kk >> 1; j > 0; j >>= 1) {
          const Key y = __shfl_xor_sync(0xffffffffu, key, j);
          const bool keep_min = ((lane & j) == 0) == ((lane & kk) == 0);
          key = keep_min == (key < y) ? key : y;
        }
      if (valid) rcols[s0 + lane] = (int32_t)(uint32_t)(key & (((Key)1 << kIdBits) - 1));
      c = last + 1;
    }
  }
}

// Ascending bitonic sort of R * 32 values held R a lane (element i = register i / 32, lane
// i % 32).
template <int R>
__device__ __forceinline__ void warp_sort(int32_t (&x)[R], int lane) {
#pragma unroll
  for (int k = 2; k <= 32 * R; k <<= 1)
#pragma unroll
    for (int j = k >> 1; j > 0; j >>= 1) {
      if (j >= 32) {
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (!(r & (j / 32))) {
            const int q = r | (j / 32);
            const bool up = !(r & (k / 32));
            const int32_t lo = min(x[r], x[q]), hi = max(x[r], x[q]);
            x[r] = up ? lo : hi;
            x[q] = up ? hi : lo;
          }
      } else {
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int32_t y = __shfl_xor_sync(0xffffffffu, x[r], j);
          const bool up = k >= 32 ? !(r & (k / 32)) : !(lane & k);
          x[r] = up == ((lane & j) == 0) ? min(x[r], y) : max(x[r], y);
        }
      }
    }
}

template <int R>
__device__ __forceinline__ void warp_sort_row(int32_t* p, int len, int lane) {
  int32_t x[R];
#pragma unroll
  for (int r = 0; r < R; ++r) x[r] = r * 32 + lane < len ? p[r * 32 + lane] : INT32_MAX;
  warp_sort<R>(x, lane);
#pragma unroll
  for (int r = 0; r < R; ++r)
    if (r * 32 + lane < len) p[r * 32 + lane] = x[r];
}

__global__ void __launch_bounds__(256) rank_sort_mid_kernel(const int64_t* roff, const int32_t* mid, int32_t* rcols,
                                                            int* ctr) {
  const int lane = threadIdx.x & 31;
  const int total = ctr[kcMid];
  for (int it = 0, it_end = 0;; ++it) {
    if (it == it_end) {
      if (lane == 0) it = atomicAdd(&ctr[kcNextMid], kGrab);
      it = __shfl_sync(0xffffffffu, it, 0);
      it_end = it + kGrab;
    }
    if (it >= total) break;
    const int32_t u = mid[it];
    const int64_t b = __ldg(roff + u);
    const int len = (int)(__ldg(roff + u + 1) - b);
    int32_t* p = rcols + b;
    if (len <= 64) warp_sort_row<2>(p, len, lane);
    else if (len <= 128) warp_sort_row<4>(p, len, lane);
    else if (len <= 256) warp_sort_row<8>(p, len, lane);
    else if (len <= 512) warp_sort_row<16>(p, len, lane);
    else warp_sort_row<32>(p, len, lane);
  }
}

// Rows beyond kRankWarpRow, in shared memory; one beyond kRankRowMax gives the count up
// (ctr[kcTooLong]: the caller counts by whole lists instead).
__global__ void __launch_bounds__(1024) rank_sort_big_kernel(const int64_t* roff, const int32_t* big, int32_t* rcols,
                                                             int* ctr) {
  extern __shared__ __align__(16) int32_t sm[];  // kRankRowMax
  __shared__ int item;
  const int total = ctr[kcBig];
  for (;;) {
    if (threadIdx.x == 0) item = atomicAdd(&ctr[kcNextBig], 1);
    __syncthreads();
    const int it = item;
    if (it >= total) break;
    const int32_t u = big[it];
    const int64_t b = roff[u], len = roff[u + 1] - b;
    if (len > kRankRowMax) {
      if (threadIdx.x == 0) ctr[kcTooLong] = 1;
      __syncthreads();
      continue;
    }
    int pow2 = 2 * kRankWarpRow;
    while (pow2 < (int)len) pow2 <<= 1;
    for (int j = threadIdx.x; j < pow2; j += blockDim.x) sm[j] = j < len ? rcols[b + j] : INT32_MAX;
    __syncthreads();
    for (int k = 2; k <= pow2; k <<= 1)
      for (int j = k >> 1; j > 0; j >>= 1) {
        for (int t = threadIdx.x; t < pow2 / 2; t += blockDim.x) {
          const int i = (t / j) * 2 * j + (t & (j - 1)), q = i + j;
          const bool up = (i & k) == 0;
          const int32_t x = sm[i], y = sm[q];
          if ((x > y) == up) {
            sm[i] = y;
            sm[q] = x;
          }
        }
        __syncthreads();
      }
    for (int j = threadIdx.x; j < len; j += blockDim.x) rcols[b + j] = sm[j];
    __syncthreads();
  }
}

// piece_row[t] = the row that holds element 32 t.
__global__ void rank_piece_rows_kernel(const int64_t* roff, int64_t n, int32_t* piece_row) {
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n; u += (int64_t)gridDim.x * blockDim.x) {
    const int64_t b = roff[u], e = roff[u + 1];
    for (int64_t t = (b + 31) >> 5; t << 5 < e; ++t) piece_row[t] = (int32_t)u;
  }
}

// Rows of the ranks below `rows` (at most 2^15) once more as bitmaps, in pieces of 128 bits: row v
// has v / 128 + 1 of them, from dense_start(v) on.
__host__ __device__ __forceinline__ uint32_t dense_start(uint32_t v) {
  const uint32_t a = v >> 7, b = v & 127;
  return (a + 1) * (64 * a + b);
}

// Whether the prefix of len ids before target v is better tested as words, by ANDing the rows of
// the source and of v: a piece of 128 bits against kWordGain times a piece of eight ids, which costs
// a look at every id and the edge's entry.  Gains of 2, 3, 4, 6, 8, 12 and 24: 41.8, 40.2, 39.9, 39.9, 40.2,
// 40.2 and 40.3 ms at R-MAT scale 24; 3, 6, 12 and 24 at scale 20: 1.55, 1.47, 1.52 and 1.61.
constexpr int kWordGain = 6;
__device__ __forceinline__ bool words_pay(uint32_t len, uint32_t v) {
  return kWordGain * ((len + 7) >> 3) > (v >> 7) + 1;
}

constexpr int kDenseWarps = 8;
__global__ void __launch_bounds__(kDenseWarps * 32) rank_dense_kernel(const int64_t* roff, const int32_t* rcols, int rows,
                                                                      uint4* dense) {
  __shared__ __align__(16) uint32_t smem[kDenseWarps][1 << 10];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  uint32_t* T = smem[w];
  uint4* T4 = reinterpret_cast<uint4*>(T);
  const int warps = gridDim.x * kDenseWarps;
  for (int u = blockIdx.x * kDenseWarps + w; u < rows; u += warps) {
    const int pieces = (u >> 7) + 1;
    for (int j = lane; j < pieces; j += 32) T4[j] = make_uint4(0u, 0u, 0u, 0u);
    __syncwarp();
    const int64_t e = __ldg(roff + u + 1);
    for (int64_t j = __ldg(roff + u) + lane; j < e; j += 32) {
      const int32_t x = __ldg(rcols + j);
      atomicOr(&T[x >> 5], 1u << (x & 31));
    }
    __syncwarp();
    uint4* to = dense + dense_start(u);
    for (int j = lane; j < pieces; j += 32) to[j] = T4[j];
    __syncwarp();
  }
}

// Entry of every edge in its target's group: where the source's row starts and how much of it
// lies before the target.  Targets below below16 read the 16-bit copy of the rows (r16, starts in
// pieces of eight ids), written here; the others the rows themselves.  A tile's entries of the
// most contended targets take their places with one atomic per tile and target.  Edges that
// are tested as words have none: those of the first `sources` rows to targets below `rows` for
// which that pays.
constexpr int kEntryThreads = 1024;
constexpr int kEntryEach = kTile / kEntryThreads;
__global__ void __launch_bounds__(kEntryThreads, 2) rank_entries_kernel(const int64_t* roff, int64_t n, int64_t m,
                                                                     const int32_t* rcols, const int32_t* piece_row,
                                                                     const int64_t* gstart, const int64_t* roff8,
                                                                     int32_t below16, int32_t rows, int32_t sources,
                                                                     int32_t* gcur, uint16_t* r16, uint2* ent) {
  __shared__ int hub[kHubEntry];
  const int64_t tiles = (m + kTile - 1) / kTile;
  for (int64_t t = blockIdx.x; t < tiles; t += gridDim.x) {
    for (int j = threadIdx.x; j < kHubEntry; j += kEntryThreads) hub[j] = 0;
    __syncthreads();
    int32_t lo[kEntryEach];
    uint32_t st[kEntryEach], len[kEntryEach];
    int pos[kEntryEach];
#pragma unroll
    for (int q = 0; q < kEntryEach; ++q) {
      const int64_t p = t * kTile + q * kEntryThreads + threadIdx.x;
      lo[q] = -1;
      if (p < m) {
        // the last row that starts at or before p: the warp's 32 elements lie in one piece, most
        // often of one row (a search over the tile's rows instead took 5.8 ms at R-MAT scale 24)
        const int64_t pc = p >> 5;
        int32_t a = __ldg(piece_row + pc), b = (pc + 1) << 5 < m ? __ldg(piece_row + pc + 1) : (int32_t)(n - 1);
        while (a < b) {
          const int32_t mid = a + ((b - a + 1) >> 1);
          if (__ldg(roff + mid) <= p) a = mid; else b = mid - 1;
        }
        lo[q] = rcols[p];
        st[q] = (uint32_t)__ldg(roff + a);
        len[q] = (uint32_t)p - st[q];
        if (lo[q] < below16) {
          const int64_t r8 = __ldg(roff8 + a);
          st[q] = (uint32_t)r8;
          r16[8 * r8 + len[q]] = (uint16_t)lo[q];
        }
        if (a < sources && lo[q] < rows && words_pay(len[q], (uint32_t)lo[q])) lo[q] = -1;
        else pos[q] = lo[q] < kHubEntry ? atomicAdd(&hub[lo[q]], 1) : atomicAdd(&gcur[lo[q]], 1);
      }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < kHubEntry; j += kEntryThreads)
      if (hub[j]) hub[j] = atomicAdd(&gcur[j], hub[j]);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < kEntryEach; ++q)
      if (lo[q] >= 0) {
        const int at = pos[q] + (lo[q] < kHubEntry ? hub[lo[q]] : 0);
        ent[__ldg(gstart + lo[q]) + at] = make_uint2(st[q], len[q]);
      }
    __syncthreads();
  }
}

// bitmaps: targets by kind; otherwise every target as a list.  ctr[kcMaxRow] = the longest N+(v).
__global__ void rank_items_kernel(const int64_t* roff, const int64_t* gstart, const int32_t* gcur, int64_t n,
                                  RankItemLists li, bool bitmaps, int* ctr) {
  const int64_t n_pad = (n + 31) & ~31ll;
  int longest = 0;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n_pad; v += (int64_t)gridDim.x * blockDim.x) {
    int64_t ne = 0, dv = 0;
    if (v < n) {
      ne = gcur[v];
      dv = roff[v + 1] - roff[v];
    }
    const bool any = ne > 0 && dv > 0;
    const int kind = !any ? -1
                     : !bitmaps ? (dv <= li.warp_max ? kcWarp : kcBlock)
                     : v < kRank15 ? kc15
                     : v < kRank16 ? kc16
                     : v < kRank17 && ne >= li.mid_min ? kc17 : kcFilter;
    const int64_t chunk = kind == kc17 ? kRankBlockChunk : kind == kcWarp ? li.warp_chunk
                          : kind == kcBlock ? li.block_chunk : li.chunk;
    const int k = any ? (int)((ne + chunk - 1) / chunk) : 0;
    if (any) longest = max(longest, (int)dv);
#pragma unroll
    for (int q = kc15; q <= kcBlock; ++q) {
      if (!__any_sync(0xffffffffu, kind == q)) continue;
      const int at = warp_reserve(&ctr[q], kind == q ? k : 0);
      if (kind != q) continue;
      int2* to = q == kc15 ? li.t15 : q == kc16 ? li.t16 : q == kc17 ? li.t17 : q == kcFilter ? li.filter : li.list;
      for (int c = 0; c < k; ++c)
        to[q == kcBlock ? li.lcap - 1 - (at + c) : (int64_t)(at + c)] = make_int2((int32_t)v, c);
    }
  }
  longest = __reduce_max_sync(0xffffffffu, longest);
  if ((threadIdx.x & 31) == 0 && longest) atomicMax(&ctr[kcMaxRow], longest);
}

// Streams the prefixes of entries [base, base + 32) for every batch that next() hands out through
// the bitmap T of N+(v): a bit is 0 for a member, 1 otherwise (the empty table is all ones, and
// members are put back by storing whole words).  Prefixes of 32 or more are walked by the whole
// warp, up to four loads in flight per lane; lanes past the end test v itself, which is
// never a member, so no load or test is predicated.
template <class Next>
__device__ __forceinline__ unsigned stream_bitmap(const int32_t* __restrict__ cols, const uint2* __restrict__ ent,
                                                  int64_t e1, int lane, const uint32_t* T, int32_t v, Next next) {
  unsigned cnt = 0;
  auto test = [&](int32_t x) { cnt += ~(T[(uint32_t)x >> 5] >> (x & 31)) & 1u; };
  for (int64_t base = next(); base < e1; base = next()) {
    uint2 q = make_uint2(0u, 0u);
    if (base + lane < e1) q = __ldg(ent + base + lane);
    unsigned longm = __ballot_sync(0xffffffffu, q.y >= 32);
    while (longm) {
      const int k = __ffs(longm) - 1;
      longm &= longm - 1;
      const int32_t* P = cols + __shfl_sync(0xffffffffu, q.x, k) + lane;
      int left = (int)__shfl_sync(0xffffffffu, q.y, k) - lane;  // elements from this lane's first on
      const int ln = left + lane;
      for (int j0 = 0; j0 < ln; j0 += 128, P += 128, left -= 128) {
        const int32_t x0 = left > 0 ? __ldg(P) : v;
        if (j0 + 64 < ln) {
          const int32_t x1 = __ldg(P + 32);
          const int32_t x2 = left > 64 ? __ldg(P + 64) : v;
          const int32_t x3 = left > 96 ? __ldg(P + 96) : v;
          test(x0);
          test(x1);
          test(x2);
          test(x3);
        } else {
          const int32_t x1 = left > 32 ? __ldg(P + 32) : v;
          test(x0);
          test(x1);
        }
      }
    }
    const int slen = q.y < 32 ? (int)q.y : 0;
    int incl = slen;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    const int total = __shfl_sync(0xffffffffu, incl, 31);
    const int start = incl - slen;
    const uint32_t at = q.x - (uint32_t)start;
    for (int t0 = 0; t0 < total; t0 += 32) {
      const int t = t0 + lane;
      int k = 0;  // the last lane whose prefix starts at or before t
#pragma unroll
      for (int step = 16; step > 0; step >>= 1)
        if (__shfl_sync(0xffffffffu, start, k + step) <= t) k += step;
      const uint32_t kp = __shfl_sync(0xffffffffu, at, k);
      test(t < total ? __ldg(cols + (kp + (uint32_t)t)) : v);
    }
  }
  return cnt;
}

// Targets below kRank15 (BITS = 2^15) or kRank16 (2^16): a warp per chunk of entries, N+(v) as
// the warp's own bitmap.  Prefixes are read from the 16-bit rows by groups of kLanes lanes, 16
// bytes (eight ids) a lane: 32 / kLanes entries are under way at once, so that short prefixes fill
// the warp without a search for the owner of each element, and each group has the next piece
// loading while it tests the last.  Ids past a prefix's end are masked off by position.
template <int BITS, int WARPS, int kLanes>
__global__ void __launch_bounds__(WARPS * 32) rank_warp_kernel(const int64_t* __restrict__ roff,
                                                               const int32_t* __restrict__ rcols,
                                                               const uint4* __restrict__ r16,
                                                               const uint2* __restrict__ ent,
                                                               const int2* __restrict__ items,
                                                               const int64_t* __restrict__ gstart,
                                                               const int32_t* __restrict__ nids, int chunk,
                                                               const int* nitems_dev, int* next, const int* too_long,
                                                               unsigned long long* out) {
  constexpr uint32_t kBytes = BITS / 8;
  __shared__ __align__(16) unsigned char smem[WARPS * kBytes];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t base = w * kBytes;
  uint32_t* T = reinterpret_cast<uint32_t*>(smem + base);
  for (int j = lane; j < (int)(kBytes / 4); j += 32) T[j] = 0u;
  __syncwarp();
  const int nitems = *too_long ? 0 : *nitems_dev;  // an unsorted row's prefix is no prefix
  const int sub = lane % kLanes;
  // the bit of id x is bit 31 - x % 32 of word x / 32: shifting the word left by x brings it to the
  // top, and a funnel shift moves it into acc, two instructions after the load
  auto word = [&](uint32_t r) {  // r: the id in its low 16 bits
    return *reinterpret_cast<const uint32_t*>(smem + (((r >> 3) & (kBytes - 4)) | base));
  };
  auto tests = [&](const uint4& d, int valid) -> unsigned {  // members among the first `valid` ids
    const uint32_t x1 = d.x >> 16, y1 = d.y >> 16, z1 = d.z >> 16, w1 = d.w >> 16;
    const uint32_t b0 = word(d.x), b1 = word(x1), b2 = word(d.y), b3 = word(y1), b4 = word(d.z), b5 = word(z1),
                   b6 = word(d.w), b7 = word(w1);
    auto fold = [](uint32_t acc, uint32_t b, uint32_t r) {
      return __funnelshift_l(__funnelshift_l(b, b, r), acc, 1);
    };
    uint32_t acc = fold(0u, b0, d.x), acc2 = fold(0u, b4, d.z);
    acc = fold(acc, b1, x1);
    acc2 = fold(acc2, b5, z1);
    acc = fold(acc, b2, d.y);
    acc2 = fold(acc2, b6, d.w);
    acc = fold(acc, b3, y1);
    acc2 = fold(acc2, b7, w1);
    return __popc((acc << 4 | acc2) & (0xff00u >> min(max(valid, 0), 8)) & 0xffu);
  };
  unsigned long long total = 0;
  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(next, 1);
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it >= nitems) break;
    const int2 c = __ldg(items + it);
    const int32_t v = c.x;
    const int64_t g0 = __ldg(gstart + v) + (int64_t)c.y * chunk;
    const int ne = min(__ldg(nids + v) - c.y * chunk, chunk);
    const uint2* en = ent + g0;
    const int64_t hb = __ldg(roff + v);
    const int dh = (int)(__ldg(roff + v + 1) - hb);
    int i = lane / kLanes;
    uint2 nq = i < ne ? __ldg(en + i) : make_uint2(0u, 0u);
    for (int j = lane; j < dh; j += 32) {
      const int32_t x = __ldg(rcols + hb + j);
      atomicOr(&T[x >> 5], 0x80000000u >> (x & 31));
    }
    __syncwarp();
    uint32_t at = 0;  // the lane's next piece
    int left = -8 * sub;  // ids from the lane's next piece to the end of the group's prefix
    unsigned cnt = 0;
    // loads the lane's next piece; returns its valid ids (<= 0: none)
    auto fetch = [&](uint4& d) -> int {
      if (left + 8 * sub <= 0 && i < ne) {  // the group's prefix is done
        at = nq.x + sub;
        left = (int)nq.y - 8 * sub;
        i += 32 / kLanes;
        if (i < ne) nq = __ldg(en + i);
      }
      const int valid = left;
      d = make_uint4(0u, 0u, 0u, 0u);
      if (valid > 0) d = __ldg(r16 + at);
      at += kLanes;
      left -= 8 * kLanes;
      return valid;
    };
    uint4 d0, d1;
    int v0 = fetch(d0), v1;
    do {
      v1 = fetch(d1);
      cnt += tests(d0, v0);
      v0 = fetch(d0);
      cnt += tests(d1, v1);
    } while (__any_sync(0xffffffffu, v0 > 0 || left > 0 || i < ne));
    total += cnt;
    __syncwarp();
    for (int j = lane; j < dh; j += 32) T[__ldg(rcols + hb + j) >> 5] = 0u;
    __syncwarp();
  }
  warp_add_count(total, out);
}

// The edges tested as words: a warp per row u, its ids below 2^15 as a bitmap in shared memory,
// ANDed with the bitmap rows of its targets.  Eight lanes take a target, 16 bytes a lane and four
// loads in flight; the row ascends, so the four targets under way have about as many pieces.  Bits of u
// from v on meet no bit of N+(v).  The bitmap rows take 64 MB at most and stay in L2: bound by issue
// (72 % of peak at scale 20, L1 66 %, DRAM 2 %).  A target's bitmap against the sources' rows instead
// had 192 MB of them to read, at 8 TB/s, and needed entries: 42.9 ms at R-MAT scale 24 to 40.0.
__global__ void __launch_bounds__(256) rank_words_kernel(const int64_t* __restrict__ roff,
                                                         const int32_t* __restrict__ rcols,
                                                         const uint4* __restrict__ dense, int rows, int sources, int* next,
                                                         const int* too_long, unsigned long long* out) {
  __shared__ __align__(16) uint32_t smem[8][1 << 10];
  __shared__ int32_t lists[8][32];
  const int lane = threadIdx.x & 31, sub = lane & 7, grp = lane >> 3;
  int32_t* list = lists[threadIdx.x >> 5];
  uint32_t* T = smem[threadIdx.x >> 5];
  const uint4* T4 = reinterpret_cast<const uint4*>(T);
  for (int j = lane; j < (1 << 10); j += 32) T[j] = 0u;
  __syncwarp();
  if (*too_long) return;  // an unsorted row's prefix is no prefix
  unsigned long long total = 0;
  int u = -1, u_end = 0;
  for (;;) {
    if (++u >= u_end) {
      const int grab = u < rows ? 1 : kGrab;  // the longest rows one at a time
      if (lane == 0) u = atomicAdd(next, grab);
      u = __shfl_sync(0xffffffffu, u, 0);
      u_end = u + grab;
    }
    if (u >= sources) break;
    const int64_t b = __ldg(roff + u);
    const int du = (int)(__ldg(roff + u + 1) - b);
    bool filled = false;
    unsigned cnt = 0;
    for (int j0 = 0; j0 < du; j0 += 32) {
      const int32_t v = j0 + lane < du ? __ldg(rcols + b + j0 + lane) : rows;
      unsigned left = __ballot_sync(0xffffffffu, v < rows && words_pay((uint32_t)(j0 + lane), (uint32_t)v));
      if (left && !filled) {
        for (int j = lane; j < du; j += 32) {
          const int32_t x = __ldg(rcols + b + j);
          if (x < (1 << 15)) atomicOr(&T[x >> 5], 1u << (x & 31));
        }
        __syncwarp();
        filled = true;
      }
      const int nt = __popc(left);
      if ((left >> lane) & 1u) list[__popc(left & ((1u << lane) - 1))] = v;
      __syncwarp();
      for (int k = 0; k < nt; k += 4) {
        const uint32_t x = (uint32_t)list[min(k + grp, nt - 1)];
        const int most = (list[min(k + 3, nt - 1)] >> 7) + 1;  // of the four, which ascend
        const int pieces = k + grp < nt ? (int)(x >> 7) + 1 : 0;
        const uint4* row = dense + dense_start(x) + sub;
        for (int p = 0; p < most; p += 32) {
          uint4 d[4];
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (p + 8 * q < most)
              d[q] = p + 8 * q + sub < pieces ? __ldg(row + p + 8 * q) : make_uint4(0u, 0u, 0u, 0u);
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (p + 8 * q < most) {
              const uint4 m = T4[p + 8 * q + sub];
              cnt += __popc(d[q].x & m.x) + __popc(d[q].y & m.y) + __popc(d[q].z & m.z) + __popc(d[q].w & m.w);
            }
        }
      }
      __syncwarp();
      if (__shfl_sync(0xffffffffu, v, 31) >= rows) break;  // ascending
    }
    total += cnt;
    if (filled) {
      __syncwarp();
      for (int j = lane; j < du; j += 32) {
        const int32_t x = __ldg(rcols + b + j);
        if (x < (1 << 15)) T[x >> 5] = 0u;
      }
      __syncwarp();
    }
  }
  warp_add_count(total, out);
}

// Targets of larger rank: a warp per chunk of entries.  Ids below 2^14 have a bit each in the first
// half of the warp's table, the others share the bits of the second half by their low 14 bits: a
// hit there is kept on the lane's stack and looked up in the list N+(v) when a stack fills.
// Groups of kLanes lanes read a prefix, four ids a lane from the 16-byte line they lie in; ids
// outside the prefix are masked off by position.  Bound by latency (a few dozen lines per item,
// then the next): what pays are warps in flight and the next item's header loaded early.  Halves of
// 2^15 bits, six CTAs per SM instead of nine: 42.2 against 38.5 ms at R-MAT scale 24; of 2^13 39.7; eleven
// CTAs with fewer registers, or stacks of 12 and 16: 1 ms more.  Hash tables of N+(v) instead of all
// of this (31 instructions per 32 tests): 39.7 against 37.5 at scale 24, 7.0 and 6.5 at scale 22,
// Chung-Lu n = 4 M 6.6 and 6.3.
constexpr int kStack = 8;
constexpr int kLowBits = 14;
template <int WARPS, int kLanes>
__global__ void __launch_bounds__(WARPS * 32, 9) rank_filter_kernel(const int64_t* __restrict__ roff,
                                                                 const int32_t* __restrict__ rcols,
                                                                 const uint2* __restrict__ ent,
                                                                 const int2* __restrict__ items,
                                                                 const int64_t* __restrict__ gstart, int chunk,
                                                                 const int* nitems_dev, int* next, const int* too_long,
                                                                 unsigned long long* out) {
  constexpr uint32_t kHalf = (1u << kLowBits) / 8, kBytes = 2 * kHalf;
  __shared__ __align__(16) unsigned char smem[WARPS * kBytes];
  __shared__ int32_t stacks[WARPS][kStack][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t base = w * kBytes;
  const uint4* ids = reinterpret_cast<const uint4*>(rcols);
  uint32_t* T = reinterpret_cast<uint32_t*>(smem + base);
  for (int j = lane; j < (int)(kBytes / 4); j += 32) T[j] = 0u;
  __syncwarp();
  const int nitems = *too_long ? 0 : *nitems_dev;  // an unsorted row's prefix is no prefix
  const int sub = lane % kLanes;
  // byte of id x's word
  auto place = [&](uint32_t x) {
    return ((x >> 3) & (kHalf - 4)) + (x >> kLowBits ? base + kHalf : base);
  };
  auto word = [&](uint32_t x) { return *reinterpret_cast<uint32_t*>(smem + place(x)); };
  struct Head {
    int32_t v;
    int ne, dh;
    int64_t g0, hb;
  };
  int it = 0, it_end = 0;
  auto head = [&]() {
    if (it == it_end) {
      if (lane == 0) it = atomicAdd(next, kGrab);
      it = __shfl_sync(0xffffffffu, it, 0);
      it_end = it + kGrab;
    }
    Head h{-1, 0, 0, 0, 0};
    if (it < nitems) {
      const int2 c = __ldg(items + it++);
      h.v = c.x;
      h.g0 = __ldg(gstart + c.x) + (int64_t)c.y * chunk;
      h.ne = (int)min(__ldg(gstart + c.x + 1) - h.g0, (int64_t)chunk);
      h.hb = __ldg(roff + c.x);
      h.dh = (int)(__ldg(roff + c.x + 1) - h.hb);
    }
    return h;
  };
  unsigned long long total = 0;
  Head nh = head();
  while (nh.v >= 0) {
    const int ne = nh.ne, dh = nh.dh;
    const uint2* en = ent + nh.g0;
    const int64_t hb = nh.hb;
    nh = head();  // the next item's loads run under this one's
    int i = lane / kLanes;
    uint2 nq = i < ne ? __ldg(en + i) : make_uint2(0u, 0u);
    for (int j = lane; j < dh; j += 32) {
      const uint32_t x = (uint32_t)__ldg(rcols + hb + j);
      atomicOr(reinterpret_cast<uint32_t*>(smem + place(x)), 0x80000000u >> (x & 31));
    }
    __syncwarp();
    uint32_t at = 0;  // the lane's next line
    int left = -4 * sub;  // ids from its start to the end of the group's prefix
    int skip = 0;     // ids of it before the prefix
    unsigned cnt = 0;
    int sp = 0;
    // loads the lane's next line; returns its ids that count, the first as bit 3
    auto fetch = [&](uint4& d) -> unsigned {
      if (left + 4 * sub <= 0 && i < ne) {  // the group's prefix is done
        at = (nq.x >> 2) + sub;
        skip = (int)(nq.x & 3u);
        left = (int)nq.y + skip - 4 * sub;
        if (sub) skip = 0;
        i += 32 / kLanes;
        if (i < ne) nq = __ldg(en + i);
      }
      unsigned valid = 0;
      d = make_uint4(0u, 0u, 0u, 0u);
      if (left > 0) {
        d = __ldg(ids + at);
        valid = (0xf0u >> min(left, 4)) & (0xfu >> skip);
      }
      at += kLanes;
      left -= 4 * kLanes;
      skip = 0;
      return valid;
    };
    auto tests = [&](const uint4& d, unsigned valid) {
      const uint32_t b0 = word(d.x), b1 = word(d.y), b2 = word(d.z), b3 = word(d.w);
      auto fold = [](uint32_t acc, uint32_t b, uint32_t r) {
        return __funnelshift_l(__funnelshift_l(b, b, r), acc, 1);
      };
      const unsigned hit = fold(fold(fold(fold(0u, b0, d.x), b1, d.y), b2, d.z), b3, d.w) & valid;
      const unsigned high = hit & ((d.x >> kLowBits ? 8u : 0u) | (d.y >> kLowBits ? 4u : 0u) | (d.z >> kLowBits ? 2u : 0u) |
                                  (d.w >> kLowBits ? 1u : 0u));
      cnt += __popc(hit ^ high);
      if (high) {
        auto push = [&](unsigned bit, uint32_t x) {
          if (high & bit) stacks[w][sp++][lane] = (int32_t)x;
        };
        push(8u, d.x);
        push(4u, d.y);
        push(2u, d.z);
        push(1u, d.w);
      }
    };
    auto settle = [&]() {
      const int most = __reduce_max_sync(0xffffffffu, sp);
      for (int k = 0; k < most; ++k)
        if (k < sp) {
          const int32_t x = stacks[w][k][lane];
          int a = 0, b = dh;  // the first id not below x
          while (a < b) {
            const int mid = (a + b) >> 1;
            if (__ldg(rcols + hb + mid) < x) a = mid + 1; else b = mid;
          }
          cnt += a < dh && __ldg(rcols + hb + a) == x;
        }
      sp = 0;
    };
    uint4 d0, d1;
    unsigned v0 = fetch(d0), v1;
    do {
      v1 = fetch(d1);
      tests(d0, v0);
      if (__any_sync(0xffffffffu, sp > kStack - 4)) settle();
      v0 = fetch(d0);
      tests(d1, v1);
      if (__any_sync(0xffffffffu, sp > kStack - 4)) settle();
    } while (__any_sync(0xffffffffu, v0 != 0 || left > 0 || i < ne));
    settle();
    total += cnt;
    __syncwarp();
    for (int j = lane; j < dh; j += 32) *reinterpret_cast<uint32_t*>(smem + place((uint32_t)__ldg(rcols + hb + j))) = 0u;
    __syncwarp();
  }
  warp_add_count(total, out);
}

// Targets below kRank17 with many entries on wide graphs: a CTA per chunk of them, ids in 32 bits.
__global__ void __launch_bounds__(128) rank_block_kernel(CsrView g, const uint2* __restrict__ ent,
                                                         const int2* __restrict__ items,
                                                         const int64_t* __restrict__ gstart, const int* nitems_dev,
                                                         int* next, const int* too_long, unsigned long long* out) {
  constexpr uint32_t words = kRank17 / 32;
  __shared__ __align__(16) uint32_t T[words];
  __shared__ int item;
  __shared__ unsigned long long bnext;
  const int lane = threadIdx.x & 31;
  for (uint32_t j = threadIdx.x; j < words; j += blockDim.x) T[j] = ~0u;
  const int nitems = *too_long ? 0 : *nitems_dev;  // an unsorted row holds ids beyond the bitmap
  unsigned long long total = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      item = atomicAdd(next, 1);
      bnext = 0;
    }
    __syncthreads();
    const int it = item;
    if (it >= nitems) break;
    const int2 c = __ldg(items + it);
    const int32_t v = c.x;
    const int64_t b = __ldg(gstart + v) + (int64_t)c.y * kRankBlockChunk;
    const int64_t e = min(__ldg(gstart + v + 1), b + kRankBlockChunk);
    const int64_t hb = __ldg(g.off + v);
    const int dh = (int)(__ldg(g.off + v + 1) - hb);
    for (int j = threadIdx.x; j < dh; j += blockDim.x) {
      const int32_t x = __ldg(g.cols + hb + j);
      atomicAnd(&T[x >> 5], ~(1u << (x & 31)));
    }
    __syncthreads();
    total += stream_bitmap(g.cols, ent, e, lane, T, v, [&]() {
      unsigned long long r = 0;
      if (lane == 0) r = atomicAdd(&bnext, 32ull);
      return b + (int64_t)__shfl_sync(0xffffffffu, r, 0);
    });
    __syncthreads();
    for (int j = threadIdx.x; j < dh; j += blockDim.x) T[__ldg(g.cols + hb + j) >> 5] = ~0u;
    __syncthreads();
  }
  warp_add_count(total, out);
}

// Byte offsets of the buffers of one count in a single allocation.
struct Arena {
  size_t bytes = 0;
  template <class T>
  size_t add(size_t count) {
    const size_t at = bytes;
    bytes += (sizeof(T) * (count ? count : 1) + 255) & ~size_t(255);
    return at;
  }
};

}  // namespace

atc_status build_ranked(const atc_csr* csr, bool bitmaps, RankedCopy* rc, cudaStream_t s, int* launches) {
  const CsrPriv* pv = static_cast<const CsrPriv*>(csr->priv);
  const int64_t n = csr->n, m = csr->m;
  const int B = id_bits(n), db = id_bits(n);  // degrees are below n
  size_t sort_tmp = 0, scan_tmp = 0;
  ATC_TRY(sort_keys_u64_tmp(nullptr, &sort_tmp, nullptr, nullptr, (size_t)n, B, B + db, nullptr, s));
  ATC_TRY(exclusive_scan_i32_to_i64_tmp(nullptr, &scan_tmp, nullptr, nullptr, (size_t)n + 1, s));
  // a warp item holds at most 512 entries (the bitmap costs d+(v) of them to set up), fewer where
  // that would leave warps without work
  const int64_t warps = (int64_t)sm_count() * 48;
  const int chunk = (int)std::min<int64_t>(std::max<int64_t>((m / (8 * warps)) & ~31ll, 64), 512);
  auto item_cap = [&](int64_t below, int64_t per) { return std::min<int64_t>(n, below) + m / per + 1; };
  const int64_t cap15 = bitmaps ? item_cap(kRank15, chunk) : 0;
  const int64_t cap16 = bitmaps && n > kRank15 ? item_cap(kRank16, chunk) : 0;
  const bool wide = csr->wedges_min >= kWideMean * m;
  const int64_t cap17 = bitmaps && wide && n > kRank16 ? item_cap(kRank17, kRankBlockChunk) : 0;
  const int64_t cap_filter = bitmaps && n > kRank16 ? item_cap(n, chunk) : 0;
  const int64_t lcap = !bitmaps ? max_items(n, m, chunk) : 0;
  // Bitmaps of rows take no more room than the ids once more: rows^2 / 16 against 4 m bytes.
  int rows = 0, sources = 0;
  if (bitmaps) rows = (int)std::min<double>(8.0 * std::sqrt((double)m), (double)std::min<int64_t>(n, kDenseRows));
  Arena ar;
  const size_t a_ka = ar.add<uint64_t>(n), a_kb = ar.add<uint64_t>(n);
  const size_t a_tmp = ar.add<char>(std::max(sort_tmp, scan_tmp));
  const size_t a_rank = ar.add<int32_t>(n);
  const size_t a_zero = ar.bytes;  // from here on zeroed
  const size_t a_ctr = ar.add<int>(kcCount), a_deg = ar.add<int32_t>(n + 1), a_cnt = ar.add<int32_t>(n + 1),
               a_gcur = ar.add<int32_t>(n);
  const size_t zero_end = ar.bytes;
  const size_t a_roff = ar.add<int64_t>(n + 1), a_gstart = ar.add<int64_t>(n + 1);
  const size_t a_rcols = ar.add<int32_t>(m + 16), a_ent = ar.add<uint2>(m), a_piece = ar.add<int32_t>((m >> 5) + 1);
  const size_t a_mid = ar.add<int32_t>(m / 33 + 1), a_big = ar.add<int32_t>(m / (kRankWarpRow + 1) + 1);
  const size_t a_15 = ar.add<int2>(cap15), a_16 = ar.add<int2>(cap16), a_17 = ar.add<int2>(cap17),
               a_filter = ar.add<int2>(cap_filter), a_list = ar.add<int2>(lcap);
  const size_t a_pieces = ar.add<int32_t>(bitmaps ? n + 1 : 0), a_roff8 = ar.add<int64_t>(bitmaps ? n + 1 : 0);
  const size_t a_r16 = ar.add<uint16_t>(bitmaps ? m + 8 * std::min(n, m) : 0);
  const size_t plain = ar.bytes, a_dense = ar.add<uint4>(rows ? dense_start(rows) : 0);
  if (rc->mem.alloc(ar.bytes, s) != ATC_OK) {
    cudaGetLastError();
    rows = 0;
    if (rc->mem.alloc(plain, s) != ATC_OK) {  // no room for the copy: the caller counts in place
      cudaGetLastError();
      return ATC_OK;
    }
  }
  char* p = rc->mem.p;
  uint64_t* ka = reinterpret_cast<uint64_t*>(p + a_ka);
  uint64_t* kb = reinterpret_cast<uint64_t*>(p + a_kb);
  int32_t* rank = reinterpret_cast<int32_t*>(p + a_rank);
  int* ctr = reinterpret_cast<int*>(p + a_ctr);
  int32_t* deg = reinterpret_cast<int32_t*>(p + a_deg);
  int32_t* cnt = reinterpret_cast<int32_t*>(p + a_cnt);
  int32_t* gcur = reinterpret_cast<int32_t*>(p + a_gcur);
  uint4* dense = reinterpret_cast<uint4*>(p + a_dense);
  int64_t* roff = reinterpret_cast<int64_t*>(p + a_roff);
  int64_t* gstart = reinterpret_cast<int64_t*>(p + a_gstart);
  int32_t* rcols = reinterpret_cast<int32_t*>(p + a_rcols);
  uint2* ent = reinterpret_cast<uint2*>(p + a_ent);
  uint32_t* slot = reinterpret_cast<uint32_t*>(ent);  // until the entries are written
  int32_t* piece_row = reinterpret_cast<int32_t*>(p + a_piece);
  int32_t* mid = reinterpret_cast<int32_t*>(p + a_mid);
  int32_t* big = reinterpret_cast<int32_t*>(p + a_big);
  int32_t* pieces = reinterpret_cast<int32_t*>(p + a_pieces);
  int64_t* roff8 = reinterpret_cast<int64_t*>(p + a_roff8);
  uint16_t* r16 = reinterpret_cast<uint16_t*>(p + a_r16);
  const RankItemLists li{reinterpret_cast<int2*>(p + a_15), reinterpret_cast<int2*>(p + a_16),
                         reinterpret_cast<int2*>(p + a_17), reinterpret_cast<int2*>(p + a_filter),
                         reinterpret_cast<int2*>(p + a_list), lcap, chunk, chunk, 4 * chunk, kWarpMax,
                         wide ? kRankMidMin : INT_MAX};
  ATC_CK(cudaMemsetAsync(p + a_zero, 0, zero_end - a_zero, s));
  rank_keys_kernel<<<grid_for(n, 256), 256, 0, s>>>(csr->offsets, pv->indeg, n, B, db, ka);
  ATC_CK(cudaGetLastError());
  uint64_t* sorted = nullptr;
  ATC_TRY(sort_keys_u64_tmp(p + a_tmp, &sort_tmp, ka, kb, (size_t)n, B, B + db, &sorted, s));
  rank_scatter_kernel<<<grid_for(n, 256), 256, 0, s>>>(sorted, n, B, rank);
  rank_count_kernel<<<grid_for(m, 512, 4), 512, 0, s>>>(pv->esrc, csr->cols, m, rank, deg, cnt, slot);
  ATC_CK(cudaGetLastError());
  ATC_TRY(exclusive_scan_i32_to_i64_tmp(p + a_tmp, &scan_tmp, deg, roff, (size_t)n + 1, s));
  ATC_TRY(exclusive_scan_i32_to_i64_tmp(p + a_tmp, &scan_tmp, cnt, gstart, (size_t)n + 1, s));
  if (bitmaps) {
    rank_pieces_kernel<<<grid_for(n + 1, 256), 256, 0, s>>>(deg, n, pieces);
    ATC_TRY(exclusive_scan_i32_to_i64_tmp(p + a_tmp, &scan_tmp, pieces, roff8, (size_t)n + 1, s));
    *launches += 3;
  }
  rank_rows_kernel<<<grid_for(m, 256), 256, 0, s>>>(pv->esrc, csr->cols, m, rank, slot, roff, rcols);
  if (n <= 1 << 27) rank_sort_small_kernel<uint32_t><<<grid_for(n, 256), 256, 0, s>>>(roff, n, rcols, mid, big, ctr);
  else rank_sort_small_kernel<uint64_t><<<grid_for(n, 256), 256, 0, s>>>(roff, n, rcols, mid, big, ctr);
  rank_sort_mid_kernel<<<sm_count() * blocks_per_sm((const void*)rank_sort_mid_kernel, 256, 0), 256, 0, s>>>(
      roff, mid, rcols, ctr);
  const int64_t long_rows = m / (kRankWarpRow + 1);
  if (long_rows) {
    const size_t big_smem = sizeof(int32_t) * kRankRowMax;
    ATC_CK(cudaFuncSetAttribute((const void*)rank_sort_big_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                (int)big_smem));
    rank_sort_big_kernel<<<(unsigned)std::min<int64_t>(long_rows, sm_count() * 2), 1024, big_smem, s>>>(roff, big, rcols,
                                                                                                      ctr);
    *launches += 1;
  }
  if (rows) {
    sources = (int)std::min<int64_t>(n, (int64_t)kDenseSources * rows);
    rank_dense_kernel<<<(rows + kDenseWarps - 1) / kDenseWarps, kDenseWarps * 32, 0, s>>>(roff, rcols, rows, dense);
    *launches += 1;
  }
  rank_piece_rows_kernel<<<grid_for(n, 256), 256, 0, s>>>(roff, n, piece_row);
  rank_entries_kernel<<<grid_for(m, kTile, 2), kEntryThreads, 0, s>>>(roff, n, m, rcols, piece_row, gstart, roff8,
                                                                        bitmaps ? kRank16 : 0, rows, sources, gcur,
                                                                        r16, ent);
  rank_items_kernel<<<grid_for(n, 256), 256, 0, s>>>(roff, gstart, gcur, n, li, bitmaps, ctr);
  ATC_CK(cudaGetLastError());
  *launches += 17;
  rc->n = n;
  rc->m = m;
  rc->roff = roff;
  rc->rcols = rcols;
  rc->r16 = reinterpret_cast<const uint4*>(r16);
  rc->gstart = gstart;
  rc->ent = ent;
  rc->nids = gcur;
  rc->dense = rows ? dense : nullptr;
  rc->dense_rows = rows;
  rc->dense_sources = sources;
  rc->ctr = ctr;
  rc->li = li;
  rc->long_rows = long_rows != 0;
  return ATC_OK;
}

atc_status count_ranked(const atc_csr* csr, unsigned long long* out, bool* done, cudaStream_t s, int* launches) {
  *done = false;
  RankedCopy rc;
  std::optional<Phase> ph;
  ph.emplace("tc.group", s);
  ATC_TRY(build_ranked(csr, true, &rc, s, launches));
  if (!rc.mem.p) return ATC_OK;
  ph.reset();
  ph.emplace("tc.count", s);
  const int64_t n = rc.n, m = rc.m;
  const CsrView g = csr_view(rc.roff, rc.rcols, nullptr, n, m);
  const RankItemLists& li = rc.li;
  const int64_t* gstart = rc.gstart;
  const uint2* ent = rc.ent;
  int* ctr = rc.ctr;
  const int* too = ctr + kcTooLong;
  const bool wide = csr->wedges_min >= kWideMean * m, wide15 = csr->wedges_min >= kWideMean15 * m;
  if (n > kRank16) {
    const auto kern = wide15 ? rank_filter_kernel<4, 8> : rank_filter_kernel<4, 4>;
    kern<<<sm_count() * blocks_per_sm((const void*)kern, 128, 0), 128, 0, s>>>(
        rc.roff, rc.rcols, ent, li.filter, gstart, li.chunk, ctr + kcFilter, ctr + kcNextFilter, too, out);
    ATC_CK(cudaGetLastError());
    *launches += 1;
    if (wide) {
      rank_block_kernel<<<sm_count() * blocks_per_sm((const void*)rank_block_kernel, 128, 0), 128, 0, s>>>(
          g, ent, li.t17, gstart, ctr + kc17, ctr + kcNext17, too, out);
      ATC_CK(cudaGetLastError());
      *launches += 1;
    }
  }
  if (rc.dense) {
    rank_words_kernel<<<sm_count() * blocks_per_sm((const void*)rank_words_kernel, 256, 0), 256, 0, s>>>(
        rc.roff, rc.rcols, rc.dense, rc.dense_rows, rc.dense_sources, ctr + kcNextDense, too, out);
    ATC_CK(cudaGetLastError());
    *launches += 1;
  }
  if (n > kRank15) {
    const auto kern = wide ? rank_warp_kernel<1 << 16, 4, 16> : rank_warp_kernel<1 << 16, 4, 8>;
    kern<<<sm_count() * blocks_per_sm((const void*)kern, 128, 0), 128, 0, s>>>(
        rc.roff, rc.rcols, rc.r16, ent, li.t16, gstart, rc.nids, li.chunk, ctr + kc16, ctr + kcNext16, too, out);
    *launches += 1;
  }
  const auto kern = wide15 ? rank_warp_kernel<1 << 15, 8, 8> : rank_warp_kernel<1 << 15, 8, 4>;
  kern<<<sm_count() * blocks_per_sm((const void*)kern, 256, 0), 256, 0, s>>>(
      rc.roff, rc.rcols, rc.r16, ent, li.t15, gstart, rc.nids, li.chunk, ctr + kc15, ctr + kcNext15, too, out);
  ATC_CK(cudaGetLastError());
  *launches += 1;
  int too_long = 0;
  if (rc.long_rows) {
    ATC_CK(cudaMemcpyAsync(&too_long, ctr + kcTooLong, sizeof(int), cudaMemcpyDeviceToHost, s));
    ATC_CK(cudaStreamSynchronize(s));
  }
  *done = too_long == 0;
  return ATC_OK;
}

}  // namespace atc
