// k-clique counting on an oriented CSR (k >= 3), exact in uint64.
//
// The reference (k-clique/kcl.cu:147-215, Pangolin) materialises every level of the
// embedding list in HBM: per level it counts extensions (extend_alloc, :16-50), scans
// them (thrust::exclusive_scan, :197) and writes the next level (extend_insert,
// :115-145), counting instead of writing at level k-2.  Here a warp or a CTA takes one
// source u and builds, once for all its edges, the graph that the CSR induces on N+(u) as
// bitmap rows in shared memory: row i = the members of N+(u) that are in N+(S[i]), S = N+(u).
// Row i is then C0 = N+(u) ∩ N+(S[i]) of the edge u -> S[i], and every deeper level of the
// search is an AND / popc of rows:
//
//   cliq(1, M) = |M|,  cliq(t, M) = sum_{j in M} cliq(t - 1, M & row[j]),
//   k-cliques whose first edge is u -> S[i]: cliq(k - 2, row[i]).
//
//   rows of 2..32 and (up to k = 5) 33..64 members (kcl_rows_warp_kernel): a warp per u, 32-
//     and 64-bit rows; the induced edges are listed in shared memory as they are found and dealt over
//     the lanes, each lane counting the (k-3)-cliques of its edge's common row;
//   longer rows up to kRowMax members (kcl_rows_block_kernel): a CTA per u, rows of 64-bit
//     words; at k = 4 each induced edge is one AND / popc over the words, from k = 5 on a row's
//     C0 is renumbered into shorter rows of its own by a warp (up to kRowWarp members) or, at
//     k = 5, by the CTA; what is left goes to kcl_dense_kernel, a CTA per edge; few such rows, and
//     from k = 5 on a few of the longer half a warp takes, are split over CTAs;
//   longer rows still: a warp walks the search tree of one oriented edge depth first with
//     binary searches in global memory (kcl_kernel), its C0 of 65..1024 members counted by
//     kcl_dense_kernel from k = 5 on; every edge so where walk_pays says.  atc_tuning.kcl_dense = -1 puts every edge on that warp
//     search, without the dense kernel.
//
// Orientation is acyclic, so every k-clique is found once, from its first two vertices
// in orientation order — the same count kcl_gpu_solver accumulates.
//
// Measured (ms, one call; the per-edge walk with its dense kernel -> rows): RGG 2^20 of mean
// degree 32, k = 4 / 5 / 6 / 7: 22.0 / 25.2 / 39.7 / 72.8 -> 0.87 / 1.25 / 4.3 / 16.8; R-MAT
// scale 18, k = 4 / 5 / 6: 53.7 / 69.4 / 360 -> 2.7 / 15.0 / 171; scale 20, k = 4 / 5 / 6: 424 /
// 547 / 3697 -> 16.2 / 169 / 2464; scale 14, k = 6: 3.8 -> 2.3.  Of that, the CTA
// kernel's binary searches in all of N+(u) and its grabs of 32 lists (few of its warps had any)
// took scale 18, k = 4 from 3.8 to 2.7 when a part table and smaller grabs replaced them.
#include <algorithm>

#include "internal.cuh"
#include "parts.cuh"

namespace atc {

namespace {

__device__ __forceinline__ bool kc_has(const int32_t* a, int64_t n, int32_t x) {
  int64_t lo = 0, hi = n;
  while (lo < hi) {
    int64_t mid = (lo + hi) >> 1;
    if (a[mid] < x) lo = mid + 1; else hi = mid;
  }
  return lo < n && a[lo] == x;
}

// Writes P ∩ L (P given, L sorted) into out in P's order; returns the size (all lanes).
__device__ __forceinline__ int warp_intersect(const int32_t* P, int np, const int32_t* L, int64_t nl, int32_t* out,
                                              int lane) {
  int total = 0;
  for (int base = 0; base < np; base += 32) {
    int j = base + lane;
    bool hit = j < np && kc_has(L, nl, P[j]);
    unsigned mask = __ballot_sync(0xffffffffu, hit);
    if (hit && out) out[total + __popc(mask & ((1u << lane) - 1))] = P[j];
    total += __popc(mask);
  }
  __syncwarp();
  return total;
}

constexpr int kKcWarps = 8;
constexpr int kMaxK = 16;
constexpr int kMaskMax = 64;     // candidate sets up to this size use the warp's bitmask path
constexpr int kDenseMax = 1024;  // larger ones up to this size: a CTA per edge, bitmaps in shared memory
constexpr int kDenseWords = kDenseMax / 64;
constexpr int kDensePad = 4;
constexpr int kDenseThreads = 1024;  // 256: R-MAT s20 k = 6 4.84 s; 512: 3.81 s; 1024: 3.70 s

// d-cliques inside `mask` of the DAG whose successor sets (within C0) are adj[]:
// cliq(1, M) = |M|, cliq(d, M) = sum_{i in M} cliq(d-1, M & adj[i]).  Iterative, one
// lane, an explicit stack of (remaining mask, candidate mask) per depth.
__device__ __forceinline__ int first_bit(uint32_t x) { return __ffs((int)x) - 1; }
__device__ __forceinline__ int first_bit(unsigned long long x) { return __ffsll((long long)x) - 1; }
__device__ __forceinline__ int popc_of(uint32_t x) { return __popc(x); }
__device__ __forceinline__ int popc_of(unsigned long long x) { return __popcll(x); }

template <class M>
__device__ __forceinline__ unsigned long long mask_cliques(const M* adj, M mask, int d) {
  if (d <= 0) return 1ull;
  if (d == 1) return (unsigned long long)popc_of(mask);
  unsigned long long total = 0;
  M rem[kMaxK], cand[kMaxK];
  int top = 0;
  rem[0] = mask;
  cand[0] = mask;
  while (top >= 0) {
    if (rem[top] == 0) {
      --top;
      continue;
    }
    int i = first_bit(rem[top]);
    rem[top] &= rem[top] - 1;
    M nm = cand[top] & adj[i];
    int left = d - 1 - top;  // vertices still to choose after i
    if (left == 1) {
      total += (unsigned long long)popc_of(nm);
    } else if (popc_of(nm) >= left) {
      ++top;
      rem[top] = nm;
      cand[top] = nm;
    }
  }
  return total;
}

// Edges of sources with more than min_ud members (the shorter ones go by rows, below).
// Intersections: lanes take the elements of the candidate set (a subset of N+(u)),
// binary-search each in N+(w), and ballot/popc compact the hits in order into the next level,
// which lives in the warp's slice of a scratch buffer ((k-2) x max out-degree ints per warp).
// C0 of at most 64 members: the warp builds the 64-bit successor masks of the DAG induced on
// it with one ballot per member, and each lane counts the (k-2)-cliques of its first member.
// dense (nullable): edges whose C0 has kMaskMax < |C0| <= kDenseMax are appended to
// dense[1 + ...] (count in dense[0]) for kcl_dense_kernel instead of being walked here.
__global__ void __launch_bounds__(kKcWarps * 32) kcl_kernel(const int64_t* off, const int32_t* cols, const int32_t* esrc,
                                                          int64_t e0, int64_t e1, int k, int cap, int min_ud,
                                                          int32_t* scratch, unsigned long long* dense,
                                                          unsigned long long* out) {
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const int64_t gw = (int64_t)blockIdx.x * kKcWarps + w;
  const int64_t warps = (int64_t)gridDim.x * kKcWarps;
  const int levels = k - 2;
  int32_t* buf = scratch + gw * (int64_t)levels * cap;
  __shared__ unsigned long long adjm[kKcWarps][kMaskMax];
  unsigned long long cnt = 0, bytes = 0;
  int size[kMaxK];
  int idx[kMaxK];
  for (int64_t e = e0 + gw; e < e1; e += warps) {
    int32_t u = esrc[e], v = cols[e];
    int64_t ub = off[u], ud = off[u + 1] - ub;
    if (ud <= min_ud) continue;
    int64_t vb = off[v], vd = off[v + 1] - vb;
    bytes += 4ull * (unsigned long long)vd;
    // C0 = N+(u) ∩ N+(v), in the order of N+(u)
    int c0 = warp_intersect(cols + ub, (int)ud, cols + vb, vd, levels > 1 ? buf : nullptr, lane);
    if (levels == 1) {
      cnt += c0;
      continue;
    }
    if (c0 < levels) continue;  // not enough candidates for k-2 more vertices
    if (dense && c0 > kMaskMax && c0 <= kDenseMax) {
      if (lane == 0) dense[1 + atomicAdd(dense, 1ull)] = (unsigned long long)e;
      bytes -= 4ull * (unsigned long long)vd;  // the dense kernel reads N+(v) again and counts it
      continue;
    }
    if (c0 <= kMaskMax) {
      // bitmask path: adjm[w][i] = members of C0 that are successors of C0[i]
      for (int i = 0; i < c0; ++i) {
        int32_t x = buf[i];
        int64_t xb = off[x], xd = off[x + 1] - xb;
        bytes += 4ull * (unsigned long long)xd;
        bool h0 = lane < c0 && kc_has(cols + xb, xd, buf[lane]);
        bool h1 = lane + 32 < c0 && kc_has(cols + xb, xd, buf[lane + 32]);
        unsigned lo = __ballot_sync(0xffffffffu, h0), hi = __ballot_sync(0xffffffffu, h1);
        if (lane == 0) adjm[w][i] = ((unsigned long long)hi << 32) | lo;
      }
      __syncwarp();
      // (k-2)-cliques of the DAG on C0: lane i takes the ones whose first vertex is C0[i]
      unsigned long long part = 0;
      for (int i = lane; i < c0; i += 32) part += mask_cliques(adjm[w], adjm[w][i], levels - 1);
      for (int o = 16; o > 0; o >>= 1) part += __shfl_xor_sync(0xffffffffu, part, o);
      cnt += part;
      __syncwarp();
      continue;
    }
    size[0] = c0;
    idx[0] = 0;
    int l = 0;  // level whose candidates are being chosen from
    while (l >= 0) {
      if (idx[l] >= size[l]) {
        --l;
        if (l >= 0) ++idx[l];
        continue;
      }
      // choose x from C(l); the next level is all of C(l) ∩ N+(x) (lists are sorted by
      // id, not by orientation order, so no prefix of C(l) can be skipped)
      int32_t x = buf[(int64_t)l * cap + idx[l]];
      int64_t xb = off[x], xd = off[x + 1] - xb;
      bytes += 4ull * (unsigned long long)xd;
      const int32_t* P = buf + (int64_t)l * cap;
      if (l == levels - 2) {
        cnt += warp_intersect(P, size[l], cols + xb, xd, nullptr, lane);  // k-th vertices
        ++idx[l];
      } else {
        int c = warp_intersect(P, size[l], cols + xb, xd, buf + (int64_t)(l + 1) * cap, lane);
        if (c >= levels - 1 - l) {
          ++l;
          size[l] = c;
          idx[l] = 0;
        } else {
          ++idx[l];
        }
      }
    }
  }
  if (lane != 0) { cnt = 0; bytes = 0; }
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
  }
  if (lane == 0) {
    if (cnt) atomicAdd(out, cnt);
    if (bytes) atomicAdd(out + 1, bytes);
  }
}

// Position of the r-th (from 0) set bit of x; x has more than r set bits.
__device__ __forceinline__ int select_bit(unsigned long long x, int r) {
  int pos = 0;
#pragma unroll
  for (int s = 32; s > 0; s >>= 1) {
    const int c = __popcll(x & ((1ull << s) - 1));
    if (r >= c) {
      r -= c;
      x >>= s;
      pos += s;
    }
  }
  return pos;
}

// d-cliques (d >= 1) among the common higher neighbours of members i < j of C0, in the
// graph whose rows U (`words` uint64 each) hold every member's higher-indexed neighbours:
// cliq(1, M) = |M|, cliq(d, M) = sum_{x in M} cliq(d-1, M & U[x]).  Every set below holds
// members above the last one chosen only, so the word loops start at that member's word.
// One thread, an explicit stack of candidate sets.
__device__ unsigned long long pair_cliques(const unsigned long long* U, int words, int i, int j, int d) {
  const unsigned long long* Ri = U + (size_t)i * words;
  const unsigned long long* Rj = U + (size_t)j * words;
  const int w0 = (j + 1) >> 6;
  if (d == 1) {
    unsigned long long c = 0;
    for (int w = w0; w < words; ++w) c += __popcll(Ri[w] & Rj[w]);
    return c;
  }
  unsigned long long st[kMaxK - 4][kDenseWords];
  int pos[kMaxK - 4];
  int n0 = 0;
  for (int w = w0; w < words; ++w) {
    st[0][w] = Ri[w] & Rj[w];
    n0 += __popcll(st[0][w]);
  }
  if (n0 < d) return 0;
  pos[0] = j + 1;
  int top = 0;
  unsigned long long total = 0;
  const int nbits = words * 64;
  while (top >= 0) {
    // next member x >= pos[top] of st[top]
    int x = -1;
    for (int b = pos[top]; b < nbits;) {
      const unsigned long long word = st[top][b >> 6] >> (b & 63);
      if (word) {
        x = b + __ffsll(word) - 1;
        break;
      }
      b = (b | 63) + 1;
    }
    if (x < 0) {
      --top;
      continue;
    }
    pos[top] = x + 1;
    const unsigned long long* Rx = U + (size_t)x * words;
    const int wx = (x + 1) >> 6;
    const int left = d - 1 - top;  // members still to choose after x
    if (left == 1) {
      for (int w = wx; w < words; ++w) total += __popcll(st[top][w] & Rx[w]);
    } else {
      int c = 0;
      for (int w = wx; w < words; ++w) {
        st[top + 1][w] = st[top][w] & Rx[w];
        c += __popcll(st[top + 1][w]);
      }
      if (c >= left) {
        ++top;
        pos[top] = x + 1;
      }
    }
  }
  return total;
}

// The same count with the candidate sets in registers: rows of at most W words, D members to
// choose from M.  Rows hold higher members only, so every set below is above the last one chosen.
// Words past a row's end are read (the rows are padded) and masked off by M's zero words.
template <int W, int D>
__device__ __forceinline__ unsigned long long word_cliques(const unsigned long long* U, int stride,
                                                           const unsigned long long (&M)[W]) {
  unsigned c = 0;
  if constexpr (D == 1) {
#pragma unroll
    for (int w = 0; w < W; ++w) c += __popcll(M[w]);
    return c;
  } else {
    unsigned long long total = 0;
#pragma unroll
    for (int w = 0; w < W; ++w)
      for (unsigned long long r = M[w]; r; r &= r - 1) {
        const unsigned long long* Rx = U + (size_t)(w * 64 + first_bit(r)) * stride;
        unsigned long long N[W];
#pragma unroll
        for (int v = 0; v < W; ++v) N[v] = v < w ? 0ull : M[v] & Rx[v];
        total += word_cliques<W, D - 1>(U, stride, N);
      }
    return total;
  }
}
template <int W>
__device__ __forceinline__ unsigned long long pair_word_cliques(const unsigned long long* U, int stride, int i, int j,
                                                                int d) {
  unsigned long long M[W];
#pragma unroll
  for (int w = 0; w < W; ++w) M[w] = U[(size_t)i * stride + w] & U[(size_t)j * stride + w];
  if (stride < W)
#pragma unroll
    for (int w = 0; w < W; ++w)
      if (w >= stride) M[w] = 0ull;
  if (d == 1) return word_cliques<W, 1>(U, stride, M);
  if (d == 2) return word_cliques<W, 2>(U, stride, M);
  return word_cliques<W, 3>(U, stride, M);
}

// Edges whose C0 = N+(u) ∩ N+(v) holds kMaskMax < |C0| <= kDenseMax members, a CTA per
// edge.  C0 goes to shared memory (sorted by id, as N+(u) is) and the graph induced on it
// to bitmap rows: row i = the members above i adjacent to C0[i] (each oriented edge
// x -> y inside C0 found by a binary search of y in C0, recorded at the lower index of the
// two).  A (k-2)-clique of C0 is then counted once, from its two lowest members i < j:
// the CTA deals the adjacent pairs (i, j) over its threads by a prefix sum of the row
// popcounts, and each thread counts the (k-4)-cliques of row i AND row j with AND / popc
// over 64-member words.  The pairs, not the rows, are the unit, so a dense core's few
// heavy rows are spread over every thread.
constexpr int kDenseRows = kDenseMax / kDenseThreads;  // rows a thread sums in the row scan
static_assert(kDenseRows * kDenseThreads == kDenseMax, "the row scan covers kDenseMax rows");
// DEEP: k >= 6, short rows with the candidate sets in registers (their code in the kernel of k = 5 cost it 20 %).
template <bool DEEP>
__global__ void __launch_bounds__(kDenseThreads) kcl_dense_kernel(const int64_t* off, const int32_t* cols,
                                                                  const int32_t* esrc, const unsigned long long* dense,
                                                                  int k, int cmax, unsigned long long* next,
                                                                  unsigned long long* out) {
  extern __shared__ unsigned long long dsm[];  // rows: cmax * words, and kDensePad words read past them
  __shared__ int32_t C[kDenseMax];
  __shared__ int pre[kDenseMax + 1];
  __shared__ int wcount[kDenseThreads / 32];
  __shared__ int csize;
  __shared__ unsigned long long item;
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = kDenseThreads / 32;
  const unsigned long long nitems = dense[0];
  unsigned long long cnt = 0, bytes = 0;
  for (;;) {
    if (threadIdx.x == 0) item = atomicAdd(next, 1ull);
    __syncthreads();
    const unsigned long long it = item;
    if (it >= nitems) break;
    const int64_t e = (int64_t)dense[1 + it];
    const int32_t u = esrc[e], v = cols[e];
    const int64_t ub = off[u], ud = off[u + 1] - ub, vb = off[v], vd = off[v + 1] - vb;
    if (threadIdx.x == 0) {
      csize = 0;
      bytes += 4ull * (unsigned long long)vd;
    }
    __syncthreads();
    // C0 in the order of N+(u): block-wide compaction of the hits, chunk by chunk
    for (int64_t base = 0; base < ud; base += kDenseThreads) {
      const int64_t j = base + threadIdx.x;
      const int32_t x = j < ud ? cols[ub + j] : 0;
      const bool hit = j < ud && kc_has(cols + vb, vd, x);
      const unsigned b = __ballot_sync(0xffffffffu, hit);
      if (lane == 0) wcount[w] = __popc(b);
      __syncthreads();
      int before = csize;
      for (int q = 0; q < w; ++q) before += wcount[q];
      if (hit) C[before + __popc(b & ((1u << lane) - 1))] = x;
      __syncthreads();
      if (threadIdx.x == 0) {
        int t = csize;
        for (int q = 0; q < nw; ++q) t += wcount[q];
        csize = t;
      }
      __syncthreads();
    }
    const int c = csize;
    const int words = (c + 63) >> 6;
    for (int t = threadIdx.x; t < c * words; t += kDenseThreads) dsm[t] = 0ull;
    __syncthreads();
    // the edges inside C0: a warp per member x = C[i], lanes over N+(x)
    for (int i = w; i < c; i += nw) {
      const int64_t xb = off[C[i]], xd = off[C[i] + 1] - xb;
      if (lane == 0) bytes += 4ull * (unsigned long long)xd;
      for (int64_t j = lane; j < xd; j += 32) {
        const int32_t y = cols[xb + j];
        int lo = 0, hi = c;  // y's position in C, if any
        while (lo < hi) {
          const int mid = (lo + hi) >> 1;
          if (C[mid] < y) lo = mid + 1; else hi = mid;
        }
        if (lo < c && C[lo] == y) {
          const int a = min(i, lo), z = max(i, lo);
          atomicOr(&dsm[(size_t)a * words + (z >> 6)], 1ull << (z & 63));
        }
      }
    }
    __syncthreads();
    // pre[i] = adjacent pairs in rows below i: kDenseRows rows a thread, a warp scan, warp sums
    int rc[kDenseRows], mine = 0;
#pragma unroll
    for (int q = 0; q < kDenseRows; ++q) {
      const int i = kDenseRows * threadIdx.x + q;
      rc[q] = 0;
      if (i < c)
        for (int x = (i + 1) >> 6; x < words; ++x) rc[q] += __popcll(dsm[(size_t)i * words + x]);
      mine += rc[q];
    }
    int incl = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      const int y = __shfl_up_sync(0xffffffffu, incl, o);
      if (lane >= o) incl += y;
    }
    if (lane == 31) wcount[w] = incl;
    __syncthreads();
    int run = incl - mine;
    for (int q = 0; q < w; ++q) run += wcount[q];
#pragma unroll
    for (int q = 0; q < kDenseRows; ++q) {
      const int i = kDenseRows * threadIdx.x + q;
      if (i < c) pre[i] = run;
      run += rc[q];
    }
    if (threadIdx.x == kDenseThreads - 1) pre[c] = run;  // every pair
    __syncthreads();
    const int npairs = pre[c];
    for (int p = threadIdx.x; p < npairs; p += kDenseThreads) {
      // row i: the last with pre[i] <= p (pre[c] > p); j = its (p - pre[i])-th member
      int lo = 0, hi = c;
      while (hi - lo > 1) {
        const int mid = (lo + hi) >> 1;
        if (pre[mid] <= p) lo = mid; else hi = mid;
      }
      const int i = lo;
      const unsigned long long* Ri = dsm + (size_t)i * words;
      int r = p - pre[i];
      int x = (i + 1) >> 6;
      for (;; ++x) {
        const int pc = __popcll(Ri[x]);
        if (r < pc) break;
        r -= pc;
      }
      const int j = x * 64 + select_bit(Ri[x], r);
      if (DEEP && words <= 2 && k <= 7) cnt += pair_word_cliques<2>(dsm, words, i, j, k - 4);
      else if (DEEP && words <= 4 && k <= 7) cnt += pair_word_cliques<4>(dsm, words, i, j, k - 4);
      else cnt += pair_cliques(dsm, words, i, j, k - 4);
    }
    __syncthreads();
  }
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
  }
  if (lane == 0) {
    if (cnt) atomicAdd(out, cnt);
    if (bytes) atomicAdd(out + 1, bytes);
  }
}

// ============================== rows of one source ===================================
// What bounds these kernels: building the rows streams N+(x) for every member x of N+(u) (W
// elements over the graph, mostly L2 hits) with one search in shared memory each, and is issue
// bound; the counting after it is AND / popc on shared memory.  Every search per edge that
// the walk above makes in global memory (dependent loads) is gone.
constexpr int kRowMax = 960;       // rows of 960 x 15 words (115 KB) and everything below fit
constexpr int kRowWarp = 128;      // C0 up to this size is renumbered and counted by one warp
constexpr int kRowBlock = 512;     // k = 5: C0 up to this size by the CTA that holds its rows
constexpr int kRowThreads = 512;
constexpr int kRowParts = 2048;    // part table of N+(u): two parts a member
constexpr int kRowBuckets = 4;     // lists by length, longest first (row_bucket)
constexpr int kRowCounts = 4;      // the first of their counts among the queues
// Sources of the longer half that a warp each would take, up to which they are split over CTAs
// instead, from k = 5 on: one such row's search held a whole count up where the GPU had little else to
// do.  Chung-Lu n = 128 000, 0.9 M edges: k = 5 517 -> 202 us, k = 6 850 -> 345; R-MAT scale 11 of 31 000
// edges 307 -> 182 and 752 -> 456.  k >= 6: with 2048 instead Chung-Lu n = 7000 k = 6 takes 511 us (188);
// with 65536 RGG n = 128 000 5.6 ms (2.6); Chung-Lu n = 32 000 of 0.5 M edges 970 with 8192, 650 with 16384.
constexpr int kFewRows = 2048;       // k = 5, or n / 32 (Chung-Lu n = 300 000 of mean degree 14 1.46 -> 0.60 ms)
constexpr int kFewRowsDeep = 16384;  // k >= 6, or n / 16
constexpr int kRowSearch = 128;    // lists longer than this are searched for the members of
                                   // N+(u), not streamed, where N+(u) fits one warp's masks

// D-cliques inside m of the DAG with successor rows `rows` (D levels unrolled into nested
// loops, nothing on a stack); D > kRowUnroll: `d` levels by mask_cliques' explicit stack.
constexpr int kRowUnroll = 5;
template <int D, class M>
__device__ __forceinline__ unsigned long long row_cliques(const M* rows, M m, int d) {
  if constexpr (D == 0) {
    return 1ull;
  } else if constexpr (D == 1) {
    return (unsigned long long)popc_of(m);
  } else if constexpr (D == 2) {
    unsigned c = 0;
    for (M r = m; r; r &= r - 1) c += popc_of((M)(m & rows[first_bit(r)]));
    return c;
  } else if constexpr (D <= kRowUnroll) {
    unsigned long long c = 0;
    for (M r = m; r; r &= r - 1) {
      const M nm = m & rows[first_bit(r)];
      if (popc_of(nm) >= D - 1) c += row_cliques<D - 1, M>(rows, nm, d);
    }
    return c;
  } else {
    return mask_cliques(rows, m, d);
  }
}

// Position of y in the sorted S[0, d), padded to R = 2^j entries with INT_MAX; -1 if absent.
template <int R>
__device__ __forceinline__ int member_of(const int32_t* S, int d, int32_t y) {
  int p = 0;
#pragma unroll
  for (int step = R / 2; step > 0; step >>= 1)
    if (S[p + step - 1] < y) p += step;
  return p < d && S[p] == y ? p : -1;
}

// Calls f(y, k, valid) on all 32 lanes for every element y of the lists [xb, xb + xd) held by
// the lanes (k = the lane holding y's list): lists of 32 or more elements are walked by the
// whole warp, shorter ones laid end to end and dealt 32 elements a round.
template <class F>
__device__ __forceinline__ void for_members(const int32_t* cols, int64_t xb, int xd, int lane, F f) {
  unsigned longm = __ballot_sync(0xffffffffu, xd >= 32);
  while (longm) {
    const int k = __ffs(longm) - 1;
    longm &= longm - 1;
    const int32_t* P = cols + __shfl_sync(0xffffffffu, xb, k);
    const int ln = __shfl_sync(0xffffffffu, xd, k);
    int j0 = 0;
    for (; j0 + 64 <= ln; j0 += 64) {
      const int32_t y0 = __ldg(P + j0 + lane), y1 = __ldg(P + j0 + 32 + lane);
      f(y0, k, true);
      f(y1, k, true);
    }
    for (; j0 < ln; j0 += 32) {
      const bool v = j0 + lane < ln;
      f(v ? __ldg(P + j0 + lane) : 0, k, v);
    }
  }
  const int slen = xd < 32 ? xd : 0;
  int incl = slen;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  const int total = __shfl_sync(0xffffffffu, incl, 31);
  const int start = incl - slen;
  for (int t0 = 0; t0 < total; t0 += 32) {
    const int t = t0 + lane;
    int k = 0;  // the last lane whose list starts at or before t
#pragma unroll
    for (int step = 16; step > 0; step >>= 1)
      if (__shfl_sync(0xffffffffu, start, k + step) <= t) k += step;
    const int64_t kb = __shfl_sync(0xffffffffu, xb, k);
    const int ks = __shfl_sync(0xffffffffu, start, k);
    const bool v = t < total;
    f(v ? __ldg(cols + kb + (t - ks)) : 0, k, v);
  }
}

// A warp per source u with lo < |N+(u)| <= R (R = bits of M), k - 1 <= |N+(u)|, over the edges
// of [e0, e1).  Sources above few_lo are left to kcl_rows_block_kernel where they are few (*few).  KD = k - 3: the members to choose below an induced edge (0: k = 3; above
// kRowUnroll: any k).  Sources are taken `grab` (<= 32, or a multiple of 32) at a time from `queue`.
template <class M, int KD>
__global__ void __launch_bounds__(kKcWarps * 32) kcl_rows_warp_kernel(const int64_t* off, const int32_t* cols, int64_t n,
                                                                    int64_t e0, int64_t e1, int k, int lo, int few_lo,
                                                                    const int* few, int few_max, int grab, int* queue,
                                                                    unsigned long long* out) {
  constexpr int R = 8 * (int)sizeof(M);
  constexpr int kPairs = R * (R - 1) / 2;  // induced edges of a DAG; other digraphs may hold more
  __shared__ int32_t Ssm[kKcWarps][R];
  __shared__ M rsm[kKcWarps][R];
  __shared__ uint16_t psm[kKcWarps][KD ? kPairs : 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  int32_t* S = Ssm[w];
  M* rows = rsm[w];
  uint32_t* row32 = reinterpret_cast<uint32_t*>(rows);
  uint16_t* pairs = psm[w];
  const unsigned below = (1u << lane) - 1;
  unsigned long long cnt = 0, bytes = 0;
  const int hi = *few <= few_max ? min(few_lo, R) : R;
  if (hi <= lo) return;
  int64_t row0 = 0, row_end = 0;  // sources grabbed
  for (;; row0 += 32) {
    if (row0 >= row_end) {
      int chunk = 0;
      if (lane == 0) chunk = atomicAdd(queue, 1);
      row0 = (int64_t)__shfl_sync(0xffffffffu, chunk, 0) * grab;
      row_end = min(row0 + grab, n);
      if (row0 >= n) break;
    }
    const int64_t row = min(row0 + lane, n);
    const int64_t rb = __ldg(off + row), re = __ldg(off + min(row + 1, n));
    unsigned todo = __ballot_sync(0xffffffffu, row < row_end && re - rb > lo && re - rb <= hi && re - rb >= k - 1 &&
                                                   min(re, e1) > max(rb, e0));
    while (todo) {
      const int q = __ffs(todo) - 1;
      todo &= todo - 1;
      const int64_t ub = __shfl_sync(0xffffffffu, rb, q);
      const int d = (int)(__shfl_sync(0xffffffffu, re, q) - ub);
      const int ia = (int)max(e0 - ub, (int64_t)0), ib = (int)min(e1 - ub, (int64_t)d);  // edges counted
      for (int j = lane; j < R; j += 32) {
        S[j] = j < d ? __ldg(cols + ub + j) : INT32_MAX;
        rows[j] = 0;
      }
      __syncwarp();
      int np = 0;
      // an induced edge S[i] -> S[j] on the lanes with `hit` (all 32 lanes call)
      auto found = [&](bool hit, int i, int j) {
        if constexpr (KD == 0) {
          cnt += hit && i >= ia && i < ib;
        } else {
          if (hit) atomicOr(&row32[R == 32 ? i : 2 * i + (j >> 5)], 1u << (j & 31));
          hit = hit && i >= ia && i < ib;
          const unsigned b = __ballot_sync(0xffffffffu, hit);
          const int at = np + __popc(b & below);
          if (hit && at < kPairs) pairs[at] = (uint16_t)(i << 8 | j);
          np += __popc(b);
        }
      };
      for (int base = 0; base < d; base += 32) {
        int64_t xb = 0;
        int xd = 0;
        if (base + lane < d) {
          const int32_t x = S[base + lane];
          xb = __ldg(off + x);
          xd = (int)(__ldg(off + x + 1) - xb);
        }
        bytes += 4ull * (unsigned long long)xd;
        unsigned far = __ballot_sync(0xffffffffu, xd > kRowSearch);
        while (far) {  // long lists: the members of N+(u) are searched in them
          const int kk = __ffs(far) - 1;
          far &= far - 1;
          const int64_t kb = __shfl_sync(0xffffffffu, xb, kk);
          const int kd = __shfl_sync(0xffffffffu, xd, kk);
          for (int j = lane; j < R; j += 32)
            found(j < d && kc_has(cols + kb, kd, S[j]), base + kk, j);
        }
        for_members(cols, xb, xd > kRowSearch ? 0 : xd, lane, [&](int32_t y, int kk, bool v) {
          const int j = member_of<R>(S, d, y);
          found(v && j >= 0, base + kk, j & (R - 1));
        });
      }
      __syncwarp();
      if constexpr (KD > 0) {
        if (np <= kPairs) {
          for (int p = lane; p < np; p += 32) {
            const int ij = pairs[p];
            cnt += row_cliques<KD, M>(rows, rows[ij >> 8] & rows[ij & 255], k - 3);
          }
        } else {  // not a DAG: every bit of every row
          for (int i = ia; i < ib; ++i)
            for (int j = lane; j < R; j += 32)
              if ((rows[i] >> j) & 1) cnt += row_cliques<KD, M>(rows, rows[i] & rows[j], k - 3);
        }
        __syncwarp();
      }
    }
  }
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
  }
  if (lane == 0) {
    if (cnt) atomicAdd(out, cnt);
    if (bytes) atomicAdd(out + 1, bytes);
  }
}

// Sources with mid < |N+(u)| <= hi and an edge in [e0, e1), longest bucket first: lists[b * cap ...],
// counts[b].  Those with lo < |N+(u)| <= mid, which a warp each takes where they are many, are
// counted in counts[kRowBuckets] and listed (lists[kRowBuckets * cap ...]) up to few_max.
__device__ __forceinline__ int row_bucket(int64_t d) { return d > 384 ? 0 : d > 192 ? 1 : d > 96 ? 2 : 3; }
__global__ void kcl_rows_list_kernel(const int64_t* off, int64_t n, int64_t e0, int64_t e1, int lo, int mid, int hi,
                                     int64_t cap, int few_max, int32_t* lists, int* counts) {
  const int lane = threadIdx.x & 31;
  const int64_t n_pad = (n + 31) & ~31ll;
  for (int64_t u = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; u < n_pad; u += (int64_t)gridDim.x * blockDim.x) {
    int mine = -1;
    if (u < n) {
      const int64_t b = off[u], e = off[u + 1];
      if (e - b > lo && e - b <= hi && min(e, e1) > max(b, e0)) mine = e - b > mid ? row_bucket(e - b) : kRowBuckets;
    }
    for (int q = 0; q <= kRowBuckets; ++q) {  // one atomic per warp and bucket
      const unsigned m = __ballot_sync(0xffffffffu, mine == q);
      int at = 0;
      if (m && lane == 0) at = atomicAdd(&counts[q], __popc(m));
      at = __shfl_sync(0xffffffffu, at, 0);
      at += __popc(m & ((1u << lane) - 1));
      if (mine == q && (q < kRowBuckets || at < few_max)) lists[q * cap + at] = (int32_t)u;
    }
  }
}

// Shared memory of kcl_rows_block_kernel for sources of up to dmax members.  MODE as there.
__host__ __device__ inline int row_stride(int d) { return ((d + 63) >> 6) | 1; }  // odd: rows of random j spread over the banks
constexpr int kRowWarpWords = kRowWarp * 3;  // rows of two words, three apart
struct RowsSmem {
  size_t rows, rows2, wrows, s, wmem, mem, rcnt, bytes;  // byte offsets of the parts, and their end
  __host__ __device__ RowsSmem(int dmax, int mode) {
    const int d2 = dmax < kRowBlock ? dmax : kRowBlock;
    const size_t list = (size_t)((dmax + 8) & ~7);
    rows = 0;
    rows2 = rows + sizeof(unsigned long long) * (size_t)dmax * row_stride(dmax);
    wrows = rows2 + (mode == 2 ? sizeof(unsigned long long) * (size_t)d2 * row_stride(d2) : 0);
    s = wrows + (mode >= 2 ? sizeof(unsigned long long) * kRowWarpWords * (kRowThreads / 32) : 0);
    wmem = s + sizeof(int32_t) * list;
    mem = wmem + (mode >= 2 ? sizeof(uint16_t) * kRowWarp * (kRowThreads / 32) : 0);
    rcnt = mem + (mode == 2 ? sizeof(uint16_t) * kRowBlock : 0);
    bytes = rcnt + (mode == 2 ? sizeof(uint16_t) * list : 0);
  }
};

// The members of row `Ri` (32-bit halves r32, `halves` of them) in order, by one warp.
__device__ __forceinline__ void row_members(const uint32_t* r32, int halves, uint16_t* M, int lane) {
  for (int h = 0, at = 0; h < halves; ++h) {
    const uint32_t bits = r32[h];
    if ((bits >> lane) & 1) M[at + __popc(bits & ((1u << lane) - 1))] = (uint16_t)(h * 32 + lane);
    at += __popc(bits);
  }
  __syncwarp();
}

// A CTA per source u too long for a warp.  MODE 0: k = 3 (the hits are the count), 1:
// k = 4, 2: k = 5, 3: k >= 6.  Rows are built from the lists of the members, a batch of 32
// members a warp.  From k = 5 on, with few sources, each is split over several CTAs (every
// nsplit-th of its edges): the rows are cheap to build again next to the search below them, and
// a dense core's few sources would otherwise leave most CTAs idle.  Edges whose row is too long
// for the warps (and at k = 5 for the CTA) go on the dense list.
template <int MODE>
__global__ void __launch_bounds__(kRowThreads) kcl_rows_block_kernel(const int64_t* off, const int32_t* cols, int64_t e0,
                                                                    int64_t e1, int k, const int32_t* lists, int64_t cap,
                                                                    const int* counts, int few_max, int dmax, int* queue,
                                                                    unsigned long long* dense,
                                                                    unsigned long long* out) {
  extern __shared__ __align__(16) unsigned char rsm[];
  const RowsSmem at(dmax, MODE);
  unsigned long long* rows = reinterpret_cast<unsigned long long*>(rsm + at.rows);
  int32_t* S = reinterpret_cast<int32_t*>(rsm + at.s);
  __shared__ int item, next_batch, next_row;
  __shared__ uint32_t ptab[kRowParts];
  __shared__ uint16_t part_start[kRowParts + 1];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5, nw = kRowThreads / 32;
  int first[kRowBuckets + 2];
  first[0] = 0;
#pragma unroll
  for (int b = 0; b < kRowBuckets; ++b) first[b + 1] = first[b] + counts[b];
  first[kRowBuckets + 1] = first[kRowBuckets] + (counts[kRowBuckets] <= few_max ? counts[kRowBuckets] : 0);
  // the long sources (the lists but the last) and the others are split by their own numbers
  const int sources = first[kRowBuckets + 1], longs = first[kRowBuckets];
  // Parts of fewer than four edges only build the rows once more: four of a CTA's sixteen warps
  // already have a scheduler each.
  const int split_long = MODE < 2 ? 1 : min(max(6 * (int)gridDim.x / max(longs, 1), 1), min(max(dmax / 4, 1), 32));
  const int split_few = MODE < 2 ? 1 : min(max(3 * (int)gridDim.x / max(sources - longs, 1), 1), 8);
  unsigned long long cnt = 0, bytes = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      item = atomicAdd(queue, 1);
      next_batch = 0;
      next_row = 0;
    }
    __syncthreads();
    const bool is_long = item < longs * split_long;
    const int nsplit = is_long ? split_long : split_few, at_item = is_long ? item : item - longs * split_long;
    const int it = at_item / nsplit + (is_long ? 0 : longs), part = at_item % nsplit;
    if (it >= sources) break;
    int b = 0, fb = 0;
#pragma unroll
    for (int q = 1; q <= kRowBuckets; ++q)
      if (it >= first[q]) {
        b = q;
        fb = first[q];
      }
    const int64_t u = lists[b * cap + (it - fb)];
    const int64_t ub = off[u];
    const int d = (int)(off[u + 1] - ub);
    const int ia = (int)max(e0 - ub, (int64_t)0), ib = (int)min(e1 - ub, (int64_t)d);
    const int words = (d + 63) >> 6, st = row_stride(d);
    for (int j = threadIdx.x; j < d; j += kRowThreads) S[j] = __ldg(cols + ub + j);
    if (MODE > 0)
      for (int t = threadIdx.x; t < d * st; t += kRowThreads) rows[t] = 0ull;
    __syncthreads();
    const int shift = build_parts(S, d, kRowParts, part_start, ptab, threadIdx.x, kRowThreads, [] { __syncthreads(); });
    const int32_t s_lo = S[0];
    const uint32_t s_range = (uint32_t)(S[d - 1] - s_lo);
    // lists a warp takes at a time: at least two rounds for every warp, where there are that many
    const int grab = min(max(d / (2 * nw), 1), 32);
    uint32_t* r32 = reinterpret_cast<uint32_t*>(rows);
    for (;;) {
      int base = 0;
      if (lane == 0) base = atomicAdd(&next_batch, grab);
      base = __shfl_sync(0xffffffffu, base, 0);
      if (base >= d) break;
      int64_t xb = 0;
      int xd = 0;
      if (lane < grab && base + lane < d) {
        const int32_t x = S[base + lane];
        xb = __ldg(off + x);
        xd = (int)(__ldg(off + x + 1) - xb);
      }
      bytes += 4ull * (unsigned long long)xd;
      for_members(cols, xb, xd, lane, [&](int32_t y, int kk, bool v) {
        const uint32_t r = (uint32_t)(y - s_lo);
        if (!v || r > s_range) return;
        const uint32_t pe = ptab[r >> shift];
        int lo = (int)(pe & 0xffffu), len = (int)(pe >> 16) - lo;
        if (len == 0) return;
        while (len > 1) {  // branch-free lower bound inside the part
          const int half = len >> 1;
          lo = S[lo + half - 1] < y ? lo + half : lo;
          len -= half;
        }
        if (S[lo] != y) return;
        const int i = base + kk;
        if constexpr (MODE == 0) cnt += i >= ia && i < ib;
        else atomicOr(&r32[2 * ((size_t)i * st + (lo >> 6)) + ((lo >> 5) & 1)], 1u << (lo & 31));
      });
    }
    __syncthreads();
    if constexpr (MODE == 1) {
      // a warp per row: the lanes holding a successor j take |row i AND row j|
      for (int i = ia + w; i < ib; i += nw) {
        const unsigned long long* Ri = rows + (size_t)i * st;
        for (int h = 0; h < 2 * words; ++h) {
          const uint32_t bits = r32[2 * (size_t)i * st + h];
          if ((bits >> lane) & 1) {
            const unsigned long long* Rj = rows + (size_t)(h * 32 + lane) * st;
            unsigned c = 0;
            for (int x = 0; x < words; ++x) c += __popcll(Ri[x] & Rj[x]);
            cnt += c;
          }
        }
      }
    }
    if constexpr (MODE >= 2) {
      auto has = [&](int i, int j) { return (r32[2 * ((size_t)i * st) + (j >> 5)] >> (j & 31)) & 1u; };
      uint16_t* rcnt = reinterpret_cast<uint16_t*>(rsm + at.rcnt);
      // a warp per row: its members renumbered into rows A of one or two words, then the
      // (k-2)-cliques of the induced graph: an edge a -> c a lane, with the (k-4)-cliques of
      // the two rows' common members
      unsigned long long* A = reinterpret_cast<unsigned long long*>(rsm + at.wrows) + w * kRowWarpWords;
      uint16_t* Mw = reinterpret_cast<uint16_t*>(rsm + at.wmem) + w * kRowWarp;
      for (;;) {
        int t = 0;
        if (lane == 0) t = atomicAdd(&next_row, 1);
        t = __shfl_sync(0xffffffffu, t, 0);
        const int i = ia + part + t * nsplit;
        if (i >= ib) break;
        const int r = __reduce_add_sync(0xffffffffu, lane < words ? __popcll(rows[(size_t)i * st + lane]) : 0);
        if (MODE == 2 && lane == 0) rcnt[i] = (uint16_t)r;
        const bool two = r > kMaskMax && r <= kRowWarp && k <= 7;
        if (r > kMaskMax && !two && (MODE == 3 || r > kRowBlock) && lane == 0)
          dense[1 + atomicAdd(dense, 1ull)] = (unsigned long long)(ub + i);
        if (r < k - 2 || (r > kMaskMax && !two)) continue;
        row_members(r32 + 2 * (size_t)i * st, 2 * words, Mw, lane);
        if (!two) {
          const int m0 = lane < r ? Mw[lane] : -1, m1 = lane + 32 < r ? Mw[lane + 32] : -1;
          for (int a = 0; a < r; ++a) {
            const int ma = Mw[a];
            const unsigned lo = __ballot_sync(0xffffffffu, m0 >= 0 && has(ma, m0));
            const unsigned hi = __ballot_sync(0xffffffffu, m1 >= 0 && has(ma, m1));
            if (lane == 0) A[a] = ((unsigned long long)hi << 32) | lo;
          }
          __syncwarp();
          for (int a = 0; a < r; ++a) {
            const unsigned long long Ra = A[a];
            if (__popcll(Ra) < k - 3) continue;
            for (int c = lane; c < r; c += 32)
              if ((Ra >> c) & 1) {
                const unsigned long long m = Ra & A[c];
                if (MODE == 2) cnt += __popcll(m);
                else if (k == 6) cnt += row_cliques<2, unsigned long long>(A, m, 0);
                else if (k == 7) cnt += row_cliques<3, unsigned long long>(A, m, 0);
                else cnt += mask_cliques(A, m, k - 4);
              }
          }
        } else {  // an induced edge is kept at the lower position of the two, as kcl_dense_kernel does
          uint32_t* A32 = reinterpret_cast<uint32_t*>(A);
          for (int a = 0; a < r; ++a) {
            const int ma = Mw[a];
            for (int h = 0; h < 4; ++h) {
              const int c = h * 32 + lane;
              bool in = false;
              if (c >= a && c < r) {
                const int mc = Mw[c];
                in = has(ma, mc) || has(mc, ma);
              }
              const unsigned bits = __ballot_sync(0xffffffffu, in);
              if (lane == 0) A32[6 * a + h] = bits;
            }
          }
          __syncwarp();
          for (int a = 0; a < r; ++a)
            for (int c = (a & ~31) + lane; c < r; c += 32)
              if ((A32[6 * a + (c >> 5)] >> (c & 31)) & 1) {
                if (MODE == 2) {
                  cnt += (unsigned)(__popcll(A[3 * a] & A[3 * c]) + __popcll(A[3 * a + 1] & A[3 * c + 1]));
                } else {
                  cnt += pair_word_cliques<2>(A, 3, a, c, k - 4);
                }
              }
        }
        __syncwarp();
      }
    }
    if constexpr (MODE == 2) {
      // longer rows by the whole CTA, renumbered the same way; an induced edge is one AND / popc
      auto has = [&](int i, int j) { return (r32[2 * ((size_t)i * st) + (j >> 5)] >> (j & 31)) & 1u; };
      const uint16_t* rcnt = reinterpret_cast<const uint16_t*>(rsm + at.rcnt);
      uint16_t* mem = reinterpret_cast<uint16_t*>(rsm + at.mem);
      unsigned long long* rows2 = reinterpret_cast<unsigned long long*>(rsm + at.rows2);
      uint32_t* q32 = reinterpret_cast<uint32_t*>(rows2);
      __syncthreads();
      for (int i = ia + part; i < ib; i += nsplit) {
        const int r = rcnt[i];
        if (r <= kRowWarp || r > kRowBlock) continue;
        const unsigned long long* Ri = rows + (size_t)i * st;
        for (int j = threadIdx.x; j < d; j += kRowThreads)
          if (has(i, j)) {
            int pos = __popcll(Ri[j >> 6] & ((1ull << (j & 63)) - 1));
            for (int x = 0; x < (j >> 6); ++x) pos += __popcll(Ri[x]);
            mem[pos] = (uint16_t)j;
          }
        __syncthreads();
        const int w2 = (r + 63) >> 6, st2 = row_stride(r);
        for (int a = w; a < r; a += nw) {
          const int ma = mem[a];
          for (int h = 0; h < 2 * w2; ++h) {
            const int c = h * 32 + lane;
            bool in = false;
            if (c >= a && c < r) {
              const int mc = mem[c];
              in = has(ma, mc) || has(mc, ma);
            }
            const unsigned bits = __ballot_sync(0xffffffffu, in);
            if (lane == 0) q32[2 * (size_t)a * st2 + h] = bits;
          }
        }
        __syncthreads();
        for (int a = w; a < r; a += nw) {
          const unsigned long long* Ra = rows2 + (size_t)a * st2;
          for (int c = (a & ~31) + lane; c < r; c += 32)
            if ((q32[2 * (size_t)a * st2 + (c >> 5)] >> (c & 31)) & 1) {
              const unsigned long long* Rc = rows2 + (size_t)c * st2;
              unsigned n = 0;
              for (int x = c >> 6; x < w2; ++x) n += __popcll(Ra[x] & Rc[x]);
              cnt += n;
            }
        }
        __syncthreads();
      }
    }
    __syncthreads();
  }
  for (int o = 16; o > 0; o >>= 1) {
    cnt += __shfl_xor_sync(0xffffffffu, cnt, o);
    bytes += __shfl_xor_sync(0xffffffffu, bytes, o);
  }
  if (lane == 0) {
    if (cnt) atomicAdd(out, cnt);
    if (bytes) atomicAdd(out + 1, bytes);
  }
}

}  // namespace

}  // namespace atc

using namespace atc;

// Rows of up to R = 32 or 64 members (M's bits): one warp launch for the given k.
template <class M>
static atc_status launch_rows_warp(const atc_csr* csr, int64_t e0, int64_t e1, int k, int lo, int few_lo, const int* few,
                                   int few_max, int* queue,
                                   unsigned long long* out, cudaStream_t s) {
  using Kernel = void (*)(const int64_t*, const int32_t*, int64_t, int64_t, int64_t, int, int, int, const int*, int,
                          int, int*, unsigned long long*);
  static const Kernel kernels[kRowUnroll + 2] = {
      kcl_rows_warp_kernel<M, 0>, kcl_rows_warp_kernel<M, 1>, kcl_rows_warp_kernel<M, 2>, kcl_rows_warp_kernel<M, 3>,
      kcl_rows_warp_kernel<M, 4>, kcl_rows_warp_kernel<M, 5>, kcl_rows_warp_kernel<M, kRowUnroll + 1>};
  const Kernel kern = kernels[std::min(k - 3, kRowUnroll + 1)];
  int bps = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kern, kKcWarps * 32, 0);
  // a grab of 32 sources (one coalesced read of their offsets) unless that would leave warps
  // without work; more, about 32 edges, where most vertices have none (the queue's one address takes an
  // atomic in 0.7 ns: 4.2 ms a launch for 10^8 vertices with grabs of 32)
  const int64_t warps = (int64_t)sm_count() * std::max(bps, 1) * kKcWarps;
  const int64_t most = std::max<int64_t>(csr->n / (4 * warps), 1);
  const int64_t sparse = std::max<int64_t>(csr->n / std::max<int64_t>(csr->m, 1), 1) * 32;
  const int grab = (int)(most <= 32 ? most : std::min<int64_t>({most & ~31ll, sparse, 1 << 20}));
  const int64_t grid = std::min<int64_t>(warps, (csr->n + grab - 1) / grab) / kKcWarps + 1;
  kern<<<(unsigned)grid, kKcWarps * 32, 0, s>>>(csr->offsets, csr->cols, csr->n, e0, e1, k, lo, few_lo, few,
                                                    few_max, grab, queue, out);
  ATC_CK(cudaGetLastError());
  return ATC_OK;
}

template <int MODE>
static atc_status launch_rows_block(const atc_csr* csr, int64_t e0, int64_t e1, int k, int dmax, const int32_t* lists,
                                    int64_t cap, int* counts, int few_max, int* queue, unsigned long long* dense,
                                    unsigned long long* out, cudaStream_t s) {
  const size_t smem = RowsSmem(dmax, MODE).bytes;
  ATC_CK(cudaFuncSetAttribute((const void*)kcl_rows_block_kernel<MODE>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)smem));
  int bps = 0;
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kcl_rows_block_kernel<MODE>, kRowThreads, smem);
  kcl_rows_block_kernel<MODE><<<(unsigned)(sm_count() * std::max(bps, 1)), kRowThreads, smem, s>>>(
      csr->offsets, csr->cols, e0, e1, k, lists, cap, counts, few_max, dmax, queue, dense, out);
  ATC_CK(cudaGetLastError());
  return ATC_OK;
}

// Whether the edges of a window are better walked (with the dense kernel from k = 5 on) than counted by rows:
// by predicted times (ps) of the two.  The walk takes one launch or two, a little per edge (more where most
// wedges close, as W near W_min tells) and dependent searches per wedge, more the longer the lists; rows take up
// to six launches, a pass over all vertices, and less per wedge.  From k = 7 on the enumeration below the edges
// is nearly all of either, which a warp per edge spreads better than a warp or CTA per source: rows are left to
// graphs with hardly a wedge, at k = 7 also to those of few hubs (W below 2 W_min).
// Fitted to 118 graphs of 8K to 2M edges (R-MAT, Chung-Lu, RGG, stars; ids spread by 1 to 256; every orientation), each
// counted both ways, and tried on 94 others: k = 4..9 one call in ten or fewer is more than 5 % slower than by
// the walk; by the windows of m and W that the choice was made with before, one in three.  Walk / rows in us, k = 4:
// Chung-Lu of 1.4M edges (W = 3.2 m) 257 / 61, RGG of 1.5M (2.2 m) 344 / 75, of 96 000 (11 m) 175 / 69, R-MAT of 60 000 (42 m) 296 /
// 135, of 32 000 (19 m) 85 / 131, a star of 39 000 36 / 62.
static bool walk_pays(const atc_csr* csr, int k, int64_t edges) {
  struct Cost {
    double closed;           // walk: per edge where wedges close
    double walk, walk_long;  // per wedge, and per wedge and 100 ids of the longest list
    double rows, rows_long;
  };
  static const Cost costs[] = {{0.0, 5.4, 0.09, 4.5, 0.05}, {220.0, 16.0, 6.6, 7.5, 0.64}, {170.0, 18.6, 4.2, 11.7, 3.4},
                               {130.0, 20.0, 14.0, 16.0, 12.2}, {130.0, 20.0, 126.0, 16.0, 112.0}};
  const Cost& c = costs[std::min(k, 7) - 3];
  const double n = (double)csr->n, m = (double)edges, longest = csr->max_outdeg, wmin = (double)csr->wedges_min;
  const double w = (double)csr->wedges * m / (double)csr->m, lw = w * longest / 100.0;
  const double close = wmin > 0.0 ? std::min(std::max((1.3 - (double)csr->wedges / wmin) / 0.2, 0.0), 1.0) : 0.0;
  const double walk = 4.0e7 + (95.0 + c.closed * close) * m + c.walk * w + c.walk_long * lw;
  double rows = 5.5e7 + 2.5 * n + 8.0 * m + c.rows * w + c.rows_long * lw;
  if (k == 3) rows += (longest > 32 ? 1.5e7 : 0.0) + (longest > 64 ? 3.0e7 : 0.0);  // its launches
  if (rows >= walk) return true;
  return k >= 7 && w > 5.0 * m && (k > 7 || csr->wedges >= 2 * csr->wedges_min);
}

// k-cliques whose first two vertices (in orientation order) form an edge of [e0, e1).  by_rows:
// where walk_pays says no, sources of up to kRowMax members by rows and longer ones by the walk;
// otherwise every edge by the walk alone.
static atc_status kcl_window(const atc_csr* csr, uint32_t k, int64_t e0, int64_t e1, uint64_t* count, atc_stats* stats,
                             cudaStream_t s, bool by_rows = true) {
  *count = 0;
  unsigned long long h[2] = {0, 0};
  EventTimer tm;
  int launches = 0;
  if (e1 > e0) {
    CsrPriv* pv = static_cast<CsrPriv*>(csr->priv);
    const int cap = std::max(csr->max_outdeg, 1);
    const int levels = (int)k - 2;
    DevBuf<int> q;  // queues: 32-bit rows, 64-bit rows, block rows; from kRowCounts on the block lists' counts
    DevBuf<int32_t> scratch, lists;
    // k >= 6: the search below one source of 33..64 members is long enough for a CTA (one warp
    // of it held R-MAT scale 14's k = 6 count at 12.8 ms, 3.8 by the walk)
    const int warp_max = k >= 6 ? 32 : kMaskMax;  // longest rows a warp takes
    // from k = 5 on the upper half of them goes to CTAs too where they are few
    const int few_lo = k >= 5 ? warp_max / 2 : warp_max;
    const int few_max =
        (int)(k >= 6 ? std::max<int64_t>(kFewRowsDeep, csr->n / 16) : std::max<int64_t>(kFewRows, csr->n / 32));
    const int64_t lcap = csr->m / (warp_max + 1) + 1;
    bool walk_dense = by_rows && walk_pays(csr, (int)k, e1 - e0);
    if (by_rows && !walk_dense &&
        (q.alloc(kRowCounts + kRowBuckets + 1, s) != ATC_OK ||
         (cap > few_lo && lists.alloc((size_t)lcap * kRowBuckets + few_max, s) != ATC_OK))) {
      cudaGetLastError();  // no room for the lists of rows: the walk needs none
      walk_dense = true;
    }
    if (walk_dense) by_rows = false;
    const int row_max = by_rows ? kRowMax : 0;
    const bool walk = cap > row_max;  // some source is too long for rows
    int64_t grid = 0;
    DevBuf<unsigned long long> dense;
    if (walk) {
      int bps = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, kcl_kernel, kKcWarps * 32, 0);
      if (bps < 1) bps = 1;
      grid = (int64_t)sm_count() * bps;
      // keep the scratch within 4 GiB
      int64_t per_warp = (int64_t)levels * cap * 4;
      while (grid > sm_count() && grid * kKcWarps * per_warp > (4ll << 30)) grid /= 2;
      ATC_TRY(scratch.alloc((size_t)grid * kKcWarps * levels * cap, s));
    }
    // edges with 65..1024 members in C0 go to the dense kernel from k = 5 on (at k = 4 the walk
    // does one intersection per member of C0 as fast)
    const bool use_dense = (by_rows || walk_dense) && k >= 5 && cap > kMaskMax;
    if (use_dense) ATC_TRY(dense.alloc((size_t)csr->m + 2, s));
    const bool blocks = by_rows && cap > few_lo;
    tm.start(s);
    ATC_CK(cudaMemsetAsync(pv->counter, 0, 2 * sizeof(unsigned long long), s));
    if (by_rows) ATC_CK(cudaMemsetAsync(q.p, 0, (kRowCounts + kRowBuckets + 1) * sizeof(int), s));
    if (use_dense) ATC_CK(cudaMemsetAsync(dense.p, 0, 2 * sizeof(unsigned long long), s));
    if (walk) {
      kcl_kernel<<<(unsigned)grid, kKcWarps * 32, 0, s>>>(csr->offsets, csr->cols, pv->esrc, e0, e1, (int)k, cap,
                                                           row_max, scratch.p, use_dense ? dense.p + 1 : nullptr,
                                                           pv->counter);
      ATC_CK(cudaGetLastError());
      ++launches;
    }
    if (blocks) {
      const int dmax = std::min(cap, row_max);
      kcl_rows_list_kernel<<<grid_for(csr->n, 256), 256, 0, s>>>(csr->offsets, csr->n, e0, e1, few_lo, warp_max, row_max,
                                                                lcap, few_max, lists.p, q.p + kRowCounts);
      ATC_CK(cudaGetLastError());
      const auto launch = k == 3 ? launch_rows_block<0> : k == 4 ? launch_rows_block<1>
                          : k == 5 ? launch_rows_block<2> : launch_rows_block<3>;
      ATC_TRY(launch(csr, e0, e1, (int)k, dmax, lists.p, lcap, q.p + kRowCounts, few_max, q.p + 2, use_dense ? dense.p + 1 : nullptr,
                     pv->counter, s));
      launches += 2;
    }
    if (use_dense) {
      // rows for the largest C0 this graph can have
      const int cmax = std::min(cap, kDenseMax);
      const size_t smem = sizeof(unsigned long long) * ((size_t)cmax * ((cmax + 63) / 64) + kDensePad);
      const auto kern = k >= 6 ? kcl_dense_kernel<true> : kcl_dense_kernel<false>;
      ATC_CK(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                  (int)smem));
      int dbps = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&dbps, kern, kDenseThreads, smem);
      if (dbps < 1) dbps = 1;
      kern<<<(unsigned)(sm_count() * dbps), kDenseThreads, smem, s>>>(
          csr->offsets, csr->cols, pv->esrc, dense.p + 1, (int)k, cmax, dense.p, pv->counter);
      ATC_CK(cudaGetLastError());
      ++launches;
    }
    if (by_rows && cap > 32 && warp_max > 32) {
      ATC_TRY(launch_rows_warp<unsigned long long>(csr, e0, e1, (int)k, 32, few_lo, q.p + kRowCounts + kRowBuckets, few_max, q.p + 1,
                                                   pv->counter, s));
      ++launches;
    }
    if (by_rows) {
      ATC_TRY(launch_rows_warp<uint32_t>(csr, e0, e1, (int)k, 0, few_lo, q.p + kRowCounts + kRowBuckets, few_max, q.p,
                                         pv->counter, s));
      ++launches;
    }
    tm.stop(s);
    ATC_CK(cudaMemcpyAsync(h, pv->counter, sizeof(h), cudaMemcpyDeviceToHost, s));
    ATC_CK(cudaStreamSynchronize(s));
    *count = h[0];
  }
  if (stats) {
    stats->kernel_ms = e1 > e0 ? tm.ms() : 0.0f;
    stats->total_ms = stats->kernel_ms;
    stats->alg_bytes = h[1];
    stats->wedges = (uint64_t)csr->wedges;
    stats->alg_bytes_min = h[1];
    stats->kernel_used = 0;
    stats->launches = launches;
  }
  return ATC_OK;
}

extern "C" atc_status atc_kcl(const atc_csr* csr, uint32_t k, uint64_t* count, atc_stats* stats, atc_stream st) try {
  ATC_CHECK_ARG(csr != nullptr && count != nullptr, "NULL argument");
  ATC_CHECK_ARG(k >= 3 && k <= (uint32_t)kMaxK, "k must be in [3, 16]");
  ATC_CHECK_ARG(csr->priv != nullptr || csr->m == 0, "csr was not built by atc_pretc");
  Phase ph("kcl", as_stream(st));
  return kcl_window(csr, k, 0, csr->m, count, stats, as_stream(st));
} ATC_CATCH

extern "C" atc_status atc_kcl_part(const atc_csr* csr, uint32_t k, uint32_t part, uint32_t nparts, uint64_t* count,
                                   int64_t* edge_range, atc_stats* stats, atc_stream st) try {
  return atc_kcl_part_tuned(csr, k, nullptr, part, nparts, count, edge_range, stats, st);
} ATC_CATCH

extern "C" atc_status atc_kcl_part_tuned(const atc_csr* csr, uint32_t k, const atc_tuning* tuning, uint32_t part,
                                         uint32_t nparts, uint64_t* count, int64_t* edge_range, atc_stats* stats,
                                         atc_stream st) try {
  ATC_CHECK_ARG(csr != nullptr && count != nullptr, "NULL argument");
  ATC_CHECK_ARG(k >= 3 && k <= (uint32_t)kMaxK, "k must be in [3, 16]");
  ATC_CHECK_ARG(csr->priv != nullptr || csr->m == 0, "csr was not built by atc_pretc");
  ATC_CHECK_ARG(nparts >= 1 && part < nparts, "part must be in [0, nparts)");
  cudaStream_t s = as_stream(st);
  *count = 0;
  int64_t b[2];
  ATC_TRY(part_edge_range(csr, part, nparts, b, s));
  if (edge_range) {
    edge_range[0] = b[0];
    edge_range[1] = b[1];
  }
  ATC_CHECK_ARG(!tuning || tuning->kcl_dense == 0 || tuning->kcl_dense == -1, "kcl_dense must be 0 or -1");
  Phase ph("kcl", s);
  return kcl_window(csr, k, b[0], b[1], count, stats, s, !(tuning && tuning->kcl_dense == -1));
} ATC_CATCH
