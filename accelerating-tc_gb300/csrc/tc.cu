// Triangle counting on an oriented CSR: the four kernel families of the reference,
// re-designed for sm_103a.  All count sum_u sum_{v in N+(u)} |N+(u) ∩ N+(v)| exactly in
// uint64; every warp reduces its lanes with shuffles and adds once to a 64-bit counter.
//
//   Hu-style      Hu/tc.cu:22-201       wedge walk: N+(u) staged in shared memory once
//                                        per work item (chunk of N+(u)), every N+(v),
//                                        v in N+(u), streamed through it (W tests);
//                                        sorted copy + branch-free search for short
//                                        N+(u), hash table above.
//   Bisson-style  Bisson/tc.cu:18-104   every edge handed to the endpoint h with the
//                                        longer list (grouping passes); N+(h) as a hash
//                                        table, bitmap or sorted copy in shared memory,
//                                        the partner's shorter list streamed through it
//                                        (sum of min(d+u, d+v) tests).  Kernels in
//                                        bisson.cuh.  Whole counts of CSRs that preTC built:
//                                        a degree-ranked copy (ranked.cu) where it pays.
//   Fox-style     Fox/tc.cu:18-125,     per-edge work min*log2(max+2); edges binned on
//                 316-384                the device into 1,2,4,...,32 threads per edge;
//                                        each thread searches a slice of the shorter list
//                                        in the longer one.
//   TriCore-style tricount_gpu.cu:215-290  the longer list staged in shared memory, a table
//                                        over its id range brackets each element of the
//                                        shorter list, then a binary search inside the
//                                        bracket.
// The Fox- and TriCore-style searches are staged per group item too, and run on the ranked copy under the same
// conditions; the reference's forms of both, a warp or 1..32 threads per edge searching global memory, stay
// behind atc_tuning.edge_kernels.
#include <cmath>
#include <mutex>
#include <vector>

#include "parts.cuh"
#include "ranked.cuh"

namespace atc {


namespace {


// ============================== part split ===========================================
// Work of edge e for cutting the edges into parts: the shorter list it streams, plus one.
// work[m] = 0, so that an exclusive scan of m + 1 entries ends with the total.
__global__ void edge_work_kernel(CsrView g, int64_t* work) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e <= g.m; e += stride) {
    int64_t w = 0;
    if (e < g.m) {
      const int32_t u = g.esrc[e], v = g.cols[e];
      const int64_t du = g.off[u + 1] - g.off[u], dv = g.off[v + 1] - g.off[v];
      w = (du < dv ? du : dv) + 1;
    }
    work[e] = w;
  }
}

// bounds[t] (t = 0, 1) = the first edge whose work prefix reaches total * (part + t) / nparts.
__global__ void part_bounds_kernel(const int64_t* prefix, int64_t m, uint32_t part, uint32_t nparts, int64_t* bounds) {
  const int t = threadIdx.x;
  if (t > 1) return;
  const uint32_t k = part + t;
  if (k == 0 || k >= nparts) {
    bounds[t] = k == 0 ? 0 : m;
    return;
  }
  const int64_t target = (int64_t)((__int128)prefix[m] * k / nparts);
  int64_t lo = 0, hi = m;
  while (lo < hi) {
    const int64_t mid = (lo + hi) >> 1;
    if (prefix[mid] < target) lo = mid + 1; else hi = mid;
  }
  bounds[t] = lo;
}

// ============================== TriCore-style ======================================
constexpr int kTriWarps = 8;

__global__ void __launch_bounds__(kTriWarps * 32) tricore_kernel(CsrView g, unsigned long long* out) {
  __shared__ int32_t piv[kTriWarps][32];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  unsigned long long cnt = 0;
  const int64_t warps = (int64_t)gridDim.x * kTriWarps;
  for (int64_t e = g.e0 + (int64_t)blockIdx.x * kTriWarps + w; e < g.e1; e += warps) {
    int32_t u = g.esrc[e], v = g.cols[e];
    int64_t au = g.off[u], du = g.off[u + 1] - au;
    int64_t av = g.off[v], dv = g.off[v + 1] - av;
    const int32_t* A = g.cols + (du >= dv ? au : av);
    const int32_t* Bl = g.cols + (du >= dv ? av : au);
    int64_t da = du >= dv ? du : dv, db = du >= dv ? dv : du;
    if (db == 0) continue;
    piv[w][lane] = A[(int64_t)lane * da / 32];
    __syncwarp();
    // a lane's elements ascend: `prev` = where its previous element's search ended, a
    // lower bound for the next one inside any bracket
    int64_t prev = 0;
    for (int64_t j = lane; j < db; j += 32) {
      int32_t x = __ldg(Bl + j);
      // k = number of pivots <= x
      int lo = 0, hi = 32;
      while (lo < hi) {
        int mid = (lo + hi) >> 1;
        if (piv[w][mid] <= x) lo = mid + 1; else hi = mid;
      }
      if (lo == 0) continue;                 // x < A[0]
      if (piv[w][lo - 1] == x) { ++cnt; continue; }
      int64_t b = (int64_t)(lo - 1) * da / 32 + 1;  // strictly inside the bracket
      int64_t e2 = lo == 32 ? da : (int64_t)lo * da / 32;
      if (prev > b) b = prev;
      while (b < e2) {  // lower bound of x in A[b, e2)
        const int64_t mid = (b + e2) >> 1;
        if (__ldg(A + mid) < x) b = mid + 1; else e2 = mid;
      }
      cnt += b < da && __ldg(A + b) == x;
      prev = b;
    }
    __syncwarp();
  }
  warp_add_count(cnt, out);
}

// ============================== Fox-style ==========================================
// Work of an edge (Fox/tc.cu:22-31): min(d+u, d+v) * log2(max + 2), as an int.
__device__ __forceinline__ int fox_work(int64_t du, int64_t dv) {
  int64_t big = du > dv ? du : dv, small = du > dv ? dv : du;
  double wv = (double)small * log2((double)big + 2.0);
  return wv > 2147483647.0 ? 2147483647 : (int)wv;
}

__global__ void fox_maxwork_kernel(CsrView g, int* maxw) {
  int best = 0;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = g.e0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < g.e1; e += stride) {
    int32_t u = g.esrc[e], v = g.cols[e];
    best = max(best, fox_work(g.off[u + 1] - g.off[u], g.off[v + 1] - g.off[v]));
  }
  for (int o = 16; o > 0; o >>= 1) best = max(best, __shfl_xor_sync(0xffffffffu, best, o));
  if ((threadIdx.x & 31) == 0) atomicMax(maxw, best);
}

struct FoxBins {
  int bound[7];  // work thresholds: bin b holds work in [bound[b], bound[b+1])
};

__device__ __forceinline__ int fox_bin(const FoxBins& fb, int wk) {
  int b = 0;
#pragma unroll
  for (int i = 1; i < 6; ++i) b += wk >= fb.bound[i];
  return b;
}

__global__ void fox_hist_kernel(CsrView g, FoxBins fb, unsigned long long* hist) {
  __shared__ unsigned int h[6];
  if (threadIdx.x < 6) h[threadIdx.x] = 0;
  __syncthreads();
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t e = g.e0 + blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < g.e1; e += stride) {
    int32_t u = g.esrc[e], v = g.cols[e];
    atomicAdd(&h[fox_bin(fb, fox_work(g.off[u + 1] - g.off[u], g.off[v + 1] - g.off[v]))], 1u);
  }
  __syncthreads();
  if (threadIdx.x < 6 && h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], (unsigned long long)h[threadIdx.x]);
}

// Edges into their bins; the lanes of a warp that share a bin reserve their slots with one
// atomic (six cursors taken by every edge would serialise on a handful of addresses).  The
// loop is padded to whole warps for __match_any_sync.
__global__ void fox_scatter_kernel(CsrView g, FoxBins fb, unsigned long long* cursor, int64_t* list) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t w_pad = (g.e1 - g.e0 + 31) & ~31ll;
  const int lane = threadIdx.x & 31;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < w_pad; i += stride) {
    const int64_t e = g.e0 + i;
    int b = -1;
    if (e < g.e1) {
      const int32_t u = g.esrc[e], v = g.cols[e];
      b = fox_bin(fb, fox_work(g.off[u + 1] - g.off[u], g.off[v + 1] - g.off[v]));
    }
    const unsigned same = __match_any_sync(0xffffffffu, b);
    const int lead = __ffs(same) - 1;
    unsigned long long base = 0;
    if (b >= 0 && lane == lead) base = atomicAdd(&cursor[b], (unsigned long long)__popc(same));
    base = __shfl_sync(0xffffffffu, base, lead);
    if (b >= 0) list[base + __popc(same & ((1u << lane) - 1))] = e;
  }
}

// T threads per edge (Fox/tc.cu:64-125): each thread takes every T-th element of the
// shorter list and searches it in the longer list (exponential search from the previous
// element's position, then binary search).
template <int T>
__global__ void __launch_bounds__(256) fox_kernel(CsrView g, const int64_t* list, int64_t cnt_edges,
                                                  unsigned long long* out) {
  unsigned long long cnt = 0;
  const int64_t gid = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const int sub = (int)(gid % T);
  const int64_t groups = (int64_t)gridDim.x * blockDim.x / T;
  for (int64_t i = gid / T; i < cnt_edges; i += groups) {
    int64_t e = list[i];
    int32_t u = g.esrc[e], v = g.cols[e];
    int64_t au = g.off[u], du = g.off[u + 1] - au;
    int64_t av = g.off[v], dv = g.off[v + 1] - av;
    const int32_t* L = g.cols + (du >= dv ? au : av);   // longer
    const int32_t* S = g.cols + (du >= dv ? av : au);   // shorter
    int64_t dl = du >= dv ? du : dv, ds = du >= dv ? dv : du;
    // a thread's elements ascend, so each search resumes where the previous one ended:
    // gallop forward from there, then binary-search the last step
    int64_t lo = 0;
    for (int64_t j = sub; j < ds; j += T) {
      const int32_t x = __ldg(S + j);
      int64_t a = lo, b = lo, step = 1;  // every L[i], i < a, is < x
      while (b < dl && __ldg(L + b) < x) {
        a = b + 1;
        b = a + step;
        step <<= 1;
      }
      if (b > dl) b = dl;
      while (a < b) {  // L[b] >= x or b == dl
        const int64_t mid = (a + b) >> 1;
        if (__ldg(L + mid) < x) a = mid + 1; else b = mid;
      }
      cnt += a < dl && __ldg(L + a) == x;
      lo = a;
    }
  }
  warp_add_count(cnt, out);
}

// Fox's interleave (Fox/tc.cu:127-183): a bin's edges are sorted by the length of
// their longer list, cut into groups of 32 and dealt round-robin over `nblk` blocks, so
// every block gets a mix of long and short edges.  Group g = sec*nblk + first moves to
// rank first*q + min(first, r) + sec (q, r = ngroups / nblk, ngroups % nblk): a
// bijection on the groups; the tail of fewer than 32 edges stays in place.
__global__ void fox_lenkey_kernel(CsrView g, const int64_t* list, int64_t nb, uint64_t* keys) {
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nb; i += stride) {
    int64_t e = list[i];
    int32_t u = g.esrc[e], v = g.cols[e];
    int64_t du = g.off[u + 1] - g.off[u], dv = g.off[v + 1] - g.off[v];
    uint64_t mx = (uint64_t)(du > dv ? du : dv);
    if (mx > 0x7fffffffull) mx = 0x7fffffffull;
    keys[i] = (mx << 32) | (uint64_t)i;
  }
}

__global__ void fox_deal_kernel(const uint64_t* keys, const int64_t* list, int64_t nb, int64_t nblk, int64_t* out) {
  int64_t ngroups = nb / 32;
  int64_t q = nblk > 0 ? ngroups / nblk : 0, r = nblk > 0 ? ngroups % nblk : 0;
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < nb; i += stride) {
    int64_t src = list[keys[i] & 0xffffffffull];
    int64_t grp = i / 32, dst = i;
    if (grp < ngroups && nblk > 1) {
      int64_t first = grp % nblk, sec = grp / nblk;
      dst = (first * q + (first < r ? first : r) + sec) * 32 + (i % 32);
    }
    out[dst] = src;
  }
}

// ============================== small counts =======================================
// Graphs of a few thousand edges are counted before a launch's items could be made: G lanes take
// an edge, each every G-th element of the shorter list, and binary-search it in the longer
// one, where both lists sit in L1 or L2 (Hu/tc.cu:69-201 searches a staged run the same way).  One
// launch, no item lists, no wait before the result and no memset: every block stores its sum to a
// place of its own in memory of the call, and the host adds them up, so that nothing outlives the call
// and calls that overlap share nothing.
// Measured, the whole call, items -> this kernel (us): R-MAT of 4.9K, 23K, 102K, 441K edges 55 -> 30,
// 78 -> 31, 118 -> 50, 232 -> 175; Chung-Lu of 35K, 380K 93 -> 31, 115 -> 69; RGG of 45K, 473K
// 80 -> 30, 106 -> 70, 1.6M 160 -> 180; the sums stored to the caller's memory instead of copied
// take another 5 to 10 us off (R-MAT scale 10 26; 441K edges 125).  Bound by launches below 50K edges, then by the searches'
// dependent loads.
// An edge whose shorter list has more than kSmallEach elements a lane is left to the whole block, four
// searches a thread under way at once: one group's chain of dependent searches would hold the call up
// (two hubs with the same 2000, 10 000, 100 000 neighbours: 0.20, 1.02, 11.3 ms by one group, 0.030, 0.035, 0.115 so; work
// items 0.08, 0.09, 0.37).  Edges of one row lie in several blocks, so that a hub's long ones do not meet in one.
constexpr int64_t kSmallEdges = 1 << 19;
constexpr int kSmallEach = 16;
constexpr int kSmallLong = 128;  // edges a block can keep for all of it
template <int G>
__global__ void __launch_bounds__(1024, 2) small_edges_kernel(CsrView g, volatile unsigned long long* sums) {
  __shared__ int32_t held[kSmallLong];
  __shared__ int nheld;
  if (threadIdx.x == 0) nheld = 0;
  __syncthreads();
  const int sub = threadIdx.x % G;
  const int threads = blockDim.x;
  const int64_t groups = (int64_t)gridDim.x * threads / G;
  const int64_t warp = (threadIdx.x >> 5) * (int64_t)gridDim.x + blockIdx.x;
  const unsigned group = 0xffffffffu >> (32 - G) << ((threadIdx.x & 31) - sub);
  unsigned cnt = 0;
  struct Lists {
    const int32_t *L, *S;
    int dl, ds;
  };
  auto lists = [&](int64_t e) {
    const int32_t u = __ldg(g.esrc + e), v = __ldg(g.cols + e);
    const int64_t au = __ldg(g.off + u), av = __ldg(g.off + v);
    const int du = (int)(__ldg(g.off + u + 1) - au), dv = (int)(__ldg(g.off + v + 1) - av);
    return Lists{g.cols + (du >= dv ? au : av), g.cols + (du >= dv ? av : au), max(du, dv), min(du, dv)};
  };
  for (int64_t e = g.e0 + warp * (32 / G) + (threadIdx.x & 31) / G; e < g.e1; e += groups) {
    const Lists x = lists(e);
    if (x.ds > kSmallEach * G) {
      int at = kSmallLong;
      if (sub == 0) at = atomicAdd(&nheld, 1);
      at = __shfl_sync(group, at, (threadIdx.x & 31) - sub);
      if (at < kSmallLong) {
        if (sub == 0) held[at] = (int32_t)(e - g.e0);
        continue;
      }
    }
    for (int j = sub; j < x.ds; j += G) {
      const int32_t y = __ldg(x.S + j);
      int lo = 0, n = x.dl;
      while (n > 1) {  // branch-free lower bound
        const int half = n >> 1;
        lo = __ldg(x.L + lo + half - 1) < y ? lo + half : lo;
        n -= half;
      }
      cnt += __ldg(x.L + lo) == y;
    }
  }
  __syncthreads();
  for (int h = 0; h < min(nheld, kSmallLong); ++h) {
    const Lists x = lists(g.e0 + held[h]);
    for (int j = threadIdx.x; j < x.ds; j += 4 * threads) {
      int32_t y[4];
      int lo[4], n = x.dl;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        y[q] = j + threads * q < x.ds ? __ldg(x.S + j + threads * q) : -1;  // no id
        lo[q] = 0;
      }
      while (n > 1) {
        const int half = n >> 1;
#pragma unroll
        for (int q = 0; q < 4; ++q) lo[q] = __ldg(x.L + lo[q] + half - 1) < y[q] ? lo[q] + half : lo[q];
        n -= half;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) cnt += __ldg(x.L + lo[q]) == y[q];
    }
  }
  __shared__ unsigned part[32];
  const unsigned w = __reduce_add_sync(0xffffffffu, cnt);
  if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = w;
  __syncthreads();
  if (threadIdx.x < 32) {
    unsigned long long t = (int)threadIdx.x < threads / 32 ? part[threadIdx.x] : 0u;
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (threadIdx.x == 0) sums[blockIdx.x] = t;
  }
}

// ============================== sorted-copy searches ===============================
// TriCore-style and Fox-style counts on the Bisson-style grouping: every edge goes to its
// endpoint h with the longer list and the partner's shorter list is streamed (sum of
// min(d+u, d+v) searches).  N+(h), the longer list of every edge of an item, is staged once
// per item as a sorted copy in shared memory, and every streamed element is searched in
// it.  The reference kernels search the longer list in global memory, one dependent load
// per step, per edge; here only lists too long for shared memory are searched there.
//   KIND 0, TriCore-style (tricount_gpu.cu:215-290): the reference's pivot cache (32 samples of
//     the longer list per warp) becomes a table over the list's id range: the range is cut into
//     up to kPivots equal parts, twice as many as the list has elements, and the table gives the
//     elements of each part.  One read brackets an element to a part, whose few elements are
//     then binary-searched.  (Samples at equal positions took five steps to find the bracket
//     and log2(d/32) + 1 more inside it, each a shared load with bank conflicts.)
//   KIND 1, Fox-style (Fox/tc.cu:64-125): a lane's successive elements of a list ascend, so
//     each search gallops forward from where the lane's previous one ended (restarting
//     when the element is smaller than the previous one), then binary-searches the last
//     step.
constexpr int kWarpPivots = 256;    // parts of a warp item's table (lists of up to kWarpMax)
constexpr int kBlockPivots = 2048;  // and of a block item's

template <int KIND>
struct SortedProber {
  const int32_t* T;     // sorted N+(h) (shared memory, or global for lists beyond it)
  const uint32_t* part; // TriCore: first element | end << 16 of every part (null: the whole list)
  int d;
  int32_t hi;    // T[d - 1]
  int32_t base;  // TriCore: T[0]
  uint32_t range;  // TriCore: T[d - 1] - T[0]
  int shift;     // TriCore: log2 of a part's ids
  int prev;      // Fox: lower bound of the lane's previous element
  int32_t last;  // Fox: the lane's previous element
  int gap;       // Fox: how far the lane's previous forward search moved
  __device__ __forceinline__ unsigned probe(int32_t x, bool valid) {
    if (!valid) return 0u;
    if constexpr (KIND == 0) {
      const uint32_t r = (uint32_t)(x - base);
      if (r > range) return 0u;  // outside the longer list: no search
      int lo = 0, n = d;
      if (part) {
        const uint32_t pe = part[r >> shift];
        lo = (int)(pe & 0xffffu);
        n = (int)(pe >> 16) - lo;
      }
      while (n > 1) {  // branch-free lower bound inside the part
        const int half = n >> 1;
        lo = T[lo + half - 1] < x ? lo + half : lo;
        n -= half;
      }
      return n == 1 && T[lo] == x;
    } else {
      if (x > hi) return 0u;  // above the longer list: no search
      if (x < last) {
        // a new list (or an earlier element): its lower bound lies in [0, prev]
        int a = 0, b = prev;
        while (a < b) {
          const int mid = (a + b) >> 1;
          if (T[mid] < x) a = mid + 1; else b = mid;
        }
        prev = a;
        last = x;
        return a < d && T[a] == x;
      }
      last = x;
      // every T[i], i < a, is < x; the first step is half the lane's previous move, so a
      // lane walking one list at a steady stride settles in about log2(stride) steps
      int a = prev, step = gap > 1 ? gap >> 1 : 1;
      int b = a + step - 1;
      while (b < d && T[b] < x) {
        a = b + 1;
        step <<= 1;
        b = a + step - 1;
      }
      if (b > d) b = d;
      while (a < b) {  // T[b] >= x, or b == d
        const int mid = (a + b) >> 1;
        if (T[mid] < x) a = mid + 1; else b = mid;
      }
      gap = a - prev;
      prev = a;
      return a < d && T[a] == x;
    }
  }
  __device__ __forceinline__ unsigned finish() { return 0u; }
};

// ---- 1-D bulk copies into shared memory (the TMA unit's untiled mode) -------------
// One thread issues cp.async.bulk of a whole list; its completion is counted in bytes on an
// mbarrier that every thread of the copy's group waits on.  Source and destination start on
// 16-byte boundaries and the size is a multiple of 16 bytes: a list is copied from the
// 16-byte boundary at or below its first element to the one at or above its end (the CSR's
// cols carry 16 ints of padding, so the rounded end stays inside the allocation), and read
// from the offset of its first element.  Every wait is bounded in time: a wait that runs out
// records an error for the host (ATC_ERR_TIMEOUT) and the kernel stops counting.
constexpr uint64_t kBulkWaitNs = 1000000000ull;  // one second without the copy landing

__device__ __forceinline__ uint64_t global_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void mbar_init(uint64_t* bar) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(smem_u32(bar)) : "memory");
  asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
}

// Issued by one thread: the byte count the barrier's current phase waits for, then the copy.
// The proxy fence orders the group's earlier ordinary reads of `dst` before the async write.
__device__ __forceinline__ void bulk_list_to_smem(int32_t* dst, const int32_t* src, uint32_t bytes, uint64_t* bar) {
  asm volatile("fence.proxy.async.shared::cta;\n" ::: "memory");
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(bar)), "r"(bytes)
               : "memory");
  asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];\n" ::"r"(
                   smem_u32(dst)),
               "l"(src), "r"(bytes), "r"(smem_u32(bar))
               : "memory");
}

// Waits for phase `parity` of the barrier to complete; false if it did not within limit_ns.
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, uint64_t limit_ns = kBulkWaitNs) {
  const uint64_t t0 = global_ns();
  for (;;) {
    uint32_t done;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(done)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    if (done) return true;
    if (global_ns() - t0 > limit_ns) return false;
  }
}

// The bounded wait's failure path, for tests: a barrier whose phase announces 16 bytes that
// no copy delivers (one arrival, its transaction count never reached), waited on with
// limit_ns.  err = 1 when the wait gave up, as it must; nothing is in flight at exit.
__global__ void wait_timeout_check_kernel(uint64_t limit_ns, int* err) {
  __shared__ __align__(8) uint64_t bar;
  if (threadIdx.x == 0) {
    mbar_init(&bar);
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(smem_u32(&bar)), "r"(16u)
                 : "memory");
  }
  __syncthreads();
  const bool ok = mbar_wait(&bar, 0, limit_ns);
  if (!ok && threadIdx.x == 0) *err = 1;
}

// The 16-byte-aligned window [a0, a1) of cols holding the list [hb, hb + dh).
__device__ __forceinline__ void bulk_window(int64_t hb, int64_t dh, int64_t* a0, uint32_t* bytes) {
  *a0 = hb & ~3ll;
  *bytes = (uint32_t)(((hb + dh + 3) & ~3ll) - *a0) * 4u;
}

// bulk: stage N+(h) with bulk copies (device-resident cols); otherwise with loads (cols in
// mapped host memory).  err: set to 1 when a bulk wait runs out.
template <int KIND, class Items, class Partners>
__global__ void __launch_bounds__(kBgWarps * 32) sorted_warp_kernel(CsrView g, Partners partners, Items items,
                                                                    int nitems, int* next, bool bulk, int* err,
                                                                    unsigned long long* out) {
  __shared__ __align__(16) int32_t T[kBgWarps][kWarpMax + 8];
  __shared__ uint32_t part[kBgWarps][KIND == 0 ? kWarpPivots : 1];
  __shared__ uint16_t start[kBgWarps][KIND == 0 ? kWarpPivots + 1 : 1];
  __shared__ __align__(8) uint64_t bar[kBgWarps];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  if (lane == 0) mbar_init(&bar[w]);
  __syncwarp();
  uint32_t phase = 0;
  unsigned long long total = 0;
  for (;;) {
    int it = 0;
    if (lane == 0) it = atomicAdd(next, 1);
    it = __shfl_sync(0xffffffffu, it, 0);
    if (it >= nitems) break;
    const GroupItem gi = items.get(g, it);
    const int64_t hb = g.off[gi.h];
    const int dh = (int)(g.off[gi.h + 1] - hb);  // 1 .. kWarpMax
    const int32_t* L = T[w];
    if (bulk) {
      int64_t a0;
      uint32_t bytes;
      bulk_window(hb, dh, &a0, &bytes);
      if (lane == 0) bulk_list_to_smem(T[w], g.cols + a0, bytes, &bar[w]);
      const bool ok = mbar_wait(&bar[w], phase);
      phase ^= 1u;
      if (!__all_sync(0xffffffffu, ok)) {
        if (lane == 0) atomicExch(err, 1);
        mbar_wait(&bar[w], phase ^ 1u);  // once more for the copy in flight, then stop
        break;
      }
      L = T[w] + (hb - a0);
    } else {
      for (int j = lane; j < dh; j += 32) T[w][j] = __ldg(g.cols + hb + j);
      __syncwarp();
    }
    int shift = 0;
    if (KIND == 0) shift = build_parts(L, dh, kWarpPivots, start[w], part[w], lane, 32, [] { __syncwarp(); });
    int64_t cur = gi.b;
    auto nb = [&]() { int64_t r = cur; cur += 32; return r; };
    SortedProber<KIND> pr{L, part[w], dh, L[dh - 1], L[0], (uint32_t)(L[dh - 1] - L[0]), shift, 0, INT32_MIN, 16};
    total += stream_partners(g, partners, gi.e, lane, nb, pr);
    __syncwarp();  // the next item overwrites the copy
  }
  warp_add_count(total, out);
}

template <int KIND, class Items, class Partners>
__global__ void __launch_bounds__(kBgWarps * 32) sorted_block_kernel(CsrView g, Partners partners, Items items,
                                                                     int nitems, int* next, uint32_t tab_words,
                                                                     bool bulk, int* err, unsigned long long* out) {
  extern __shared__ __align__(16) int32_t T[];  // tab_words + 8
  __shared__ uint32_t part[KIND == 0 ? kBlockPivots : 1];
  __shared__ uint16_t start[KIND == 0 ? kBlockPivots + 1 : 1];
  __shared__ int cur_item;
  __shared__ unsigned long long bnext;
  __shared__ __align__(8) uint64_t bar;
  const int lane = threadIdx.x & 31;
  if (threadIdx.x == 0) mbar_init(&bar);
  __syncthreads();
  uint32_t phase = 0;
  unsigned long long total = 0;
  for (;;) {
    if (threadIdx.x == 0) {
      cur_item = atomicAdd(next, 1);
      bnext = 0;
    }
    __syncthreads();
    const int it = cur_item;
    if (it >= nitems) break;
    const GroupItem gi = items.get(g, it);
    const int64_t hb = g.off[gi.h];
    const int64_t dh = g.off[gi.h + 1] - hb;
    const bool staged = dh <= (int64_t)tab_words;
    const int32_t* L = g.cols + hb;
    if (staged && bulk) {
      int64_t a0;
      uint32_t bytes;
      bulk_window(hb, dh, &a0, &bytes);
      if (threadIdx.x == 0) bulk_list_to_smem(T, g.cols + a0, bytes, &bar);
      const bool ok = __syncthreads_and(mbar_wait(&bar, phase));
      phase ^= 1u;
      if (!ok) {
        if (threadIdx.x == 0) atomicExch(err, 1);
        mbar_wait(&bar, phase ^ 1u);  // once more for the copy in flight, then stop
        break;
      }
      L = T + (hb - a0);
    } else if (staged) {
      for (int64_t j = threadIdx.x; j < dh; j += blockDim.x) T[j] = __ldg(g.cols + hb + j);
      L = T;
    }
    if (staged && !bulk) __syncthreads();
    int shift = 0;
    if (KIND == 0 && staged)
      shift = build_parts(L, (int)dh, kBlockPivots, start, part, threadIdx.x, kBgWarps * 32, [] { __syncthreads(); });
    auto nb = [&]() {
      unsigned long long r = 0;
      if (lane == 0) r = atomicAdd(&bnext, 32ull);
      return gi.b + (int64_t)__shfl_sync(0xffffffffu, r, 0);
    };
    const int32_t t0 = __ldg(g.cols + hb), t1 = __ldg(g.cols + hb + dh - 1);
    SortedProber<KIND> pr{L, KIND == 0 && staged ? part : nullptr, (int)dh, t1, t0, (uint32_t)(t1 - t0), shift, 0,
                          INT32_MIN, 16};
    total += stream_partners(g, partners, gi.e, lane, nb, pr);
    __syncthreads();  // the next item overwrites the copy
  }
  warp_add_count(total, out);
}

}  // namespace

// ---- family drivers ----------------------------------------------------------------
static atc_status run_tricore(const CsrView& g, const atc_tuning* t, unsigned long long* ctr, cudaStream_t s,
                              int* launches) {
  Phase ph("tc.count", s);
  int grid = t && t->tricore_blocks > 0 ? t->tricore_blocks
                                        : sm_count() * blocks_per_sm((const void*)tricore_kernel, kTriWarps * 32, 0);
  tricore_kernel<<<grid, kTriWarps * 32, 0, s>>>(g, ctr);
  ATC_CK(cudaGetLastError());
  *launches += 1;
  return ATC_OK;
}

static atc_status run_fox(const CsrView& g, const atc_tuning* t, unsigned long long* ctr, cudaStream_t s,
                          int* launches) {
  DevBuf<int> mx;
  DevBuf<unsigned long long> hist, cursor;
  std::optional<Phase> ph;
  ph.emplace("tc.bins", s);
  ATC_TRY(mx.alloc(1, s));
  ATC_TRY(hist.alloc(6, s));
  ATC_TRY(cursor.alloc(6, s));
  ATC_CK(cudaMemsetAsync(mx.p, 0, sizeof(int), s));
  ATC_CK(cudaMemsetAsync(hist.p, 0, sizeof(unsigned long long) * 6, s));
  fox_maxwork_kernel<<<grid_for(g.e1 - g.e0, 256), 256, 0, s>>>(g, mx.p);
  ATC_CK(cudaGetLastError());
  int maxw = 0;
  ATC_CK(cudaMemcpyAsync(&maxw, mx.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  // Bin boundaries of Fox/tc.cu:318-331: partition points 8^((log8(max)-1)(i-1)/32 + 1)
  // for i = 2, 4, ..., 32; bin i threads holds work in [pp(i), pp(2i)).
  int wpt = t && t->fox_work_per_thread > 1 ? t->fox_work_per_thread : 8;
  FoxBins fb;
  fb.bound[0] = INT32_MIN;
  double maxPow = maxw > 0 ? std::log((double)maxw) / std::log((double)wpt) : 0.0;
  int k = 1;
  for (int i = 2; i <= 32; i *= 2, ++k) {
    double index = (maxPow - 1) * (i - 1) / 32.0 + 1;
    long double pp = powl((long double)wpt, (long double)index);
    fb.bound[k] = pp > 2147483647.0L ? 2147483647 : (int)pp;
  }
  fb.bound[6] = INT32_MAX;
  fox_hist_kernel<<<grid_for(g.e1 - g.e0, 256), 256, 0, s>>>(g, fb, hist.p);
  ATC_CK(cudaGetLastError());
  unsigned long long h[6];
  ATC_CK(cudaMemcpyAsync(h, hist.p, sizeof(h), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  unsigned long long start[7];
  start[0] = 0;
  for (int b = 0; b < 6; ++b) start[b + 1] = start[b] + h[b];
  ATC_CK(cudaMemcpyAsync(cursor.p, start, sizeof(unsigned long long) * 6, cudaMemcpyHostToDevice, s));
  DevBuf<int64_t> list, list2;
  ATC_TRY(list.alloc(g.e1 - g.e0, s));
  fox_scatter_kernel<<<grid_for(g.e1 - g.e0, 256), 256, 0, s>>>(g, fb, cursor.p, list.p);
  ATC_CK(cudaGetLastError());
  *launches += 3;
  const int64_t* L = list.p;
  if (t && t->fox_rearrange) {
    ATC_TRY(list2.alloc(g.e1 - g.e0, s));
    for (int b = 0; b < 6; ++b) {
      int64_t nb = (int64_t)h[b];
      if (nb == 0) continue;
      DevBuf<uint64_t> k1, k2;
      ATC_TRY(k1.alloc(nb, s));
      ATC_TRY(k2.alloc(nb, s));
      fox_lenkey_kernel<<<grid_for(nb, 256), 256, 0, s>>>(g, list.p + start[b], nb, k1.p);
      ATC_CK(cudaGetLastError());
      uint64_t* ka = k1.p;
      uint64_t* kb = k2.p;
      ATC_TRY(sort_keys_u64(ka, kb, nb, 0, 63, s));
      int64_t edges_per_block = 256 >> b;
      int64_t nblk = nb / edges_per_block;
      fox_deal_kernel<<<grid_for(nb, 256), 256, 0, s>>>(ka, list.p + start[b], nb, nblk, list2.p + start[b]);
      ATC_CK(cudaGetLastError());
      *launches += 2;
    }
    L = list2.p;
  }
  ph.reset();
  ph.emplace("tc.count", s);
  int sms = sm_count();
  for (int b = 0; b < 6; ++b) {
    int64_t nb = (int64_t)h[b];
    if (nb == 0) continue;
    const int64_t* Lb = L + start[b];
    int64_t threads = nb << b;
    unsigned grid = (unsigned)std::min<int64_t>((threads + 255) / 256, (int64_t)sms * 8);
    switch (b) {
      case 0: fox_kernel<1><<<grid, 256, 0, s>>>(g, Lb, nb, ctr); break;
      case 1: fox_kernel<2><<<grid, 256, 0, s>>>(g, Lb, nb, ctr); break;
      case 2: fox_kernel<4><<<grid, 256, 0, s>>>(g, Lb, nb, ctr); break;
      case 3: fox_kernel<8><<<grid, 256, 0, s>>>(g, Lb, nb, ctr); break;
      case 4: fox_kernel<16><<<grid, 256, 0, s>>>(g, Lb, nb, ctr); break;
      default: fox_kernel<32><<<grid, 256, 0, s>>>(g, Lb, nb, ctr); break;
    }
    ATC_CK(cudaGetLastError());
    *launches += 1;
  }
  ATC_CK(cudaStreamSynchronize(s));  // `start` / `h` live on this frame
  return ATC_OK;
}

// Launches the block and warp kernels over work items; S = hash slots per bucket.
// hc = {warp items, block items, -, longest hashed block list}.
template <int S>
static atc_status launch_bisson(const CsrView& g, const int32_t* plist, const GroupItem* witems,
                                const GroupItem* bitems, const int* hc, int* counters, unsigned long long* ctr,
                                cudaStream_t s, int* launches) {
  if (hc[1]) {
    // block table: enough slots for the longest hashed list at load factor 1/4, or the
    // full bitmap when some list needs it
    uint32_t words = 64;
    while (words < 4u * (uint32_t)hc[3]) words <<= 1;
    if (words > (uint32_t)kTabWords) words = kTabWords;
    size_t smem = sizeof(int32_t) * words;
    ATC_CK(cudaFuncSetAttribute((const void*)bisson_block_kernel<FullItems, S>,
                                cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int bps = blocks_per_sm((const void*)bisson_block_kernel<FullItems, S>, kBgWarps * 32, smem);
    int grid = std::min(hc[1], sm_count() * bps);
    bisson_block_kernel<FullItems, S><<<grid, kBgWarps * 32, smem, s>>>(
        g, ListPartners{plist}, FullItems{bitems}, hc[1], nullptr, counters + 5, words, GraphTags{nullptr, 0, nullptr}, ctr);
    ATC_CK(cudaGetLastError());
    *launches += 1;
  }
  if (hc[0]) {
    int bps = blocks_per_sm((const void*)bisson_warp_kernel<FullItems, S>, kBgWarps * 32, 0);
    int grid = (int)std::min<int64_t>((hc[0] + kBgWarps - 1) / kBgWarps, (int64_t)sm_count() * bps);
    bisson_warp_kernel<FullItems, S><<<grid, kBgWarps * 32, 0, s>>>(g, ListPartners{plist}, FullItems{witems}, hc[0], nullptr,
                                                                   counters + 4, GraphTags{nullptr, 0, nullptr}, ctr);
    ATC_CK(cudaGetLastError());
    *launches += 1;
  }
  return ATC_OK;
}

static atc_status launch_slots(int slots, const CsrView& g, const int32_t* plist, const GroupItem* witems,
                               const GroupItem* bitems, const int* hc, int* counters, unsigned long long* ctr,
                               cudaStream_t s, int* launches) {
  if (slots == 1) return launch_bisson<1>(g, plist, witems, bitems, hc, counters, ctr, s, launches);
  if (slots == 2) return launch_bisson<2>(g, plist, witems, bitems, hc, counters, ctr, s, launches);
  return launch_bisson<4>(g, plist, witems, bitems, hc, counters, ctr, s, launches);
}

// Item shape: the defaults, overridden field by field by the tuning (chunks >= 32 partners).
static atc_status item_shape(const atc_tuning* t, ItemShape* sh, int* slots) {
  *sh = default_shape(32);
  *slots = kDefaultSlots;
  if (!t) return ATC_OK;
  ATC_CHECK_ARG(t->bisson_slots == 0 || t->bisson_slots == 1 || t->bisson_slots == 2 || t->bisson_slots == 4,
                "bisson_slots must be 0, 1, 2 or 4");
  if (t->bisson_cutover > 0) sh->cutover = std::min(t->bisson_cutover, kWarpMax);
  if (t->bisson_warp_max > 0) sh->warp_max = std::min(t->bisson_warp_max, kWarpHashMax);
  if (t->bisson_warp_chunk > 0) sh->warp_chunk = std::max(t->bisson_warp_chunk, 32);
  if (t->bisson_block_chunk > 0) sh->block_chunk = std::max(t->bisson_block_chunk, 32);
  if (t->bisson_slots > 0) *slots = t->bisson_slots;
  return ATC_OK;
}

// Hu-style (Hu/tc.cu:69-201): every wedge u -> v -> w is tested against N+(u), which a
// work item stages in shared memory once and which every N+(v), v in N+(u), streams
// through: W tests in all.  The reference binary-searches a sorted run of N+(u); here the
// staged set is the sorted copy searched branch-free for d+(u) <= 32 and a hash table
// above (the Bisson-style kernels' sets).  The reference's 30 000 vertex ranges of equal
// wedge work (Hu/tc.cu:22-67,263-301) become chunks of N+(u) drained from a device queue,
// which balances dynamically.  No grouping pass: the items index the CSR itself.
static atc_status run_hu(const CsrView& g, const atc_tuning* t, unsigned long long* ctr, cudaStream_t s,
                         int* launches) {
  ItemShape sh;
  int slots;
  ATC_TRY(item_shape(t, &sh, &slots));
  // the sorted copy only for N+(u) of at most 8 (every N+(v) is searched in it; the hash
  // takes one probe): 4 % faster than 32 at R-MAT scale 24
  if (!t || t->bisson_cutover <= 0) sh.cutover = 8;
  std::optional<Phase> ph;
  ph.emplace("tc.items", s);
  DevBuf<int> counters;  // warp items, block items, (unused), longest block list, warp next, block next
  ATC_TRY(counters.alloc(8, s));
  ATC_CK(cudaMemsetAsync(counters.p, 0, sizeof(int) * 8, s));
  const int64_t mi = max_items(g.n, g.e1 - g.e0, std::min(sh.warp_chunk, sh.block_chunk));
  DevBuf<GroupItem> witems, bitems;
  ATC_TRY(witems.alloc(mi, s));
  ATC_TRY(bitems.alloc(mi, s));
  // the partner range of u is its own CSR row
  group_items_kernel<<<grid_for(g.n, 256), 256, 0, s>>>(g, g.off, witems.p, bitems.p, counters.p, sh, g.e0, g.e1);
  ATC_CK(cudaGetLastError());
  int hc[4];
  ATC_CK(cudaMemcpyAsync(hc, counters.p, sizeof(hc), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  *launches += 1;
  ph.reset();
  ph.emplace("tc.count", s);
  return launch_slots(slots, g, g.cols, witems.p, bitems.p, hc, counters.p, ctr, s, launches);
}

// Whether the window's Hu-style count goes to the small kernel: 5.5 ps per element of W_min and 60
// ps per edge (dependent loads) against 2 ps per wedge, 45 ps per edge and 47 us more of launches
// and waits.  Dense graphs of few edges (K_1000: 0.9 ms here, 0.4 by items) are not small.
static bool small_pays(const atc_csr* csr, int64_t edges) {
  if (edges > kSmallEdges) return false;
  const double part = (double)edges / (double)csr->m;
  return part * (5.5 * (double)csr->wedges_min + 15.0 * (double)csr->m) < part * 2.0 * (double)csr->wedges + 4.7e7;
}

// Counts the window into *count and waits for it; tm is stopped behind the kernel.  The blocks' sums
// go to host memory where the kernel can store there, else to device memory of the call.
static atc_status run_small(const CsrView& g, int64_t mean_min, uint64_t* count, EventTimer* tm, cudaStream_t s,
                            int* launches) {
  const int lanes = mean_min <= 8 ? 8 : mean_min <= 32 ? 16 : 32;
  // blocks of 256 up to two an SM, then of 1024: the fewer sums, the less the host has to add up (1216 of them
  // took 3 us)
  const int64_t all = (g.e1 - g.e0) * lanes, two = (int64_t)sm_count() * 2;
  const int threads = all <= 256 * two ? 256 : 1024;
  const unsigned grid = (unsigned)std::min<int64_t>((all + threads - 1) / threads, two);
  const bool stored = host_stores();
  std::vector<unsigned long long> sums(grid);
  DevBuf<unsigned long long> dev;
  if (!stored) ATC_TRY(dev.alloc(grid, s));
  unsigned long long* to = stored ? sums.data() : dev.p;
  {
    Phase ph("tc.count", s);
    if (lanes == 8) small_edges_kernel<8><<<grid, threads, 0, s>>>(g, to);
    else if (lanes == 16) small_edges_kernel<16><<<grid, threads, 0, s>>>(g, to);
    else small_edges_kernel<32><<<grid, threads, 0, s>>>(g, to);
  }
  *launches += 1;
  tm->stop(s);
  Phase ph("tc.readback", s);
  ATC_TRY(read_bytes(sums.data(), dev.p, sizeof(unsigned long long) * grid, stored, s));
  const volatile unsigned long long* v = sums.data();
  uint64_t t = 0;
  for (unsigned i = 0; i < grid; ++i) t += v[i];
  *count = t;
  return ATC_OK;
}

// The Bisson-style grouping of the edges of [e0, e1): every edge {u, v} at its endpoint h
// with the longer list, the partners of each h contiguous in plist, cut into warp and block
// items.  hc = {warp items, block items, -, longest hashed block list}.
struct Grouping {
  DevBuf<int32_t> cnt, cur, plist, deg;
  DevBuf<int64_t> gstart;
  DevBuf<int> counters;  // warp items, block items, (unused), longest block list, warp next, block next
  DevBuf<GroupItem> witems, bitems;
  int hc[4] = {0, 0, 0, 0};
};

// The device memory that group_edges allocates for `edges` edges.
static atc_status grouping_bytes(const CsrView& g, int64_t edges, const ItemShape& sh, size_t* bytes, cudaStream_t s) {
  ATC_TRY(exclusive_scan_i32_to_i64_tmp(nullptr, bytes, nullptr, nullptr, (size_t)g.n + 1, s));
  const int64_t items = max_items(g.n, edges, std::min(sh.warp_chunk, sh.block_chunk));
  *bytes += sizeof(int32_t) * (3 * (size_t)g.n + 2 + (size_t)edges + 32) + sizeof(int64_t) * ((size_t)g.n + 1) +
            sizeof(int) * 8 + 2 * sizeof(GroupItem) * (size_t)items;
  return ATC_OK;
}

static atc_status group_edges(const CsrView& g, const ItemShape& sh, Grouping* gr, cudaStream_t s, int* launches) {
  ATC_TRY(gr->cnt.alloc(g.n + 1, s));
  ATC_TRY(gr->cur.alloc(g.n, s));
  ATC_TRY(gr->gstart.alloc(g.n + 1, s));
  ATC_TRY(gr->counters.alloc(8, s));
  ATC_CK(cudaMemsetAsync(gr->cnt.p, 0, sizeof(int32_t) * (g.n + 1), s));
  ATC_CK(cudaMemsetAsync(gr->cur.p, 0, sizeof(int32_t) * g.n, s));
  ATC_CK(cudaMemsetAsync(gr->counters.p, 0, sizeof(int) * 8, s));
  ATC_TRY(gr->deg.alloc(g.n + 1, s));
  csr_outdeg_kernel<<<grid_for(g.n, 256), 256, 0, s>>>(g, gr->deg.p);
  ATC_CK(cudaGetLastError());
  group_count_kernel<<<grid_for(g.e1 - g.e0, 256), 256, 0, s>>>(g, gr->cnt.p, gr->deg.p);
  ATC_CK(cudaGetLastError());
  ATC_TRY(exclusive_scan_i32_to_i64(gr->cnt.p, gr->gstart.p, g.n + 1, s));
  int64_t total = 0;
  ATC_CK(cudaMemcpyAsync(&total, gr->gstart.p + g.n, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  ATC_TRY(gr->plist.alloc(total + 32, s));
  group_scatter_kernel<<<grid_for(g.e1 - g.e0, 256), 256, 0, s>>>(g, gr->gstart.p, gr->cur.p, gr->plist.p,
                                                                   gr->deg.p);
  ATC_CK(cudaGetLastError());
  // items: at most one per group plus one per chunk boundary
  int64_t max_items = g.n + total / std::min(sh.warp_chunk, sh.block_chunk) + 1;
  ATC_TRY(gr->witems.alloc(max_items, s));
  ATC_TRY(gr->bitems.alloc(max_items, s));
  group_items_kernel<<<grid_for(g.n, 256), 256, 0, s>>>(g, gr->gstart.p, gr->witems.p, gr->bitems.p,
                                                         gr->counters.p, sh, 0, INT64_MAX);
  ATC_CK(cudaGetLastError());
  ATC_CK(cudaMemcpyAsync(gr->hc, gr->counters.p, sizeof(gr->hc), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  *launches += 5;
  return ATC_OK;
}

// Predicted times (ps) of a whole count by grouped lists and on the ranked copy, per family: launches and
// waits, per vertex, per edge, per element of the shorter lists; and for lists, where W well above W_min
// tells of hubs, their contended group cursors and the longest item, whose 512 partners one warp streams.
// Fitted to 150 graphs of 16K to 16M edges (R-MAT, Chung-Lu, RGG, stars; ids spread by 1 to 256; every orientation), each
// counted both ways: following the faster prediction costs 1 % of the sum of the faster times, no graph more
// than half its own, and is 17 (Bisson), 29 (TriCore) and 27 % (Fox) faster in the mean than lists.  Lists / ranked
// in us, Bisson, stars (no wedge) of 3 M leaves 125 / 406, 4 M edges 173 / 554; R-MAT of 0.5 M edges on ids up to 7e7 1350 / 3800; RGG
// (W = 1.06 W_min) of 0.5 M 151 / 291; R-MAT of 0.7 M, 3.1 M, 11 M 528 / 300, 1058 / 474, 2652 / 1026, scale 24
// 117500 / 35700; Chung-Lu of 0.6 M, 14 M 387 / 295, 2232 / 1332; Fox, R-MAT scale 12 of 80 000 733 / 287.
static double lists_ps(const atc_csr* csr, atc_kernel kernel) {
  const double n = (double)csr->n, m = (double)csr->m, w = (double)csr->wedges, wmin = (double)csr->wedges_min;
  const double test = kernel == ATC_KERNEL_TRICORE ? 3.9 : kernel == ATC_KERNEL_FOX ? 4.2 : 1.0;
  const double tail = kernel == ATC_KERNEL_TRICORE ? 9.7e6 : kernel == ATC_KERNEL_FOX ? 1.44e7 : 4.6e6;
  const double hubs = wmin > 0.0 ? std::min(std::max(2.0 * (w / wmin - 1.0), 0.0), 1.0) : 0.0;
  return 9.2e7 + 15.0 * n + 32.0 * m + test * wmin +
         hubs * (2.9e5 * std::sqrt(m) + tail * wmin / m * std::min(m / 20000.0, 1.0));
}
static double ranked_ps(const atc_csr* csr, atc_kernel kernel) {
  const double test = kernel == ATC_KERNEL_TRICORE ? 1.1 : kernel == ATC_KERNEL_FOX ? 3.4 : 0.3;
  return 1.95e8 + 52.0 * (double)csr->n + 87.0 * (double)csr->m + test * (double)csr->wedges_min;
}
static bool ranked_pays(const atc_csr* csr, atc_kernel kernel) { return ranked_ps(csr, kernel) < lists_ps(csr, kernel); }

// The ranked count (csrc/ranked.cu) takes whole counts of CSRs that preTC built and that live on
// the device.  Parts keep the CSR's own orientation (their counts are defined by it), as do CSRs
// read from files (any sorted rows are accepted there); CSRs in host memory count in bounded
// scratch; an item shape asked for by tuning is one of the grouped lists.  Entries hold 32-bit
// positions.
static bool shaped(const atc_tuning* t) {  // an item shape is asked for
  return t && (t->bisson_cutover > 0 || t->bisson_warp_max > 0 || t->bisson_warp_chunk > 0 ||
               t->bisson_block_chunk > 0 || t->bisson_slots != 0);
}
static bool ranked_applies(const atc_csr* csr, int64_t e0, int64_t e1, const atc_tuning* t) {
  const CsrPriv* pv = static_cast<const CsrPriv*>(csr->priv);
  if (!pv->indeg || pv->host_cols || e0 != 0 || e1 != csr->m || csr->m > (int64_t)INT32_MAX) return false;
  return !shaped(t);
}

static atc_status run_bisson(const CsrView& g, const atc_tuning* t, unsigned long long* ctr, cudaStream_t s,
                             int* launches) {
  ItemShape sh;
  int slots;
  ATC_TRY(item_shape(t, &sh, &slots));
  std::optional<Phase> ph;
  ph.emplace("tc.group", s);
  Grouping gr;
  ATC_TRY(group_edges(g, sh, &gr, s, launches));
  ph.reset();
  ph.emplace("tc.count", s);
  return launch_slots(slots, g, gr.plist.p, gr.witems.p, gr.bitems.p, gr.hc, gr.counters.p, ctr, s, launches);
}

// Launches the searched kernels of one family over warp items [0, hc0) and block items
// [0, hc1), and checks their bulk waits.  next: the items' cursors (warp, block); err: zeroed.
template <int KIND, class Items, class Partners>
static atc_status launch_sorted(const CsrView& g, const Partners& partners, const Items& witems, const Items& bitems,
                                int hc0, int hc1, int max_row, bool bulk, int* next_w, int* next_b, int* err_d,
                                unsigned long long* ctr, cudaStream_t s, int* launches) {
  if (hc1) {
    const auto kern = sorted_block_kernel<KIND, Items, Partners>;
    uint32_t words = (uint32_t)std::min(std::max(max_row, kWarpMax + 1), kTabWords);
    words = (words + 31) & ~31u;
    const size_t smem = sizeof(int32_t) * (words + 8);  // + the bulk window's rounding
    ATC_CK(cudaFuncSetAttribute((const void*)kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    const int bps = blocks_per_sm((const void*)kern, kBgWarps * 32, smem);
    const int grid = std::min(hc1, sm_count() * bps);
    kern<<<grid, kBgWarps * 32, smem, s>>>(g, partners, bitems, hc1, next_b, words, bulk, err_d, ctr);
    ATC_CK(cudaGetLastError());
    *launches += 1;
  }
  if (hc0) {
    const auto kern = sorted_warp_kernel<KIND, Items, Partners>;
    const int bps = blocks_per_sm((const void*)kern, kBgWarps * 32, 0);
    const int grid = (int)std::min<int64_t>((hc0 + kBgWarps - 1) / kBgWarps, (int64_t)sm_count() * bps);
    kern<<<grid, kBgWarps * 32, 0, s>>>(g, partners, witems, hc0, next_w, bulk, err_d, ctr);
    ATC_CK(cudaGetLastError());
    *launches += 1;
  }
  int err = 0;
  ATC_CK(cudaMemcpyAsync(&err, err_d, sizeof(int), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  if (err) {
    set_error("a bulk copy into shared memory did not complete within its wait limit");
    return ATC_ERR_TIMEOUT;
  }
  return ATC_OK;
}

// TriCore-style (KIND 0) and Fox-style (KIND 1) searches of the staged longer lists, on the
// Bisson-style grouping of whole lists.
// max_outdeg sizes the block kernels' shared copy (lists above kTabWords stay in global).
// bulk: the lists are staged by TMA bulk copies (cols in device memory); with cols in mapped
// host memory they are staged with loads.
template <int KIND>
static atc_status run_sorted(const CsrView& g, int max_outdeg, bool bulk, unsigned long long* ctr, cudaStream_t s,
                             int* launches) {
  ItemShape sh = default_shape(kWarpMax);
  std::optional<Phase> ph;
  ph.emplace("tc.group", s);
  Grouping gr;
  ATC_TRY(group_edges(g, sh, &gr, s, launches));
  ph.reset();
  ph.emplace("tc.count", s);
  return launch_sorted<KIND>(g, ListPartners{gr.plist.p}, FullItems{gr.witems.p}, FullItems{gr.bitems.p}, gr.hc[0],
                             gr.hc[1], max_outdeg, bulk, gr.counters.p + 4, gr.counters.p + 5, gr.counters.p + 7, ctr,
                             s, launches);
}

// The same searches on the degree-ranked copy: for every edge u -> v the part of row u before v is
// searched in N+(v) (sum of C(d+(u), 2) searches instead of the sum of min(d+u, d+v), in lists
// that are shorter too).  TriCore-style with the part tables, R-MAT scale 20: 10.4 ms by whole lists
// and 32 samples, 8.7 with the tables, 6.9 on the ranked copy with samples, 3.6 with both; scale 24:
// 290 -> 97 ms.  Fox-style: 11.8 -> 7.6 and 304 -> 200 ms.  Both are bound by the shared-memory
// reads of the searches (three to four a test, with conflicts).
// *done = false: no room for the copy, or a row too long for it.
template <int KIND>
static atc_status run_sorted_ranked(const atc_csr* csr, unsigned long long* ctr, bool* done, cudaStream_t s,
                                    int* launches) {
  *done = false;
  std::optional<Phase> ph;
  ph.emplace("tc.group", s);
  RankedCopy rc;
  ATC_TRY(build_ranked(csr, false, &rc, s, launches));
  if (!rc.mem.p) return ATC_OK;
  int h[kcCount];
  ATC_CK(cudaMemcpyAsync(h, rc.ctr, sizeof(h), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  if (h[kcTooLong]) return ATC_OK;
  ph.reset();
  ph.emplace("tc.count", s);
  const CsrView g = csr_view(rc.roff, rc.rcols, nullptr, rc.n, rc.m);
  const RankItemLists& li = rc.li;
  ATC_TRY(launch_sorted<KIND>(g, PrefixPartners{rc.ent}, RankedItems{li.list, rc.gstart, li.lcap, li.warp_chunk, false},
                              RankedItems{li.list, rc.gstart, li.lcap, li.block_chunk, true}, h[kcWarp], h[kcBlock],
                              h[kcMaxRow], true, rc.ctr + kcNextWarp, rc.ctr + kcNextBlock, rc.ctr + kcError, ctr, s,
                              launches));
  *done = true;
  return ATC_OK;
}

// ---- counting without device allocation ------------------------------------------
// Some callers cannot call cudaMalloc: a host whose device memory is all owned by
// another allocator or runtime (a framework's caching pool, a memory manager that
// reserves the device up front), or a real-time loop that must not block in the
// driver's allocator.  atc_tc_noalloc runs the Bisson-style count above with every
// scratch buffer (edge sources, group counts, grouped partner list, work items,
// counters) carved out of one file-scope device array of kNoAllocBytes, fixed in size,
// which every GPU that loads this library keeps until the process exits.  Graphs above
// kNoAllocMaxN vertices or kNoAllocMaxM edges are refused.  The call synchronises its
// stream: it reads the CSR check, the item counts and the count back to the host.  All
// calls share the one array: calls that overlap on the GPU (concurrent streams or host
// threads on one device) race and must be serialised by the caller.
constexpr int64_t kNoAllocMaxN = 1 << 17;  // 131072 vertices
constexpr int64_t kNoAllocMaxM = 1 << 20;  // 1048576 oriented edges
constexpr int64_t kNoAllocItems = kNoAllocMaxN + kNoAllocMaxM / kWarpChunk + 1;

constexpr size_t align256(size_t x) { return (x + 255) & ~size_t(255); }
constexpr size_t kNaEsrc = 0;
constexpr size_t kNaCnt = kNaEsrc + align256(sizeof(int32_t) * (kNoAllocMaxM + 32));
constexpr size_t kNaCur = kNaCnt + align256(sizeof(int32_t) * (kNoAllocMaxN + 1));
constexpr size_t kNaGstart = kNaCur + align256(sizeof(int32_t) * kNoAllocMaxN);
constexpr size_t kNaPlist = kNaGstart + align256(sizeof(int64_t) * (kNoAllocMaxN + 1));
constexpr size_t kNaWitems = kNaPlist + align256(sizeof(int32_t) * (kNoAllocMaxM + 32));
constexpr size_t kNaBitems = kNaWitems + align256(sizeof(GroupItem) * kNoAllocItems);
constexpr size_t kNaCounters = kNaBitems + align256(sizeof(GroupItem) * kNoAllocItems);
constexpr size_t kNaCount = kNaCounters + align256(sizeof(int) * 8);
constexpr size_t kNoAllocBytes = kNaCount + align256(sizeof(unsigned long long));

static __device__ __align__(256) unsigned char g_noalloc_scratch[kNoAllocBytes];

namespace {

// Device address of g_noalloc_scratch for each device, looked up once per device (with
// that device current) and kept for the life of the process.  cudaDeviceReset destroys
// the context that holds the array, so after a reset of a device this entry point must
// not be called on it again in the same process.
atc_status noalloc_scratch(unsigned char** out) {
  static std::mutex mu;
  static unsigned char* addr[64] = {};
  int dev = 0;
  ATC_CK(cudaGetDevice(&dev));
  ATC_CHECK_ARG(dev >= 0 && dev < 64, "device index above 63");
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    void* p = nullptr;
    cudaError_t e = cudaGetSymbolAddress(&p, g_noalloc_scratch);
    if (e != cudaSuccess) {
      set_error("cudaGetSymbolAddress(g_noalloc_scratch): %s", cudaGetErrorString(e));
      return ATC_ERR_CUDA;
    }
    addr[dev] = static_cast<unsigned char*>(p);
  }
  *out = addr[dev];
  return ATC_OK;
}

// Checks a caller's CSR before any kernel indexes with it: offsets start at 0, end at m
// and never decrease; every row is strictly increasing with ids in [0, n).  Sets
// *bad = 1 on the first violation found by each warp.
__global__ void csr_check_kernel(const int64_t* off, const int32_t* cols, int64_t n, int64_t m, int* bad) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  if (blockIdx.x == 0 && threadIdx.x == 0 && (off[0] != 0 || off[n] != m)) *bad = 1;
  for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < n; u += warps) {
    int64_t b = off[u], e = off[u + 1];
    bool ok = b <= e && b >= 0 && e <= m;
    if (ok) {
      for (int64_t j = b + lane; j < e; j += 32) {
        int32_t x = cols[j];
        if (x < 0 || x >= n || (j + 1 < e && cols[j + 1] <= x)) ok = false;
      }
    }
    if (__any_sync(0xffffffffu, !ok) && lane == 0) *bad = 1;
  }
}

__global__ void esrc_fill_kernel(const int64_t* off, int64_t n, int32_t* esrc) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t u = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; u < n; u += warps)
    for (int64_t j = off[u] + lane; j < off[u + 1]; j += 32) esrc[j] = (int32_t)u;
}

// Exclusive scan of cnt[0, len) into out (int64), one block of 1024 threads, no
// temporary storage: each thread scans a contiguous slice, slices are combined in
// shared memory.
__global__ void __launch_bounds__(1024) scan_one_block_kernel(const int32_t* cnt, int64_t len, int64_t* out) {
  __shared__ int64_t part[1024];
  const int t = threadIdx.x;
  const int64_t per = (len + 1023) / 1024;
  const int64_t b = t * per, e = b + per < len ? b + per : len;
  int64_t s = 0;
  for (int64_t i = b; i < e; ++i) s += cnt[i];
  part[t] = s;
  __syncthreads();
  for (int o = 1; o < 1024; o <<= 1) {
    int64_t y = t >= o ? part[t - o] : 0;
    __syncthreads();
    part[t] += y;
    __syncthreads();
  }
  int64_t run = part[t] - s;
  for (int64_t i = b; i < e; ++i) {
    out[i] = run;
    run += cnt[i];
  }
}

}  // namespace

static atc_status tc_noalloc_impl(const int64_t* off, const int32_t* cols, int64_t n, int64_t m, uint64_t* count,
                                  cudaStream_t s) {
  unsigned char* base = nullptr;
  ATC_TRY(noalloc_scratch(&base));
  int32_t* esrc = reinterpret_cast<int32_t*>(base + kNaEsrc);
  int32_t* cnt = reinterpret_cast<int32_t*>(base + kNaCnt);
  int32_t* cur = reinterpret_cast<int32_t*>(base + kNaCur);
  int64_t* gstart = reinterpret_cast<int64_t*>(base + kNaGstart);
  int32_t* plist = reinterpret_cast<int32_t*>(base + kNaPlist);
  GroupItem* witems = reinterpret_cast<GroupItem*>(base + kNaWitems);
  GroupItem* bitems = reinterpret_cast<GroupItem*>(base + kNaBitems);
  int* counters = reinterpret_cast<int*>(base + kNaCounters);
  unsigned long long* total_ctr = reinterpret_cast<unsigned long long*>(base + kNaCount);
  // what the kernels accumulate into starts at zero; the rest is overwritten
  ATC_CK(cudaMemsetAsync(cnt, 0, sizeof(int32_t) * (n + 1), s));
  ATC_CK(cudaMemsetAsync(cur, 0, sizeof(int32_t) * n, s));
  ATC_CK(cudaMemsetAsync(counters, 0, sizeof(int) * 8, s));
  ATC_CK(cudaMemsetAsync(total_ctr, 0, sizeof(unsigned long long), s));
  csr_check_kernel<<<grid_for(n * 32, 256), 256, 0, s>>>(off, cols, n, m, counters + 6);
  ATC_CK(cudaGetLastError());
  int bad = 0;
  ATC_CK(cudaMemcpyAsync(&bad, counters + 6, sizeof(int), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  if (bad) {
    set_error("atc_tc_noalloc: offsets/cols are not an oriented CSR with sorted rows of ids in [0, n)");
    return ATC_ERR_INVALID;
  }
  esrc_fill_kernel<<<grid_for(n * 32, 256), 256, 0, s>>>(off, n, esrc);
  ATC_CK(cudaGetLastError());
  CsrView g = csr_view(off, cols, esrc, n, m);
  group_count_kernel<<<grid_for(m, 256), 256, 0, s>>>(g, cnt, nullptr);
  scan_one_block_kernel<<<1, 1024, 0, s>>>(cnt, n + 1, gstart);
  group_scatter_kernel<<<grid_for(m, 256), 256, 0, s>>>(g, gstart, cur, plist, nullptr);
  group_items_kernel<<<grid_for(n, 256), 256, 0, s>>>(g, gstart, witems, bitems, counters, default_shape(32), 0,
                                                       INT64_MAX);
  ATC_CK(cudaGetLastError());
  int hc[4];
  ATC_CK(cudaMemcpyAsync(hc, counters, sizeof(hc), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  int launches = 0;
  ATC_TRY(launch_bisson<kDefaultSlots>(g, plist, witems, bitems, hc, counters, total_ctr, s, &launches));
  unsigned long long h = 0;
  ATC_CK(cudaMemcpyAsync(&h, total_ctr, sizeof(h), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  *count = h;
  return ATC_OK;
}

}  // namespace atc

using namespace atc;

atc_status atc::part_edge_range(const atc_csr* csr, uint32_t part, uint32_t nparts, int64_t* range, cudaStream_t s) {
  range[0] = 0;
  range[1] = csr->m;
  if (nparts <= 1 || csr->m == 0) return ATC_OK;
  CsrPriv* pv = static_cast<CsrPriv*>(csr->priv);
  CsrView g = csr_view(csr->offsets, csr->cols, pv->esrc, csr->n, csr->m);
  DevBuf<int64_t> work, prefix, bounds;
  ATC_TRY(work.alloc(csr->m + 1, s));
  ATC_TRY(prefix.alloc(csr->m + 1, s));
  ATC_TRY(bounds.alloc(2, s));
  edge_work_kernel<<<grid_for(csr->m + 1, 256), 256, 0, s>>>(g, work.p);
  ATC_CK(cudaGetLastError());
  ATC_TRY(exclusive_scan_i64(work.p, prefix.p, csr->m + 1, s));
  part_bounds_kernel<<<1, 32, 0, s>>>(prefix.p, csr->m, part, nparts, bounds.p);
  ATC_CK(cudaGetLastError());
  ATC_CK(cudaMemcpyAsync(range, bounds.p, 2 * sizeof(int64_t), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  return ATC_OK;
}

// ATC_KERNEL_AUTO: the Bisson-style or the Hu-style count, whichever is predicted faster.  Against the ranked
// copy: Hu-style 2.3 ps per wedge (W; 1.2 at scale 20 and above, where it loses anyway) + 45 ps per edge + 9 ps
// per vertex + 0.06 ms, or the small count.  Against grouped lists (parts, loaded CSRs, graphs that the copy does not pay
// for): 1.097 ps per wedge + 103.5 ps per edge against 1.232 ps per element of W_min + 117.5 ps per edge + 0.3 ms, the fit
// of the two that it was made with.  Measured Hu / ranked in ms: R-MAT scale 14 0.09 / 0.23, 15 0.18 / 0.24, 16 0.39 / 0.27, 18 1.32 /
// 0.47, 20 6.4 / 1.35; Chung-Lu 1.3M edges 0.27 / 0.34, 4.0M 0.68 / 0.53, 9.6M 1.52 / 0.98.
static atc_kernel auto_kernel(const atc_csr* csr, bool ranked) {
  const double n = (double)csr->n, m = (double)csr->m, w = (double)csr->wedges, wmin = (double)csr->wedges_min;
  const double bisson_ps = ranked ? ranked_ps(csr, ATC_KERNEL_BISSON) : 1.232 * wmin + 117.5 * m + 3.0e8;
  double hu_ps = ranked ? 2.3 * w + 45.0 * m + 9.0 * n + 6.0e7 : 1.097 * w + 103.5 * m;
  if (small_pays(csr, csr->m)) hu_ps = std::min(hu_ps, 5.5 * wmin + 60.0 * m + 1.3e7);
  return hu_ps < bisson_ps ? ATC_KERNEL_HU : ATC_KERNEL_BISSON;
}

// Counts the edges [e0, e1) of the CSR (every edge for the whole count).
static atc_status tc_window(const atc_csr* csr, atc_kernel kernel, const atc_tuning* tuning, int64_t e0, int64_t e1,
                            uint64_t* count, atc_stats* stats, cudaStream_t s) {
  CsrPriv* pv = static_cast<CsrPriv*>(csr->priv);
  const bool applies = pv && ranked_applies(csr, e0, e1, tuning), chosen = kernel == ATC_KERNEL_AUTO;
  if (chosen) kernel = auto_kernel(csr, applies && ranked_pays(csr, ATC_KERNEL_BISSON));
  const bool ranked = applies && ranked_pays(csr, kernel);
  int launches = 0;
  EventTimer tm;
  if (e1 > e0) {
    CsrView g = csr_view(csr->offsets, csr->cols, pv->esrc, csr->n, csr->m);
    g.e0 = e0;
    g.e1 = e1;
    unsigned long long* ctr = pv->counter;
    Phase ph("tc", s);
    tm.start(s);
    if (kernel == ATC_KERNEL_HU && !shaped(tuning) && small_pays(csr, e1 - e0)) {
      ATC_TRY(run_small(g, csr->wedges_min / csr->m, count, &tm, s, &launches));
    } else {
      ATC_CK(cudaMemsetAsync(ctr, 0, sizeof(unsigned long long), s));
      switch (kernel) {
        case ATC_KERNEL_HU: ATC_TRY(run_hu(g, tuning, ctr, s, &launches)); break;
        case ATC_KERNEL_BISSON: {
          bool done = false;
          if (ranked) ATC_TRY(count_ranked(csr, ctr, &done, s, &launches));
          if (done) break;
          if (ranked) ATC_CK(cudaMemsetAsync(ctr, 0, sizeof(unsigned long long), s));
          // the choice was the library's: where the lists find no room, the Hu-style count, which groups none
          atc_status st = ATC_OK;
          if (chosen && alloc_budget_left() >= 0) {
            ItemShape sh;
            int slots;
            size_t need = 0;
            ATC_TRY(item_shape(tuning, &sh, &slots));
            ATC_TRY(grouping_bytes(g, e1 - e0, sh, &need, s));
            if ((size_t)alloc_budget_left() < need) st = ATC_ERR_OOM;
          }
          if (st == ATC_OK) st = run_bisson(g, tuning, ctr, s, &launches);
          if (st == ATC_ERR_OOM && chosen) {
            cudaGetLastError();
            kernel = ATC_KERNEL_HU;
            st = run_hu(g, tuning, ctr, s, &launches);
          }
          ATC_TRY(st);
          break;
        }
        default: {
          const bool fox = kernel == ATC_KERNEL_FOX;
          if (tuning && tuning->edge_kernels) {
            ATC_TRY(fox ? run_fox(g, tuning, ctr, s, &launches) : run_tricore(g, tuning, ctr, s, &launches));
            break;
          }
          bool done = false;
          if (ranked)
            ATC_TRY(fox ? run_sorted_ranked<1>(csr, ctr, &done, s, &launches)
                        : run_sorted_ranked<0>(csr, ctr, &done, s, &launches));
          if (!done) {
            const bool bulk = pv->host_cols == nullptr;
            ATC_TRY(fox ? run_sorted<1>(g, csr->max_outdeg, bulk, ctr, s, &launches)
                        : run_sorted<0>(g, csr->max_outdeg, bulk, ctr, s, &launches));
          }
          break;
        }
      }
      tm.stop(s);
      Phase ph_rb("tc.readback", s);
      unsigned long long h = 0;
      ATC_TRY(read_bytes(&h, ctr, sizeof(h), false, s));
      *count = h;
    }
  }
  if (stats) {
    stats->kernel_ms = e1 > e0 ? tm.ms() : 0.0f;
    stats->total_ms = stats->kernel_ms;
    stats->wedges = (uint64_t)csr->wedges;
    stats->alg_bytes = 4ull * (uint64_t)(csr->n + 1) + 4ull * (uint64_t)csr->m + 4ull * (uint64_t)csr->wedges + 8ull;
    stats->alg_bytes_min =
        4ull * (uint64_t)(csr->n + 1) + 4ull * (uint64_t)csr->m + 4ull * (uint64_t)csr->wedges_min + 8ull;
    stats->kernel_used = (int32_t)kernel;
    stats->launches = launches;
  }
  return ATC_OK;
}

extern "C" atc_status atc_tc(const atc_csr* csr, atc_kernel kernel, const atc_tuning* tuning, uint64_t* count,
                             atc_stats* stats, atc_stream st) try {
  ATC_CHECK_ARG(csr != nullptr && count != nullptr, "NULL argument");
  ATC_CHECK_ARG(csr->priv != nullptr || csr->m == 0, "csr was not built by atc_pretc");
  ATC_CHECK_ARG(kernel >= ATC_KERNEL_AUTO && kernel <= ATC_KERNEL_TRICORE, "unknown atc_kernel");
  *count = 0;
  return tc_window(csr, kernel, tuning, 0, csr->m, count, stats, as_stream(st));
} ATC_CATCH

extern "C" atc_status atc_tc_part(const atc_csr* csr, atc_kernel kernel, const atc_tuning* tuning, uint32_t part,
                                  uint32_t nparts, uint64_t* count, int64_t* edge_range, atc_stats* stats,
                                  atc_stream st) try {
  ATC_CHECK_ARG(csr != nullptr && count != nullptr, "NULL argument");
  ATC_CHECK_ARG(csr->priv != nullptr || csr->m == 0, "csr was not built by atc_pretc");
  ATC_CHECK_ARG(kernel >= ATC_KERNEL_AUTO && kernel <= ATC_KERNEL_TRICORE, "unknown atc_kernel");
  ATC_CHECK_ARG(nparts >= 1 && part < nparts, "part must be in [0, nparts)");
  cudaStream_t s = as_stream(st);
  *count = 0;
  int64_t b[2];
  ATC_TRY(part_edge_range(csr, part, nparts, b, s));
  if (edge_range) {
    edge_range[0] = b[0];
    edge_range[1] = b[1];
  }
  return tc_window(csr, kernel, tuning, b[0], b[1], count, stats, s);
} ATC_CATCH

extern "C" atc_status atc_tc_noalloc(const int64_t* offsets, const int32_t* cols, int64_t n, int64_t m,
                                     uint64_t* count, atc_stream st) try {
  ATC_CHECK_ARG(count != nullptr, "count is NULL");
  ATC_CHECK_ARG(n >= 0 && m >= 0, "negative size");
  if (n > kNoAllocMaxN || m > kNoAllocMaxM) {
    set_error("graph too large for atc_tc_noalloc: n=%lld m=%lld, limits n<=%lld m<=%lld (scratch %zu bytes)",
              (long long)n, (long long)m, (long long)kNoAllocMaxN, (long long)kNoAllocMaxM, kNoAllocBytes);
    return ATC_ERR_INVALID;
  }
  *count = 0;
  if (m == 0 || n == 0) return ATC_OK;
  ATC_CHECK_ARG(offsets != nullptr && cols != nullptr, "NULL CSR array");
  return tc_noalloc_impl(offsets, cols, n, m, count, as_stream(st));
} ATC_CATCH

extern "C" atc_status atc_check_wait_timeout(atc_stream st) try {
  cudaStream_t s = as_stream(st);
  DevBuf<int> err;
  ATC_TRY(err.alloc(1, s));
  ATC_CK(cudaMemsetAsync(err.p, 0, sizeof(int), s));
  atc::wait_timeout_check_kernel<<<1, 32, 0, s>>>(1000000ull, err.p);  // a 1 ms limit
  ATC_CK(cudaGetLastError());
  int h = 0;
  ATC_CK(cudaMemcpyAsync(&h, err.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  if (h) {
    atc::set_error("a bulk-copy wait gave up after its time limit (the check's barrier never completes)");
    return ATC_ERR_TIMEOUT;
  }
  return ATC_OK;
} ATC_CATCH
