// Batched triangle counting: many graphs of uneven sizes counted together.
//
// The reference runs one program per graph.  Here the graphs of a batch are kept as one
// disjoint union on the device (graph g owns vertices [vbase[g], vbase[g+1])), and one
// replay of a CUDA graph counts all of them: the Bisson-style grouping passes run once
// over the union, the persistent counting kernels drain its work items from device
// counters, and every item adds its triangles to its own graph's counter.  Nothing in
// the replay waits on the host, so small graphs cost no launch or synchronisation of
// their own — the overhead a per-graph loop pays 4096 times.
//
// Memory, per union vertex / edge: offsets 8 B, cols 4 B, group count / cursor 8 B,
// group starts 8 B, grouped partner list <= 4 B per edge, work items 8 B each.  No
// per-edge source array is kept (the grouping passes walk rows).
#include <algorithm>
#include <cstring>
#include <vector>

#include "bisson.cuh"

struct atc_batch {
  int64_t n = 0, m = 0;        // vertices / edges held
  int64_t vcap = 0, ecap = 0;  // allocated
  int64_t* off = nullptr;      // vcap + 1
  int32_t* cols = nullptr;     // ecap + 16
  std::vector<int64_t> vbase{0};
  std::vector<int64_t> gm, gw, gwmin;  // per graph: edges, W, sum of min(d+u, d+v)
  std::vector<int32_t> gmax;           // per graph: longest list
  int32_t max_outdeg = 0;
  bool dirty = true;
  int rows_graphs = 0;  // graphs of the last built pipeline counted by rows
  int launches = 0;     // kernel launches of one replay of the built pipeline
  atc::ItemShape shape = atc::default_shape(32);
  // counting pipeline, sized for the union when built
  int32_t* cnt = nullptr;
  int32_t* cur = nullptr;
  int64_t* gstart = nullptr;
  int32_t* plist = nullptr;
  int2* items = nullptr;
  int* counters = nullptr;
  int2* items_r = nullptr;   // mode 2: the rows items of the graphs counted by rows
  int* counters_r = nullptr;
  int2* big = nullptr;       // block items of lists longer than kBlockSmallList
  int2* big_r = nullptr;     // the same for the rows items
  int64_t big_cap = 0;
  uint8_t* vrows = nullptr;  // mode 2: 1 for the vertices of graphs counted by rows
  int64_t* vbase_d = nullptr;
  unsigned long long* gcounts = nullptr;
  void* scan_tmp = nullptr;
  int64_t built_n = -1, built_m = -1, items_cap = 0, rows_cap = 0, plist_cap = 0;
  int built_graphs = -1;
  atc::ItemShape built_shape{};
  cudaStream_t cap_stream = nullptr;
  cudaGraph_t graph = nullptr;
  cudaGraphExec_t exec = nullptr;
  // event nodes of the replay: stage k runs from stage_ev[k] to stage_ev[k + 1]
  std::vector<cudaEvent_t> stage_ev;
  std::vector<const char*> stage_name;
};

namespace atc {
namespace {

// counters of one replay: [0] warp items, [1] block items, [2] block items of long lists,
// [3] longest list among [1], [4..6] the counting kernels' item cursors, [8], [9] the
// grouping passes' row-block queues
constexpr int kBatchCounters = 16;

__global__ void batch_copy_kernel(const int64_t* off_g, const int32_t* cols_g, int64_t n_g, int64_t m_g,
                                  int64_t vbase, int64_t ebase, int64_t* off_u, int32_t* cols_u) {
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n_g || i < m_g; i += stride) {
    if (i < n_g) off_u[vbase + i] = off_g[i] + ebase;
    if (i < m_g) cols_u[ebase + i] = cols_g[i] + (int32_t)vbase;
  }
}

void free_pipeline(atc_batch* b) {
  if (b->exec) cudaGraphExecDestroy(b->exec);
  if (b->graph) cudaGraphDestroy(b->graph);
  b->exec = nullptr;
  b->graph = nullptr;
  void* bufs[] = {b->cnt, b->cur, b->gstart, b->plist, b->items, b->counters, b->vbase_d, b->gcounts, b->scan_tmp,
                  b->items_r, b->counters_r, b->vrows, b->big, b->big_r};
  for (void* p : bufs)
    if (p) cudaFree(p);
  b->cnt = b->cur = b->plist = nullptr;
  b->gstart = b->vbase_d = nullptr;
  b->items = nullptr;
  b->counters = nullptr;
  b->items_r = nullptr;
  b->counters_r = nullptr;
  b->vrows = nullptr;
  b->big = b->big_r = nullptr;
  b->big_cap = 0;
  b->gcounts = nullptr;
  b->scan_tmp = nullptr;
  b->built_n = b->built_m = -1;
  b->built_graphs = -1;
}

template <class T>
atc_status dev_alloc(T** p, size_t count) {
  if (!alloc_budget_take(sizeof(T) * (count ? count : 1))) {
    *p = nullptr;
    set_error("device allocation of %zu bytes for the batch refused: the allocation budget (atc_set_alloc_budget) "
              "is spent", sizeof(T) * count);
    return ATC_ERR_OOM;
  }
  cudaError_t e = cudaMalloc(reinterpret_cast<void**>(p), sizeof(T) * (count ? count : 1));
  if (e != cudaSuccess) {
    *p = nullptr;
    set_error("cudaMalloc(%zu bytes) for the batch: %s", sizeof(T) * count, cudaGetErrorString(e));
    return e == cudaErrorMemoryAllocation ? ATC_ERR_OOM : ATC_ERR_CUDA;
  }
  return ATC_OK;
}

// Grows the union arrays to hold n vertices and m edges (keeping the contents).
atc_status ensure_union(atc_batch* b, int64_t n, int64_t m, cudaStream_t s) {
  if (n <= b->vcap && m <= b->ecap) return ATC_OK;
  int64_t vcap = std::max(n, b->vcap ? 2 * b->vcap : n);
  int64_t ecap = std::max(m, b->ecap ? 2 * b->ecap : m);
  int64_t* off = nullptr;
  int32_t* cols = nullptr;
  ATC_TRY(dev_alloc(&off, (size_t)vcap + 1));
  atc_status st = dev_alloc(&cols, (size_t)ecap + 16);
  if (st != ATC_OK) {
    cudaFree(off);
    return st;
  }
  ATC_CK(cudaMemsetAsync(cols + ecap, 0, sizeof(int32_t) * 16, s));
  if (b->n) ATC_CK(cudaMemcpyAsync(off, b->off, sizeof(int64_t) * b->n, cudaMemcpyDeviceToDevice, s));
  if (b->m) ATC_CK(cudaMemcpyAsync(cols, b->cols, sizeof(int32_t) * b->m, cudaMemcpyDeviceToDevice, s));
  ATC_CK(cudaStreamSynchronize(s));
  if (b->off) cudaFree(b->off);
  if (b->cols) cudaFree(b->cols);
  b->off = off;
  b->cols = cols;
  b->vcap = vcap;
  b->ecap = ecap;
  return ATC_OK;
}

}  // namespace
}  // namespace atc

using namespace atc;

extern "C" atc_status atc_batch_create(atc_batch** out) try {
  ATC_CHECK_ARG(out != nullptr, "out is NULL");
  *out = new atc_batch();
  return ATC_OK;
} ATC_CATCH

extern "C" atc_status atc_batch_reserve(atc_batch* b, int64_t n, int64_t m, atc_stream s) try {
  ATC_CHECK_ARG(b != nullptr && n >= 0 && m >= 0, "bad argument");
  return ensure_union(b, n, m, as_stream(s));
} ATC_CATCH

extern "C" atc_status atc_batch_add(atc_batch* b, const atc_csr* csr, int32_t* index, atc_stream st) try {
  ATC_CHECK_ARG(b != nullptr && csr != nullptr, "NULL argument");
  ATC_CHECK_ARG(b->n + csr->n < (int64_t)INT32_MAX, "batch would exceed 2^31 vertices");
  cudaStream_t s = as_stream(st);
  ATC_TRY(ensure_union(b, b->n + csr->n, b->m + csr->m, s));
  int64_t work = std::max(csr->n, csr->m);
  if (work > 0) {
    batch_copy_kernel<<<grid_for(work, 256), 256, 0, s>>>(csr->offsets, csr->cols, csr->n, csr->m, b->n, b->m,
                                                          b->off, b->cols);
    ATC_CK(cudaGetLastError());
  }
  ATC_CK(cudaStreamSynchronize(s));
  if (index) *index = (int32_t)(b->vbase.size() - 1);
  b->n += csr->n;
  b->m += csr->m;
  b->vbase.push_back(b->n);
  b->gm.push_back(csr->m);
  b->gw.push_back(csr->wedges);
  b->gwmin.push_back(csr->wedges_min);
  b->gmax.push_back(csr->max_outdeg);
  b->max_outdeg = std::max(b->max_outdeg, csr->max_outdeg);
  b->dirty = true;
  return ATC_OK;
} ATC_CATCH

extern "C" atc_status atc_batch_info(const atc_batch* b, int32_t* graphs, int64_t* n, int64_t* m) try {
  ATC_CHECK_ARG(b != nullptr, "NULL batch");
  if (graphs) *graphs = (int32_t)(b->vbase.size() - 1);
  if (n) *n = b->n;
  if (m) *m = b->m;
  return ATC_OK;
} ATC_CATCH

extern "C" atc_status atc_batch_destroy(atc_batch* b) try {
  if (!b) return ATC_OK;
  free_pipeline(b);
  if (b->off) cudaFree(b->off);
  if (b->cols) cudaFree(b->cols);
  if (b->cap_stream) cudaStreamDestroy(b->cap_stream);
  for (cudaEvent_t e : b->stage_ev) cudaEventDestroy(e);
  delete b;
  return ATC_OK;
} ATC_CATCH

namespace atc {
namespace {

// Rows items: a warp per chunk of row u's members, whose lists are tested against N+(u), held in
// 4 KB of shared memory per warp.  The ids of a graph are consecutive, which makes three forms of it:
//   - up to 2^15 vertices: a bit per id;
//   - more: 1024 words of four 8-bit tags, or three of 10 or two of 16 where the graph's ids need
//     them.  The word is id + (id / 1024 + 1) * odd mod 1024 and the tag id / 1024 + 1 (ids from the
//     graph's first), which together name the id;
//   - rows of which more members share a word than it has tags (and graphs above 2^26 vertices): a bit
//     by the low 15 bits of the id, and the members among the hits looked up in the list, from a stack
//     per lane.
// Groups of kLanes lanes read a list, four ids a lane from the 16-byte line they lie in; ids
// outside the list are masked off by position.
// The lists are short (20 ids in the mean), so what counts is that the groups stay busy: the warp
// loads 32 members' list bounds at once and a group whose list is done takes the next.  48 Chung-Lu
// graphs, 25 M edges, 9e8 tests: hash tables and 32 elements a round 2.95 ms; this with members dealt
// out in advance and every hit looked up 2.33, dealt out in turn 2.17 (8 lanes 2.22, 2 lanes 2.45), with
// tags 1.75 (1.34 if no hit had to be told from a shared bit).  Bound by issue.
constexpr int kRowsChunk = 64;  // members an item: one row's members, so the longest rows set the tail
constexpr int kRowsLanes = 4;
constexpr int kRowStack = 12;
template <int kLanes>
__global__ void __launch_bounds__(128, 9) rows_kernel(CsrView g, CompactItems items, const int* nitems_dev, int* next,
                                                      GraphTags tags) {
  constexpr uint32_t kBytes = 1 << 12;
  __shared__ __align__(16) unsigned char smem[4 * kBytes];
  __shared__ int32_t stacks[4][kRowStack][32];
  __shared__ GraphAccSlot acc[4];
  const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
  const uint32_t base = w * kBytes;
  const uint4* ids = reinterpret_cast<const uint4*>(g.cols);
  uint32_t* T = reinterpret_cast<uint32_t*>(smem + base);
  for (int j = lane; j < (int)(kBytes / 4); j += 32) T[j] = 0u;
  graph_acc_init(&acc[w]);
  const int nitems = *nitems_dev;
  const int sub = lane % kLanes;
  auto word = [&](uint32_t x) {
    return reinterpret_cast<uint32_t*>(smem + (((x >> 3) & (kBytes - 4)) | base));
  };
  int it = 0, it_end = 0;
  auto take = [&]() {
    if (it == it_end) {
      int first = 0;
      if (lane == 0) first = atomicAdd(next, kWarpGrab);
      it = __shfl_sync(0xffffffffu, first, 0);
      it_end = it + kWarpGrab;
    }
    return it < nitems ? items.get(g, it++) : GroupItem{-1, 0, 0, 0};
  };
  GroupItem ni = take();
  while (ni.h >= 0) {
    const GroupItem gi = ni;
    const int64_t hb = __ldg(g.off + gi.h);
    const int dh = (int)(__ldg(g.off + gi.h + 1) - hb);
    ni = take();  // the next item's loads run under this one's
    if (dh < 2) continue;
    graph_acc_enter(tags, &acc[w], gi.h);
    const int size = acc[w].hi - acc[w].lo;
    const bool exact = size <= (1 << 15);
    // four times (id - the graph's first + 1024)
    const uint32_t shift4 = 4u * (1024u - (uint32_t)acc[w].lo);
    auto tag_word = [&](uint32_t x4, uint32_t tag) {
      return reinterpret_cast<uint32_t*>(smem + (((x4 + tag * (4u * 661u)) & (kBytes - 4)) | base));
    };
    // tags of `bits` bits: one in each field, and each field's top bit
    const int bits = size <= 255 << 10 ? 8 : size <= 1023 << 10 ? 10 : 16;
    const uint32_t ones = bits == 8 ? 0x01010101u : bits == 10 ? 0x00100401u : 0x00010001u;
    const uint32_t tops = ones << (bits - 1);
    bool tagged = !exact && size <= 65535 << 10;
    const int ne = (int)(gi.e - gi.b);
    const int32_t* en = g.cols + gi.b;
    if (tagged) {
      bool full = false;
      for (int j = lane; j < dh; j += 32) {
        const uint32_t x4 = 4u * (uint32_t)__ldg(g.cols + hb + j) + shift4, tag = x4 >> 12;
        uint32_t* at = tag_word(x4, tag);
        uint32_t old = 0;
        for (int k = 0;;) {  // into the first free field, counting from the low end
          if (k + bits > 32) {
            full = true;
            break;
          }
          if (old >> k & ((1u << bits) - 1)) {
            k += bits;
            continue;
          }
          const uint32_t seen = atomicCAS(at, old, old | tag << k);
          if (seen == old) break;
          old = seen;
        }
      }
      if (__any_sync(0xffffffffu, full)) {
        for (int j = lane; j < dh; j += 32) {
          const uint32_t x4 = 4u * (uint32_t)__ldg(g.cols + hb + j) + shift4;
          *tag_word(x4, x4 >> 12) = 0u;
        }
        tagged = false;
      }
      __syncwarp();
    }
    if (!tagged)
      for (int j = lane; j < dh; j += 32) {
        const uint32_t x = (uint32_t)__ldg(g.cols + hb + j);
        atomicOr(word(x), 0x80000000u >> (x & 31));
      }
    __syncwarp();
    // 32 members' lists at a time, one per lane: first line, and ids from its start to the list's end
    // (times four, plus those before the list)
    uint32_t line = 0, span = 0;
    int from = 0, lim = 0, given = 0;  // next members to load; lists loaded, and handed out
    uint32_t at = 0;  // the lane's next line
    int left = -4 * sub;  // ids from its start to the end of the group's list
    int skip = 0;     // ids of it before the list
    unsigned cnt = 0;
    int sp = 0;
    // Loads the lane's next line; returns its ids that count, the first as bit 3.  Groups whose list
    // is done take the next ones in turn, so that lists of uneven lengths keep all of them busy.
    auto fetch = [&](uint4& d) -> unsigned {
      const bool need = left + 4 * sub <= 0;
      const unsigned groups = __ballot_sync(0xffffffffu, need && sub == 0);
      if (groups) {
        if (given >= lim && from < ne) {
          span = 0;
          if (from + lane < ne) {
            const int32_t v = __ldg(en + from + lane);
            const int64_t b = __ldg(g.off + v), e = __ldg(g.off + v + 1);
            line = (uint32_t)(b >> 2);
            if (e > b) span = (uint32_t)(e - (b & ~3ll)) << 2 | (uint32_t)(b & 3);
          }
          lim = min(ne - from, 32);
          from += 32;
          given = 0;
        }
        const int k = given + __popc(groups & ((1u << (lane - sub)) - 1));
        const uint32_t l = __shfl_sync(0xffffffffu, line, k), sk = __shfl_sync(0xffffffffu, span, k);
        if (need) {
          const bool some = k < lim;
          at = l + sub;
          skip = some && sub == 0 ? (int)(sk & 3u) : 0;
          left = (some ? (int)(sk >> 2) : 0) - 4 * sub;
        }
        given = min(given + __popc(groups), lim);
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
      if (tagged) {
        auto in = [&](uint32_t x) {
          const uint32_t x4 = 4u * x + shift4, tag = x4 >> 12, y = *tag_word(x4, tag) ^ tag * ones;
          return ((y - ones) & ~y & tops) != 0;  // a field of zeros
        };
        cnt += __popc(valid & ((in(d.x) ? 8u : 0u) | (in(d.y) ? 4u : 0u) | (in(d.z) ? 2u : 0u) | (in(d.w) ? 1u : 0u)));
        return;
      }
      const uint32_t b0 = *word(d.x), b1 = *word(d.y), b2 = *word(d.z), b3 = *word(d.w);
      auto fold = [](uint32_t a, uint32_t b, uint32_t r) { return __funnelshift_l(__funnelshift_l(b, b, r), a, 1); };
      const unsigned hit = fold(fold(fold(fold(0u, b0, d.x), b1, d.y), b2, d.z), b3, d.w) & valid;
      if (exact) {
        cnt += __popc(hit);
      } else if (hit) {
        auto push = [&](unsigned bit, uint32_t x) {
          if (hit & bit) stacks[w][sp++][lane] = (int32_t)x;
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
          int a = 0, b = dh;  // the first member not below x
          while (a < b) {
            const int mid = (a + b) >> 1;
            if (__ldg(g.cols + hb + mid) < x) a = mid + 1; else b = mid;
          }
          cnt += a < dh && __ldg(g.cols + hb + a) == x;
        }
      sp = 0;
    };
    uint4 d0, d1;
    unsigned v0 = fetch(d0), v1;
    do {
      v1 = fetch(d1);
      tests(d0, v0);
      v0 = fetch(d0);
      tests(d1, v1);
      if (!exact && !tagged && __any_sync(0xffffffffu, sp > kRowStack - 8)) settle();
    } while (__any_sync(0xffffffffu, v0 != 0 || left > 0) || given < lim || from < ne);
    if (!exact && !tagged) settle();
    cnt = __reduce_add_sync(0xffffffffu, cnt);
    if (lane == 0) acc[w].part += cnt;
    for (int j = lane; j < dh; j += 32) {
      const uint32_t x = (uint32_t)__ldg(g.cols + hb + j), x4 = 4u * x + shift4;
      *(tagged ? tag_word(x4, x4 >> 12) : word(x)) = 0u;
    }
    __syncwarp();
  }
  graph_acc_flush(tags, &acc[w]);
}

bool same_shape(const ItemShape& a, const ItemShape& b) {
  return a.cutover == b.cutover && a.warp_max == b.warp_max && a.warp_chunk == b.warp_chunk &&
         a.block_chunk == b.block_chunk && a.by_source == b.by_source;
}

ItemShape shape_from(const atc_tuning* t, const ItemShape& base) {
  ItemShape sh = base;
  if (!t) return sh;
  if (t->bisson_cutover > 0) sh.cutover = std::min(t->bisson_cutover, kWarpMax);
  if (t->bisson_warp_max > 0) sh.warp_max = std::min(t->bisson_warp_max, kWarpHashMax);
  if (t->bisson_warp_chunk > 0) sh.warp_chunk = t->bisson_warp_chunk;
  if (t->bisson_block_chunk > 0) sh.block_chunk = t->bisson_block_chunk;
  if (t->group_by_source > 0) sh.by_source = t->group_by_source >= 2 ? 2 : 1;
  if (sh.cutover > sh.warp_max) sh.cutover = sh.warp_max;
  return sh;
}

// The shape of rows items for an asked-for shape: their kernel has no sorted copy, so a cutover means
// nothing to it, and chunks beyond kRowsChunk only lengthen its tail (six R-MAT graphs of scale 19 11.1 ms,
// with chunks of 512 12.9).
ItemShape rows_shape(ItemShape sh) {
  sh.by_source = 1;
  sh.cutover = 0;
  sh.warp_chunk = std::min(sh.warp_chunk, kRowsChunk);
  return sh;
}

// Mode 2: the graphs counted by rows.  ps, fitted to 105 batches of 1 to 48 R-MAT, Chung-Lu and random geometric
// graphs, each in both modes: rows cost per wedge (more in graphs of many ids, whose tags are wider), edge
// and vertex; grouping per element of the shorter lists, edge and vertex, and once for the whole batch
// what its hubs' cursors take, 8 us per member of the longest list (R-MAT scale 18, grouped, 1, 2 and 6 graphs 3.7,
// 4.3 and 7.5 ms).  In no batch slower than the choice by 1.097 W + 103.5 m against 1.232 W_min + 117.5 m that the
// earlier kernels were given; R-MAT scale 20 by rows / grouped: of 15.7M edges 17.1 / 8.6 ms, of 4.1M 1.65 / 2.3, six of those
// 7.1 / 5.4; 48 Chung-Lu graphs 2.3 / 5.2.
std::vector<bool> rows_graphs(const atc_batch* b) {
  constexpr double kHubPs = 8.0e6;
  const size_t ng = b->gm.size();
  std::vector<bool> rows(ng, true);
  double gain = 0.0;
  int32_t longest = 0;
  for (size_t q = 0; q < ng; ++q) {
    const double n = (double)(b->vbase[q + 1] - b->vbase[q]), m = (double)b->gm[q];
    const double by_rows = (n > 300000.0 ? 2.1 : 1.3) * (double)b->gw[q] + 10.0 * m + 350.0 * n;
    const double grouped = 1.2 * (double)b->gwmin[q] + 100.0 * m + 60.0 * n;
    if (by_rows <= grouped) continue;
    rows[q] = false;
    gain += by_rows - grouped;
    longest = std::max(longest, b->gmax[q]);
  }
  if (gain <= kHubPs * longest) rows.assign(ng, true);
  return rows;
}

// Sizes the scratch for the union and records the counting pipeline into a CUDA graph
// on the batch's own stream (capture is not allowed on the legacy default stream).
atc_status build_pipeline(atc_batch* b, const ItemShape& sh, cudaStream_t s) {  // by_source == 1: of rows_shape
  const int64_t n = b->n, m = b->m;
  const int ng = (int)(b->vbase.size() - 1);
  const bool mixed = sh.by_source == 2;
  const std::vector<bool> rows = mixed ? rows_graphs(b) : std::vector<bool>();
  int64_t nr = 0, mr = 0;  // vertices and edges of mode 2's rows graphs, which have no groups and items of their own
  for (int q = 0; mixed && q < ng; ++q)
    if (rows[q]) {
      nr += b->vbase[q + 1] - b->vbase[q];
      mr += b->gm[q];
    }
  const int64_t cap_items = max_items(n - nr, m - mr, std::min(sh.warp_chunk, sh.block_chunk));
  const int64_t cap_plist = sh.by_source == 1 ? 0 : m - mr;
  // block items of lists longer than kBlockSmallList: one per such list (at most
  // m / (kBlockSmallList + 1) of them) plus one per chunk boundary
  const int64_t big_cap = m / (kBlockSmallList + 1) + m / sh.block_chunk + 1;
  const ItemShape shr = rows_shape(sh);  // rows items of mode 2
  const int64_t cap_rows = mixed ? max_items(nr, mr, std::min(shr.warp_chunk, shr.block_chunk)) : 0;
  const bool same = b->built_n == n && b->built_m == m && b->built_graphs == ng;
  if (!same || b->items_cap < cap_items || b->rows_cap < cap_rows || b->plist_cap < cap_plist ||
      b->big_cap < big_cap) {
    // room for the shapes of before too, so that a change back and forth allocates once
    const int64_t items_cap = std::max(cap_items, same ? b->items_cap : 0);
    const int64_t rows_cap = std::max(cap_rows, same ? b->rows_cap : 0);
    const int64_t plist_cap = std::max(cap_plist, same ? b->plist_cap : 0);
    free_pipeline(b);
    ATC_TRY(dev_alloc(&b->cnt, (size_t)n + 1));
    ATC_TRY(dev_alloc(&b->cur, (size_t)n + 1));
    ATC_TRY(dev_alloc(&b->gstart, (size_t)n + 1));
    ATC_TRY(dev_alloc(&b->plist, (size_t)plist_cap + 32));
    ATC_TRY(dev_alloc(&b->items, (size_t)items_cap));
    ATC_TRY(dev_alloc(&b->counters, kBatchCounters));
    ATC_TRY(dev_alloc(&b->items_r, (size_t)rows_cap));
    ATC_TRY(dev_alloc(&b->counters_r, 8));
    ATC_TRY(dev_alloc(&b->vrows, (size_t)n + 1));
    ATC_TRY(dev_alloc(&b->big, (size_t)big_cap));
    ATC_TRY(dev_alloc(&b->big_r, (size_t)big_cap));
    ATC_TRY(dev_alloc(&b->vbase_d, (size_t)ng + 1));
    ATC_TRY(dev_alloc(&b->gcounts, (size_t)ng));
    size_t bytes = 0;
    ATC_TRY(exclusive_scan_i32_to_i64_tmp(nullptr, &bytes, b->cnt, b->gstart, (size_t)n + 1, s));
    ATC_TRY(dev_alloc(reinterpret_cast<char**>(&b->scan_tmp), bytes));
    ATC_CK(cudaMemcpyAsync(b->vbase_d, b->vbase.data(), sizeof(int64_t) * (ng + 1), cudaMemcpyHostToDevice, s));
    b->built_n = n;
    b->built_m = m;
    b->built_graphs = ng;
    b->items_cap = items_cap;
    b->rows_cap = rows_cap;
    b->plist_cap = plist_cap;
    b->big_cap = big_cap;
  } else if (b->exec) {
    cudaGraphExecDestroy(b->exec);
    cudaGraphDestroy(b->graph);
    b->exec = nullptr;
    b->graph = nullptr;
  }
  ATC_CK(cudaMemcpyAsync(b->off + n, &b->m, sizeof(int64_t), cudaMemcpyHostToDevice, s));
  ATC_CK(cudaStreamSynchronize(s));
  if (!b->cap_stream) ATC_CK(cudaStreamCreateWithFlags(&b->cap_stream, cudaStreamNonBlocking));

  // block tables: lists up to kBlockSmallList at load factor 1/4 (at most 32 KB), and the
  // full 64 KB table for the longer lists, launched apart so that the short lists' CTAs are
  // not held to the occupancy of the largest table
  const void* kblock = (const void*)bisson_block_kernel<CompactItems, kDefaultSlots>;
  uint32_t words = 64;
  const uint32_t want = 4u * (uint32_t)std::min(std::max(b->max_outdeg, 1), kBlockSmallList);
  while (words < want) words <<= 1;
  const bool any_big = b->max_outdeg > kBlockSmallList;
  const uint32_t words_big = kTabWords;
  const size_t smem = sizeof(int32_t) * words, smem_big = sizeof(int32_t) * words_big;
  ATC_CK(cudaFuncSetAttribute(kblock, cudaFuncAttributeMaxDynamicSharedMemorySize,
                              (int)(any_big ? smem_big : smem)));
  const int grid_block = sm_count() * blocks_per_sm(kblock, kBgWarps * 32, smem);
  const int grid_big = sm_count() * blocks_per_sm(kblock, kBgWarps * 32, smem_big);
  const int grid_warp = sm_count() * blocks_per_sm((const void*)bisson_warp_kernel<CompactItems, kDefaultSlots>, kBgWarps * 32, 0);

  CsrView g = csr_view(b->off, b->cols, nullptr, n, m);
  GraphTags tags{b->vbase_d, ng, b->gcounts};
  // grouped at the source, a vertex's partners are its own row: the items index the CSR
  // itself and the grouping passes are skipped
  const int64_t* gstart = sh.by_source == 1 ? b->off : b->gstart;
  const int32_t* plist = sh.by_source == 1 ? b->cols : b->plist;
  CompactItems witems{b->items, gstart, cap_items, false, false, sh};
  CompactItems bitems{b->items, gstart, cap_items, true, true, sh};
  CompactItems litems{b->big, gstart, big_cap, false, true, sh};
  // mode 2: each graph counts by rows (every wedge tested at its source, W tests, no grouping)
  // or grouped at the longer endpoint (sum of min(d+u, d+v) tests plus the grouping passes): rows_graphs
  CompactItems witems_r{b->items_r, b->off, cap_rows, false, false, shr};
  CompactItems bitems_r{b->items_r, b->off, cap_rows, true, true, shr};
  CompactItems litems_r{b->big_r, b->off, big_cap, false, true, shr};
  int nrows = 0;
  if (mixed) {
    ATC_CK(cudaMemsetAsync(b->vrows, 0, (size_t)n + 1, s));
    for (int q = 0; q < ng; ++q)
      if (rows[q] && b->vbase[q + 1] > b->vbase[q]) {
        ATC_CK(cudaMemsetAsync(b->vrows + b->vbase[q], 1, (size_t)(b->vbase[q + 1] - b->vbase[q]), s));
        ++nrows;
      }
    ATC_CK(cudaStreamSynchronize(s));
  }
  b->rows_graphs = mixed ? nrows : (sh.by_source == 1 ? ng : 0);
  const uint8_t* skip = mixed ? b->vrows : nullptr;
  cudaStream_t c = b->cap_stream;
  size_t bytes = 0;
  ATC_TRY(exclusive_scan_i32_to_i64_tmp(nullptr, &bytes, b->cnt, b->gstart, (size_t)n + 1, s));

  // event nodes between the stages (read by atc_phase_times after a replay)
  constexpr int kMaxStages = 12;
  while (b->stage_ev.size() < (size_t)kMaxStages + 1) {
    cudaEvent_t e = nullptr;
    ATC_CK(cudaEventCreate(&e));
    b->stage_ev.push_back(e);
  }
  b->stage_name.clear();
  int kernels = 0;
  auto stage = [&](const char* name) {
    b->stage_name.push_back(name);
    cudaEventRecordWithFlags(b->stage_ev[b->stage_name.size()], c, cudaEventRecordExternal);
  };

  ATC_CK(cudaStreamBeginCapture(c, cudaStreamCaptureModeThreadLocal));
  cudaEventRecordWithFlags(b->stage_ev[0], c, cudaEventRecordExternal);
  cudaMemsetAsync(b->cnt, 0, sizeof(int32_t) * (n + 1), c);
  cudaMemsetAsync(b->cur, 0, sizeof(int32_t) * (n + 1), c);
  cudaMemsetAsync(b->counters, 0, sizeof(int) * kBatchCounters, c);
  cudaMemsetAsync(b->gcounts, 0, sizeof(unsigned long long) * ng, c);
  stage("batch.reset");
  if (sh.by_source != 1) {
    group_count_vc_kernel<<<grid_for(n * 32, 256), 256, 0, c>>>(g, b->cnt, skip, b->counters + 8);
    exclusive_scan_i32_to_i64_tmp(b->scan_tmp, &bytes, b->cnt, b->gstart, (size_t)n + 1, c);
    group_scatter_vc_kernel<<<grid_for(n * 32, 256), 256, 0, c>>>(g, b->gstart, b->cur, b->plist, skip,
                                                                 b->counters + 9);
    kernels += 4;  // two grouping passes and the scan's two kernels
    stage("batch.group");
  }
  group_items_compact_kernel<<<grid_for(n, 256), 256, 0, c>>>(g, gstart, b->items, cap_items, b->big, b->counters, sh,
                                                              skip, 0);
  kernels += 3;  // items, block, warp
  stage("batch.items");
  bisson_block_kernel<CompactItems, kDefaultSlots><<<grid_block, kBgWarps * 32, smem, c>>>(g, ListPartners{plist}, bitems, 0, b->counters + 1,
                                                                            b->counters + 5, words, tags, b->gcounts);
  stage("batch.block");
  if (any_big) {
    bisson_block_kernel<CompactItems, kDefaultSlots><<<grid_big, kBgWarps * 32, smem_big, c>>>(
        g, ListPartners{plist}, litems, 0, b->counters + 2, b->counters + 6, words_big, tags, b->gcounts);
    kernels += 1;
    stage("batch.block.long");
  }
  const int grid_rows = sm_count() * blocks_per_sm((const void*)rows_kernel<kRowsLanes>, 128, 0);
  if (sh.by_source == 1)
    rows_kernel<kRowsLanes><<<grid_rows, 128, 0, c>>>(g, witems, b->counters, b->counters + 4, tags);
  else
    bisson_warp_kernel<CompactItems, kDefaultSlots><<<grid_warp, kBgWarps * 32, 0, c>>>(
        g, ListPartners{plist}, witems, 0, b->counters, b->counters + 4, tags, b->gcounts);
  stage("batch.warp");
  if (mixed && nrows > 0) {
    cudaMemsetAsync(b->counters_r, 0, sizeof(int) * 8, c);
    group_items_compact_kernel<<<grid_for(n, 256), 256, 0, c>>>(g, b->off, b->items_r, cap_rows, b->big_r,
                                                                b->counters_r, shr, b->vrows, 1);
    kernels += 3;
    stage("batch.rows.items");
    bisson_block_kernel<CompactItems, kDefaultSlots><<<grid_block, kBgWarps * 32, smem, c>>>(
        g, ListPartners{b->cols}, bitems_r, 0, b->counters_r + 1, b->counters_r + 5, words, tags, b->gcounts);
    stage("batch.rows.block");
    if (any_big) {
      bisson_block_kernel<CompactItems, kDefaultSlots><<<grid_big, kBgWarps * 32, smem_big, c>>>(
          g, ListPartners{b->cols}, litems_r, 0, b->counters_r + 2, b->counters_r + 6, words_big, tags, b->gcounts);
      kernels += 1;
      stage("batch.rows.block.long");
    }
    rows_kernel<kRowsLanes><<<grid_rows, 128, 0, c>>>(g, witems_r, b->counters_r, b->counters_r + 4, tags);
    stage("batch.rows.warp");
  }
  cudaError_t launch_err = cudaGetLastError();
  cudaError_t end_err = cudaStreamEndCapture(c, &b->graph);
  if (launch_err != cudaSuccess || end_err != cudaSuccess) {
    set_error("capturing the batch pipeline: %s", cudaGetErrorString(launch_err != cudaSuccess ? launch_err : end_err));
    if (b->graph) cudaGraphDestroy(b->graph);
    b->graph = nullptr;
    return ATC_ERR_CUDA;
  }
  ATC_CK(cudaGraphInstantiate(&b->exec, b->graph, 0));
  b->built_shape = sh;
  b->launches = kernels;
  b->dirty = false;
  return ATC_OK;
}

atc_status run_once(atc_batch* b, const ItemShape& asked, uint64_t* counts, float* ms, cudaStream_t s) {
  const ItemShape sh = asked.by_source == 1 ? rows_shape(asked) : asked;
  if (b->dirty || !b->exec || !same_shape(sh, b->built_shape)) ATC_TRY(build_pipeline(b, sh, s));
  EventTimer tm;
  tm.start(s);
  ATC_CK(cudaGraphLaunch(b->exec, s));
  tm.stop(s);
  const int ng = (int)(b->vbase.size() - 1);
  if (counts && ng) ATC_CK(cudaMemcpyAsync(counts, b->gcounts, sizeof(uint64_t) * ng, cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  if (ms) *ms = tm.ms();
  if (phase_timing_on()) {
    for (size_t k = 0; k < b->stage_name.size(); ++k) {
      float t = 0.f;
      ATC_CK(cudaEventElapsedTime(&t, b->stage_ev[k], b->stage_ev[k + 1]));
      phase_add(b->stage_name[k], t);
    }
  }
  return ATC_OK;
}

}  // namespace
}  // namespace atc

extern "C" atc_status atc_batch_run(atc_batch* b, const atc_tuning* t, uint64_t* counts, atc_stats* stats,
                                    atc_stream st) try {
  ATC_CHECK_ARG(b != nullptr, "NULL batch");
  const int ng = (int)(b->vbase.size() - 1);
  ATC_CHECK_ARG(counts != nullptr || ng == 0, "counts is NULL");
  if (ng == 0 || b->m == 0) {
    for (int i = 0; i < ng; ++i) counts[i] = 0;
    if (stats) memset(stats, 0, sizeof(*stats));
    return ATC_OK;
  }
  atc::ItemShape sh = atc::shape_from(t, b->shape);
  float ms = 0;
  atc::Phase ph("batch", as_stream(st));
  ATC_TRY(atc::run_once(b, sh, counts, &ms, as_stream(st)));
  if (stats) {
    memset(stats, 0, sizeof(*stats));
    stats->kernel_ms = ms;
    stats->total_ms = ms;
    stats->kernel_used = sh.by_source ? ATC_KERNEL_HU : ATC_KERNEL_BISSON;
    stats->launches = b->launches;
  }
  return ATC_OK;
} ATC_CATCH

extern "C" atc_status atc_batch_tune(atc_batch* b, const atc_tuning* cands, int32_t ncand, int32_t* best, float* ms,
                                     atc_stream st) try {
  ATC_CHECK_ARG(b != nullptr && cands != nullptr && ncand > 0 && best != nullptr, "bad argument");
  cudaStream_t s = as_stream(st);
  const int ng = (int)(b->vbase.size() - 1);
  if (ng == 0 || b->m == 0) {
    *best = 0;
    return ATC_OK;
  }
  std::vector<uint64_t> scratch(ng);
  float best_ms = 0;
  *best = 0;
  for (int i = 0; i < ncand; ++i) {
    atc::ItemShape sh = atc::shape_from(&cands[i], atc::default_shape(32));
    float t0 = 0, t1 = 0;
    ATC_TRY(atc::run_once(b, sh, scratch.data(), &t0, s));  // builds and warms
    ATC_TRY(atc::run_once(b, sh, scratch.data(), &t0, s));
    ATC_TRY(atc::run_once(b, sh, scratch.data(), &t1, s));
    float avg = 0.5f * (t0 + t1);
    if (ms) ms[i] = avg;
    if (i == 0 || avg < best_ms) {
      best_ms = avg;
      *best = i;
    }
  }
  b->shape = atc::shape_from(&cands[*best], atc::default_shape(32));
  return ATC_OK;
} ATC_CATCH
