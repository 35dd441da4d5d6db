// A-direction peel on the GPU, level-synchronous.
//
// The reference peels serially (edge_directing/A-direction-seri.cpp:35-153): each outer
// step admits every unpeeled vertex whose runtime degree rt (twice its remaining degree)
// is <= a float threshold, then repeats waves in which every frontier vertex lowers rt of
// each unpeeled neighbour by 2 and a neighbour that reaches the threshold joins the next
// wave with the next priority.  Which vertices cross in a wave depends only on the set
// of frontier vertices (rt falls by exactly 2 per frontier neighbour until it crosses),
// never on the order the serial loop visits them, and the rt of already-peeled vertices
// (changed by the tie rule at :99-103) never feeds back into a priority.  A wave is
// therefore one parallel pass: atomicSub(rt[y], 2) on each unpeeled neighbour; the one
// subtraction that takes rt from above the threshold to at or below it admits y.  The
// float threshold arithmetic is the reference's (:37, :77, :127), in the same types.
#include <algorithm>
#include <climits>
#include <vector>

#include "internal.cuh"

namespace atc {

namespace {

// Symmetric adjacency from the sorted keys (a < b).  Keys of one smaller endpoint are
// contiguous, so a warp reserves each run's slots with one atomic (the loop is padded to
// whole warps for __match_any_sync); the larger endpoints are scattered one by one.
__global__ void sym_scatter_kernel(const uint64_t* keys, int64_t m, int B, unsigned long long* cur, int32_t* adj) {
  const uint64_t mask = (1ull << B) - 1;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  const int64_t m_pad = (m + 31) & ~31ll;
  const int lane = threadIdx.x & 31;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m_pad; i += stride) {
    int64_t a = -1;
    int32_t b = 0;
    if (i < m) {
      const uint64_t k = keys[i];
      a = (int64_t)(k >> B);
      b = (int32_t)(k & mask);
      adj[atomicAdd(&cur[b], 1ull)] = (int32_t)a;
    }
    const unsigned same = __match_any_sync(0xffffffffu, a);
    const int lead = __ffs(same) - 1;
    unsigned long long base = 0;
    if (a >= 0 && lane == lead) base = atomicAdd(&cur[a], (unsigned long long)__popc(same));
    base = __shfl_sync(0xffffffffu, base, lead);
    if (a >= 0) adj[base + __popc(same & ((1u << lane) - 1))] = b;
  }
}

__global__ void peel_init_kernel(const int32_t* deg, int64_t n, int32_t* rt, int32_t* prio) {
  int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += stride) {
    rt[v] = 2 * deg[v];
    prio[v] = -1;
  }
}

// ---- the peel loop as one persistent kernel ------------------------------------------------
// Both peels here (A-direction's and the k-core's) are a chain of short dependent steps: an outer
// scan that admits every unpeeled vertex at or below the limit, then waves until one admits
// nobody.  A step is a few microseconds of work, so launching each and reading its count back
// cost more than the work, and a wave whose frontier is one hub took as long as one warp needs to
// walk the hub's list.  Here one cooperative kernel runs all of them, its blocks meeting at a
// barrier after each step, and
//   - the frontier is a queue of (vertex, piece of kPeelPiece neighbours), so that a hub's list
//     is spread over as many warps as it has pieces; a warp lays several pieces' neighbours end to
//     end over its lanes, four rounds of loads and atomics in flight;
//   - a scan goes over the vertices that the last scan left unpeeled, and finds their smallest
//     remaining degree: the outer steps that would admit nobody are passed over;
//   - every wait at the barrier is bounded by the time it has polled: a block that gives up records it
//     and returns, and so do the others, one after another.
// Data that other blocks write is read past L1 (ld.global.cg).
// Measured, the whole peel (adjacency and loop): R-MAT scale 22 12.3 -> 4.0 ms (89 waves and 57
// scans; the loop 2.8, the adjacency 1.2), scale 20 5.0 -> 1.4, scale 17 2.3 -> 0.7.
constexpr int kPeelThreads = 512;
constexpr int kPeelPiece = 256;
constexpr uint64_t kPeelWaitNs = 2000000000ull;  // two seconds for one step of the other blocks
// The time between two looks at the clock counts as at most this: they are microseconds apart, unless the
// whole kernel was off the GPU in between (time slices of other processes, a debugger), which is no block's delay.
constexpr uint64_t kPeelPollNs = 1000000ull;
constexpr unsigned kPeelPolls = 16;  // polls per look at the clock

struct PeelStep {  // what one step's blocks count
  int admitted, alive, smallest;
  unsigned queued;
};
struct PeelState {
  PeelStep step[3];      // step t uses [t % 3] and clears [(t + 1) % 3]
  unsigned arrived;      // barrier
  int timed_out;         // a barrier wait ran out
  int stuck;             // the threshold stopped growing (A-direction)
  int waves;
  float threshold;
  long long peeled;
};

struct PeelArgs {
  const int64_t* off;
  const int32_t* adj;
  int64_t n;
  int32_t* rt;       // remaining degree (A-direction: twice it)
  int32_t* label;    // -1, then the priority (A-direction) or core number
  int2* queue;       // (vertex, piece)
  int32_t* alive[2];
  float threshold;   // A-direction
  int grow;          // A-direction: what the threshold grows by
  uint64_t wait_ns;  // limit of a wait at the barrier
  PeelState* st;
};

// A wait's time, poll by poll.
struct PeelWait {
  uint64_t last, waited;
  __host__ __device__ bool over(uint64_t now, uint64_t limit) {
    const uint64_t gap = now - last;
    waited += gap < kPeelPollNs ? gap : kPeelPollNs;
    last = now;
    return waited > limit;
  }
};

__device__ __forceinline__ uint64_t peel_clock_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

// All blocks of the (cooperative) launch; false when the wait ran out.
__device__ __forceinline__ bool peel_barrier(PeelState* st, uint64_t limit, unsigned* epoch) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    *epoch += gridDim.x;
    __threadfence();
    atomicAdd(&st->arrived, 1u);
    PeelWait wait{peel_clock_ns(), 0};
    ok = 1;
    for (unsigned polls = 1;; ++polls) {
      unsigned a;
      asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(a) : "l"(&st->arrived) : "memory");
      if ((int)(a - *epoch) >= 0) break;
      // the clock only now and then: on each poll it made a step of 3.6 us 3.9
      if (polls % kPeelPolls == 0 && wait.over(peel_clock_ns(), limit)) {
        st->timed_out = 1;
        ok = 0;
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

// Slots of a counter for k items on each lane, one atomic a warp (all 32 lanes call).
__device__ __forceinline__ unsigned peel_reserve(unsigned* ctr, int k) {
  const int lane = threadIdx.x & 31;
  int incl = k;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const int y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  unsigned base = 0;
  if (lane == 31 && incl) base = atomicAdd(ctr, (unsigned)incl);
  return __shfl_sync(0xffffffffu, base, 31) + (unsigned)(incl - k);
}

__device__ __forceinline__ int peel_pieces(const PeelArgs& a, int32_t v) {
  return (int)((__ldg(a.off + v + 1) - __ldg(a.off + v) + kPeelPiece - 1) / kPeelPiece);
}

// Queues the pieces of every v >= 0 from `tail` on, in step c (all 32 lanes call).
__device__ __forceinline__ void peel_enqueue(const PeelArgs& a, PeelStep* c, unsigned tail, int32_t v) {
  const int k = v >= 0 ? peel_pieces(a, v) : 0;
  const unsigned at = tail + peel_reserve(&c->queued, k);
  for (int j = 0; j < k; ++j) __stcg(a.queue + at + j, make_int2(v, j));
}

// CORE: k-core numbers (a neighbour loses 1, the limit jumps to the smallest remaining degree);
// otherwise A-direction priorities (a neighbour loses 2, the limit is the float threshold).
template <bool CORE>
__global__ void __launch_bounds__(kPeelThreads, 2) peel_kernel(PeelArgs a) {
  constexpr int kLoss = CORE ? 1 : 2;
  const int lane = threadIdx.x & 31;
  const int64_t threads = (int64_t)gridDim.x * kPeelThreads, tid = blockIdx.x * (int64_t)kPeelThreads + threadIdx.x;
  const unsigned warps = (unsigned)(threads >> 5), gw = (unsigned)(tid >> 5);
  PeelState* st = a.st;
  unsigned epoch = 0, head = 0, tail = 0;  // the frontier is queue[head, tail)
  int t = 0, waves = 0, cur = 0;  // cur: which alive list holds the unpeeled vertices
  int64_t n_alive = a.n, peeled = 0;
  bool first = true;
  float thr = a.threshold;
  int32_t k = 0, p = 0;
  auto within = [&](int32_t r) { return CORE ? r <= k : (float)r <= thr; };
  // ends step t: the blocks' counts of it
  auto finish_step = [&](int admitted, PeelStep* got) -> bool {
    PeelStep* c = &st->step[t % 3];
    admitted = __reduce_add_sync(0xffffffffu, admitted);
    if (lane == 0 && admitted) atomicAdd(&c->admitted, admitted);
    if (!peel_barrier(st, a.wait_ns, &epoch)) return false;
    got->admitted = __ldcg(&c->admitted);
    got->alive = __ldcg(&c->alive);
    got->smallest = __ldcg(&c->smallest);
    head = tail;
    tail += __ldcg(&c->queued);
    ++t;
    return true;
  };
  auto clear_next = [&]() {
    if (tid == 0) st->step[(t + 1) % 3] = PeelStep{0, 0, INT_MAX, 0u};
  };
  for (;;) {
    // outer step: admit every unpeeled vertex within the limit, keep the others
    clear_next();
    PeelStep got;
    {
      PeelStep* c = &st->step[t % 3];
      const int32_t* from = a.alive[cur];
      int32_t* to = a.alive[cur ^ 1];
      int admitted = 0, smallest = INT_MAX;
      const int64_t n_pad = (n_alive + 31) & ~31ll;
      for (int64_t i0 = tid; i0 < n_pad; i0 += 4 * threads) {
        int32_t v[4];
        bool keep[4];
        int kept = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int64_t i = i0 + q * threads;
          v[q] = -1;
          keep[q] = false;
          if (i < n_alive) v[q] = first ? (int32_t)i : __ldcg(from + i);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          int32_t in = -1;
          if (v[q] >= 0 && __ldcg(a.label + v[q]) == -1) {
            const int32_t r = __ldcg(a.rt + v[q]);
            if (within(r)) {
              in = v[q];
              __stcg(a.label + in, CORE ? k : p);
              ++admitted;
            } else {
              keep[q] = true;
              ++kept;
              smallest = min(smallest, r);
            }
          }
          if (__any_sync(0xffffffffu, in >= 0)) peel_enqueue(a, c, tail, in);
        }
        unsigned at = peel_reserve(reinterpret_cast<unsigned*>(&c->alive), kept);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (keep[q]) __stcg(to + at++, v[q]);
      }
      smallest = __reduce_min_sync(0xffffffffu, smallest);
      if (lane == 0 && smallest != INT_MAX) atomicMin(&c->smallest, smallest);
      if (!finish_step(admitted, &got)) return;
      first = false;
      cur ^= 1;
      n_alive = got.alive;
    }
    peeled += got.admitted;
    ++p;
    int32_t smallest = got.smallest;  // of the vertices left; stale once a wave lowers them
    while (got.admitted > 0) {  // also after a scan that admitted isolated vertices only
      // one wave: every unpeeled neighbour of a frontier vertex loses kLoss; the loss that takes
      // it from above the limit to within it admits it.  label only ever moves from -1, so a stale
      // -1 costs at most a harmless extra loss of an admitted vertex.
      clear_next();
      PeelStep* c = &st->step[t % 3];
      int admitted = 0;
      const unsigned nf = tail - head;
      const unsigned batch = min(max(nf / warps, 1u), 32u);
      for (unsigned b0 = gw * batch; b0 < nf; b0 += warps * batch) {
        int64_t xb = 0;
        int xd = 0;
        if (lane < (int)batch && b0 + lane < nf) {
          const int2 e = __ldcg(a.queue + head + b0 + lane);
          xb = __ldg(a.off + e.x) + (int64_t)e.y * kPeelPiece;
          xd = (int)min(__ldg(a.off + e.x + 1) - xb, (int64_t)kPeelPiece);
        }
        int incl = xd;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const int y = __shfl_up_sync(0xffffffffu, incl, o);
          if (lane >= o) incl += y;
        }
        const int total = __shfl_sync(0xffffffffu, incl, 31);
        const int start = incl - xd;
        for (int t0 = 0; t0 < total; t0 += 128) {
          int32_t y[4];
          int32_t old[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            y[q] = -1;
            if (t0 + 32 * q < total) {
              const int at = t0 + 32 * q + lane;
              int w = 0;  // the last lane whose piece starts at or before `at`
#pragma unroll
              for (int step = 16; step > 0; step >>= 1)
                if (__shfl_sync(0xffffffffu, start, w + step) <= at) w += step;
              const int64_t wb = __shfl_sync(0xffffffffu, xb, w);
              const int ws = __shfl_sync(0xffffffffu, start, w);
              if (at < total) y[q] = __ldg(a.adj + wb + (at - ws));
            }
          }
#pragma unroll
          for (int q = 0; q < 4; ++q)
            if (y[q] >= 0 && __ldcg(a.label + y[q]) != -1) y[q] = -1;
#pragma unroll
          for (int q = 0; q < 4; ++q) old[q] = y[q] >= 0 ? atomicSub(a.rt + y[q], kLoss) : INT_MIN;
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const bool in = y[q] >= 0 && !within(old[q]) && within(old[q] - kLoss);
            if (in) {
              __stcg(a.label + y[q], CORE ? k : p);
              ++admitted;
            }
            if (__any_sync(0xffffffffu, in)) peel_enqueue(a, c, tail, in ? y[q] : -1);
          }
        }
      }
      if (!finish_step(admitted, &got)) return;
      peeled += got.admitted;
      ++p;
      ++waves;
      smallest = -1;
    }
    if (peeled >= a.n) break;
    if (CORE) {
      // the smallest remaining degree is known when no wave has run since the scan; otherwise the
      // next level admits what it finds
      k = smallest > k ? smallest : k + 1;
    } else {
      // the outer steps up to the first that admits a vertex (one, when that is not known)
      do {
        const float grown = __fadd_rn(thr, (float)a.grow);
        if (!(grown > thr)) {
          if (tid == 0) {
            st->stuck = 1;
            st->threshold = thr;
            st->peeled = peeled;
          }
          return;
        }
        thr = grown;
        if (smallest < 0 || (float)smallest <= thr) break;
        ++p;
      } while (true);
    }
  }
  if (tid == 0) st->waves = waves;
}

// Symmetric adjacency of the simple graph (lists unsorted) and the peel loop over it.  rt and
// label are set up by the caller.
struct PeelGraph {
  DevBuf<int64_t> off;
  DevBuf<int32_t> adj;
  DevBuf<unsigned long long> cur;  // n: the scatter's cursors, then the peel's lists of the unpeeled
};

atc_status sym_graph(const SimpleEdges& e, const int32_t* deg, PeelGraph* g, cudaStream_t s) {
  const int64_t n = e.n_in, m = e.m, total = 2 * m;
  ATC_TRY(g->off.alloc(n + 1, s));
  ATC_TRY(exclusive_scan_i32_to_i64(deg, g->off.p, n, s));
  ATC_CK(cudaMemcpyAsync(g->off.p + n, &total, sizeof(total), cudaMemcpyHostToDevice, s));
  ATC_TRY(g->cur.alloc(n, s));
  ATC_CK(cudaMemcpyAsync(g->cur.p, g->off.p, sizeof(int64_t) * n, cudaMemcpyDeviceToDevice, s));
  ATC_TRY(g->adj.alloc(total, s));
  if (m) sym_scatter_kernel<<<grid_for(m, 256), 256, 0, s>>>(e.keys.p, m, e.bits, g->cur.p, g->adj.p);
  ATC_CK(cudaGetLastError());
  return ATC_OK;
}

template <bool CORE>
atc_status run_peel(const SimpleEdges& e, const PeelGraph& g, int32_t* rt, int32_t* label, float threshold, int grow,
                    PeelState* out, cudaStream_t s, uint64_t wait_ns = kPeelWaitNs) {
  const int64_t n = e.n_in, m = e.m;
  DevBuf<int2> queue;
  DevBuf<PeelState> st;
  // every vertex is queued once, in at most one piece more than its list has full ones
  ATC_TRY(queue.alloc((size_t)(n + 2 * m / kPeelPiece + 1), s));
  ATC_TRY(st.alloc(1, s));
  *out = PeelState{};
  out->step[0].smallest = INT_MAX;
  ATC_CK(cudaMemcpyAsync(st.p, out, sizeof(PeelState), cudaMemcpyHostToDevice, s));
  int32_t* const alive = reinterpret_cast<int32_t*>(g.cur.p);
  PeelArgs a{g.off.p, g.adj.p, n, rt, label, queue.p, {alive, alive + n}, threshold, grow, wait_ns, st.p};
  int bps = 0;
  ATC_CK(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&bps, peel_kernel<CORE>, kPeelThreads, 0));
  // about four vertices or sixteen neighbours a thread: more blocks only make the barrier dearer
  const int64_t want = (n / 4 + m / 8) / kPeelThreads + 1;
  unsigned grid = (unsigned)std::min<int64_t>(want, (int64_t)sm_count() * std::min(std::max(bps, 1), 2));
  void* args[] = {&a};
  for (;;) {
    const cudaError_t launched =
        cudaLaunchCooperativeKernel((const void*)peel_kernel<CORE>, dim3(grid), dim3(kPeelThreads), args, 0, s);
    // the stream may have fewer SMs than the device (a green context's): fewer blocks do as well
    if (launched != cudaErrorCooperativeLaunchTooLarge || grid == 1) {
      ATC_CK(launched);
      break;
    }
    cudaGetLastError();
    grid = (grid + 1) / 2;
  }
  ATC_CK(cudaMemcpyAsync(out, st.p, sizeof(PeelState), cudaMemcpyDeviceToHost, s));
  ATC_CK(cudaStreamSynchronize(s));
  if (out->timed_out) {
    set_error("a peel step did not end within its wait limit");
    return ATC_ERR_TIMEOUT;
  }
  return ATC_OK;
}

}  // namespace

atc_status peel_priorities(const SimpleEdges& e, const int32_t* deg, int32_t* prio, int* waves_out, cudaStream_t s) {
  Phase ph("peel", s);
  const int64_t n = e.n_in;
  *waves_out = 0;
  if (n == 0) return ATC_OK;
  PeelGraph g;  // the peel only needs neighbour sets
  ATC_TRY(sym_graph(e, deg, &g, s));
  DevBuf<int32_t> rt;
  ATC_TRY(rt.alloc(n, s));
  peel_init_kernel<<<grid_for(n, 256), 256, 0, s>>>(deg, n, rt.p, prio);
  ATC_CK(cudaGetLastError());
  // threshold arithmetic as A-direction-seri.cpp:37,77,127 (edgeNum = 2m as unsigned, nodeNum =
  // max id + 1 as int); the kernel goes on with the same float additions
  const unsigned edgeNum = (unsigned)(2 * e.m);
  const int nodeNum = (int)n;
  const float threshold = ((float)edgeNum) / nodeNum + 1;
  const int threshold_old = threshold;
  PeelState st;
  ATC_TRY(run_peel<false>(e, g, rt.p, prio, threshold, threshold_old, &st, s));
  if (st.stuck) {
    // float addition no longer moves the threshold: the serial reference would loop
    // forever here (runtime degrees above 2^24 are needed to get this far)
    set_error("A-direction threshold stopped growing at %g with %lld vertices unpeeled", (double)st.threshold,
              (long long)(n - st.peeled));
    return ATC_ERR_UNSUPPORTED;
  }
  *waves_out = st.waves;
  return ATC_OK;
}

// ---- Bisson's A-direction relabelling (Bisson/A-direction.cpp:43-163, 283-292) ----------
// The program peels serially over a doubled adjacency list and numbers the outer selection
// and every wave with one priority each (:91-126); the new ids sort the vertices by
// (priority, degreeRecord, id) and reverse the rank (:283-292).  degreeRecord is written at
// the selected vertex in the outer scan but at the frontier POSITION in the waves (:118),
// so it depends on the order in which the serial loop admits vertices.  That order is
// rebuilt here wave by wave, in parallel:
//   - the list of x (allEdges, :69-80) holds N(x) ∩ [0, x), then N(x), then N(x) ∩ (x, n),
//     each ascending, so a neighbour y sits at two known entries of it (first, second);
//   - an unpeeled y loses 1 per entry processed and is admitted at its k-th loss,
//     k = rt(y) - floor(threshold) (rt > threshold while unpeeled, so the loss that crosses
//     leaves rt exactly at the floor): that is entry (k odd ? first : second) of its
//     ceil(k/2)-th frontier neighbour in frontier order;
//   - the next frontier lists the admitted vertices by (position of that neighbour, entry);
//   - every admission writes degreeRecord[position] = floor(threshold); writes happen in
//     program order across waves, so the last one wins as in the serial program.
// Pairs (y, position of an adjacent frontier vertex) are radix-sorted per wave to find
// each y's ceil(k/2)-th frontier neighbour.
namespace {

__global__ void both_dir_keys_kernel(const uint64_t* keys, int64_t m, int B, uint64_t* out) {
  const uint64_t mask = (1ull << B) - 1;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m; i += stride) {
    const uint64_t k = keys[i], a = k >> B, b = k & mask;
    out[2 * i] = (a << B) | b;
    out[2 * i + 1] = (b << B) | a;
  }
}

// adj[j] = the low half of the sorted both-direction keys; nlow[x] = |N(x) ∩ [0, x)|.
__global__ void sorted_adj_kernel(const uint64_t* sk, int64_t m2, int B, int32_t* adj) {
  const uint64_t mask = (1ull << B) - 1;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < m2; i += stride)
    adj[i] = (int32_t)(sk[i] & mask);
}

__global__ void nlow_kernel(const int64_t* off, const int32_t* adj, int64_t n, int32_t* nlow) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t x = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; x < n; x += stride) {
    int64_t lo = off[x], hi = off[x + 1];
    const int64_t b = lo;
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (adj[mid] < (int32_t)x) lo = mid + 1; else hi = mid;
    }
    nlow[x] = (int32_t)(lo - b);
  }
}

__global__ void bis_init_kernel(const int32_t* deg, int64_t n, int32_t* rt, int32_t* prio, int32_t* drec) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += stride) {
    rt[v] = 2 * deg[v];
    prio[v] = -1;
    drec[v] = 0;
  }
}

// Outer selection (:89-98), in id order: flag, then (after a scan) place.
__global__ void bis_flag_kernel(const int32_t* rt, const int32_t* prio, int64_t n, float thr, int32_t* flag) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += stride)
    flag[v] = prio[v] == -1 && (float)rt[v] <= thr;
}

__global__ void bis_place_kernel(const int32_t* flag, const int64_t* pos, const int32_t* rt, int64_t n, int32_t P,
                                 int32_t* prio, int32_t* drec, int32_t* F) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += stride)
    if (flag[v]) {
      F[pos[v]] = (int32_t)v;
      prio[v] = P;
      drec[v] = rt[v];
    }
}

__global__ void bis_fdeg_kernel(const int32_t* F, int64_t nf, const int32_t* deg, int32_t* fd) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t p = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; p < nf; p += stride) fd[p] = deg[F[p]];
}

// (y << 32 | position, rank of y in N(x)) for every unpeeled neighbour y of frontier
// position p; peeled neighbours get the all-ones key, which sorts last.
__global__ void bis_emit_kernel(const int32_t* F, int64_t nf, const int64_t* fstart, const int64_t* off,
                                const int32_t* adj, const int32_t* prio, uint64_t* keys, int32_t* vals) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t p = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; p < nf; p += warps) {
    const int32_t x = F[p];
    const int64_t b = off[x], d = off[x + 1] - b, at = fstart[p];
    for (int64_t j = lane; j < d; j += 32) {
      const int32_t y = adj[b + j];
      keys[at + j] = prio[y] == -1 ? (((uint64_t)(uint32_t)y << 32) | (uint64_t)p) : ~0ull;
      vals[at + j] = (int32_t)j;
    }
  }
}

// One thread per segment start of the sorted pairs: admit y at its k-th loss, or take
// away 2 per adjacent frontier vertex.  cand gets (position << 32 | entry, y).
__global__ void bis_admit_kernel(const uint64_t* keys, const int32_t* vals, int64_t total, const int32_t* F,
                                 const int32_t* deg, const int32_t* nlow, int32_t T, int32_t P, int32_t* rt,
                                 int32_t* prio, int32_t* drec, uint64_t* ckeys, int32_t* cvals, int* ccount) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < total; i += stride) {
    const uint64_t key = keys[i];
    if (key == ~0ull) continue;
    const uint32_t y = (uint32_t)(key >> 32);
    if (i > 0 && (uint32_t)(keys[i - 1] >> 32) == y) continue;  // not a segment start
    int64_t lo = i + 1, hi = total;  // first pair of another vertex (the sentinels too)
    while (lo < hi) {
      const int64_t mid = (lo + hi) >> 1;
      if (keys[mid] != ~0ull && (uint32_t)(keys[mid] >> 32) == y) lo = mid + 1; else hi = mid;
    }
    const int64_t c = lo - i;
    const int32_t k = rt[y] - T;  // >= 1
    if (2 * c >= (int64_t)k) {
      const int64_t cross = i + (k + 1) / 2 - 1;
      const uint32_t p = (uint32_t)(keys[cross] & 0xffffffffull);
      const int32_t r = vals[cross];
      const int32_t x = F[p];
      const int32_t nl = nlow[x];
      const int32_t entry = (k & 1) ? ((int32_t)y < x ? r : nl + r) : ((int32_t)y < x ? nl + r : deg[x] + r);
      prio[y] = P;
      rt[y] = T;
      drec[p] = T;  // :118 writes at the frontier position
      const int at = atomicAdd(ccount, 1);
      ckeys[at] = ((uint64_t)p << 32) | (uint32_t)entry;
      cvals[at] = (int32_t)y;
    } else {
      rt[y] -= (int32_t)(2 * c);
    }
  }
}

__global__ void bis_rank_keys_kernel(const int32_t* prio, const int32_t* drec, int64_t n, uint64_t* keys, int32_t* ids) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += stride) {
    keys[v] = ((uint64_t)(uint32_t)prio[v] << 32) | (uint32_t)drec[v];
    ids[v] = (int32_t)v;
  }
}

__global__ void bis_lookup_kernel(const int32_t* ids, int64_t n, int32_t* lookup) {
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += stride)
    lookup[ids[i]] = (int32_t)(n - 1 - i);
}

}  // namespace

atc_status bisson_adirection_lookup(const SimpleEdges& e, const int32_t* deg, int32_t* lookup, cudaStream_t s) {
  Phase ph("bisson_adirection", s);
  const int64_t n = e.n_in, m = e.m, m2 = 2 * m;
  if (n == 0) return ATC_OK;
  DevBuf<int64_t> off, fstart, pos;
  DevBuf<int32_t> adj, nlow, rt, prio, drec, fa, fb, flag, fd, va, vb, cva, cvb;
  DevBuf<uint64_t> ka, kb, cka, ckb;
  DevBuf<int> cnt;
  // sorted symmetric adjacency
  ATC_TRY(off.alloc(n + 1, s));
  ATC_TRY(exclusive_scan_i32_to_i64(deg, off.p, n, s));
  ATC_CK(cudaMemcpyAsync(off.p + n, &m2, sizeof(m2), cudaMemcpyHostToDevice, s));
  // ka/kb/va/vb: the both-direction keys, each wave's (y, position) pairs (at most 2m) and
  // the final (priority, degreeRecord) keys of all n vertices
  const int64_t cap = std::max(m2, n) + 1;
  ATC_TRY(adj.alloc(m2 + 1, s));
  ATC_TRY(ka.alloc(cap, s));
  ATC_TRY(kb.alloc(cap, s));
  if (m) {
    both_dir_keys_kernel<<<grid_for(m, 256), 256, 0, s>>>(e.keys.p, m, e.bits, ka.p);
    ATC_CK(cudaGetLastError());
    uint64_t* k0 = ka.p;
    uint64_t* k1 = kb.p;
    ATC_TRY(sort_keys_u64(k0, k1, m2, 0, 2 * e.bits, s));
    sorted_adj_kernel<<<grid_for(m2, 256), 256, 0, s>>>(k0, m2, e.bits, adj.p);
    ATC_CK(cudaGetLastError());
  }
  ATC_TRY(nlow.alloc(n, s));
  nlow_kernel<<<grid_for(n, 256), 256, 0, s>>>(off.p, adj.p, n, nlow.p);
  ATC_TRY(rt.alloc(n, s));
  ATC_TRY(prio.alloc(n, s));
  ATC_TRY(drec.alloc(n, s));
  bis_init_kernel<<<grid_for(n, 256), 256, 0, s>>>(deg, n, rt.p, prio.p, drec.p);
  ATC_CK(cudaGetLastError());
  ATC_TRY(fa.alloc(n + 1, s));
  ATC_TRY(fb.alloc(n + 1, s));
  ATC_TRY(flag.alloc(n + 1, s));
  ATC_TRY(pos.alloc(n + 1, s));
  ATC_TRY(fd.alloc(n + 1, s));
  ATC_TRY(fstart.alloc(n + 1, s));
  ATC_TRY(va.alloc(cap, s));
  ATC_TRY(vb.alloc(cap, s));
  ATC_TRY(cka.alloc(n + 1, s));
  ATC_TRY(ckb.alloc(n + 1, s));
  ATC_TRY(cva.alloc(n + 1, s));
  ATC_TRY(cvb.alloc(n + 1, s));
  ATC_TRY(cnt.alloc(1, s));

  // threshold arithmetic of :45, :83, :138 on the host (edgeNum = 2m, nodeNum = max id + 1)
  const unsigned edgeNum = (unsigned)m2;
  const int nodeNum = (int)n;
  float threshold = ((float)edgeNum) / nodeNum + 1;
  const int threshold_old = threshold;
  int32_t P = 0;
  int64_t peeled = 0;
  int32_t* F = fa.p;
  int32_t* N = fb.p;
  for (;;) {
    // outer selection in id order
    ATC_CK(cudaMemsetAsync(flag.p + n, 0, sizeof(int32_t), s));
    bis_flag_kernel<<<grid_for(n, 256), 256, 0, s>>>(rt.p, prio.p, n, threshold, flag.p);
    ATC_CK(cudaGetLastError());
    ATC_TRY(exclusive_scan_i32_to_i64(flag.p, pos.p, n + 1, s));
    bis_place_kernel<<<grid_for(n, 256), 256, 0, s>>>(flag.p, pos.p, rt.p, n, P, prio.p, drec.p, F);
    ATC_CK(cudaGetLastError());
    int64_t nf = 0;
    ATC_CK(cudaMemcpyAsync(&nf, pos.p + n, sizeof(nf), cudaMemcpyDeviceToHost, s));
    ATC_CK(cudaStreamSynchronize(s));
    peeled += nf;
    ++P;
    const int32_t T = (int32_t)floorf(threshold);
    while (nf > 0) {
      // pairs (y, position) of the unpeeled neighbours of the frontier
      bis_fdeg_kernel<<<grid_for(nf, 256), 256, 0, s>>>(F, nf, deg, fd.p);
      ATC_CK(cudaMemsetAsync(fd.p + nf, 0, sizeof(int32_t), s));
      ATC_CK(cudaGetLastError());
      ATC_TRY(exclusive_scan_i32_to_i64(fd.p, fstart.p, nf + 1, s));
      int64_t total = 0;
      ATC_CK(cudaMemcpyAsync(&total, fstart.p + nf, sizeof(total), cudaMemcpyDeviceToHost, s));
      ATC_CK(cudaStreamSynchronize(s));
      ATC_CK(cudaMemsetAsync(cnt.p, 0, sizeof(int), s));
      if (total > 0) {
        bis_emit_kernel<<<grid_for(nf * 32, 256), 256, 0, s>>>(F, nf, fstart.p, off.p, adj.p, prio.p, ka.p, va.p);
        ATC_CK(cudaGetLastError());
        uint64_t* k0 = ka.p;
        uint64_t* k1 = kb.p;
        int32_t* v0 = va.p;
        int32_t* v1 = vb.p;
        ATC_TRY(sort_pairs_u64_i32(k0, k1, v0, v1, total, 0, 64, s));
        bis_admit_kernel<<<grid_for(total, 256), 256, 0, s>>>(k0, v0, total, F, deg, nlow.p, T, P, rt.p, prio.p,
                                                              drec.p, cka.p, cva.p, cnt.p);
        ATC_CK(cudaGetLastError());
      }
      int hc = 0;
      ATC_CK(cudaMemcpyAsync(&hc, cnt.p, sizeof(int), cudaMemcpyDeviceToHost, s));
      ATC_CK(cudaStreamSynchronize(s));
      // the next frontier in admission order
      uint64_t* c0 = cka.p;
      uint64_t* c1 = ckb.p;
      int32_t* w0 = cva.p;
      int32_t* w1 = cvb.p;
      ATC_TRY(sort_pairs_u64_i32(c0, c1, w0, w1, (size_t)hc, 0, 64, s));
      if (hc) ATC_CK(cudaMemcpyAsync(N, w0, sizeof(int32_t) * hc, cudaMemcpyDeviceToDevice, s));
      std::swap(F, N);
      nf = hc;
      peeled += nf;
      ++P;
    }
    if (peeled >= n) break;
    const float grown = threshold + threshold_old;
    if (!(grown > threshold)) {
      set_error("Bisson A-direction threshold stopped growing at %g with %lld vertices unpeeled", (double)threshold,
                (long long)(n - peeled));
      return ATC_ERR_UNSUPPORTED;
    }
    threshold = grown;
  }
  // new id = nodeNum - 1 - rank of (priority, degreeRecord, id)
  {
    uint64_t* k0 = ka.p;
    uint64_t* k1 = kb.p;
    int32_t* v0 = va.p;
    int32_t* v1 = vb.p;
    bis_rank_keys_kernel<<<grid_for(n, 256), 256, 0, s>>>(prio.p, drec.p, n, k0, v0);
    ATC_CK(cudaGetLastError());
    ATC_TRY(sort_pairs_u64_i32(k0, k1, v0, v1, n, 0, 64, s));
    bis_lookup_kernel<<<grid_for(n, 256), 256, 0, s>>>(v0, n, lookup);
    ATC_CK(cudaGetLastError());
  }
  ATC_CK(cudaStreamSynchronize(s));
  return ATC_OK;
}

// ---- k-core numbers (for the k-core direction, edge_directing/kcore_direction.cpp:91-146) ----
// Level-synchronous peeling: at level k every vertex whose remaining degree is <= k
// leaves with core number k, each leaving vertex lowers its remaining neighbours by 1,
// and the level repeats until nothing more leaves; k then jumps to the smallest
// remaining degree.  Which vertices leave at a level does not depend on the order, so
// the core numbers equal the sequential Batagelj-Zaversnik result.  (The reference tool
// counts degrees over the first node_num edges only, :35-38; this uses the true degrees.)
atc_status core_numbers(const SimpleEdges& e, const int32_t* deg, int32_t* core, cudaStream_t s) {
  const int64_t n = e.n_in;
  if (n == 0) return ATC_OK;
  PeelGraph g;
  ATC_TRY(sym_graph(e, deg, &g, s));
  DevBuf<int32_t> rt;
  ATC_TRY(rt.alloc(n, s));
  ATC_CK(cudaMemcpyAsync(rt.p, deg, sizeof(int32_t) * n, cudaMemcpyDeviceToDevice, s));
  ATC_CK(cudaMemsetAsync(core, 0xff, sizeof(int32_t) * n, s));
  PeelState st;
  return run_peel<true>(e, g, rt.p, core, 0.0f, 0, &st, s);
}

// ---- approximate parallel peel (edge_directing/A-direction-parallel/peel.cu:130-317) ----
// Frontier-synchronous: a frontier is every unpeeled vertex whose runtime degree (simple
// degree minus peeled neighbours, uint32) is <= a limit; it gets the iteration number as
// its major priority and its runtime degree as minor priority.  The limit starts at
// (uint32)(m / n) and grows by that step when a frontier comes out empty or small
// (peel.cu:239-246, 255); the loop stops at 90 % of the vertices, depth 255 or 50
// iterations (:217), and the vertices left keep flag 0xFFFFFFFF and their simple degree.
// Which vertices join a frontier depends only on the set of the previous frontier, so
// the atomic order inside a pass does not matter.
namespace {

constexpr uint32_t kUnpeeled = 0xFFFFFFFFu;

__global__ void apeel_init_kernel(const int32_t* deg, int64_t n, uint32_t* rd, uint32_t* flags, uint32_t* minor) {
  for (int64_t v = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; v < n; v += (int64_t)gridDim.x * blockDim.x) {
    rd[v] = (uint32_t)deg[v];
    minor[v] = (uint32_t)deg[v];
    flags[v] = kUnpeeled;
  }
}

// peel.cu:95-117 (advance + back_nbr_count): every unpeeled neighbour w of a frontier
// vertex loses one runtime degree per frontier neighbour.  The lists are symmetric and
// duplicate-free, so counting from the frontier side gives the same sums.
__global__ void apeel_lower_kernel(const int32_t* frontier, int nf, const int64_t* off, const int32_t* adj,
                                   const uint32_t* flags, uint32_t* rd) {
  const int lane = threadIdx.x & 31;
  const int64_t warps = ((int64_t)gridDim.x * blockDim.x) >> 5;
  for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < nf; i += warps) {
    const int32_t u = frontier[i];
    for (int64_t j = off[u] + lane; j < off[u + 1]; j += 32) {
      const int32_t w = adj[j];
      if (flags[w] == kUnpeeled) atomicSub(&rd[w], 1u);
    }
  }
}

// peel.cu:239-262: frontier = {v : rd[v] <= limit} (peeled vertices hold rd = 0xFFFFFFFF);
// each member takes flag `it`, minor = rd, rd = 0xFFFFFFFF.  Counts only when `assign` is 0.
// Whole warps step through the ids together so the ballot covers all 32 lanes.
__global__ void apeel_select_kernel(uint32_t* rd, uint32_t* flags, uint32_t* minor, int64_t n, uint32_t limit,
                                    uint32_t it, int assign, int32_t* frontier, int* count) {
  const int lane = threadIdx.x & 31;
  const int64_t stride = (int64_t)gridDim.x * blockDim.x;
  for (int64_t v0 = blockIdx.x * (int64_t)blockDim.x + threadIdx.x - lane; v0 < n; v0 += stride) {
    const int64_t v = v0 + lane;
    const uint32_t r = v < n ? rd[v] : 0u;
    const bool in = v < n && r <= limit;
    const unsigned ballot = __ballot_sync(0xffffffffu, in);
    if (!ballot) continue;
    int base = 0;
    if (lane == 0) base = atomicAdd(count, __popc(ballot));
    base = __shfl_sync(0xffffffffu, base, 0);
    if (in && assign) {
      frontier[base + __popc(ballot & ((1u << lane) - 1))] = (int32_t)v;
      flags[v] = it;
      minor[v] = r;
      rd[v] = kUnpeeled;
    }
  }
}

}  // namespace

atc_status approx_peel(const SimpleEdges& e, const int32_t* deg, uint32_t* flags, uint32_t* minor, int* iters_out,
                       cudaStream_t s) {
  const int64_t n = e.n_in, m = e.m;
  if (iters_out) *iters_out = 0;
  if (n == 0) return ATC_OK;
  PeelGraph g;
  DevBuf<int32_t> fr;
  DevBuf<uint32_t> rd;
  DevBuf<int> cnt;
  ATC_TRY(sym_graph(e, deg, &g, s));
  ATC_TRY(rd.alloc(n, s));
  ATC_TRY(fr.alloc(n, s));
  ATC_TRY(cnt.alloc(1, s));
  apeel_init_kernel<<<grid_for(n, 256), 256, 0, s>>>(deg, n, rd.p, flags, minor);
  ATC_CK(cudaGetLastError());

  // host arithmetic in the reference's types: float threshold, uint32 limits and counts
  const uint32_t node_num = (uint32_t)n, edge_num = (uint32_t)(2 * m);
  const float deg_thre = (float)edge_num / 2 / node_num;
  const uint32_t step = (uint32_t)deg_thre;
  const uint32_t stop_at = node_num * 9 / 10;
  int hcnt = 0;
  auto select = [&](uint32_t limit, uint32_t it, int assign, int* nf) -> atc_status {
    ATC_CK(cudaMemsetAsync(cnt.p, 0, sizeof(int), s));
    apeel_select_kernel<<<grid_for(n, 256), 256, 0, s>>>(rd.p, flags, minor, n, limit, it, assign, fr.p, cnt.p);
    ATC_CK(cudaGetLastError());
    ATC_CK(cudaMemcpyAsync(&hcnt, cnt.p, sizeof(int), cudaMemcpyDeviceToHost, s));
    ATC_CK(cudaStreamSynchronize(s));
    *nf = hcnt;
    return ATC_OK;
  };
  int f_size = 0;
  ATC_TRY(select(step, 1, 1, &f_size));
  uint32_t visited = (uint32_t)f_size;
  uint32_t depth = 1, it = 1;
  while (visited < stop_at && depth < 0xFF && it < 50) {
    ++it;
    if (f_size)
      apeel_lower_kernel<<<grid_for((int64_t)f_size * 32, 256), 256, 0, s>>>(fr.p, f_size, g.off.p, g.adj.p, flags, rd.p);
    ATC_CK(cudaGetLastError());
    int cand = 0;
    ATC_TRY(select(step * depth, it, 0, &cand));
    while (cand == 0 && depth < 0xFF && visited < stop_at) {
      ++depth;
      ATC_TRY(select(step * depth, it, 0, &cand));
    }
    ATC_TRY(select(step * depth, it, 1, &f_size));
    visited += (uint32_t)f_size;
    if ((uint32_t)f_size <= node_num / 500) ++depth;
  }
  if (iters_out) *iters_out = (int)it;
  return ATC_OK;
}

}  // namespace atc
