// Least-significant-digit radix sort of 64-bit keys, one pass over memory per eight bits: the published
// one-sweep method (Adinets and Merrill, "Onesweep: A Faster Least Significant Digit Radix Sort for GPUs",
// 2022; the decoupled look-back is Merrill and Garland's, 2016), in code of its own.
//
// preTC sorts its edges as 64-bit keys, which was half of its time.  Each pass reads and writes the
// keys once: a CTA takes a tile (tiles are handed out in order), ranks its keys by digit, learns
// where its keys of every digit go from the tiles before it (each tile publishes its digit counts,
// then their running sums; a thread per digit looks back, kLook tiles at a time, until it meets a
// running sum), and writes the tile out digit by digit through shared memory, so that the writes are
// runs of 32 keys on average.  The digits' totals of all passes come from one histogram pass.
// Stable.
//
// What bounds a pass is the ranking, not memory (9.1 ms for 2^28 keys in six passes; the bytes
// alone take 4.1).  With one warp match per key a pass took 1.8 times as long as with the table in
// shared memory that the lanes of one digit put their bits into; eight ballots were between the
// two.  A look at eight earlier tiles per step gave 3-7 % over one; 512 x 16 keys in two CTAs per SM
// and 384 x 16 in three are equal, nine-bit digits gain at 44 bits and lose at 40 and 48.
// Measured against CUB's sort (ms): 2^24 keys of 40 bits 0.58 to 0.89, 2^26 of 44 2.3 to 3.9, 2^28 of
// 48 9.1 to 15.4; 1.5 M of 34 0.11 to 0.15; 200 000 of 28 0.050 to 0.073, 8000 of 20 0.035 to 0.042, 4000 0.033
// to 0.038; fewer are one launch in CUB (2000 keys: 0.031 to 0.010).
//
// A wait for an earlier tile's counts ends by itself: tiles start in order and publish before they
// wait.  A thread that has still waited kWaitNs counts the tile's keys of its digit from the
// input, and goes on; no wait is without an end and no result depends on one.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

namespace atc {

namespace radix {

constexpr int kDigitBits = 8;
constexpr int kDigits = 1 << kDigitBits;
constexpr int kThreads = 512;
// Keys a thread: 16, or four up to kSmallSort keys, where tiles of 8192 would leave most SMs idle (200 000
// keys of 28 bits 58 -> 50 us, 32 000 of 20 bits 46 -> 35; 400 000 of 34 bits 70 and 70, 800 000 78 -> 91).
constexpr int kSmallItems = 4;
constexpr size_t kSmallSort = 1 << 18;
constexpr int kWarps = kThreads / 32;
constexpr int kMaxPasses = 8;
constexpr int kLook = 8;
constexpr uint64_t kWaitNs = 10000000ull;

struct Passes {
  int n;
  int shift[kMaxPasses], bits[kMaxPasses];
};

// [begin, end) cut into the fewest passes of at most eight bits, as even as can be.
inline Passes cut(int begin, int end) {
  Passes p{};
  p.n = (end - begin + kDigitBits - 1) / kDigitBits;
  for (int i = 0, at = begin; i < p.n; ++i) {
    p.bits[i] = (end - at + p.n - i - 1) / (p.n - i);
    p.shift[i] = at;
    at += p.bits[i];
  }
  return p;
}

__global__ void __launch_bounds__(512) histogram_kernel(const uint64_t* __restrict__ keys, uint64_t n, Passes ps,
                                                        unsigned long long* hist) {
  __shared__ unsigned h[kMaxPasses][kDigits];
  for (int i = threadIdx.x; i < kMaxPasses * kDigits; i += blockDim.x) (&h[0][0])[i] = 0;
  __syncthreads();
  const uint64_t stride = (uint64_t)gridDim.x * blockDim.x;
  for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n; i += stride) {
    const uint64_t k = keys[i];
#pragma unroll
    for (int p = 0; p < kMaxPasses; ++p)
      if (p < ps.n) atomicAdd(&h[p][(k >> ps.shift[p]) & ((1u << ps.bits[p]) - 1)], 1u);
  }
  __syncthreads();
  for (int i = threadIdx.x; i < ps.n * kDigits; i += blockDim.x)
    if ((&h[0][0])[i]) atomicAdd(&hist[i], (unsigned long long)(&h[0][0])[i]);
}

// hist[p] becomes its exclusive prefix sums: a CTA of kDigits threads per pass.
__global__ void __launch_bounds__(kDigits) offsets_kernel(unsigned long long* hist) {
  __shared__ unsigned long long s[kDigits];
  const int t = threadIdx.x;
  const unsigned long long v = hist[blockIdx.x * kDigits + t];
  s[t] = v;
  __syncthreads();
  for (int o = 1; o < kDigits; o <<= 1) {
    const unsigned long long y = t >= o ? s[t - o] : 0ull;
    __syncthreads();
    s[t] += y;
    __syncthreads();
  }
  hist[blockIdx.x * kDigits + t] = s[t] - v;
}

__device__ __forceinline__ uint64_t clock_ns() {
  uint64_t t;
  asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
  return t;
}

template <int kItems>
struct PassSmem {
  static constexpr int kTileKeys = kThreads * kItems;
  // a warp's match table (a word per digit, zero between uses) while ranking, then the tile's keys
  union {
    uint64_t keys[kTileKeys];
    unsigned match[kWarps][kDigits];
  };
  uint16_t cnt[kWarps][kDigits];     // keys of each digit per warp, then where the warp's keys of it start
  unsigned long long dest[kDigits];  // global position of keys[0] if it were of that digit
  unsigned wsum[kWarps];
  unsigned tile;
};

// state[tile * kDigits + digit]: the tile's keys of the digit with flag kCount, then those of all
// tiles up to it with kSum; the flags are S's top bits, and n < 2^(bits of S - 2).  ticket: the
// next tile.  next: the state of the next pass, cleared here when it is a buffer of its own.
template <typename S, int kItems>
__global__ void __launch_bounds__(kThreads, 2)
    pass_kernel(const uint64_t* __restrict__ in, uint64_t* __restrict__ out, uint64_t n, int shift, int bits,
                const unsigned long long* __restrict__ offsets, S* state, S* next, unsigned* ticket,
                uint64_t wait_ns) {
  constexpr int kTileKeys = kThreads * kItems;
  constexpr S kSum = (S)1 << (8 * sizeof(S) - 1), kCount = kSum >> 1, kValue = kCount - 1;
  extern __shared__ __align__(16) unsigned char raw[];
  PassSmem<kItems>& sm = *reinterpret_cast<PassSmem<kItems>*>(raw);
  const int t = threadIdx.x, lane = t & 31, w = t >> 5;
  const unsigned below = (1u << lane) - 1, mask = (1u << bits) - 1;
  if (t == 0) sm.tile = atomicAdd(ticket, 1u);
  for (int i = t; i < kWarps * kDigits; i += kThreads) (&sm.cnt[0][0])[i] = 0;
  for (int i = t; i < kWarps * kDigits; i += kThreads) (&sm.match[0][0])[i] = 0;
  __syncthreads();
  const uint64_t tile = sm.tile, base = tile * kTileKeys;
  const int valid = (int)min((uint64_t)kTileKeys, n - base);
  // a warp's keys are contiguous: key i of a lane is w * 32 kItems + 32 i + lane.  Those past the
  // end are all ones: last in the tile and of the last digit, so they rank behind every other
  uint64_t key[kItems];
  unsigned rank[kItems / 2];  // two 16-bit ranks
  const int first = w * 32 * kItems + lane;
  if (valid == kTileKeys) {
#pragma unroll
    for (int i = 0; i < kItems; ++i) key[i] = in[base + first + 32 * i];
  } else {
#pragma unroll
    for (int i = 0; i < kItems; ++i) key[i] = first + 32 * i < valid ? in[base + first + 32 * i] : ~0ull;
  }
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const unsigned d = (unsigned)(key[i] >> shift) & mask;
    atomicOr(&sm.match[w][d], 1u << lane);
    __syncwarp();
    const unsigned same = sm.match[w][d], at = sm.cnt[w][d];
    __syncwarp();
    if ((same & below) == 0) {
      sm.match[w][d] = 0;
      sm.cnt[w][d] = (uint16_t)(at + __popc(same));
    }
    const unsigned r = at + __popc(same & below);
    rank[i / 2] = i & 1 ? rank[i / 2] | r << 16 : r;
    __syncwarp();
  }
  __syncthreads();
  // a thread per digit: the warps' starts, the tile's count, the tiles before
  unsigned mine = 0;
  if (t < kDigits) {
#pragma unroll
    for (int q = 0; q < kWarps; ++q) {
      const unsigned c = sm.cnt[q][t];
      sm.cnt[q][t] = (uint16_t)mine;
      mine += c;
    }
    if (t == (int)mask) mine -= kTileKeys - valid;
    *(volatile S*)(state + tile * kDigits + t) = (tile == 0 ? kSum : kCount) | (S)mine;
    if (next) next[tile * kDigits + t] = 0;
  }
  // exclusive scan of the digits' counts over the first kDigits threads
  unsigned incl = mine;
#pragma unroll
  for (int o = 1; o < 32; o <<= 1) {
    const unsigned y = __shfl_up_sync(0xffffffffu, incl, o);
    if (lane >= o) incl += y;
  }
  if (lane == 31) sm.wsum[w] = incl;
  __syncthreads();
  if (t < kDigits) {
    unsigned start = incl - mine;
    for (int q = 0; q < w; ++q) start += sm.wsum[q];
#pragma unroll
    for (int q = 0; q < kWarps; ++q) sm.cnt[q][t] = (uint16_t)(sm.cnt[q][t] + start);
    S before = 0;
    if (tile > 0) {
      uint64_t t0 = clock_ns();
      int64_t p = (int64_t)tile - 1;
      for (bool found = false; !found;) {
        S v[kLook];
#pragma unroll
        for (int j = 0; j < kLook; ++j) v[j] = *(volatile S*)(state + max(p - j, (int64_t)0) * kDigits + t);
        int used = 0;
#pragma unroll
        for (int j = 0; j < kLook; ++j)
          if (!found && used == j && v[j]) {
            before += v[j] & kValue;
            ++used;
            found = (v[j] & kSum) != 0;  // tile 0 publishes a sum, so the walk ends there
          }
        p -= used;
        if (used) {
          t0 = clock_ns();
        } else if (clock_ns() - t0 > wait_ns) {
          const uint64_t* const q = in + p * kTileKeys;  // a tile before this one is full
          for (int j = 0; j < kTileKeys; ++j) before += ((unsigned)(q[j] >> shift) & mask) == (unsigned)t;
          found = --p < 0;
        }
      }
      *(volatile S*)(state + tile * kDigits + t) = kSum | (S)(before + mine);
    }
    sm.dest[t] = offsets[t] + before - start;
  }
  __syncthreads();
#pragma unroll
  for (int i = 0; i < kItems; ++i) {
    const unsigned d = (unsigned)(key[i] >> shift) & mask;
    sm.keys[sm.cnt[w][d] + (i & 1 ? rank[i / 2] >> 16 : rank[i / 2] & 0xffffu)] = key[i];
  }
  __syncthreads();
  if (valid == kTileKeys) {
#pragma unroll
    for (int i = 0; i < kItems; ++i) {
      const int j = t + i * kThreads;
      const uint64_t k = sm.keys[j];
      out[sm.dest[(unsigned)(k >> shift) & mask] + j] = k;
    }
  } else {
    for (int j = t; j < valid; j += kThreads) {
      const uint64_t k = sm.keys[j];
      out[sm.dest[(unsigned)(k >> shift) & mask] + j] = k;
    }
  }
}

}  // namespace radix

// Sorts n keys by bits [begin, end), end > begin; *sorted = the buffer holding the result.  tmp ==
// nullptr: *bytes receives the scratch needed.  wide: 64-bit tile states whatever n, for tests, as wait_ns is.
inline cudaError_t radix_sort_keys(void* tmp, size_t* bytes, uint64_t* keys, uint64_t* alt, size_t n, int begin, int end,
                                   uint64_t** sorted, cudaStream_t s, bool wide = false,
                                   uint64_t wait_ns = radix::kWaitNs) {
  using namespace radix;
  const Passes ps = cut(begin, end);
  wide = wide || n >= (1ull << 30);
  const int items = n <= kSmallSort && !wide ? kSmallItems : 16;
  const size_t tile = (size_t)kThreads * items, tiles = (n + tile - 1) / tile;
  const size_t head = 256;  // a ticket per pass
  const size_t hist = sizeof(unsigned long long) * kMaxPasses * kDigits;
  const size_t state = (wide ? 8 : 4) * kDigits * tiles;
  // Up to 2^20 keys a launch to clear the state costs more than a second buffer; beyond, one
  // buffer (an eighth of a byte per key) is cleared between passes.
  const bool two = n <= (1u << 20);
  if (!tmp) {
    *bytes = head + hist + (two ? 2 : 1) * state;
    return cudaSuccess;
  }
  char* p = static_cast<char*>(tmp);
  unsigned* ticket = reinterpret_cast<unsigned*>(p);
  unsigned long long* h = reinterpret_cast<unsigned long long*>(p + head);
  char* st = p + head + hist;
  cudaError_t e = cudaMemsetAsync(tmp, 0, head + hist + state, s);
  if (e != cudaSuccess) return e;
  int dev = 0, sms = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const size_t hgrid = (n + 512 * 16 - 1) / (512 * 16);
  histogram_kernel<<<(unsigned)(hgrid < (size_t)sms * 4 ? hgrid : (size_t)sms * 4), 512, 0, s>>>(keys, n, ps, h);
  offsets_kernel<<<ps.n, kDigits, 0, s>>>(h);
  uint64_t *a = keys, *b = alt;
  auto run = [&](auto kernel, auto zero, size_t smem) -> cudaError_t {
    using S = decltype(zero);
    const cudaError_t r =
        cudaFuncSetAttribute((const void*)kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
    if (r != cudaSuccess) return r;
    for (int i = 0; i < ps.n; ++i) {
      S* const mine = reinterpret_cast<S*>(st + (two && (i & 1) ? state : 0));
      S* const next = two ? reinterpret_cast<S*>(st + (i & 1 ? 0 : state)) : nullptr;
      if (!two && i > 0) {
        const cudaError_t c = cudaMemsetAsync(st, 0, state, s);
        if (c != cudaSuccess) return c;
      }
      kernel<<<(unsigned)tiles, kThreads, smem, s>>>(a, b, n, ps.shift[i], ps.bits[i], h + i * kDigits, mine,
                                         next, ticket + i, wait_ns);
      uint64_t* x = a;
      a = b;
      b = x;
    }
    return cudaSuccess;
  };
  e = items != 16 ? run(pass_kernel<unsigned, kSmallItems>, 0u, sizeof(PassSmem<kSmallItems>))
      : wide      ? run(pass_kernel<unsigned long long, 16>, 0ull, sizeof(PassSmem<16>))
                  : run(pass_kernel<unsigned, 16>, 0u, sizeof(PassSmem<16>));
  if (e != cudaSuccess) return e;
  if (sorted) *sorted = a;
  return cudaGetLastError();
}

}  // namespace atc
