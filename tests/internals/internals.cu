// Parts of the library that no call reaches at a test's size: rules that show in times only (a batch's item
// shapes, and which of its graphs are counted by rows), the sort's wide tile states and its recount of an
// earlier tile, the 64-bit row sort of the ranked copy, and a peel whose barrier wait runs out.  One
// section per argument; prints "ok" or what differs.
#include <cstdint>
#include <cstdio>
#include <cstring>
#include <random>
#include <vector>

#include "batch.cu"
#include "peel.cu"
#include "radix.cuh"
#include "ranked.cu"

using namespace atc;

#define REQUIRE(cond)                                   \
  do {                                                  \
    if (!(cond)) {                                      \
      std::printf("line %d: %s\n", __LINE__, #cond);    \
      return 1;                                         \
    }                                                   \
  } while (0)

// ---- no device needed ----------------------------------------------------------------
static int shapes() {
  const ItemShape base = default_shape(32);
  atc_tuning rows{}, mixed{}, wide{};
  rows.group_by_source = 1;
  mixed.group_by_source = 2;
  wide.group_by_source = 1;
  wide.bisson_cutover = 64;
  wide.bisson_warp_chunk = 2048;
  // a batch tuned to rows items and then run in the other mode has that mode's items
  const ItemShape tuned = shape_from(&rows, base), then = shape_from(&mixed, tuned);
  REQUIRE(same_shape(then, shape_from(&mixed, base)));
  // what rows items do not use makes no other shape; what they use does
  REQUIRE(same_shape(rows_shape(tuned), rows_shape(shape_from(&wide, base))));
  rows.bisson_warp_chunk = 32;
  REQUIRE(!same_shape(rows_shape(tuned), rows_shape(shape_from(&rows, base))));
  return 0;
}

// Which graphs of a batch are counted by rows, for batches of `graphs` equal graphs whose two modes were
// measured (ms by rows / grouped beside each).
static bool by_rows(int graphs, int64_t n, int64_t m, double w, double wmin, int32_t longest) {
  atc_batch b;
  for (int q = 0; q < graphs; ++q) {
    b.vbase.push_back(b.vbase.back() + n);
    b.gm.push_back(m);
    b.gw.push_back((int64_t)(w * (double)m));
    b.gwmin.push_back((int64_t)(wmin * (double)m));
    b.gmax.push_back(longest);
  }
  const std::vector<bool> rows = rows_graphs(&b);
  return rows.size() == (size_t)graphs && rows[0] && rows[graphs - 1];
}

static int choice() {
  REQUIRE(!by_rows(1, 1048576, 15701789, 286.8, 127.6, 615));  // R-MAT scale 20: 17.1 / 8.6
  REQUIRE(!by_rows(2, 1048576, 15700815, 292.3, 129.6, 615));  // 33.1 / 12.9
  REQUIRE(by_rows(1, 1048576, 4087819, 94.7, 39.3, 200));      // 1.65 / 2.34
  REQUIRE(!by_rows(6, 1048576, 4087656, 96.1, 39.7, 204));     // 7.1 / 5.4
  REQUIRE(by_rows(1, 262144, 3805211, 178.7, 86.9, 375));      // scale 18: 2.1 / 3.7
  REQUIRE(by_rows(6, 262144, 3805306, 181.6, 87.8, 375));      // 6.6 / 7.5
  REQUIRE(!by_rows(6, 262144, 7253730, 300.3, 150.4, 588));    // 18.9 / 16.5
  REQUIRE(by_rows(1, 2000000, 38453316, 51.3, 23.2, 136));     // Chung-Lu: 3.1 / 6.0
  REQUIRE(by_rows(48, 20000, 357849, 29.1, 18.9, 54));         // 1.0 / 2.6
  REQUIRE(by_rows(12, 500000, 5979693, 8.8, 8.4, 24));         // RGG: 4.0 / 5.5
  atc_batch none;
  REQUIRE(rows_graphs(&none).empty());
  return 0;
}

static int wait() {
  const uint64_t limit = 2000000000ull;
  PeelWait w{1000, 0};
  uint64_t now = 1000;
  // polls a microsecond apart reach the limit after that time
  int64_t polls = 0;
  while (!w.over(now += 1000, limit)) REQUIRE(++polls < 3000000);
  REQUIRE(now - 1000 > limit && now - 1000 <= limit + 2000);
  // a gap of any length between two polls is no delay of the other blocks
  w = PeelWait{1000, 0};
  REQUIRE(!w.over(60000000000ull, limit));
  REQUIRE(!w.over(60000001000ull, limit));
  return 0;
}

// ---- on the device -------------------------------------------------------------------
static int sort_case(size_t n, int bits, bool wide, uint64_t wait_ns, unsigned seed) {
  std::mt19937_64 rng(seed);
  std::vector<uint64_t> h(n);
  for (auto& x : h) x = rng() & ((1ull << bits) - 1);
  DevBuf<uint64_t> a, b;
  REQUIRE(a.alloc(n, nullptr) == ATC_OK && b.alloc(n, nullptr) == ATC_OK);
  REQUIRE(cudaMemcpy(a.p, h.data(), 8 * n, cudaMemcpyHostToDevice) == cudaSuccess);
  size_t bytes = 0;
  uint64_t* sorted = nullptr;
  REQUIRE(radix_sort_keys(nullptr, &bytes, a.p, b.p, n, 0, bits, nullptr, nullptr, wide, wait_ns) == cudaSuccess);
  DevBuf<char> tmp;
  REQUIRE(tmp.alloc(bytes, nullptr) == ATC_OK);
  REQUIRE(radix_sort_keys(tmp.p, &bytes, a.p, b.p, n, 0, bits, &sorted, nullptr, wide, wait_ns) == cudaSuccess);
  std::vector<uint64_t> got(n);
  REQUIRE(cudaMemcpy(got.data(), sorted, 8 * n, cudaMemcpyDeviceToHost) == cudaSuccess);
  std::sort(h.begin(), h.end());
  REQUIRE(got == h);
  return 0;
}

static int sorts() {
  for (size_t n : {size_t(1), size_t(2047), size_t(2049), size_t(1) << 18, (size_t(1) << 18) + 1, size_t(700001),
                   (size_t(1) << 20) + 8193, size_t(3) << 20})
    for (int wide = 0; wide < 2; ++wide)
      for (uint64_t wait_ns : {radix::kWaitNs, uint64_t(0)})
        if (sort_case(n, 21, wide != 0, wait_ns, (unsigned)n)) return 1;
  return 0;
}

// Rows of 0..40 ids (those above 32 are left to other kernels, as lists) by both key widths.
template <class Key>
static int row_sort(const std::vector<int64_t>& off, std::vector<int32_t> cols) {
  const int64_t n = (int64_t)off.size() - 1;
  DevBuf<int64_t> roff;
  DevBuf<int32_t> rcols, mid, big;
  DevBuf<int> ctr;
  REQUIRE(roff.alloc(n + 1, nullptr) == ATC_OK && rcols.alloc(cols.size(), nullptr) == ATC_OK &&
          mid.alloc(n, nullptr) == ATC_OK && big.alloc(n, nullptr) == ATC_OK && ctr.alloc(kcCount, nullptr) == ATC_OK);
  cudaMemcpy(roff.p, off.data(), 8 * off.size(), cudaMemcpyHostToDevice);
  cudaMemcpy(rcols.p, cols.data(), 4 * cols.size(), cudaMemcpyHostToDevice);
  cudaMemset(ctr.p, 0, sizeof(int) * kcCount);
  rank_sort_small_kernel<Key><<<grid_for(n, 256), 256>>>(roff.p, n, rcols.p, mid.p, big.p, ctr.p);
  REQUIRE(cudaDeviceSynchronize() == cudaSuccess);
  std::vector<int32_t> got(cols.size());
  cudaMemcpy(got.data(), rcols.p, 4 * cols.size(), cudaMemcpyDeviceToHost);
  for (int64_t u = 0; u < n; ++u)
    if (off[u + 1] - off[u] <= 32) std::sort(cols.begin() + off[u], cols.begin() + off[u + 1]);
  REQUIRE(got == cols);
  return 0;
}

static int rows() {
  std::mt19937 rng(5);
  for (int64_t n : {1, 31, 33, 5000}) {
    std::vector<int64_t> off(1, 0);
    std::vector<int32_t> cols;
    for (int64_t u = 0; u < n; ++u) {
      const int len = rng() % 4 ? rng() % 9 : rng() % 41;
      for (int j = 0; j < len; ++j) cols.push_back((int32_t)(rng() & 0x7ffffff));
      off.push_back((int64_t)cols.size());
    }
    cols.push_back(0);  // no row is empty-handed
    off.push_back((int64_t)cols.size());
    if (row_sort<uint32_t>(off, cols) || row_sort<uint64_t>(off, cols)) return 1;
    for (auto& x : cols) x |= 0x40000000;  // beyond the 27 bits of the narrow keys
    if (row_sort<uint64_t>(off, cols)) return 1;
  }
  return 0;
}

// A ring of n vertices with chords; its cores by the peel, with a wait that runs out and without.
static int peel() {
  const int64_t n = 1 << 18;
  SimpleEdges e;
  e.n_in = n;
  e.bits = id_bits(n);
  std::vector<uint64_t> keys;
  std::vector<int32_t> deg(n, 0);
  for (int64_t a = 0; a < n; ++a)
    for (int64_t s : {1, 2, 5}) {
      const int64_t b = a + s;
      if (b >= n) continue;
      keys.push_back((uint64_t)a << e.bits | (uint64_t)b);
      ++deg[a];
      ++deg[b];
    }
  e.m = (int64_t)keys.size();
  DevBuf<int32_t> d, rt, core;
  REQUIRE(e.keys.alloc(e.m, nullptr) == ATC_OK && d.alloc(n, nullptr) == ATC_OK && rt.alloc(n, nullptr) == ATC_OK &&
          core.alloc(n, nullptr) == ATC_OK);
  cudaMemcpy(e.keys.p, keys.data(), 8 * e.m, cudaMemcpyHostToDevice);
  cudaMemcpy(d.p, deg.data(), 4 * n, cudaMemcpyHostToDevice);
  std::vector<int32_t> want, got(n);
  for (int round = 0; round < 3; ++round) {
    PeelGraph g;
    REQUIRE(sym_graph(e, d.p, &g, nullptr) == ATC_OK);
    cudaMemcpy(rt.p, deg.data(), 4 * n, cudaMemcpyHostToDevice);
    cudaMemset(core.p, 0xff, 4 * n);
    PeelState st;
    const atc_status s = run_peel<true>(e, g, rt.p, core.p, 0.0f, 0, &st, nullptr, round == 1 ? 0 : kPeelWaitNs);
    REQUIRE(s == (round == 1 ? ATC_ERR_TIMEOUT : ATC_OK));
    if (round == 1) continue;
    cudaMemcpy(got.data(), core.p, 4 * n, cudaMemcpyDeviceToHost);
    if (round == 0) want = got;
    REQUIRE(got == want);
  }
  for (int64_t v = 1; v < n - 1; ++v) REQUIRE(want[v] == want[n / 2]);
  REQUIRE(want[n / 2] == 3);
  return 0;
}

int main(int argc, char** argv) {
  const char* const what = argc > 1 ? argv[1] : "";
  int r = 2;
  if (!strcmp(what, "shapes")) r = shapes();
  if (!strcmp(what, "choice")) r = choice();
  if (!strcmp(what, "wait")) r = wait();
  if (!strcmp(what, "sorts")) r = sorts();
  if (!strcmp(what, "rows")) r = rows();
  if (!strcmp(what, "peel")) r = peel();
  if (r == 0) std::printf("ok\n");
  return r;
}
