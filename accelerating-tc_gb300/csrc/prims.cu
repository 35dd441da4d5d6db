// Device-wide sort / unique / scan used by preTC.  The key sort is radix.cuh's; the rest are plain
// library primitives (CUB, shipped with the CUDA toolkit), in the role thrust::sort /
// thrust::unique / thrust::exclusive_scan play in the reference preprocessing
// (Hu/preTC.cu:208-212, tricount_gpu.cu:172-174, kcl.cu:197).
#include <cub/device/device_radix_sort.cuh>
#include <cub/device/device_scan.cuh>
#include <cub/device/device_select.cuh>
#include <thrust/iterator/transform_iterator.h>

#include "internal.cuh"
#include "radix.cuh"

namespace atc {

// The framework's own sort (radix.cuh) from here on; fewer keys are a single launch in CUB, against a
// clearing, a histogram, an offsets launch and the passes (figures in radix.cuh).
constexpr size_t kOwnSort = 1 << 12;

static atc_status library_sort(void* tmp, size_t* bytes, uint64_t* keys, uint64_t* alt, size_t n, int begin_bit,
                               int end_bit, uint64_t** sorted, cudaStream_t s) {
  cub::DoubleBuffer<uint64_t> db(keys, alt);
  ATC_CK(cub::DeviceRadixSort::SortKeys(tmp, *bytes, db, (int64_t)n, begin_bit, end_bit, s));
  if (sorted) *sorted = db.Current();
  return ATC_OK;
}

// Sorts with caller-provided temporary storage; *sorted = the buffer that holds the result.
// tmp == nullptr: *bytes receives the size needed.
atc_status sort_keys_u64_tmp(void* tmp, size_t* bytes, uint64_t* keys, uint64_t* alt, size_t n, int begin_bit,
                             int end_bit, uint64_t** sorted, cudaStream_t s) {
  if (n < kOwnSort || end_bit <= begin_bit) return library_sort(tmp, bytes, keys, alt, n, begin_bit, end_bit, sorted, s);
  ATC_CK(radix_sort_keys(tmp, bytes, keys, alt, n, begin_bit, end_bit, sorted, s));
  return ATC_OK;
}

atc_status sort_keys_u64(uint64_t*& keys, uint64_t*& alt, size_t n, int begin_bit, int end_bit, cudaStream_t s) {
  if (n <= 1) return ATC_OK;
  size_t tmp = 0, lib = 0;
  ATC_TRY(sort_keys_u64_tmp(nullptr, &tmp, keys, alt, n, begin_bit, end_bit, nullptr, s));
  DevBuf<char> t;
  uint64_t* sorted = nullptr;
  // up to 2^20 keys the library's scratch is the smaller one (0.18 bytes a key to 0.25 or, up to 2^18, one):
  // taken where the own one is refused, and under a budget, whose bytes do not come back
  const bool capped = alloc_budget_left() >= 0;
  if (capped) ATC_TRY(library_sort(nullptr, &lib, keys, alt, n, begin_bit, end_bit, nullptr, s));
  if ((!capped || tmp <= lib) && t.alloc(tmp, s) == ATC_OK) {
    ATC_TRY(sort_keys_u64_tmp(t.p, &tmp, keys, alt, n, begin_bit, end_bit, &sorted, s));
  } else {
    cudaGetLastError();
    ATC_TRY(library_sort(nullptr, &lib, keys, alt, n, begin_bit, end_bit, nullptr, s));
    ATC_TRY(t.alloc(lib, s));
    ATC_TRY(library_sort(t.p, &lib, keys, alt, n, begin_bit, end_bit, &sorted, s));
  }
  if (sorted != keys) {
    alt = keys;
    keys = sorted;
  }
  return ATC_OK;
}

atc_status sort_pairs_u64_i32(uint64_t*& keys, uint64_t*& kalt, int32_t*& vals, int32_t*& valt, size_t n, int begin_bit,
                             int end_bit, cudaStream_t s) {
  if (n <= 1) return ATC_OK;
  cub::DoubleBuffer<uint64_t> dk(keys, kalt);
  cub::DoubleBuffer<int32_t> dv(vals, valt);
  size_t tmp = 0;
  ATC_CK(cub::DeviceRadixSort::SortPairs(nullptr, tmp, dk, dv, (int64_t)n, begin_bit, end_bit, s));
  DevBuf<char> t;
  ATC_TRY(t.alloc(tmp, s));
  ATC_CK(cub::DeviceRadixSort::SortPairs(t.p, tmp, dk, dv, (int64_t)n, begin_bit, end_bit, s));
  if (dk.Current() != keys) {
    kalt = keys;
    keys = dk.Current();
  }
  if (dv.Current() != vals) {
    valt = vals;
    vals = dv.Current();
  }
  return ATC_OK;
}

atc_status unique_u64_async(const uint64_t* in, uint64_t* out, size_t n, int64_t* count, cudaStream_t s) {
  size_t tmp = 0;
  ATC_CK(cub::DeviceSelect::Unique(nullptr, tmp, in, out, count, (int64_t)n, s));
  DevBuf<char> t;
  ATC_TRY(t.alloc(tmp, s));
  ATC_CK(cub::DeviceSelect::Unique(t.p, tmp, in, out, count, (int64_t)n, s));
  return ATC_OK;
}

atc_status exclusive_scan_i64(const int64_t* in, int64_t* out, size_t n, cudaStream_t s) {
  if (n == 0) return ATC_OK;
  size_t tmp = 0;
  ATC_CK(cub::DeviceScan::ExclusiveSum(nullptr, tmp, in, out, (int64_t)n, s));
  DevBuf<char> t;
  ATC_TRY(t.alloc(tmp, s));
  ATC_CK(cub::DeviceScan::ExclusiveSum(t.p, tmp, in, out, (int64_t)n, s));
  return ATC_OK;
}

struct I32ToI64 {
  __host__ __device__ int64_t operator()(int32_t x) const { return (int64_t)x; }
};

atc_status exclusive_scan_i32_to_i64(const int32_t* in, int64_t* out, size_t n, cudaStream_t s) {
  if (n == 0) return ATC_OK;
  thrust::transform_iterator<I32ToI64, const int32_t*, int64_t> it(in, I32ToI64());
  size_t tmp = 0;
  ATC_CK(cub::DeviceScan::ExclusiveSum(nullptr, tmp, it, out, (int64_t)n, s));
  DevBuf<char> t;
  ATC_TRY(t.alloc(tmp, s));
  ATC_CK(cub::DeviceScan::ExclusiveSum(t.p, tmp, it, out, (int64_t)n, s));
  return ATC_OK;
}

// The same scan with caller-provided temporary storage (no allocation, so it can be
// recorded into a CUDA graph).  tmp == nullptr: *bytes receives the size needed.
atc_status exclusive_scan_i32_to_i64_tmp(void* tmp, size_t* bytes, const int32_t* in, int64_t* out, size_t n,
                                         cudaStream_t s) {
  thrust::transform_iterator<I32ToI64, const int32_t*, int64_t> it(in, I32ToI64());
  ATC_CK(cub::DeviceScan::ExclusiveSum(tmp, *bytes, it, out, (int64_t)n, s));
  return ATC_OK;
}

}  // namespace atc
