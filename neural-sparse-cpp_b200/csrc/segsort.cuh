// Segmented sorts of the SEISMIC build (CUB), their scratch from an arena.
#ifndef NSP_SEGSORT_CUH
#define NSP_SEGSORT_CUH

#include <cub/device/device_segmented_sort.cuh>
#include <cuda_runtime.h>

#include <cstdint>
#include <stdexcept>

#include "engine.h"

namespace nsp {

template <class K, class V>
void segmented_sort_pairs(const K* kin, K* kout, const V* vin, V* vout, int64_t n,
                          int64_t segs, const int32_t* off, cudaStream_t s, bool stable,
                          Arena& scratch) {
    if (n == 0 || segs == 0) return;
    if (n > INT32_MAX || segs > INT32_MAX) throw std::invalid_argument("build batch too large");
    size_t tmp = 0;
    if (stable)
        cuda_check(cub::DeviceSegmentedSort::StableSortPairs(nullptr, tmp, kin, kout, vin, vout,
                                                             static_cast<int>(n), static_cast<int>(segs),
                                                             off, off + 1, s), "cub sort");
    else
        cuda_check(cub::DeviceSegmentedSort::SortPairs(nullptr, tmp, kin, kout, vin, vout,
                                                       static_cast<int>(n), static_cast<int>(segs),
                                                       off, off + 1, s), "cub sort");
    const Arena::Mark m = scratch.mark();
    uint8_t* t = scratch.take<uint8_t>(tmp + 16);
    if (stable)
        cuda_check(cub::DeviceSegmentedSort::StableSortPairs(t, tmp, kin, kout, vin, vout,
                                                             static_cast<int>(n), static_cast<int>(segs),
                                                             off, off + 1, s), "cub sort");
    else
        cuda_check(cub::DeviceSegmentedSort::SortPairs(t, tmp, kin, kout, vin, vout,
                                                       static_cast<int>(n), static_cast<int>(segs),
                                                       off, off + 1, s), "cub sort");
    scratch.release(m);
}

template <class K>
void segmented_sort_keys(const K* kin, K* kout, int64_t n, int64_t segs, const int32_t* off,
                         cudaStream_t s, Arena& scratch) {
    if (n == 0 || segs == 0) return;
    if (n > INT32_MAX || segs > INT32_MAX) throw std::invalid_argument("build batch too large");
    size_t tmp = 0;
    cuda_check(cub::DeviceSegmentedSort::SortKeys(nullptr, tmp, kin, kout, static_cast<int>(n),
                                                  static_cast<int>(segs), off, off + 1, s),
               "cub sort");
    const Arena::Mark m = scratch.mark();
    uint8_t* t = scratch.take<uint8_t>(tmp + 16);
    cuda_check(cub::DeviceSegmentedSort::SortKeys(t, tmp, kin, kout, static_cast<int>(n),
                                                  static_cast<int>(segs), off, off + 1, s),
               "cub sort");
    scratch.release(m);
}

}  // namespace nsp

#endif  // NSP_SEGSORT_CUH
