// Segmented sorts of the SEISMIC build (CUB), with an optional pooled scratch.
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
                          DevArray<uint8_t>* pool = nullptr) {
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
    DevArray<uint8_t> own;
    DevArray<uint8_t>& t = pool != nullptr ? *pool : own;
    t.grow(tmp + 16);
    if (stable)
        cuda_check(cub::DeviceSegmentedSort::StableSortPairs(t.data(), tmp, kin, kout, vin, vout,
                                                             static_cast<int>(n), static_cast<int>(segs),
                                                             off, off + 1, s), "cub sort");
    else
        cuda_check(cub::DeviceSegmentedSort::SortPairs(t.data(), tmp, kin, kout, vin, vout,
                                                       static_cast<int>(n), static_cast<int>(segs),
                                                       off, off + 1, s), "cub sort");
    if (pool == nullptr) cuda_check(cudaStreamSynchronize(s), "sort sync");
}

template <class K>
void segmented_sort_keys(const K* kin, K* kout, int64_t n, int64_t segs, const int32_t* off,
                         cudaStream_t s, DevArray<uint8_t>* pool = nullptr) {
    if (n == 0 || segs == 0) return;
    if (n > INT32_MAX || segs > INT32_MAX) throw std::invalid_argument("build batch too large");
    size_t tmp = 0;
    cuda_check(cub::DeviceSegmentedSort::SortKeys(nullptr, tmp, kin, kout, static_cast<int>(n),
                                                  static_cast<int>(segs), off, off + 1, s),
               "cub sort");
    DevArray<uint8_t> own;
    DevArray<uint8_t>& t = pool != nullptr ? *pool : own;
    t.grow(tmp + 16);
    cuda_check(cub::DeviceSegmentedSort::SortKeys(t.data(), tmp, kin, kout, static_cast<int>(n),
                                                  static_cast<int>(segs), off, off + 1, s),
               "cub sort");
    if (pool == nullptr) cuda_check(cudaStreamSynchronize(s), "sort sync");
}

}  // namespace nsp

#endif  // NSP_SEGSORT_CUH
