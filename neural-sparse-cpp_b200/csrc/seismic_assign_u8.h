// Cluster assignment of the SEISMIC build for uint8 codes on the tensor cores
// (seismic_assign_u8.cu).
#ifndef NSP_SEISMIC_ASSIGN_U8_H
#define NSP_SEISMIC_ASSIGN_U8_H

#include <cuda_runtime.h>

#include <cstdint>
#include <vector>

#include "engine.h"

namespace nsp {

struct AssignLists {
    int32_t n_lists;
    const int64_t* kept_ptr;  // [n_lists + 1]
    const int32_t* kept;      // every list's kept docs
    const int64_t* cptr;      // [n_lists + 1]
    const int32_t* cpos;      // centroid positions within each list
    int32_t max_nc;           // most centroids in one list
    int64_t max_kept;         // longest list
    int64_t max_row;          // longest row
};

// out_key[kept position] = cluster * 2 + (centroid ? 0 : 1), as assign_kernel
// gives it. `df`: documents per term. Returns false, having written nothing,
// where the general kernel is the one to use: a row that is not strictly
// ascending, or of more than kAssignMaxRowU8 entries, more than
// kAssignMaxCentroids centroids in a list, a vocabulary past 49,152 terms, or
// terms so evenly spread that the frequent ones hold less than half of the
// products.
constexpr int kAssignMaxCentroids = 1024;
// Terms two rows can share with their sum of uint8 code products below 2^31.
constexpr int64_t kAssignMaxRowU8 = INT32_MAX / (255 * 255);
bool assign_u8(const FwdView& f, const AssignLists& lists, const std::vector<int64_t>& df,
               uint32_t* out_key, cudaStream_t s, Arena& scratch);

}  // namespace nsp

#endif  // NSP_SEISMIC_ASSIGN_U8_H
