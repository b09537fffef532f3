// Block summaries of the SEISMIC build (seismic_summaries.cu): every block's
// rows max-pooled per term, cut where the running mass reaches alpha, and
// laid out term-major per list.
#ifndef NSP_SEISMIC_SUMMARIES_H
#define NSP_SEISMIC_SUMMARIES_H

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <string>
#include <utility>
#include <vector>

#include "engine.h"

namespace nsp {

// Summary columns of all lists, in device memory: the index's final arrays,
// handed to the device image without a round trip through host memory.
struct DevColumns {
    DevArray<uint16_t> sterm, sblk;
    DevArray<int64_t> srun;  // a boundary per column, and the first
    DevArray<uint8_t> sval;
};

// Blocks of the lists, as the build's earlier phases leave them.
struct BlockSet {
    const int64_t* lbp;     // host, [n_lists + 1]: blocks before each list
    const int64_t* d_lbp;   // the same on the device
    int32_t n_lists;
    const int32_t* d_docs;  // every block's docs, block after block
    const int64_t* d_bdp;   // [n_blocks + 1]: docs before each block
    const uint16_t* d_local;  // [n_blocks]: the block's index within its list
};

// Fills `out` with every list's summary columns and appends its column prefix
// to `ltp` (which starts as {0}). `host`: the host rows of an fp32 index, whose
// blocks with equal maxima across the alpha cut take the reference's choice
// (nullptr: value descending, then term ascending, as the codes do).
// `steps`: time per step, when not null (each step then synchronizes).
void summarize_blocks(int esz, const FwdView& f, const BlockSet& blocks, float alpha,
                      const HostCsr* host, cudaStream_t s, Arena& scratch, DevColumns& out,
                      std::vector<int64_t>& ltp,
                      std::vector<std::pair<std::string, double>>* steps);

}  // namespace nsp

#endif  // NSP_SEISMIC_SUMMARIES_H
