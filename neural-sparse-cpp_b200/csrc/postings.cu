// Doc-ascending postings of an fp32 forward index, built on the device for
// the exact search's term-at-a-time kernel (search_exact.cu).
//
// The reference's InvertedIndex keeps per-term posting lists in doc order
// (invlists/inverted_lists.cpp:159-180, built from the forward index by
// inverted_index.cpp:236-252). Here they come from the resident padded rows
// in five device steps: row lengths (and a check that every row's terms are
// strictly ascending), an exclusive scan, a doc-major compaction of (term,
// value | doc) pairs, a stable radix sort by term -- which keeps each term's
// postings in doc order --, and the per-(term, doc chunk) start table.
// Terms of a large share of the docs are kept as dense rows too.
#include <cub/device/device_radix_sort.cuh>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <vector>

#include "engine.h"
#include "postings_plan.h"
#include "scan.h"

namespace nsp {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// off[d] = row d's length; *unsorted = 1 if some row's terms are not
// strictly ascending. One warp per row.
__global__ void row_lens_kernel(FwdView f, int64_t* off, int* unsorted) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t d = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
         d < f.n_docs; d += warps) {
        const uint2 ri = f.rowinfo[d];
        const int len = static_cast<int>(ri.y);
        const uint16_t* ip = f.idx + static_cast<size_t>(ri.x) * kRowAlign;
        bool bad = false;
        for (int e = lane + 1; e < len; e += 32) bad |= ip[e] <= ip[e - 1];
        if (__any_sync(kFull, bad) && lane == 0) atomicOr(unsorted, 1);
        if (lane == 0) off[d] = len;
    }
}

// keys[off[d] + e] = term, vals[off[d] + e] = value bits << 32 | doc, in
// doc-major order.
__global__ void compact_kernel(FwdView f, const int64_t* off, uint16_t* keys,
                               unsigned long long* vals) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const float* fv = static_cast<const float*>(f.val);
    for (int64_t d = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
         d < f.n_docs; d += warps) {
        const uint2 ri = f.rowinfo[d];
        const int len = static_cast<int>(ri.y);
        const size_t src = static_cast<size_t>(ri.x) * kRowAlign;
        const int64_t dst = off[d];
        for (int e = lane; e < len; e += 32) {
            keys[dst + e] = f.idx[src + e];
            vals[dst + e] = (static_cast<unsigned long long>(__float_as_uint(fv[src + e])) << 32) |
                            static_cast<uint32_t>(d);
        }
    }
}

// tstart[t] = first position of term t in the sorted keys, t = 0..dim.
__global__ void term_start_kernel(const uint16_t* keys, int64_t nnz, int dim, int32_t* tstart) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t > dim) return;
    int64_t lo = 0, hi = nnz;
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        if (static_cast<int>(keys[mid]) < t) lo = mid + 1;
        else hi = mid;
    }
    tstart[t] = static_cast<int32_t>(lo);
}

// *max_abs = the bits of the largest magnitude, NaN above all (0 on entry).
__global__ void unpack_kernel(const unsigned long long* v, int64_t nnz, int32_t* doc, float* val,
                              unsigned* max_abs) {
    unsigned mine = 0u;
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t j = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; j < nnz;
         j += stride) {
        const unsigned long long x = v[j];
        doc[j] = static_cast<int32_t>(static_cast<uint32_t>(x));
        val[j] = __uint_as_float(static_cast<uint32_t>(x >> 32));
        mine = max(mine, static_cast<uint32_t>(x >> 32) & 0x7fffffffu);
    }
    mine = __reduce_max_sync(kFull, mine);
    if ((threadIdx.x & 31) == 0 && mine > 0u) atomicMax(max_abs, mine);
}

// chunk_at[t * (nc + 1) + c] = first posting of term t with doc >= c * C.
__global__ void chunk_at_kernel(const int32_t* tstart, const int32_t* doc, int dim, int nc, int C,
                                int32_t* chunk_at) {
    const int64_t total = static_cast<int64_t>(dim) * (nc + 1);
    const int64_t stride = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < total;
         i += stride) {
        const int t = static_cast<int>(i / (nc + 1));
        const int c = static_cast<int>(i - static_cast<int64_t>(t) * (nc + 1));
        int32_t lo = tstart[t];
        int32_t hi = tstart[t + 1];
        if (c < nc) {
            const int64_t bound = static_cast<int64_t>(c) * C;
            while (lo < hi) {
                const int32_t mid = lo + ((hi - lo) >> 1);
                if (doc[mid] < bound) lo = mid + 1;
                else hi = mid;
            }
        } else {
            lo = hi;
        }
        chunk_at[i] = lo;
    }
}

// Dense rows of the frequent terms: the postings of dense term blockIdx.y
// scattered to their docs' places.
__global__ void dense_rows_kernel(const int32_t* terms, int n_dense, const int32_t* tstart,
                                  const int32_t* doc, const float* val, int C, float* dense) {
    const int j = blockIdx.y;
    const int t = terms[j];
    const int64_t first = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    each_posting(tstart[t], tstart[t + 1], first, static_cast<int64_t>(gridDim.x) * blockDim.x,
                 [&](int32_t p) {
                     const int32_t d = doc[p];
                     const int32_t c = d / C;
                     dense[(static_cast<size_t>(c) * n_dense + j) * C + (d - c * C)] = val[p];
                 });
}

int grid_for(int64_t work, int per_block) {
    const int64_t g = (work + per_block - 1) / per_block;
    return static_cast<int>(std::max<int64_t>(1, std::min<int64_t>(g, 148 * 32)));
}

}  // namespace

void PostingsDevice::build(const ForwardDevice& fwd, int chunk_docs) {
    cudaStream_t s = Workspace::get().stream();
    generation_ = fwd.generation();
    usable_ = false;
    doc_.reset();
    val_.reset();
    chunk_at_.reset();
    dense_of_.reset();
    dense_.reset();
    n_dense_ = 0;
    n_chunks_ = 0;
    chunk_docs_ = chunk_docs;
    if (fwd.empty() || fwd.esz() != 4 || chunk_docs <= 0) return;
    const FwdView f = fwd.view();
    const int32_t n = f.n_docs;

    Arena scratch(s);
    int64_t* off = scratch.take<int64_t>(static_cast<size_t>(n) + 1);
    int* flag = scratch.take<int>(1);
    cuda_check(cudaMemsetAsync(flag, 0, sizeof(int), s), "memset");
    cuda_check(cudaMemsetAsync(off + n, 0, sizeof(int64_t), s), "memset");
    row_lens_kernel<<<grid_for(static_cast<int64_t>(n) * 32, 256), 256, 0, s>>>(f, off,
                                                                                flag);
    cuda_check(cudaGetLastError(), "row_lens_kernel");
    exclusive_scan_i64(off, off, static_cast<int64_t>(n) + 1, s, scratch);
    int64_t nnz = 0;
    int unsorted = 0;
    cuda_check(cudaMemcpyAsync(&nnz, off + n, sizeof(nnz), cudaMemcpyDeviceToHost, s), "D2H");
    cuda_check(cudaMemcpyAsync(&unsorted, flag, sizeof(int), cudaMemcpyDeviceToHost, s),
               "D2H");
    cuda_check(cudaStreamSynchronize(s), "sync");
    if (unsorted != 0 || nnz > kMaxPostings) return;  // the tile kernel serves this index

    n_chunks_ = (n + chunk_docs - 1) / chunk_docs;
    const int dim = f.dim;
    int32_t* tstart = scratch.take<int32_t>(static_cast<size_t>(dim) + 1);
    unsigned* max_abs = scratch.take<unsigned>(1);
    cuda_check(cudaMemsetAsync(max_abs, 0, sizeof(unsigned), s), "memset");
    doc_.resize(static_cast<size_t>(std::max<int64_t>(nnz, 1)));
    val_.resize(static_cast<size_t>(std::max<int64_t>(nnz, 1)));
    if (nnz > 0) {
        // (given back before the arrays below are allocated)
        Arena sort(s);
        uint16_t* k_in = sort.take<uint16_t>(static_cast<size_t>(nnz));
        uint16_t* k_out = sort.take<uint16_t>(static_cast<size_t>(nnz));
        auto* v_in = sort.take<unsigned long long>(static_cast<size_t>(nnz));
        auto* v_out = sort.take<unsigned long long>(static_cast<size_t>(nnz));
        compact_kernel<<<grid_for(static_cast<int64_t>(n) * 32, 256), 256, 0, s>>>(
            f, off, k_in, v_in);
        cuda_check(cudaGetLastError(), "compact_kernel");
        size_t tmp_bytes = 0;
        cuda_check(cub::DeviceRadixSort::SortPairs(nullptr, tmp_bytes, k_in, k_out,
                                                   v_in, v_out, static_cast<int>(nnz),
                                                   0, 16, s),
                   "radix sort size");
        auto* tmp = sort.take<unsigned char>(tmp_bytes);
        cuda_check(cub::DeviceRadixSort::SortPairs(tmp, tmp_bytes, k_in, k_out,
                                                   v_in, v_out, static_cast<int>(nnz),
                                                   0, 16, s),
                   "radix sort");
        term_start_kernel<<<(dim + 1 + 255) / 256, 256, 0, s>>>(k_out, nnz, dim,
                                                                tstart);
        cuda_check(cudaGetLastError(), "term_start_kernel");
        unpack_kernel<<<grid_for(nnz, 256), 256, 0, s>>>(v_out, nnz, doc_.data(),
                                                         val_.data(), max_abs);
        cuda_check(cudaGetLastError(), "unpack_kernel");
    } else {
        cuda_check(cudaMemsetAsync(tstart, 0, (static_cast<size_t>(dim) + 1) * 4, s),
                   "memset");
    }
    chunk_at_.resize(static_cast<size_t>(dim) * (n_chunks_ + 1));
    chunk_at_kernel<<<grid_for(static_cast<int64_t>(dim) * (n_chunks_ + 1), 256), 256, 0, s>>>(
        tstart, doc_.data(), dim, n_chunks_, chunk_docs, chunk_at_.data());
    cuda_check(cudaGetLastError(), "chunk_at_kernel");
    // dense rows of the frequent terms, as far as there is memory for them
    std::vector<int32_t> h_start(static_cast<size_t>(dim) + 1);
    cuda_check(cudaMemcpyAsync(h_start.data(), tstart, h_start.size() * sizeof(int32_t),
                               cudaMemcpyDeviceToHost, s), "D2H");
    cuda_check(cudaMemcpyAsync(&max_abs_, max_abs, sizeof(max_abs_), cudaMemcpyDeviceToHost, s),
               "D2H");
    cuda_check(cudaStreamSynchronize(s), "sync");
    const size_t row_cells = static_cast<size_t>(n_chunks_) * chunk_docs;
    size_t free_b = 0, total_b = 0;
    cuda_check(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
    std::vector<int32_t> frequent = dense_terms(h_start, n, row_cells * sizeof(float), free_b);
    frequent.resize(allocate_dense_rows(frequent.size(), [&](size_t rows) {
        try {
            dense_.resize(rows * row_cells);
        } catch (...) {
            (void)cudaGetLastError();  // the failed allocation's
            throw;
        }
    }));
    n_dense_ = static_cast<int32_t>(frequent.size());
    std::vector<int16_t> of(static_cast<size_t>(std::max(dim, 1)), -1);
    for (int32_t j = 0; j < n_dense_; ++j) of[frequent[j]] = static_cast<int16_t>(j);
    dense_of_.upload(of.data(), of.size(), s);
    if (n_dense_ > 0) {
        cuda_check(cudaMemsetAsync(dense_.data(), 0, n_dense_ * row_cells * sizeof(float), s),
                   "memset");
        const int32_t* terms = scratch.put(frequent.data(), frequent.size());
        dense_rows_kernel<<<dim3(static_cast<unsigned>(grid_for(n, 256 * 8)),
                                 static_cast<unsigned>(n_dense_)), 256, 0, s>>>(
            terms, n_dense_, tstart, doc_.data(), val_.data(), chunk_docs, dense_.data());
        cuda_check(cudaGetLastError(), "dense_rows_kernel");
    }
    cuda_check(cudaStreamSynchronize(s), "sync");
    usable_ = true;
}

PostingsView PostingsDevice::view() const {
    PostingsView v;
    v.n_chunks = n_chunks_;
    v.chunk_docs = chunk_docs_;
    v.doc = doc_.data();
    v.val = val_.data();
    v.chunk_at = chunk_at_.data();
    v.n_dense = n_dense_;
    v.dense_of = dense_of_.data();
    v.dense = dense_.data();
    return v;
}

size_t PostingsDevice::device_bytes() const {
    return doc_.size() * 4 + val_.size() * 4 + chunk_at_.size() * 4 + dense_.size() * 4 +
           dense_of_.size() * 2;
}

}  // namespace nsp
