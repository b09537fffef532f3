// SEISMIC index build on the device (the reference's
// build_inverted_lists_clusters, seismic_common.h:146-184).
//
//  1. postings      one warp per document scatters its (term, doc, value)
//                   entries into per-term lists (warp-aggregated atomics);
//                   a segmented sort orders each list: by value descending,
//                   then doc ascending, when it exceeds the posting cap lambda
//                   (invlists/inverted_lists.cpp:110-132), else by doc
//                   (the order build_inverted_lists produces, :159-180).
//  2. centroids     drawn on the host with std::mt19937 and
//                   std::uniform_int_distribution<> seeded base_seed + list,
//                   the reference's own draw (cluster/random_kmeans.cpp:28-51);
//                   it depends only on list lengths, so only those come back.
//  3. assignment    uint8 codes: on the tensor cores (seismic_assign_u8.cu).
//                   Else one CTA per list: the centroids' terms are indexed term
//                   major in scratch, one warp per document accumulates its
//                   similarity to every centroid in the document's term order
//                   (cluster/kmeans_utils.cpp:131-145; fp32 products and sums
//                   rounded separately, int64 for codes) and takes the strict
//                   argmax, lowest index on ties (:147-156).
//  4. blocks        a stable segmented sort puts each centroid first and its
//                   members after it in list order.
//  5. summaries     seismic_summaries.cu: per block the per-term maxima, the
//                   mass and the alpha cut (cluster/inverted_list_clusters.cpp:
//                   37-124), then term-major per list (:230-293).
// The lists stay on the device in the search layout and come back to the host
// when they are asked for (persistence).
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstdint>
#include <cstring>
#include <random>
#include <utility>
#include <string>
#include <stdexcept>
#include <thread>
#include <vector>

#include "engine.h"
#include "index_state.h"
#include "ref_order.h"
#include "scan.h"
#include "segsort.cuh"
#include "seismic_assign_u8.h"
#include "seismic_summaries.h"

namespace nsparse {
namespace detail {
namespace {

using nsp::cuda_check;
using nsp::DevArray;
using nsp::segmented_sort_keys;
using nsp::segmented_sort_pairs;

constexpr unsigned kFull = 0xffffffffu;

// ------------------------------------------------------- parameters ------

// seismic_common.h:130-144
int calc_lambda(int lambda, size_t n_vectors) {
    if (lambda == -1)
        return std::max(static_cast<int>(0.0005F * static_cast<float>(n_vectors)), 160);
    return lambda;
}

int calc_beta(int beta, int lambda) {
    if (beta == -1) return static_cast<int>(static_cast<float>(lambda) * 0.1F);
    return beta;
}

// random_kmeans.cpp:53-63 with the caller's int beta converted to size_t.
size_t clusters_for(size_t n_docs, int beta) {
    size_t nc = static_cast<size_t>(static_cast<long long>(beta));  // wraps like the reference
    if (beta == 0) nc = static_cast<size_t>(std::sqrt(n_docs));
    nc = nc > n_docs ? n_docs : nc;
    return std::max<size_t>(1, nc);
}

// Positions (into the list's kept order) of the centroids of one list:
// random_kmeans.cpp:28-51, applied to positions instead of ids.
void draw_positions(size_t n, size_t nc, uint32_t seed, std::vector<int32_t>& perm,
                    int32_t* out) {
    perm.resize(n);
    for (size_t i = 0; i < n; ++i) perm[i] = static_cast<int32_t>(i);
    std::mt19937 gen(seed);
    for (size_t i = 0; i < nc; ++i) {
        std::uniform_int_distribution<> distrib(0, static_cast<int>(n - i - 1));
        const size_t r = static_cast<size_t>(distrib(gen));
        out[i] = perm[r];
        std::swap(perm[r], perm[n - 1 - i]);
    }
}

// ------------------------------------------------------------- keys ------

// Order-preserving map of a value to uint32 (ascending value = ascending key).
__device__ __forceinline__ uint32_t orderable(float v) {
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}

template <int ESZ>
__device__ __forceinline__ float value_at(const uint8_t* val, int64_t i) {
    if constexpr (ESZ == 4) return reinterpret_cast<const float*>(val)[i];
    if constexpr (ESZ == 2) return static_cast<float>(reinterpret_cast<const uint16_t*>(val)[i]);
    return static_cast<float>(val[i]);
}

// ------------------------------------------------------------ 1. postings --

__global__ void post_count_kernel(nsp::FwdView f, unsigned long long* cnt) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t d = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
         d < f.n_docs; d += warps) {
        const uint2 ri = f.rowinfo[d];
        const uint16_t* ip = f.idx + static_cast<size_t>(ri.x) * nsp::kRowAlign;
        for (uint32_t e0 = 0; e0 < ri.y; e0 += 32) {
            const uint32_t e = e0 + lane;
            const bool valid = e < ri.y;
            const uint32_t t = valid ? ip[e] : 0xffffffffu;
            const unsigned peers = __match_any_sync(kFull, t);
            if (valid && (__ffs(peers) - 1) == lane) atomicAdd(cnt + t, __popc(peers));
        }
    }
}

// Writes each entry's sort key into its list: (~value << 32 | doc) when the
// list is over the cap, doc otherwise.
template <int ESZ>
__global__ void post_scatter_kernel(nsp::FwdView f, const int64_t* post_ptr,
                                    unsigned long long* cursor, int64_t cap,
                                    uint64_t* keys) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    const uint8_t* vals = static_cast<const uint8_t*>(f.val);
    for (int64_t d = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
         d < f.n_docs; d += warps) {
        const uint2 ri = f.rowinfo[d];
        const int64_t base = static_cast<int64_t>(ri.x) * nsp::kRowAlign;
        for (uint32_t e0 = 0; e0 < ri.y; e0 += 32) {
            const uint32_t e = e0 + lane;
            const bool valid = e < ri.y;
            const uint32_t t = valid ? f.idx[base + e] : 0xffffffffu;
            const unsigned peers = __match_any_sync(kFull, t);
            const int leader = __ffs(peers) - 1;
            unsigned long long start = 0;
            if (valid && leader == lane) start = atomicAdd(cursor + t, __popc(peers));
            start = __shfl_sync(kFull, start, leader);
            if (valid) {
                const int rank = __popc(peers & ((1u << lane) - 1u));
                const int64_t len = post_ptr[t + 1] - post_ptr[t];
                const uint64_t key =
                    (cap > 0 && len > cap)
                        ? (static_cast<uint64_t>(~orderable(value_at<ESZ>(vals, base + e))) << 32) |
                              static_cast<uint32_t>(d)
                        : static_cast<uint64_t>(static_cast<uint32_t>(d));
                keys[post_ptr[t] + static_cast<int64_t>(start) + rank] = key;
            }
        }
    }
}

__global__ void kept_copy_kernel(const uint64_t* keys, const int64_t* post_ptr,
                                 const int64_t* kept_ptr, int32_t n_lists, int32_t* kept) {
    for (int32_t t = blockIdx.x; t < n_lists; t += gridDim.x) {
        const int64_t n = kept_ptr[t + 1] - kept_ptr[t];
        for (int64_t i = threadIdx.x; i < n; i += blockDim.x)
            kept[kept_ptr[t] + i] = static_cast<int32_t>(keys[post_ptr[t] + i] & 0xffffffffu);
    }
}

// Flags a truncated list (len > cap) whose first cap + 1 sorted keys hold two
// equal values: its kept order (and, with a tie across the cut, its kept set)
// is what the reference's unstable sort leaves, which the host reproduces.
__global__ void tie_flag_kernel(const uint64_t* keys, const int64_t* post_ptr, int32_t n_lists,
                                int64_t cap, uint8_t* flag) {
    for (int32_t t = blockIdx.x; t < n_lists; t += gridDim.x) {
        const int64_t len = post_ptr[t + 1] - post_ptr[t];
        if (cap <= 0 || len <= cap) {
            if (threadIdx.x == 0) flag[t] = 0;
            continue;
        }
        const uint64_t* k = keys + post_ptr[t];
        int tie = 0;
        for (int64_t i = threadIdx.x + 1; i <= cap; i += blockDim.x)
            tie |= (k[i] >> 32) == (k[i - 1] >> 32);
        tie = __syncthreads_or(tie);
        if (threadIdx.x == 0) flag[t] = static_cast<uint8_t>(tie);
    }
}

// ---------------------------------------------------------- 3. assignment --

struct AssignArgs {
    nsp::FwdView f;
    int32_t n_lists;
    const int64_t* kept_ptr;
    const int32_t* kept;
    const int64_t* cptr;
    const int32_t* cpos;
    uint32_t* out_key;      // per kept position: cluster * 2 + (centroid ? 0 : 1)
    int32_t* work;          // list counter
    // per-CTA scratch
    int32_t* tcnt;          // [dim] per CTA, zero between lists
    int32_t* tcur;          // [dim] per CTA
    int2* trun;             // [dim] per CTA: (start, count) of the term's centroid
                            // entries, count zero between lists
    int32_t* touched;       // [max centroid entries] per CTA
    uint16_t* ccl;          // [max centroid entries] per CTA
    uint8_t* cw;            // [max centroid entries * esz] per CTA
    uint8_t* is_centroid;   // [max kept] per CTA
    void* sims;             // per warp [max nc] (float or int64)
    int64_t max_centroid_entries;
    int64_t max_kept;
    int32_t max_nc;
    int32_t sims_in_smem;  // 1: the similarity rows are in dynamic shared memory
    // fp32: after them, rows of the list's terms that most centroids hold, a
    // value per centroid (max_nc, a multiple of 4, floats each)
    int32_t dense_rows;
};

// A term's centroid run as (start, count | (dense row + 1) << kDenseShift).
constexpr int kDenseShift = 20;  // counts are at most 65,536 centroids
constexpr int kMaxDenseRows = 64;

// Similarity accumulators: fp32 for fp32 values; for codes int64, or int for
// uint8 codes of rows so short that it holds every sum: kAnyRows is set for
// rows that repeat a term, and for uint8 rows of more than kAssignMaxRowU8
// entries.
template <int ESZ, bool kAnyRows>
using assign_acc_t = typename std::conditional<
    ESZ == 4, float,
    typename std::conditional<ESZ == 1 && !kAnyRows, int, long long>::type>::type;

template <int ESZ>
using assign_val_t = typename std::conditional<
    ESZ == 4, float, typename std::conditional<ESZ == 1, uint8_t, uint16_t>::type>::type;

__device__ __forceinline__ void add_product(float* sims, int32_t c, float dv, float w) {
    sims[c] = __fadd_rn(sims[c], __fmul_rn(dv, w));
}
template <class T>
__device__ __forceinline__ void add_product(T* sims, int32_t c, T dv, T w) {
    sims[c] += dv * w;
}

// Lane by lane the products of 32 entries of a term's run (c < 0: none), where
// a centroid may hold several: its entries are added one after another, in
// lane order. By a whole warp.
template <class T>
__device__ __forceinline__ void add_products_in_turn(T* sims, int32_t c, T dv, T w, int lane) {
    const unsigned peers = __match_any_sync(kFull, c);
    const int turn = c < 0 ? -1 : __popc(peers & ((1u << lane) - 1u));
    for (int r = 0; __any_sync(kFull, turn >= r); ++r) {
        if (turn == r) add_product(sims, c, dv, w);
        __syncwarp();
    }
}

// sims[c] += dv * row[c] for every centroid (n4 a multiple of 4).
__device__ __forceinline__ void apply_dense(float* sims, const float* row, float dv, int32_t n4,
                                            int lane) {
    const float4* w4 = reinterpret_cast<const float4*>(row);
    float4* s4 = reinterpret_cast<float4*>(sims);
    for (int32_t c = lane; c < n4 / 4; c += 32) {
        const float4 w = w4[c];
        float4 x = s4[c];
        x.x = __fadd_rn(x.x, __fmul_rn(dv, w.x));
        x.y = __fadd_rn(x.y, __fmul_rn(dv, w.y));
        x.z = __fadd_rn(x.z, __fmul_rn(dv, w.z));
        x.w = __fadd_rn(x.w, __fmul_rn(dv, w.w));
        s4[c] = x;
    }
}
template <class T>
__device__ __forceinline__ void apply_dense(T*, const float*, T, int32_t, int) {}

// kAnyRows: some row may repeat a term. A centroid then has several entries in
// one term's run, which the reference adds in the centroid's order
// (kmeans_utils.cpp:40-97): one warp indexes the centroids in order, so a run
// lists them as they come, and entries of one centroid take turns. Other
// indexes have distinct centroids in a run, whose products commute.
template <int ESZ, bool kAnyRows>
__global__ void __launch_bounds__(1024) assign_kernel(AssignArgs a) {
    using acc_t = assign_acc_t<ESZ, kAnyRows>;
    using val_t = assign_val_t<ESZ>;
    // centroid entries of one term in flight per lane: a term's run is
    // loaded kChunks * 32 entries at a time, the next hit term's first
    // chunk while the current one is applied
    constexpr int kChunks = 4;
    __shared__ int32_t s_list;
    __shared__ int32_t s_touched;
    __shared__ int32_t s_total;
    __shared__ int32_t s_dense;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    const int wpb = blockDim.x >> 5;
    const int dim = a.f.dim;
    int32_t* tcnt = a.tcnt + static_cast<size_t>(blockIdx.x) * dim;
    int32_t* tcur = a.tcur + static_cast<size_t>(blockIdx.x) * dim;
    int2* trun = a.trun + static_cast<size_t>(blockIdx.x) * dim;
    int32_t* touched = a.touched + static_cast<size_t>(blockIdx.x) * a.max_centroid_entries;
    uint16_t* ccl = a.ccl + static_cast<size_t>(blockIdx.x) * a.max_centroid_entries;
    val_t* vals = reinterpret_cast<val_t*>(
        a.cw + static_cast<size_t>(blockIdx.x) * a.max_centroid_entries * ESZ);
    uint8_t* isc = a.is_centroid + static_cast<size_t>(blockIdx.x) * a.max_kept;
    // each warp's row of similarities: shared memory when the launch gave
    // room for it (the read-modify-writes of one doc are serial), else global
    extern __shared__ __align__(16) unsigned char dyn[];
    acc_t* sims = a.sims_in_smem ? reinterpret_cast<acc_t*>(dyn) + static_cast<size_t>(warp) * a.max_nc
                                 : static_cast<acc_t*>(a.sims) +
                                       static_cast<size_t>(blockIdx.x * wpb + warp) * a.max_nc;
    // Bound by shared memory: a product is a read-modify-write of its
    // similarity, and a warp's 32 scattered ones conflict in the banks. A term
    // that at least 40% of the list's centroids hold is therefore applied as a
    // dense row of shared memory, four centroids per lane and no conflicts
    // (below that share the row's zero products cost more than the conflicts:
    // with 20% the case below takes 84 ms, with 30% 80. With 30 / 40 / 60%:
    // docs of median 120 terms, 80,000 of them, lambda 4000, beta 400 97 / 93 /
    // 96 ms; 60,000, 6000, 750 101 / 94 / 92; 40,000, 1000, 100 and 20,000,
    // 2500, 125 the same 37 and 25 with all three);
    // centroids without the term add a zero product, which leaves a sum as it
    // is while the doc's value is finite. Staging the other terms' runs in
    // shared memory as well, 32 terms at a time, was slower: the stage is more
    // of the same traffic (80,000 docs, lambda 4000, beta 400, assignment: 89
    // ms without rows, 78 with them and with four entries in flight in the
    // indexing below, 101 with the stage).
    constexpr bool kDense = ESZ == 4 && !kAnyRows;  // (a row's cell holds one entry)
    float* rows = reinterpret_cast<float*>(dyn) + static_cast<size_t>(wpb) * a.max_nc;
    const val_t* fval = static_cast<const val_t*>(a.f.val);

    for (;;) {
        if (threadIdx.x == 0) s_list = atomicAdd(a.work, 1);
        __syncthreads();
        const int32_t t = s_list;
        __syncthreads();
        if (t >= a.n_lists) break;
        const int64_t kb = a.kept_ptr[t];
        const int32_t n = static_cast<int32_t>(a.kept_ptr[t + 1] - kb);
        const int32_t nc = static_cast<int32_t>(a.cptr[t + 1] - a.cptr[t]);
        if (n == 0) continue;
        const int32_t* cp = a.cpos + a.cptr[t];
        if (n == nc) {  // every doc is a centroid
            for (int32_t c = threadIdx.x; c < nc; c += blockDim.x)
                a.out_key[kb + cp[c]] = static_cast<uint32_t>(c) * 2u;
            continue;
        }
        for (int32_t i = threadIdx.x; i < n; i += blockDim.x) isc[i] = 0;
        if (threadIdx.x == 0) {
            s_touched = 0;
            s_total = 0;
            s_dense = 0;
        }
        __syncthreads();
        for (int32_t c = threadIdx.x; c < nc; c += blockDim.x) {
            isc[cp[c]] = 1;
            a.out_key[kb + cp[c]] = static_cast<uint32_t>(c) * 2u;  // its own cluster, placed first
        }
        // index the centroid entries by term: count, ranges, scatter
        for (int32_t c = warp; c < nc; c += wpb) {
            const int32_t doc = a.kept[kb + cp[c]];
            const uint2 ri = a.f.rowinfo[doc];
            const uint16_t* ip = a.f.idx + static_cast<size_t>(ri.x) * nsp::kRowAlign;
            for (uint32_t e = lane; e < ri.y; e += 32) {
                const int32_t term = ip[e];
                if (atomicAdd(tcnt + term, 1) == 0) touched[atomicAdd(&s_touched, 1)] = term;
            }
        }
        __syncthreads();
        const int32_t nt = s_touched;
        for (int32_t i = threadIdx.x; i < nt; i += blockDim.x) {
            const int32_t term = touched[i];
            const int32_t cnt = tcnt[term];
            const int32_t st = atomicAdd(&s_total, cnt);
            tcur[term] = st;
            int32_t row = 0;
            if (kDense && a.dense_rows > 0 && 10ll * cnt >= 4ll * nc) {
                row = atomicAdd(&s_dense, 1) + 1;
                if (row > a.dense_rows) row = 0;
            }
            trun[term] = make_int2(st, cnt | (row << kDenseShift));
        }
        __syncthreads();
        const int32_t nc4 = (nc + 3) & ~3;
        if constexpr (kDense) {
            const int32_t cells = min(s_dense, a.dense_rows) * nc4;
            for (int32_t i = threadIdx.x; i < cells; i += blockDim.x) rows[i] = 0.0f;
            __syncthreads();
        }
        if constexpr (kAnyRows) {
            for (int32_t c = 0; c < nc && warp == 0; ++c) {
                const int32_t doc = a.kept[kb + cp[c]];
                const uint2 ri = a.f.rowinfo[doc];
                const int64_t rb = static_cast<int64_t>(ri.x) * nsp::kRowAlign;
                for (uint32_t e0 = 0; e0 < ri.y; e0 += 32) {
                    const uint32_t e = e0 + lane;
                    const int32_t term = e < ri.y ? a.f.idx[rb + e] : -1;
                    const unsigned peers = __match_any_sync(kFull, term);
                    const int rank = __popc(peers & ((1u << lane) - 1u));
                    const int32_t at = term >= 0 ? tcur[term] : 0;
                    __syncwarp();
                    if (term >= 0) {
                        ccl[at + rank] = static_cast<uint16_t>(c);
                        vals[at + rank] = fval[rb + e];
                        if (rank == 0) tcur[term] = at + __popc(peers);
                    }
                    __syncwarp();
                }
            }
        }
        for (int32_t c = warp; c < nc && !kAnyRows; c += wpb) {
            const int32_t doc = a.kept[kb + cp[c]];
            const uint2 ri = a.f.rowinfo[doc];
            const int64_t rb = static_cast<int64_t>(ri.x) * nsp::kRowAlign;
            for (uint32_t e0 = 0; e0 < ri.y; e0 += 128) {  // four entries in flight per lane
                int32_t pos[4], row[4];
                val_t w[4];
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    const uint32_t e = e0 + u * 32 + lane;
                    pos[u] = -1;
                    if (e < ri.y) {
                        const int32_t term = a.f.idx[rb + e];
                        w[u] = fval[rb + e];
                        pos[u] = atomicAdd(tcur + term, 1);
                        if constexpr (kDense) row[u] = trun[term].y >> kDenseShift;
                    }
                }
#pragma unroll
                for (int u = 0; u < 4; ++u) {
                    if (pos[u] < 0) continue;
                    ccl[pos[u]] = static_cast<uint16_t>(c);
                    vals[pos[u]] = w[u];
                    if constexpr (kDense)
                        if (row[u] > 0) rows[(row[u] - 1) * nc4 + c] = w[u];
                }
            }
        }
        __syncthreads();
        // assign every non-centroid doc, one warp per doc
        for (int32_t p = warp; p < n; p += wpb) {
            if (isc[p]) continue;
            const int32_t doc = a.kept[kb + p];
            for (int32_t c = lane; c < nc4; c += 32) sims[c] = 0;
            __syncwarp();
            const uint2 ri = a.f.rowinfo[doc];
            const int64_t rb = static_cast<int64_t>(ri.x) * nsp::kRowAlign;
            for (uint32_t e0 = 0; e0 < ri.y; e0 += 32) {
                const uint32_t e = e0 + lane;
                int2 run = make_int2(0, 0);
                acc_t v = 0;
                if (e < ri.y) {
                    run = trun[a.f.idx[rb + e]];
                    v = fval[rb + e];
                }
                // doc terms in order (kmeans_utils.cpp:134-145); a term's
                // centroids are distinct, so its products commute, and the
                // warp barrier between terms keeps each similarity's sum in
                // doc-term order
                unsigned m = __ballot_sync(kFull, run.y > 0);
                int32_t nc_[kChunks];
                acc_t nw[kChunks];
                int32_t s0 = 0, cnt = 0, row = 0;
                acc_t dv = 0;
                // the hit term of lane src: its value, and its dense row or
                // the first entries of its run
                auto fetch = [&](int src) {
                    s0 = __shfl_sync(kFull, run.x, src);
                    cnt = __shfl_sync(kFull, run.y, src);
                    dv = __shfl_sync(kFull, v, src);
                    row = 0;
                    if constexpr (kDense) {
                        row = isfinite(dv) ? cnt >> kDenseShift : 0;
                        cnt &= (1 << kDenseShift) - 1;
                    }
#pragma unroll
                    for (int j = 0; j < kChunks; ++j) {
                        const int32_t k = j * 32 + lane;
                        nc_[j] = -1;
                        if (row == 0 && k < cnt) {
                            nc_[j] = ccl[s0 + k];
                            nw[j] = vals[s0 + k];
                        }
                    }
                };
                if (m) fetch(__ffs(m) - 1);
                while (m) {
                    m &= m - 1;
                    int32_t cc[kChunks];
                    acc_t cwv[kChunks];
#pragma unroll
                    for (int j = 0; j < kChunks; ++j) {
                        cc[j] = nc_[j];
                        cwv[j] = nw[j];
                    }
                    const int32_t cs0 = s0, ccnt = cnt, crow = row;
                    const acc_t cdv = dv;
                    if (m) fetch(__ffs(m) - 1);
                    if (kDense && crow > 0) {
                        apply_dense(sims, rows + (crow - 1) * nc4, cdv, nc4, lane);
                        __syncwarp();
                        continue;
                    }
#pragma unroll
                    for (int j = 0; j < kChunks; ++j) {
                        if constexpr (kAnyRows)
                            add_products_in_turn(sims, cc[j], cdv, cwv[j], lane);
                        else if (cc[j] >= 0)
                            add_product(sims, cc[j], cdv, cwv[j]);
                    }
                    for (int32_t k0 = kChunks * 32; k0 < ccnt; k0 += kChunks * 32) {
#pragma unroll
                        for (int j = 0; j < kChunks; ++j) {
                            const int32_t k = k0 + j * 32 + lane;
                            cc[j] = -1;
                            if (k < ccnt) {
                                cc[j] = ccl[cs0 + k];
                                cwv[j] = vals[cs0 + k];
                            }
                        }
#pragma unroll
                        for (int j = 0; j < kChunks; ++j) {
                            if constexpr (kAnyRows)
                                add_products_in_turn(sims, cc[j], cdv, cwv[j], lane);
                            else if (cc[j] >= 0)
                                add_product(sims, cc[j], cdv, cwv[j]);
                        }
                    }
                    __syncwarp();
                }
            }
            // strict >, ascending: ties go to the lowest cluster (kmeans_utils.cpp:147-156)
            acc_t best = 0;
            int32_t bi = -1;
            for (int32_t c = lane; c < nc; c += 32) {
                const acc_t s = sims[c];
                if (bi < 0 || s > best) {
                    best = s;
                    bi = c;
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const acc_t s2 = __shfl_xor_sync(kFull, best, o);
                const int32_t i2 = __shfl_xor_sync(kFull, bi, o);
                if (i2 >= 0 && (bi < 0 || s2 > best || (s2 == best && i2 < bi))) {
                    best = s2;
                    bi = i2;
                }
            }
            if (lane == 0) a.out_key[kb + p] = static_cast<uint32_t>(bi) * 2u + 1u;
            __syncwarp();
        }
        __syncthreads();
        for (int32_t i = threadIdx.x; i < nt; i += blockDim.x) {
            tcnt[touched[i]] = 0;
            trun[touched[i]] = make_int2(0, 0);
        }
        __syncthreads();
    }
}

// *repeats = 1 when some row holds a term twice: a warp per row, a bitmap of
// the terms seen for the rows that are not strictly ascending.
constexpr int kSeenWarps = 4;
__global__ void __launch_bounds__(kSeenWarps * 32) repeats_kernel(nsp::FwdView f, int* repeats) {
    __shared__ uint32_t seen[kSeenWarps][65536 / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int i = lane; i < 65536 / 32; i += 32) seen[warp][i] = 0u;
    __syncwarp();
    for (int64_t d = static_cast<int64_t>(blockIdx.x) * kSeenWarps + warp; d < f.n_docs;
         d += static_cast<int64_t>(gridDim.x) * kSeenWarps) {
        const uint2 ri = __ldg(f.rowinfo + d);
        const uint16_t* ip = f.idx + static_cast<size_t>(ri.x) * nsp::kRowAlign;
        bool bad = false;
        for (uint32_t e = 1 + lane; e < ri.y; e += 32) bad |= __ldg(ip + e - 1) >= __ldg(ip + e);
        if (!__any_sync(kFull, bad)) continue;
        bool twice = false;
        for (uint32_t e = lane; e < ri.y; e += 32) {
            const uint32_t t = __ldg(ip + e), bit = 1u << (t & 31);
            twice |= (atomicOr(&seen[warp][t >> 5], bit) & bit) != 0u;
        }
        if (__any_sync(kFull, twice) && lane == 0) *repeats = 1;
        __syncwarp();
        for (uint32_t e = lane; e < ri.y; e += 32) seen[warp][__ldg(ip + e) >> 5] = 0u;
        __syncwarp();
    }
}

template <class T>
std::vector<T> to_host(const T* d, size_t n, cudaStream_t s) {
    std::vector<T> h(n);
    cuda_check(cudaMemcpyAsync(h.data(), d, n * sizeof(T), cudaMemcpyDeviceToHost, s), "D2H");
    cuda_check(cudaStreamSynchronize(s), "D2H");
    return h;
}

std::vector<int32_t> to_i32_offsets(const std::vector<int64_t>& v) {
    std::vector<int32_t> o(v.size());
    for (size_t i = 0; i < v.size(); ++i) {
        if (v[i] > INT32_MAX) throw std::invalid_argument("build batch too large");
        o[i] = static_cast<int32_t>(v[i]);
    }
    return o;
}

// ------------------------------------------------------------- 4. blocks --

// Block boundaries from the sorted assignment keys (cluster * 2 + member),
// CTA per list: block c of list t ends where the keys pass 2c + 1. And each
// block's index within its list.
__global__ void block_bounds_kernel(const uint32_t* key, const int64_t* kept_ptr,
                                    const int64_t* lbp, int32_t n_lists, int64_t* bdp,
                                    uint16_t* local) {
    for (int32_t t = blockIdx.x; t < n_lists; t += gridDim.x) {
        const int64_t k0 = kept_ptr[t], k1 = kept_ptr[t + 1];
        const int64_t b0 = lbp[t], nc = lbp[t + 1] - b0;
        for (int64_t c = threadIdx.x; c < nc; c += blockDim.x) {
            int64_t lo = k0, hi = k1;
            while (lo < hi) {
                const int64_t mid = (lo + hi) >> 1;
                if (key[mid] < 2u * static_cast<uint32_t>(c) + 2u) lo = mid + 1;
                else hi = mid;
            }
            bdp[b0 + c + 1] = lo;
            local[b0 + c] = static_cast<uint16_t>(c);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) bdp[0] = 0;
}

// fp32 lists whose kept postings hold tied values get the reference's kept
// order from the host (ref_order.cpp); every other list's device order
// (value desc, then doc asc) is already the reference's.
void reference_tie_order(const nsp::HostCsr& h, const std::vector<int64_t>& post,
                         const std::vector<int64_t>& kept_ptr, const std::vector<uint8_t>& tie,
                         int64_t cap, int32_t* kept, cudaStream_t s) {
    std::vector<int32_t> lists;
    for (int32_t t = 0; t < static_cast<int32_t>(tie.size()); ++t)
        if (tie[t]) lists.push_back(t);
    if (lists.empty()) return;
    std::vector<int32_t> out;
    nsp::reference_kept_order(h, post, lists, cap, out);
    for (size_t j = 0; j < lists.size(); ++j)
        cuda_check(cudaMemcpyAsync(kept + kept_ptr[lists[j]], out.data() + j * cap,
                                   static_cast<size_t>(cap) * sizeof(int32_t),
                                   cudaMemcpyHostToDevice, s),
                   "H2D kept order");
    cuda_check(cudaStreamSynchronize(s), "sync");
}

// Phase timings on stderr when NSP_VERBOSE=1 (the engine's one debug switch).
struct PhaseClock {
    cudaStream_t s;
    bool on;
    std::chrono::steady_clock::time_point t;
    explicit PhaseClock(cudaStream_t st) : s(st) {
        const char* v = std::getenv("NSP_VERBOSE");
        on = v != nullptr && v[0] == '1';
        t = std::chrono::steady_clock::now();
    }
    void mark(const char* what) {
        if (!on) return;
        cudaStreamSynchronize(s);
        const auto now = std::chrono::steady_clock::now();
        std::fprintf(stderr, "[nsparse build] %-12s %8.3f s\n", what,
                     std::chrono::duration<double>(now - t).count());
        t = now;
    }
};

// Assignment by assign_kernel: any values, any rows.
template <int ESZ, bool kAnyRows>
void assign_general(const nsp::FwdView& f, const nsp::AssignLists& l, uint32_t* out_key,
                    cudaStream_t s, nsp::Arena& scratch) {
    const int dim = f.dim;
    const int64_t max_ce = std::max<int64_t>(1, static_cast<int64_t>(l.max_nc) * l.max_row);
    const int wpb = 32;
    const size_t acc_bytes = sizeof(assign_acc_t<ESZ, kAnyRows>);
    const int32_t nc_row = (std::max(l.max_nc, 1) + 3) & ~3;
    const size_t sims_smem = static_cast<size_t>(wpb) * nc_row * acc_bytes;
    const bool sims_in_smem = sims_smem <= 160u * 1024u;
    // dense rows in what is left of 224 KB
    int32_t dense_rows = 0;
    if (ESZ == 4 && !kAnyRows && sims_in_smem)
        dense_rows = static_cast<int32_t>(std::min<size_t>(
            kMaxDenseRows, (224u * 1024u - sims_smem) / (static_cast<size_t>(nc_row) * 4)));
    const size_t smem =
        sims_in_smem ? sims_smem + static_cast<size_t>(dense_rows) * nc_row * 4 : 0;
    if (sims_in_smem)
        cuda_check(nsp::allow_opt_in_smem(assign_kernel<ESZ, kAnyRows>), "assign smem");
    // one CTA of 32 warps per SM: as many warps as four CTAs of 8 hide
    // the memory round trips with, and a quarter of the per-CTA term
    // tables (trun, tcnt, ...), which then stay in L2 (8.8M SQ docs:
    // 6.4 -> 5.5 s against four CTAs of 8 warps; two of 16: 5.7 s)
    int per_sm = 0;
    cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, assign_kernel<ESZ, kAnyRows>,
                                                             wpb * 32, smem),
               "assign occupancy");
    const size_t ctas = static_cast<size_t>(nsp::device_sm_count()) * std::max(1, std::min(per_sm, 1));
    const nsp::Arena::Mark mark = scratch.mark();
    AssignArgs a{};
    a.f = f;
    a.n_lists = l.n_lists;
    a.kept_ptr = l.kept_ptr;
    a.kept = l.kept;
    a.cptr = l.cptr;
    a.cpos = l.cpos;
    a.out_key = out_key;
    a.max_centroid_entries = max_ce;
    a.max_kept = std::max<int64_t>(l.max_kept, 1);
    a.max_nc = nc_row;
    a.dense_rows = dense_rows;
    a.sims_in_smem = sims_in_smem ? 1 : 0;
    a.work = scratch.take<int32_t>(1);
    a.tcnt = scratch.take<int32_t>(ctas * dim);
    a.tcur = scratch.take<int32_t>(ctas * dim);
    a.trun = scratch.take<int2>(ctas * dim);
    a.touched = scratch.take<int32_t>(ctas * max_ce);
    a.ccl = scratch.take<uint16_t>(ctas * max_ce);
    a.cw = scratch.take<uint8_t>(ctas * max_ce * ESZ);
    a.is_centroid = scratch.take<uint8_t>(ctas * a.max_kept);
    a.sims = scratch.take<uint8_t>(ctas * wpb * a.max_nc * 8);
    cuda_check(cudaMemsetAsync(a.tcnt, 0, ctas * dim * 4, s), "memset");
    cuda_check(cudaMemsetAsync(a.trun, 0, ctas * dim * sizeof(int2), s), "memset");
    cuda_check(cudaMemsetAsync(a.work, 0, 4, s), "memset");
    assign_kernel<ESZ, kAnyRows><<<static_cast<unsigned>(ctas), wpb * 32, smem, s>>>(a);
    cuda_check(cudaGetLastError(), "assign_kernel");
    scratch.release(mark);
}

template <int ESZ>
void build_typed(SeismicState& st, int dim, const SeismicClusterParameters& p) {
    const nsp::HostCsr& h = st.vectors.host;
    cudaStream_t s = nsp::Workspace::get().stream();
    const int64_t n_docs = h.n();
    const int lambda = calc_lambda(p.lambda, static_cast<size_t>(n_docs));
    const int beta = calc_beta(p.beta, lambda);
    const int64_t cap = lambda <= 0 ? 0 : lambda;  // 0: keep whole lists (inverted_lists.cpp:114)
    const uint32_t base_seed =
        p.seed == -1 ? std::random_device{}() : static_cast<uint32_t>(p.seed);
    st.vectors.ensure_device();
    const nsp::FwdView f = st.vectors.dev.view();
    const int32_t n_lists = dim;
    const int sms = nsp::device_sm_count();
    PhaseClock clock(s);

    // ---- 1. postings
    nsp::Arena arena(s);
    const size_t nl1 = static_cast<size_t>(n_lists) + 1;
    auto* cnt = arena.take<unsigned long long>(nl1);
    cuda_check(cudaMemsetAsync(cnt, 0, nl1 * 8, s), "memset");
    post_count_kernel<<<sms * 8, 256, 0, s>>>(f, cnt);
    cuda_check(cudaGetLastError(), "post_count_kernel");
    int64_t* post_ptr = arena.take<int64_t>(nl1);
    nsp::exclusive_scan_i64(reinterpret_cast<const int64_t*>(cnt), post_ptr, n_lists + 1, s,
                            arena);
    const std::vector<int64_t> h_post = to_host(post_ptr, n_lists + 1, s);
    const int64_t nnz = h_post.back();
    std::vector<int32_t> kept_len(n_lists);
    std::vector<int64_t> kept_ptr(n_lists + 1, 0);
    for (int32_t t = 0; t < n_lists; ++t) {
        const int64_t len = h_post[t + 1] - h_post[t];
        kept_len[t] = static_cast<int32_t>(cap > 0 && len > cap ? cap : len);
        kept_ptr[t + 1] = kept_ptr[t] + kept_len[t];
    }
    const int64_t total_kept = kept_ptr.back();
    const int64_t* d_kept_ptr = arena.put(kept_ptr.data(), nl1);
    int32_t* kept = arena.take<int32_t>(static_cast<size_t>(total_kept));
    const nsp::Arena::Mark before_keys = arena.mark();
    uint64_t* keys = arena.take<uint64_t>(static_cast<size_t>(nnz));
    uint64_t* keys2 = arena.take<uint64_t>(static_cast<size_t>(nnz));
    cuda_check(cudaMemsetAsync(cnt, 0, nl1 * 8, s), "memset");
    post_scatter_kernel<ESZ><<<sms * 8, 256, 0, s>>>(f, post_ptr, cnt, cap, keys);
    cuda_check(cudaGetLastError(), "post_scatter_kernel");
    {
        const std::vector<int32_t> off32 = to_i32_offsets(h_post);
        segmented_sort_keys(keys, keys2, nnz, n_lists, arena.put(off32.data(), nl1), s, arena);
    }
    kept_copy_kernel<<<sms * 8, 256, 0, s>>>(keys2, post_ptr, d_kept_ptr, n_lists, kept);
    cuda_check(cudaGetLastError(), "kept_copy_kernel");
    uint8_t* d_tie = nullptr;
    if (ESZ == 4 && cap > 0) {
        d_tie = arena.take<uint8_t>(static_cast<size_t>(n_lists));
        tie_flag_kernel<<<sms * 8, 256, 0, s>>>(keys2, post_ptr, n_lists, cap, d_tie);
        cuda_check(cudaGetLastError(), "tie_flag_kernel");
    }

    // ---- 2. centroid positions (host; depends on list lengths only, so the
    // device sorts the postings meanwhile)
    std::vector<int64_t> cptr(n_lists + 1, 0);
    for (int32_t t = 0; t < n_lists; ++t)
        cptr[t + 1] = cptr[t] + (kept_len[t] > 0 ? static_cast<int64_t>(clusters_for(kept_len[t], beta)) : 0);
    int32_t max_nc = 0;
    int64_t max_kept = 0;
    for (int32_t t = 0; t < n_lists; ++t) {
        max_nc = std::max<int32_t>(max_nc, static_cast<int32_t>(cptr[t + 1] - cptr[t]));
        max_kept = std::max<int64_t>(max_kept, kept_len[t]);
    }
    if (max_nc > 65536)
        throw std::invalid_argument("more than 65536 blocks in one posting list");
    std::vector<int32_t> cpos(static_cast<size_t>(std::max<int64_t>(cptr.back(), 1)));
    {
        const int nth = std::max(1u, std::min(32u, std::thread::hardware_concurrency()));
        std::vector<std::thread> pool;
        for (int w = 0; w < nth; ++w) {
            pool.emplace_back([&, w] {
                std::vector<int32_t> perm;
                for (int32_t t = w; t < n_lists; t += nth) {
                    if (kept_len[t] == 0) continue;
                    draw_positions(static_cast<size_t>(kept_len[t]),
                                   static_cast<size_t>(cptr[t + 1] - cptr[t]),
                                   base_seed + static_cast<uint32_t>(t), perm, cpos.data() + cptr[t]);
                }
            });
        }
        for (auto& th : pool) th.join();
    }
    std::vector<uint8_t> tie(static_cast<size_t>(n_lists), 0);
    if (d_tie != nullptr) tie = to_host(d_tie, tie.size(), s);
    arena.release(before_keys);
    if (ESZ == 4) reference_tie_order(h, h_post, kept_ptr, tie, cap, kept, s);
    const int64_t* d_cptr = arena.put(cptr.data(), nl1);
    const int32_t* d_cpos = arena.put(cpos.data(), cpos.size());

    clock.mark("postings, centroids");
    // ---- 3. assignment
    uint32_t* akey = arena.take<uint32_t>(static_cast<size_t>(total_kept));
    // centroid entries per list bound: max_nc rows of the longest rows
    int64_t max_row = 0;
    for (int64_t d = 0; d < n_docs; ++d)
        max_row = std::max<int64_t>(max_row, h.indptr[d + 1] - h.indptr[d]);
    bool assigned = total_kept == 0;
    const nsp::AssignLists lists{n_lists, d_kept_ptr, kept,     d_cptr,
                                 d_cpos,  max_nc,     max_kept, max_row};
    if (ESZ == 1 && !assigned) {
        std::vector<int64_t> df(static_cast<size_t>(n_lists));
        for (int32_t t = 0; t < n_lists; ++t) df[t] = h_post[t + 1] - h_post[t];
        assigned = nsp::assign_u8(f, lists, df, akey, s, arena);
    }
    if (!assigned) {
        int* repeats = arena.take<int>(1);
        cuda_check(cudaMemsetAsync(repeats, 0, sizeof(int), s), "memset");
        repeats_kernel<<<sms * 7, kSeenWarps * 32, 0, s>>>(f, repeats);
        cuda_check(cudaGetLastError(), "repeats_kernel");
        if (to_host(repeats, 1, s)[0] != 0 || (ESZ == 1 && max_row > nsp::kAssignMaxRowU8))
            assign_general<ESZ, true>(f, lists, akey, s, arena);
        else
            assign_general<ESZ, false>(f, lists, akey, s, arena);
    }

    clock.mark("assignment");
    // ---- 4. blocks: centroid first, members in list order
    // (the per-block and per-posting arrays are the index's own)
    DevArray<int32_t> bdocs(static_cast<size_t>(std::max<int64_t>(total_kept, 1)));
    uint32_t* akey2 = arena.take<uint32_t>(static_cast<size_t>(total_kept));
    {
        const std::vector<int32_t> off32 = to_i32_offsets(kept_ptr);
        segmented_sort_pairs(akey, akey2, kept, bdocs.data(), total_kept, n_lists,
                             arena.put(off32.data(), nl1), s, /*stable=*/true, arena);
    }
    // one block per centroid, block docs where the sorted keys change cluster
    const int64_t n_blocks = cptr.back();
    DevArray<int64_t> bdp(static_cast<size_t>(n_blocks) + 1);
    uint16_t* local = arena.take<uint16_t>(static_cast<size_t>(n_blocks));
    block_bounds_kernel<<<sms * 8, 128, 0, s>>>(akey2, d_kept_ptr, d_cptr, n_lists, bdp.data(),
                                                local);
    cuda_check(cudaGetLastError(), "block_bounds_kernel");

    clock.mark("blocks");
    // ---- 5. summaries
    nsp::DevColumns cols;
    std::vector<int64_t> ltp{0};
    std::vector<std::pair<std::string, double>> steps;
    const nsp::BlockSet blocks{cptr.data(), d_cptr, n_lists, bdocs.data(), bdp.data(), local};
    nsp::summarize_blocks(ESZ, f, blocks, p.alpha, ESZ == 4 ? &h : nullptr, s, arena, cols, ltp,
                          clock.on ? &steps : nullptr);

    clock.mark("summaries");
    for (const auto& st_ : steps)
        std::fprintf(stderr, "[nsparse build]   %-14s %8.3f s\n", st_.first.c_str(), st_.second);
    // ---- 6. publish: the device image takes the built arrays; the host copy
    // is filled on demand (host_lists)
    std::lock_guard<std::mutex> g(st.mu);
    st.lists_dev.adopt(cptr, std::move(bdp), ltp, ESZ, dim, std::move(bdocs),
                       std::move(cols.sterm), std::move(cols.srun), std::move(cols.sblk),
                       std::move(cols.sval));
    st.lists = nsp::SeismicHost{};
    st.lists.esz = ESZ;
    st.list_esz.assign(static_cast<size_t>(n_lists), static_cast<uint8_t>(ESZ));
    st.host_valid = false;
    st.dev_valid = true;
}

}  // namespace

void seismic_build(SeismicState& st, int dim, const SeismicClusterParameters& params) {
    if (!st.vectors.terms_in_range(dim)) throw std::invalid_argument("term_id out of range");
    const int esz = st.vectors.host.esz;
    if (st.vectors.host.n() == 0) {
        // no documents: one empty list per term
        nsp::SeismicHost L;
        L.esz = esz;
        L.lbp.assign(static_cast<size_t>(dim) + 1, 0);
        L.ltp.assign(static_cast<size_t>(dim) + 1, 0);
        std::lock_guard<std::mutex> g(st.mu);
        st.lists = std::move(L);
        st.list_esz.assign(static_cast<size_t>(dim), static_cast<uint8_t>(esz));
        st.host_valid = true;
        st.dev_valid = false;
        return;
    }
    if (esz == 4) build_typed<4>(st, dim, params);
    else if (esz == 2) build_typed<2>(st, dim, params);
    else build_typed<1>(st, dim, params);
}

}  // namespace detail
}  // namespace nsparse
