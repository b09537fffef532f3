// Limits of the exact search's device postings (postings.cu), for host and
// device.
#ifndef NSP_POSTINGS_PLAN_H
#define NSP_POSTINGS_PLAN_H

#include <algorithm>
#include <climits>
#include <cstddef>
#include <cstdint>
#include <exception>
#include <vector>

#if defined(__CUDACC__)
#define NSP_POSTINGS_HD __host__ __device__
#else
#define NSP_POSTINGS_HD
#endif

namespace nsp {

// Positions of postings are held as int32. The search kernel computes
// positions up to kPostingsAhead past a run (a thread each, eight steps of a
// CTA ahead) to compare them with its end, so the last posting stays that far
// below 2^31: larger indexes take the tile kernel.
constexpr int32_t kPostingsAhead = 4096;
constexpr int64_t kMaxPostings = INT_MAX - kPostingsAhead;

// visit(p) for p = lo + first, lo + first + step, ... below hi: positions in
// 64 bits, since a grid's step (a million and more) past a run that ends near
// 2^31 has no int32.
template <class Visit>
NSP_POSTINGS_HD inline void each_posting(int32_t lo, int32_t hi, int64_t first, int64_t step,
                                         Visit visit) {
    for (int64_t p = lo + first; p < hi; p += step) visit(static_cast<int32_t>(p));
}

// Whether no score can leave the finite numbers: a bound on every partial sum
// of products from the largest magnitude stored and a bound on the sum of a
// query's magnitudes (65,536 roundings add less than half a percent). Not so
// where either is infinite or NaN.
inline bool finite_scores(float max_abs, double query_abs) {
    return static_cast<double>(max_abs) * query_abs < 3.0e38;
}

// Which terms also get a dense row. A term's postings are applied with a
// shared-memory read-modify-write each (about 10 L1 wavefronts per 32
// postings, random banks), its dense row with 12 wavefronts per 128 docs,
// fewer in a run of dense terms: dense is cheaper from about 0.3 of the docs
// on. 256 rows bound the memory at 1 KB per doc, and a term of few postings
// gets none, since a row fills whole chunks.
constexpr double kDenseShare = 0.3;
constexpr int32_t kMinDensePostings = 512;
constexpr size_t kMaxDense = 256;

// The dense terms, most frequent first, given each term's first posting
// (dim + 1 entries): at most as many as rows of `row_bytes` fit in a quarter
// of the device's free memory. The rows only save time, so they must not take
// the memory that the index itself needs.
inline std::vector<int32_t> dense_terms(const std::vector<int32_t>& start, int32_t n_docs,
                                        size_t row_bytes, size_t free_bytes) {
    std::vector<int32_t> out;
    const auto count = [&](int32_t t) { return start[t + 1] - start[t]; };
    for (int32_t t = 0; t + 1 < static_cast<int32_t>(start.size()); ++t)
        if (count(t) >= kDenseShare * n_docs && count(t) >= kMinDensePostings) out.push_back(t);
    std::sort(out.begin(), out.end(), [&](int32_t x, int32_t y) {
        return count(x) != count(y) ? count(x) > count(y) : x < y;
    });
    const size_t room = row_bytes > 0 ? free_bytes / 4 / row_bytes : 0;
    out.resize(std::min(out.size(), std::min(kMaxDense, room)));
    return out;
}

// The rows there are after alloc(rows): none where it throws (the memory went
// to someone else meanwhile).
template <class Alloc>
size_t allocate_dense_rows(size_t rows, Alloc alloc) {
    try {
        if (rows > 0) alloc(rows);
    } catch (const std::exception&) {
        return 0;
    }
    return rows;
}

}  // namespace nsp

#endif  // NSP_POSTINGS_PLAN_H
