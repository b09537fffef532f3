// Limits of the exact search's device postings (postings.cu), for host and
// device.
#ifndef NSP_POSTINGS_PLAN_H
#define NSP_POSTINGS_PLAN_H

#include <climits>
#include <cstdint>

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

}  // namespace nsp

#endif  // NSP_POSTINGS_PLAN_H
