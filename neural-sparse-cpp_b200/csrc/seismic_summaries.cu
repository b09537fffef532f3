// Block summaries of the SEISMIC build (the reference's
// cluster/inverted_list_clusters.cpp:37-124 and :230-293), one pass over the
// rows without sorting them.
//
// A block's summary takes its docs' rows in block order: per term the running
// max (a first value clamped at 0), and the block's mass as the sum of the
// maxima's increments in entry order (:89-115); the maxima by value
// descending, term ascending, are kept up to the one where their running sum
// reaches alpha of the mass (:43-51). In shared memory per block:
//
//   1. the block's terms as a bitmap over the vocabulary and its popcount
//      prefix, so a term's rank among the block's terms is two loads and a
//      popcount, and the maxima are a dense array in term order;
//   2. the maxima and the mass. fp32 and 16-bit sums depend on their order,
//      so increments are added one at a time in entry order by one lane; a
//      block of several warps hands the turn from doc to doc (named
//      barriers), while the other warps load rows and locate their ranks.
//      uint8 mass is an exact integer sum of the final maxima, in any order;
//   3. the cut. Values: a 64-bin histogram over the top four octaves bounds
//      the prefix that must reach alpha * mass (1% of slack against the
//      rounding of the sequential sum; if it does not, everything is taken),
//      only that prefix is sorted, and one thread adds it up in order. Codes:
//      the exact 256-bin histogram gives the level and the count directly;
//   4. the kept pairs go to the block's slot of a scratch array, are packed
//      per list, sorted by (term, block) and become the list's columns.
//
// A block of one doc whose row is strictly ascending (half of all entries at
// 80,000 docs and lambda 4000, a quarter at 1M and 6000) needs no steps 1-2:
// the row is the summary.
//
// What bounds it: instruction issue (~40 warp instructions per 32 entries and
// phase), then, for the few blocks of thousands of docs, the serial sum.
// Measured, all summaries of a build: fp32, 80,000 docs, lambda 4000 (1.2G
// entries in 3.7M blocks): 0.79 s when the entries were
// sorted by term and the maxima by value (about ten passes over global
// memory), 0.08 s now, 0.06 s of it in these kernels; SEISMIC-SQ 8-bit,
// 200,000 docs, lambda 6000 (3.2G entries): 0.33 s with a hash table per block
// and two passes, 0.15 s now, 0.05 s in these kernels.
#include <cuda_runtime.h>

#include <algorithm>
#include <chrono>
#include <cstdint>
#include <stdexcept>
#include <vector>

#include "ref_order.h"
#include "scan.h"
#include "segsort.cuh"
#include "seismic_summaries.h"

namespace nsp {
namespace {

constexpr unsigned kFull = 0xffffffffu;

// Tiers of blocks, by docs and by the most distinct terms they can hold
// (entries, at most the vocabulary): one strictly ascending row of up to
// kRowCap entries, a warp per block; then one, four and eight warps per block
// with room for kSmallCap, kMidCap and all of the vocabulary's terms.
// kRowCap covers the longest rows of the SPLADE shapes (400 terms); kSmallCap
// keeps 14 one-warp blocks on an SM and kMidCap three of four warps.
constexpr int kRowCap = 512;
constexpr int kSmallCap = 1024;
constexpr int kMidCap = 8192;
constexpr int kTiers = 4;
constexpr int kRowWarps = 4;  // warps per CTA of the single-row kernel
constexpr int kMidWarps = 4;
constexpr int kBigWarps = 8;

struct SumArgs {
    FwdView f;
    const int32_t* docs;
    const int64_t* bdp;
    const uint16_t* local;
    const int64_t* slot;   // first scratch element of each block (global ids)
    int64_t slot0;         // slot of the batch's first element
    int64_t b0;            // the batch's first block
    const int32_t* ids;    // the tier's blocks, relative to b0
    const unsigned* n_ids;
    unsigned* next;        // claim counter (tiers of claimed blocks)
    int32_t* retry;        // single rows that are not strictly ascending
    unsigned* n_retry;
    float alpha;
    int64_t* keep;         // kept pairs per block, relative to b0
    uint32_t* okey;        // scratch: term << 16 | block within its list
    float* oval;
    int32_t* tied;         // blocks with equal maxima across the cut (or nullptr)
    unsigned* n_tied;
    uint64_t* spill;       // sort buffers past shared memory, spill_cap per group
    int64_t spill_cap;
    uint32_t* gvals;       // maxima and terms past shared memory (or nullptr)
    uint16_t* gterms;
    int cap;               // distinct terms a block of this tier can hold
    int sel_cap;           // sort keys in shared memory
    int words;             // bitmap words
};

__host__ __device__ inline size_t align16(size_t x) { return (x + 15) & ~size_t(15); }

// Shared-memory layout of one group (a warp or a CTA working on one block).
struct SumLayout {
    size_t vals, terms, sel, bins, bits, pre, total;
};
__host__ __device__ inline SumLayout sum_layout(int cap, int sel_cap, int words, bool vals_in_smem) {
    SumLayout L;
    size_t o = 0;
    L.vals = o;  o += vals_in_smem ? align16(static_cast<size_t>(cap) * 4) : 0;
    L.sel = o;   o += align16(static_cast<size_t>(sel_cap) * 8);
    L.bins = o;  o += 256 * 4;
    L.terms = o; o += vals_in_smem ? align16(static_cast<size_t>(cap) * 2) : 0;
    L.bits = o;  o += align16(static_cast<size_t>(words) * 4);
    L.pre = o;   o += align16(static_cast<size_t>(words) * 2);
    L.total = o;
    return L;
}

template <int ESZ>
__device__ __forceinline__ float row_value(const void* val, int64_t i) {
    if constexpr (ESZ == 4) return __ldg(static_cast<const float*>(val) + i);
    if constexpr (ESZ == 2) return static_cast<float>(__ldg(static_cast<const uint16_t*>(val) + i));
    return static_cast<float>(__ldg(static_cast<const uint8_t*>(val) + i));
}

template <int NT>
__device__ __forceinline__ void group_sync() {
    if constexpr (NT == 32) __syncwarp();
    else __syncthreads();
}

// Sum of n shared-memory floats onto `sum`, one after another (n padded with
// zeros to a multiple of 4: no increment is negative, so +0.0 changes nothing).
__device__ __forceinline__ float add_in_order(float sum, const float* x, int n) {
    const float4* x4 = reinterpret_cast<const float4*>(x);
    for (int i = 0; i < n; i += 4) {
        const float4 v = x4[i >> 2];
        sum = __fadd_rn(sum, v.x);
        sum = __fadd_rn(sum, v.y);
        sum = __fadd_rn(sum, v.z);
        sum = __fadd_rn(sum, v.w);
    }
    return sum;
}

struct SumCut {
    int keep;   // pairs kept
    int vstar;  // the level the cut falls in (-1: every pair is kept)
    int r;      // that level's pairs kept (its smallest terms)
};

// The alpha cut (inverted_list_clusters.cpp:43-51) from the histogram of a
// block's uint8 maxima, by one warp: walking the pairs by value descending,
// the first count whose running sum `addup` satisfies addup / sum >= alpha.
// The running sums are integers below 2^24, so (float) of each is the
// reference's float accumulation; the division is the same correctly rounded
// one. No such count (sum 0, or alpha above 1): every pair is kept.
__device__ SumCut sum_u8_cut(const uint32_t* hist, uint32_t mass, int n_pairs, float alpha,
                             int lane) {
    uint32_t c[8];
    uint32_t cs = 0, ss = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const int v = 255 - 8 * lane - i;  // lane 0 holds the top levels
        c[i] = hist[v];
        cs += c[i];
        ss += c[i] * static_cast<uint32_t>(v);
    }
    // counts and sums of the levels above this lane's
    uint32_t ci = cs, si = ss;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t cu = __shfl_up_sync(kFull, ci, o);
        const uint32_t su = __shfl_up_sync(kFull, si, o);
        if (lane >= o) {
            ci += cu;
            si += su;
        }
    }
    uint32_t cnt_above = ci - cs, sum_above = si - ss;
    const float fm = static_cast<float>(mass);
    int found = -1;
#pragma unroll
    for (int i = 0; i < 8; ++i) {
        const uint32_t v = static_cast<uint32_t>(255 - 8 * lane - i);
        if (found < 0 && c[i] > 0) {
            const uint32_t end = sum_above + c[i] * v;
            if (__fdiv_rn(static_cast<float>(end), fm) >= alpha) {
                found = i;
            } else {
                sum_above = end;
                cnt_above += c[i];
            }
        }
    }
    const unsigned hit = __ballot_sync(kFull, found >= 0);
    SumCut out{n_pairs, -1, 0};
    if (hit == 0u) return out;
    const int src = __ffs(hit) - 1;
    int keep = 0, vstar = 0, r = 0;
    if (lane == src) {
        uint32_t cf = 0;
#pragma unroll
        for (int i = 0; i < 8; ++i)
            if (i == found) cf = c[i];
        const uint32_t v = static_cast<uint32_t>(255 - 8 * lane - found);
        // the smallest j in [1, cf] whose sum satisfies the test (the test
        // only turns true as j grows)
        uint32_t lo = 1, hi = cf;
        while (lo < hi) {
            const uint32_t mid = (lo + hi) >> 1;
            if (__fdiv_rn(static_cast<float>(sum_above + mid * v), fm) >= alpha)
                hi = mid;
            else
                lo = mid + 1;
        }
        keep = static_cast<int>(cnt_above + lo);
        vstar = static_cast<int>(v);
        r = static_cast<int>(lo);
    }
    out.keep = __shfl_sync(kFull, keep, src);
    out.vstar = __shfl_sync(kFull, vstar, src);
    out.r = __shfl_sync(kFull, r, src);
    return out;
}

// Scalars a group shares.
struct SumShared {
    unsigned vmax, count, bin, k;
    float mass;
    unsigned umass;
    SumCut cut;
    unsigned above[kBigWarps], ties[kBigWarps];
    unsigned wtot[kBigWarps];
};

// Codes: histogram, cut, and the kept pairs in term order (a level cut in two
// keeps its smallest terms). vals[0..nu) are the maxima's float bits.
template <int NT>
__device__ void cut_codes(const SumArgs& a, const uint32_t* vals, const uint16_t* terms, int nu,
                          int64_t rb, uint32_t* hist, SumShared& sh, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    for (int i = tid; i < 256; i += NT) hist[i] = 0u;
    if (tid == 0) sh.umass = 0u;
    group_sync<NT>();
    uint32_t m = 0u;
    for (int i = tid; i < nu; i += NT) {
        const uint32_t v = static_cast<uint32_t>(__uint_as_float(vals[i]));
        m += v;
        atomicAdd(&hist[v], 1u);
    }
    m = __reduce_add_sync(kFull, m);
    if (lane == 0 && m > 0u) atomicAdd(&sh.umass, m);
    group_sync<NT>();
    if (warp == 0) {
        const SumCut c = sum_u8_cut(hist, sh.umass, nu, a.alpha, lane);
        if (lane == 0) sh.cut = c;
    }
    group_sync<NT>();
    const SumCut cut = sh.cut;
    const int64_t b = a.b0 + rb;
    const int64_t out = a.slot[b] - a.slot0;
    const uint32_t bl = a.local[b];
    // each warp a contiguous range of ranks; its kept pairs start after the
    // ranges' before it
    constexpr int kW = NT / 32;
    const int per = ((nu + kW - 1) / kW + 31) & ~31;
    const int lo = warp * per, hi = min(nu, lo + per);
    uint32_t above0 = 0u, ties0 = 0u;
    if constexpr (kW > 1) {
        uint32_t na = 0u, nt = 0u;
        for (int i0 = lo; i0 < hi; i0 += 32) {
            const int i = i0 + lane;
            const int v = i < hi ? static_cast<int>(__uint_as_float(vals[i])) : -2;
            na += __popc(__ballot_sync(kFull, v > cut.vstar));
            nt += __popc(__ballot_sync(kFull, v == cut.vstar));
        }
        if (lane == 0) {
            sh.above[warp] = na;
            sh.ties[warp] = nt;
        }
        group_sync<NT>();
        for (int w = 0; w < warp; ++w) {
            above0 += sh.above[w];
            ties0 += sh.ties[w];
        }
    }
    const uint32_t r = static_cast<uint32_t>(cut.r);
    const unsigned below = (1u << lane) - 1u;
    for (int i0 = lo; i0 < hi; i0 += 32) {
        const int i = i0 + lane;
        const int v = i < hi ? static_cast<int>(__uint_as_float(vals[i])) : -2;
        const unsigned am = __ballot_sync(kFull, v > cut.vstar);
        const unsigned tm = __ballot_sync(kFull, v == cut.vstar);
        const uint32_t ab = above0 + __popc(am & below);
        const uint32_t tb = ties0 + __popc(tm & below);
        if (v > cut.vstar || (v == cut.vstar && tb < r)) {
            const int64_t o = out + ab + min(tb, r);
            a.okey[o] = (static_cast<uint32_t>(terms[i]) << 16) | bl;
            a.oval[o] = static_cast<float>(v);
        }
        above0 += __popc(am);
        ties0 += __popc(tm);
    }
    if (tid == 0) a.keep[rb] = cut.keep;
    group_sync<NT>();
}

// Sorts buf[0..n) ascending (keys are distinct); `cap` holds the next power
// of two at least.
template <int NT>
__device__ void sort_keys(uint64_t* buf, int n, int tid) {
    constexpr int kPer = 4;
    if (n <= NT * kPer && n <= 512) {
        // by rank: every thread counts the keys below its own
        uint64_t k[kPer];
        int r[kPer];
#pragma unroll
        for (int u = 0; u < kPer; ++u) {
            const int i = u * NT + tid;
            k[u] = i < n ? buf[i] : 0ull;
            r[u] = 0;
        }
        if (n <= NT) {
            for (int j = 0; j < n; ++j) r[0] += buf[j] < k[0] ? 1 : 0;
        } else {
            for (int j = 0; j < n; ++j) {
                const uint64_t x = buf[j];
#pragma unroll
                for (int u = 0; u < kPer; ++u) r[u] += x < k[u] ? 1 : 0;
            }
        }
        group_sync<NT>();
#pragma unroll
        for (int u = 0; u < kPer; ++u)
            if (u * NT + tid < n) buf[r[u]] = k[u];
        group_sync<NT>();
        return;
    }
    int p2 = 1;
    while (p2 < n) p2 <<= 1;
    for (int i = n + tid; i < p2; i += NT) buf[i] = ~0ull;
    group_sync<NT>();
    for (int k = 2; k <= p2; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            for (int i = tid; i < p2; i += NT) {
                const int o = i ^ j;
                if (o > i) {
                    const uint64_t x = buf[i], y = buf[o];
                    if (((i & k) == 0) == (x > y)) {
                        buf[i] = y;
                        buf[o] = x;
                    }
                }
            }
            group_sync<NT>();
        }
    }
}

// Values: the cut by the sorted prefix, and the kept pairs in sorted order.
template <int NT>
__device__ void cut_values(const SumArgs& a, const uint32_t* vals, const uint16_t* terms, int nu,
                           int64_t rb, float mass, uint64_t* sel, uint64_t* spill, uint32_t* bins,
                           SumShared& sh, int tid) {
    const int lane = tid & 31, warp = tid >> 5;
    constexpr int kShift = 19;  // bins of 1/16 octave
    for (int i = tid; i < 64; i += NT) bins[i] = 0u;
    if (tid == 0) {
        sh.vmax = 0u;
        sh.bin = 63u;
    }
    group_sync<NT>();
    uint32_t vm = 0u;  // maxima are >= 0: their bits order as they do
    for (int i = tid; i < nu; i += NT) vm = max(vm, vals[i]);
    vm = __reduce_max_sync(kFull, vm);
    if constexpr (NT > 32) {
        if (lane == 0) atomicMax(&sh.vmax, vm);
        group_sync<NT>();
        vm = sh.vmax;
    }
    // fixed-point sums (each bin's is rounded down): 65536 terms of at most
    // 65000 units stay below 2^32
    const float scale = 65000.0f / __uint_as_float(vm);
    const float need = a.alpha * mass * scale * 1.01f + 1.0f;
    const bool part = vm > 0u && vm < 0x7f800000u && mass < 3.0e38f && scale < 3.0e38f;
    if (part) {
        for (int i = tid; i < nu; i += NT) {
            const uint32_t v = vals[i];
            atomicAdd(&bins[min((vm - v) >> kShift, 63u)],
                      static_cast<uint32_t>(__uint_as_float(v) * scale));
        }
        group_sync<NT>();
        if (warp == 0) {
            const uint32_t c0 = bins[2 * lane], c1 = bins[2 * lane + 1];
            uint32_t incl = c0 + c1;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += y;
            }
            const bool h1 = static_cast<float>(incl) >= need;
            const bool h0 = static_cast<float>(incl - c1) >= need;
            const unsigned m = __ballot_sync(kFull, h1);
            if (m != 0u && lane == __ffs(m) - 1)
                sh.bin = static_cast<unsigned>(2 * lane + (h0 ? 0 : 1));
        }
        group_sync<NT>();
    }
    unsigned bin = sh.bin;
    uint64_t* buf = sel;
    int n = 0, k = 0;
    for (;;) {
        // the pairs of the first `bin` + 1 bins (63: all), as (~value, rank)
        const bool all = bin >= 63u;
        for (int room = a.sel_cap;; room = INT32_MAX) {
            if constexpr (NT > 32) {
                if (tid == 0) sh.count = 0u;
                group_sync<NT>();
            }
            n = 0;
            for (int i0 = 0; i0 < nu; i0 += NT) {
                const int i = i0 + tid;
                const uint32_t v = i < nu ? vals[i] : 0u;
                const bool in = i < nu && (all || ((vm - v) >> kShift) <= bin);
                const unsigned m = __ballot_sync(kFull, in);
                int base = n;
                if constexpr (NT > 32) {
                    if (lane == 0 && m != 0u) base = static_cast<int>(atomicAdd(&sh.count, __popc(m)));
                    base = __shfl_sync(kFull, base, 0);
                }
                const int p = base + __popc(m & ((1u << lane) - 1u));
                if (in && p < room)
                    buf[p] = (static_cast<uint64_t>(~v) << 32) | static_cast<uint32_t>(i);
                n += __popc(m);
            }
            if constexpr (NT > 32) {
                group_sync<NT>();
                n = static_cast<int>(sh.count);
            }
            if (n <= room) break;
            buf = spill;
            group_sync<NT>();
        }
        group_sync<NT>();
        sort_keys<NT>(buf, n, tid);
        // the reference's running sum; the division only where it can matter
        if (tid == 0) {
            const float guard = a.alpha * mass * 0.999999f;
            float addup = 0.0f;
            int kk = 0;
            const uint32_t* hi = reinterpret_cast<const uint32_t*>(buf) + 1;
            for (int i = 0; i < n; ++i) {
                addup = __fadd_rn(addup, __uint_as_float(~hi[2 * i]));
                if (!(addup < guard) && __fdiv_rn(addup, mass) >= a.alpha) {
                    kk = i + 1;
                    break;
                }
            }
            sh.k = static_cast<unsigned>(kk);
        }
        group_sync<NT>();
        k = static_cast<int>(sh.k);
        if (k > 0 || all) break;
        bin = 63u;
        group_sync<NT>();
    }
    if (k == 0) k = nu;
    const int64_t b = a.b0 + rb;
    const int64_t out = a.slot[b] - a.slot0;
    const uint32_t bl = a.local[b];
    for (int i = tid; i < k; i += NT) {
        const uint64_t x = buf[i];
        a.okey[out + i] =
            (static_cast<uint32_t>(terms[static_cast<uint32_t>(x)]) << 16) | bl;
        a.oval[out + i] = __uint_as_float(~static_cast<uint32_t>(x >> 32));
    }
    if (tid == 0) {
        a.keep[rb] = k;
        if (a.tied != nullptr && k < n && (buf[k - 1] >> 32) == (buf[k] >> 32))
            a.tied[atomicAdd(a.n_tied, 1u)] = static_cast<int32_t>(rb);
    }
    group_sync<NT>();
}

// Blocks of one doc: the row is the summary when its terms are strictly
// ascending (others are handed to the next tier).
template <int ESZ>
__global__ void __launch_bounds__(kRowWarps * 32) sum_rows_kernel(SumArgs a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SumShared shared[kRowWarps];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const SumLayout L = sum_layout(a.cap, a.sel_cap, 0, true);
    unsigned char* sm = smem + warp * L.total;
    uint32_t* vals = reinterpret_cast<uint32_t*>(sm + L.vals);
    uint16_t* terms = reinterpret_cast<uint16_t*>(sm + L.terms);
    SumShared& sh = shared[warp];
    const int64_t w0 = static_cast<int64_t>(blockIdx.x) * kRowWarps + warp;
    const int64_t nw = static_cast<int64_t>(gridDim.x) * kRowWarps;
    const int64_t n = *a.n_ids;
    for (int64_t j = w0; j < n; j += nw) {
        const int64_t rb = a.ids[j];
        const uint2 ri = __ldg(a.f.rowinfo + a.docs[a.bdp[a.b0 + rb]]);
        const int64_t row = static_cast<int64_t>(ri.x) * kRowAlign;
        const int len = static_cast<int>(ri.y);
        // 8 elements per lane: rows are padded to 64 elements, so the 16-byte
        // loads stay inside them
        bool asc = true;
        uint32_t last = 0u;  // the last term before this step, plus 1
        for (int e0 = 0; e0 < len; e0 += 256) {
            const int e = e0 + 8 * lane;
            uint4 t4 = make_uint4(0u, 0u, 0u, 0u);
            float v[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) v[u] = 0.0f;
            if (e < len) {
                t4 = __ldg(reinterpret_cast<const uint4*>(a.f.idx + row + e));
                if constexpr (ESZ == 4) {
                    const float4* p = reinterpret_cast<const float4*>(
                        static_cast<const float*>(a.f.val) + row + e);
                    const float4 x = __ldg(p), y = __ldg(p + 1);
                    v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
                    v[4] = y.x; v[5] = y.y; v[6] = y.z; v[7] = y.w;
                } else if constexpr (ESZ == 2) {
                    const uint4 x = __ldg(reinterpret_cast<const uint4*>(
                        static_cast<const uint16_t*>(a.f.val) + row + e));
                    const uint32_t w[4] = {x.x, x.y, x.z, x.w};
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        v[u] = static_cast<float>((w[u >> 1] >> (16 * (u & 1))) & 0xffffu);
                } else {
                    const uint2 x = __ldg(reinterpret_cast<const uint2*>(
                        static_cast<const uint8_t*>(a.f.val) + row + e));
#pragma unroll
                    for (int u = 0; u < 8; ++u)
                        v[u] = static_cast<float>(((u < 4 ? x.x : x.y) >> (8 * (u & 3))) & 0xffu);
                }
            }
            const uint32_t tw[4] = {t4.x, t4.y, t4.z, t4.w};
            uint32_t t[8];
#pragma unroll
            for (int u = 0; u < 8; ++u) t[u] = (tw[u >> 1] >> (16 * (u & 1))) & 0xffffu;
            uint32_t prev = __shfl_up_sync(kFull, t[7] + 1u, 1);
            if (lane == 0) prev = last;
#pragma unroll
            for (int u = 0; u < 8; ++u) {
                if (e + u < len) {
                    asc = asc && t[u] + 1u > prev;
                    prev = t[u] + 1u;
                }
                // the first value of a term: max(0, v)
                if (!(e + u < len && v[u] > 0.0f)) v[u] = 0.0f;
            }
            last = __shfl_sync(kFull, t[7] + 1u, 31);
            if (e < a.cap) {
                uint4* vp = reinterpret_cast<uint4*>(vals + e);
                vp[0] = make_uint4(__float_as_uint(v[0]), __float_as_uint(v[1]),
                                   __float_as_uint(v[2]), __float_as_uint(v[3]));
                vp[1] = make_uint4(__float_as_uint(v[4]), __float_as_uint(v[5]),
                                   __float_as_uint(v[6]), __float_as_uint(v[7]));
                *reinterpret_cast<uint4*>(terms + e) = t4;
            }
        }
        if (!__all_sync(kFull, asc)) {
            if (lane == 0) a.retry[atomicAdd(a.n_retry, 1u)] = static_cast<int32_t>(rb);
            continue;
        }
        __syncwarp();
        uint32_t* bins = reinterpret_cast<uint32_t*>(sm + L.bins);
        if constexpr (ESZ == 1) {
            cut_codes<32>(a, vals, terms, len, rb, bins, sh, lane);
        } else {
            float mass = 0.0f;
            if (lane == 0)
                mass = add_in_order(0.0f, reinterpret_cast<const float*>(vals), (len + 3) & ~3);
            mass = __shfl_sync(kFull, mass, 0);
            cut_values<32>(a, vals, terms, len, rb, mass,
                           reinterpret_cast<uint64_t*>(sm + L.sel), a.spill + w0 * a.spill_cap,
                           bins, sh, lane);
        }
    }
}

// Named barriers 1..W hand the turn from the warp of one doc to the next's.
__device__ __forceinline__ void turn_wait(int id) {
    asm volatile("bar.sync %0, 64;" ::"r"(id) : "memory");
}
__device__ __forceinline__ void turn_pass(int id) {
    __threadfence_block();
    asm volatile("bar.arrive %0, 64;" ::"r"(id) : "memory");
}

// Any block of up to a.cap distinct terms, by a CTA of W warps.
template <int ESZ, int W>
__global__ void __launch_bounds__(W * 32) sum_blocks_kernel(SumArgs a) {
    constexpr int NT = W * 32;
    constexpr int kChunks = W > 1 ? 8 : 4;  // of 32 entries, in registers at once
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ SumShared sh;
    __shared__ __align__(16) float inc[W][kChunks * 32 + 4];  // increments, in entry order
    __shared__ unsigned s_job;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const bool in_smem = a.gvals == nullptr;
    const SumLayout L = sum_layout(a.cap, a.sel_cap, a.words, in_smem);
    uint32_t* vals = in_smem ? reinterpret_cast<uint32_t*>(smem + L.vals)
                             : a.gvals + static_cast<size_t>(blockIdx.x) * a.cap;
    uint16_t* terms = in_smem ? reinterpret_cast<uint16_t*>(smem + L.terms)
                              : a.gterms + static_cast<size_t>(blockIdx.x) * a.cap;
    uint64_t* sel = reinterpret_cast<uint64_t*>(smem + L.sel);
    uint32_t* bins = reinterpret_cast<uint32_t*>(smem + L.bins);
    uint32_t* bits = reinterpret_cast<uint32_t*>(smem + L.bits);
    uint16_t* pre = reinterpret_cast<uint16_t*>(smem + L.pre);
    const unsigned n = *a.n_ids;
    for (;;) {
        if (tid == 0) s_job = atomicAdd(a.next, 1u);
        for (int i = tid; i < a.words; i += NT) bits[i] = 0u;
        __syncthreads();
        const unsigned job = s_job;
        if (job >= n) break;
        const int64_t rb = a.ids[job];
        const int64_t d0 = a.bdp[a.b0 + rb];
        const int nd = static_cast<int>(a.bdp[a.b0 + rb + 1] - d0);
        // 1. the block's terms: 8 row elements per lane; a bit already set
        // costs no atomic
        for (int j = warp; j < nd; j += W) {
            const uint2 ri = __ldg(a.f.rowinfo + __ldg(a.docs + d0 + j));
            const int64_t row = static_cast<int64_t>(ri.x) * kRowAlign;
            const int len = static_cast<int>(ri.y);
            for (int e = 8 * lane; e < len; e += 256) {
                const uint4 t4 = __ldg(reinterpret_cast<const uint4*>(a.f.idx + row + e));
                const uint32_t tw[4] = {t4.x, t4.y, t4.z, t4.w};
#pragma unroll
                for (int u = 0; u < 8; ++u) {
                    const uint32_t t = (tw[u >> 1] >> (16 * (u & 1))) & 0xffffu;
                    const uint32_t bit = 1u << (t & 31);
                    if (e + u < len && !(bits[t >> 5] & bit)) atomicOr(&bits[t >> 5], bit);
                }
            }
        }
        __syncthreads();
        // ranks: exclusive popcount prefix of the bitmap's words
        const int per = (a.words + NT - 1) / NT;
        const int wl = min(a.words, tid * per), wh = min(a.words, wl + per);
        int mine = 0;
        for (int i = wl; i < wh; ++i) mine += __popc(bits[i]);
        int incl = mine;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        int run = incl - mine, nu = 0;
        if constexpr (W > 1) {
            if (lane == 31) sh.wtot[warp] = static_cast<unsigned>(incl);
            __syncthreads();
            for (int w = 0; w < W; ++w) {
                run += w < warp ? static_cast<int>(sh.wtot[w]) : 0;
                nu += static_cast<int>(sh.wtot[w]);
            }
        } else {
            nu = __shfl_sync(kFull, incl, 31);
        }
        for (int i = wl; i < wh; ++i) {
            pre[i] = static_cast<uint16_t>(run);
            run += __popc(bits[i]);
        }
        for (int i = tid; i < nu; i += NT) vals[i] = 0u;
        if (tid == 0) sh.mass = 0.0f;
        __syncthreads();
        // 2. maxima, and (values) the mass in entry order
        for (int j = warp; j < nd; j += W) {
            const uint2 ri = __ldg(a.f.rowinfo + __ldg(a.docs + d0 + j));
            const int64_t row = static_cast<int64_t>(ri.x) * kRowAlign;
            const int len = static_cast<int>(ri.y);
            uint32_t last = 0u;  // the last term of the step before, plus 1
            bool turn = W == 1 || ESZ == 1 || j == 0;
            float mass = 0.0f;
            for (int e0 = 0; e0 < len; e0 += kChunks * 32) {
                uint32_t t[kChunks];
                float v[kChunks];
                int r[kChunks];
                bool asc = true;
#pragma unroll
                for (int c = 0; c < kChunks; ++c) {
                    const int e = e0 + c * 32 + lane;
                    t[c] = 0u;
                    v[c] = 0.0f;
                    r[c] = -1;
                    if (e < len) {
                        t[c] = __ldg(a.f.idx + row + e);
                        v[c] = row_value<ESZ>(a.f.val, row + e);
                    }
                }
#pragma unroll
                for (int c = 0; c < kChunks; ++c) {
                    if (e0 + c * 32 + lane < len) {
                        const uint32_t w = t[c] >> 5;
                        r[c] = pre[w] + __popc(bits[w] & ((1u << (t[c] & 31)) - 1u));
                    }
                }
                if constexpr (ESZ == 1) {
                    // codes: maxima in any order
#pragma unroll
                    for (int c = 0; c < kChunks; ++c) {
                        if (r[c] >= 0) {
                            atomicMax(&vals[r[c]], __float_as_uint(v[c]));
                            terms[r[c]] = static_cast<uint16_t>(t[c]);
                        }
                    }
                } else {
#pragma unroll
                    for (int c = 0; c < kChunks; ++c) {
                        uint32_t prev = __shfl_up_sync(kFull, t[c] + 1u, 1);
                        if (lane == 0) prev = last;
                        asc = asc && (r[c] < 0 || t[c] + 1u > prev);
                        last = __shfl_sync(kFull, t[c] + 1u, 31);
                    }
                    asc = __all_sync(kFull, asc);
                    if (!turn) {
                        turn_wait(1 + warp);
                        turn = true;
                    }
                    float d[kChunks];
                    if (asc) {
                        // distinct terms: every maximum is read before any is written
                        float m[kChunks];
#pragma unroll
                        for (int c = 0; c < kChunks; ++c)
                            m[c] = r[c] >= 0 ? __uint_as_float(vals[r[c]]) : 0.0f;
#pragma unroll
                        for (int c = 0; c < kChunks; ++c) {
                            d[c] = 0.0f;
                            if (r[c] >= 0) {
                                if (v[c] > m[c]) {
                                    d[c] = __fsub_rn(v[c], m[c]);
                                    vals[r[c]] = __float_as_uint(v[c]);
                                }
                                terms[r[c]] = static_cast<uint16_t>(t[c]);
                            }
                        }
                    } else {
                        // a term may repeat: one entry at a time
#pragma unroll
                        for (int c = 0; c < kChunks; ++c) {
                            d[c] = 0.0f;
                            for (int l = 0; l < 32; ++l) {
                                if (l == lane && r[c] >= 0) {
                                    const float m = __uint_as_float(vals[r[c]]);
                                    if (v[c] > m) {
                                        d[c] = __fsub_rn(v[c], m);
                                        vals[r[c]] = __float_as_uint(v[c]);
                                    }
                                    terms[r[c]] = static_cast<uint16_t>(t[c]);
                                }
                                __syncwarp();
                            }
                        }
                    }
                    // the increments in entry order, then their sum
                    int ni = 0;
#pragma unroll
                    for (int c = 0; c < kChunks; ++c) {
                        const unsigned m = __ballot_sync(kFull, d[c] > 0.0f);
                        if (d[c] > 0.0f) inc[warp][ni + __popc(m & ((1u << lane) - 1u))] = d[c];
                        ni += __popc(m);
                    }
                    if (lane < 4) inc[warp][ni + lane] = 0.0f;
                    __syncwarp();
                    if (lane == 0 && ni > 0) {
                        if (e0 == 0) mass = sh.mass;
                        mass = add_in_order(mass, inc[warp], (ni + 3) & ~3);
                        sh.mass = mass;
                    } else if (lane == 0 && e0 == 0) {
                        mass = sh.mass;
                    }
                    __syncwarp();
                }
            }
            if constexpr (ESZ != 1 && W > 1) {
                if (!turn) turn_wait(1 + warp);  // an empty row passes the turn on
                if (j + 1 < nd) turn_pass(1 + (warp + 1 == W ? 0 : warp + 1));
            }
        }
        __syncthreads();
        // 3. the cut
        if constexpr (ESZ == 1)
            cut_codes<NT>(a, vals, terms, nu, rb, bins, sh, tid);
        else
            cut_values<NT>(a, vals, terms, nu, rb, sh.mass, sel,
                           a.spill + static_cast<size_t>(blockIdx.x) * a.spill_cap, bins, sh, tid);
        __syncthreads();
    }
}

// ------------------------------------------------------ blocks and tiers --

// ucap[b] = the most distinct terms block b can hold: its docs' row lengths
// summed, at most `dim`. A warp takes 32 blocks: a lane each, long blocks
// together.
__global__ void block_terms_kernel(FwdView f, const int32_t* docs, const int64_t* bdp, int64_t nb,
                                   int64_t* ucap) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t w = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5;
         w * 32 < nb; w += nw) {
        const int64_t b = w * 32 + lane;
        int64_t lo = 0, hi = 0;
        if (b < nb) {
            lo = bdp[b];
            hi = bdp[b + 1];
        }
        int64_t e = 0;
        const bool big = hi - lo > 16;
        if (!big)
            for (int64_t j = lo; j < hi; ++j) e += f.rowinfo[docs[j]].y;
        unsigned m = __ballot_sync(kFull, big);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const int64_t l = __shfl_sync(kFull, lo, src), h = __shfl_sync(kFull, hi, src);
            int64_t x = 0;
            for (int64_t j = l + lane; j < h; j += 32) x += f.rowinfo[docs[j]].y;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
            if (lane == src) e = x;
        }
        if (b < nb) ucap[b] = e < f.dim ? e : f.dim;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) ucap[nb] = 0;
}

__global__ void gather_i64_kernel(const int64_t* src, const int64_t* at, int32_t n, int64_t at0,
                                  int64_t* out64, int32_t* out32) {
    for (int32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const int64_t v = src[at[i] - at0];
        if (out64 != nullptr) out64[i] = v;
        if (out32 != nullptr) out32[i] = static_cast<int32_t>(v);
    }
}

// The batch's blocks by tier; an empty block keeps nothing.
__global__ void tier_kernel(const int64_t* bdp, const int64_t* slot, int64_t b0, int64_t nb,
                            int32_t* ids, unsigned* n_ids, int64_t* keep) {
    const int lane = threadIdx.x & 31;
    const int64_t step = static_cast<int64_t>(gridDim.x) * blockDim.x;
    for (int64_t i0 = blockIdx.x * static_cast<int64_t>(blockDim.x); i0 < nb; i0 += step) {
        const int64_t i = i0 + threadIdx.x;
        int tier = -1;
        if (i < nb) {
            const int64_t cap = slot[b0 + i + 1] - slot[b0 + i];
            if (cap == 0) keep[i] = 0;
            else if (cap <= kRowCap && bdp[b0 + i + 1] - bdp[b0 + i] == 1) tier = 0;
            else tier = cap <= kSmallCap ? 1 : (cap <= kMidCap ? 2 : 3);
        }
#pragma unroll
        for (int t = 0; t < kTiers; ++t) {
            const unsigned m = __ballot_sync(kFull, tier == t);
            if (m == 0u) continue;
            unsigned base = 0;
            if (lane == 0) base = atomicAdd(n_ids + t, __popc(m));
            base = __shfl_sync(kFull, base, 0);
            if (tier == t)
                ids[static_cast<int64_t>(t) * nb + base + __popc(m & ((1u << lane) - 1u))] =
                    static_cast<int32_t>(i);
        }
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) keep[nb] = 0;
}

// Kept pairs from the blocks' scratch slots to their packed places, a warp
// per block.
__global__ void pack_pairs_kernel(const int64_t* slot, int64_t slot0, int64_t b0,
                                  const int64_t* kept_off, int64_t nb, const uint32_t* okey,
                                  const float* oval, uint32_t* tkey, float* tval) {
    const int lane = threadIdx.x & 31;
    const int64_t nw = (static_cast<int64_t>(gridDim.x) * blockDim.x) >> 5;
    for (int64_t b = (blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x) >> 5; b < nb;
         b += nw) {
        const int64_t src = slot[b0 + b] - slot0, dst = kept_off[b];
        const int n = static_cast<int>(kept_off[b + 1] - dst);
        for (int i = lane; i < n; i += 32) {
            tkey[dst + i] = okey[src + i];
            tval[dst + i] = oval[src + i];
        }
    }
}

// --------------------------------------------------------------- columns --

// Per kept summary pair (sorted by (term, block) within each list): its block
// id, its value as the index stores it, and a flag where a new term starts.
template <int ESZ>
__global__ void columns_kernel(const uint32_t* key, const float* val, int64_t n, uint16_t* blk,
                               uint8_t* out_val, int64_t* flag) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        blk[i] = static_cast<uint16_t>(key[i] & 0xffffu);
        const float v = val[i];
        if constexpr (ESZ == 4) {
            reinterpret_cast<float*>(out_val)[i] = v;
        } else if constexpr (ESZ == 2) {
            reinterpret_cast<uint16_t*>(out_val)[i] = static_cast<uint16_t>(v);
        } else {
            out_val[i] = static_cast<uint8_t>(v);
        }
        flag[i] = (i == 0 || (key[i] >> 16) != (key[i - 1] >> 16)) ? 1 : 0;
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) flag[n] = 0;
}

// A list's first pair always starts a column (its term may equal the last
// term of the list before).
__global__ void list_start_kernel(const int32_t* list_off, int32_t nl, int64_t n, int64_t* flag) {
    const int32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l < nl && list_off[l] < list_off[l + 1] && list_off[l] < n) flag[list_off[l]] = 1;
}

__global__ void column_compact_kernel(const uint32_t* key, const int64_t* flag, const int64_t* pos,
                                      int64_t n, uint16_t* term, int64_t* start) {
    for (int64_t i = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; i < n;
         i += static_cast<int64_t>(gridDim.x) * blockDim.x) {
        if (flag[i]) {
            term[pos[i]] = static_cast<uint16_t>(key[i] >> 16);
            start[pos[i]] = i;
        }
    }
}

// Columns before each list boundary.
__global__ void list_cols_kernel(const int32_t* list_off, int32_t nl, const int64_t* pos,
                                 int64_t* cols) {
    const int32_t l = blockIdx.x * blockDim.x + threadIdx.x;
    if (l <= nl) cols[l] = pos[list_off[l]];
}

// Column boundaries of a batch: column c > 0 starts where column c-1 ends;
// the last ends after the batch's n_kept entries; all offset by `ebase`.
__global__ void column_bounds_kernel(const int64_t* start, int64_t n_cols, int64_t ebase,
                                     int64_t n_kept, int64_t* srun_tail) {
    for (int64_t c = blockIdx.x * static_cast<int64_t>(blockDim.x) + threadIdx.x; c < n_cols;
         c += static_cast<int64_t>(gridDim.x) * blockDim.x)
        srun_tail[c] = ebase + (c + 1 < n_cols ? start[c + 1] : n_kept);
}

// A batch's columns, held until all batches are done.
struct Piece {
    const uint16_t* term;
    const int64_t* start;
    const uint16_t* blk;
    const uint8_t* val;
    int64_t n_cols, n_kept;
};

struct Steps {
    std::vector<std::pair<std::string, double>>* out;
    cudaStream_t s;
    std::chrono::steady_clock::time_point t = std::chrono::steady_clock::now();
    void mark(const char* name) {
        if (out == nullptr) return;
        cudaStreamSynchronize(s);
        const auto now = std::chrono::steady_clock::now();
        const double dt = std::chrono::duration<double>(now - t).count();
        t = now;
        for (auto& a : *out)
            if (a.first == name) {
                a.second += dt;
                return;
            }
        out->emplace_back(name, dt);
    }
};

// Kept pairs of `nl` lists (tkey, tval; list_koff[l] the first of list l)
// become the lists' summary columns, term-major per list (build_transpose,
// inverted_list_clusters.cpp:230-293), in memory of `keep`.
Piece emit_columns(int esz, int32_t nl, int64_t n_kept, const uint32_t* tkey, const float* tval,
                   const int32_t* list_koff, size_t cols_before, cudaStream_t s, Arena& scratch,
                   Arena& keep, Steps& steps, std::vector<int64_t>& ltp) {
    const int sms = device_sm_count();
    const size_t nk = static_cast<size_t>(n_kept);
    uint32_t* key = scratch.take<uint32_t>(nk);
    float* val = scratch.take<float>(nk);
    segmented_sort_pairs(tkey, key, tval, val, n_kept, nl, list_koff, s, /*stable=*/false, scratch);
    steps.mark("transpose sort");
    // block ids, values, and one run per (list, term) with its start
    uint16_t* blk = keep.take<uint16_t>(nk);
    uint8_t* out_val = keep.take<uint8_t>(nk * esz);
    int64_t* flag = scratch.take<int64_t>(nk + 1);
    int64_t* pos = scratch.take<int64_t>(nk + 1);
    int64_t* lcol = scratch.take<int64_t>(static_cast<size_t>(nl) + 1);
    auto* columns = esz == 4 ? columns_kernel<4> : (esz == 2 ? columns_kernel<2> : columns_kernel<1>);
    columns<<<sms * 8, 256, 0, s>>>(key, val, n_kept, blk, out_val, flag);
    cuda_check(cudaGetLastError(), "columns_kernel");
    list_start_kernel<<<std::max(1, (nl + 255) / 256), 256, 0, s>>>(list_koff, nl, n_kept, flag);
    cuda_check(cudaGetLastError(), "list_start_kernel");
    exclusive_scan_i64(flag, pos, n_kept + 1, s, scratch);
    list_cols_kernel<<<std::max(1, (nl + 1 + 255) / 256), 256, 0, s>>>(list_koff, nl, pos, lcol);
    cuda_check(cudaGetLastError(), "list_cols_kernel");
    // only the per-list column counts come back to the host
    std::vector<int64_t> h_lcol(static_cast<size_t>(nl) + 1);
    cuda_check(cudaMemcpyAsync(h_lcol.data(), lcol, h_lcol.size() * 8, cudaMemcpyDeviceToHost, s),
               "D2H");
    cuda_check(cudaStreamSynchronize(s), "D2H");
    const int64_t n_cols = h_lcol.back();
    uint16_t* term = keep.take<uint16_t>(static_cast<size_t>(n_cols));
    int64_t* start = keep.take<int64_t>(static_cast<size_t>(n_cols));
    column_compact_kernel<<<sms * 8, 256, 0, s>>>(key, flag, pos, n_kept, term, start);
    cuda_check(cudaGetLastError(), "column_compact_kernel");
    for (int32_t l = 0; l < nl; ++l)
        ltp.push_back(static_cast<int64_t>(cols_before) + h_lcol[l + 1]);
    steps.mark("columns");
    return {term, start, blk, out_val, n_cols, n_kept};
}

// The batches' columns one after another, in arrays of exactly their size.
void join_columns(int esz, const std::vector<Piece>& pieces, cudaStream_t s, DevColumns& out) {
    size_t cols = 0, entries = 0;
    for (const Piece& p : pieces) {
        cols += static_cast<size_t>(p.n_cols);
        entries += static_cast<size_t>(p.n_kept);
    }
    out.sterm.resize(cols);
    out.srun.resize(cols + 1);
    out.sblk.resize(entries);
    out.sval.resize(entries * esz);
    cuda_check(cudaMemsetAsync(out.srun.data(), 0, sizeof(int64_t), s), "memset");
    size_t cb = 0, eb = 0;
    auto copy = [&](void* dst, const void* src, size_t bytes) {
        if (bytes > 0)
            cuda_check(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToDevice, s), "D2D");
    };
    for (const Piece& p : pieces) {
        const size_t nk = static_cast<size_t>(p.n_kept), nc = static_cast<size_t>(p.n_cols);
        copy(out.sterm.data() + cb, p.term, nc * sizeof(uint16_t));
        copy(out.sblk.data() + eb, p.blk, nk * sizeof(uint16_t));
        copy(out.sval.data() + eb * esz, p.val, nk * esz);
        if (nc > 0)
            column_bounds_kernel<<<device_sm_count() * 4, 256, 0, s>>>(
                p.start, p.n_cols, static_cast<int64_t>(eb), p.n_kept, out.srun.data() + cb + 1);
        cuda_check(cudaGetLastError(), "column_bounds_kernel");
        cb += nc;
        eb += nk;
    }
}

// fp32 blocks whose alpha cut falls between equal maxima keep the terms the
// reference's unstable sort keeps: for each, the reference's own sort on the
// host gives them (the count is the same: equal values give equal running
// sums), and the pairs written at the cut's value take those terms.
void settle_ties(const HostCsr& host, const BlockSet& blocks, const SumArgs& a, int64_t nb,
                 std::vector<int32_t> tied, cudaStream_t s) {
    std::sort(tied.begin(), tied.end());
    std::vector<int64_t> bdp(static_cast<size_t>(nb) + 1), slot(static_cast<size_t>(nb) + 1),
        keep(static_cast<size_t>(nb));
    auto fetch = [&](void* dst, const void* src, size_t bytes) {
        cuda_check(cudaMemcpyAsync(dst, src, bytes, cudaMemcpyDeviceToHost, s), "D2H");
    };
    fetch(bdp.data(), blocks.d_bdp + a.b0, bdp.size() * 8);
    fetch(slot.data(), a.slot + a.b0, slot.size() * 8);
    fetch(keep.data(), a.keep, keep.size() * 8);
    cuda_check(cudaStreamSynchronize(s), "D2H");
    std::vector<int32_t> docs(static_cast<size_t>(bdp.back() - bdp.front()));
    fetch(docs.data(), blocks.d_docs + bdp.front(), docs.size() * sizeof(int32_t));
    cuda_check(cudaStreamSynchronize(s), "D2H");
    std::vector<uint32_t> key;
    std::vector<float> val;
    std::vector<uint8_t> want(65536, 0);
    for (const int32_t b : tied) {
        const size_t k = static_cast<size_t>(keep[b]);
        const int64_t at = slot[b] - a.slot0;
        const std::vector<uint16_t> kept = reference_summary_kept(
            host, docs.data() + (bdp[b] - bdp[0]), static_cast<size_t>(bdp[b + 1] - bdp[b]),
            a.alpha);
        if (kept.size() != k)
            throw std::runtime_error("summary cut differs from the reference's count");
        key.resize(k);
        val.resize(k);
        fetch(key.data(), a.okey + at, k * sizeof(uint32_t));
        fetch(val.data(), a.oval + at, k * sizeof(float));
        cuda_check(cudaStreamSynchronize(s), "D2H");
        const float cut = val[k - 1];  // pairs are written by value descending
        for (const uint16_t t : kept) want[t] = 1;
        for (size_t i = 0; i < k; ++i)
            if (val[i] != cut) want[key[i] >> 16] = 0;
        // what is left are the reference's terms at the cut's value
        size_t i = 0;
        while (val[i] != cut) ++i;
        for (const uint16_t t : kept)
            if (want[t]) {
                want[t] = 0;
                if (i < k) key[i] = (static_cast<uint32_t>(t) << 16) | (key[i] & 0xffffu);
                ++i;
            }
        if (i != k) throw std::runtime_error("summary cut differs from the reference's terms");
        cuda_check(cudaMemcpyAsync(a.okey + at, key.data(), k * sizeof(uint32_t),
                                   cudaMemcpyHostToDevice, s), "H2D");
        cuda_check(cudaStreamSynchronize(s), "sync");
    }
}

int pow2_at_least(int64_t n) {
    int p = 1;
    while (p < n) p <<= 1;
    return p;
}

template <int ESZ>
void summarize_typed(const FwdView& f, const BlockSet& blocks, float alpha, const HostCsr* host,
                     cudaStream_t s, Arena& scratch, DevColumns& out, std::vector<int64_t>& ltp,
                     Steps& steps) {
    const int sms = device_sm_count();
    const int32_t n_lists = blocks.n_lists;
    const int64_t n_blocks = blocks.lbp[n_lists];
    const int words = (f.dim + 31) / 32;
    int dev = 0, optin = 0;
    cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    cuda_check(cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev),
               "cudaDeviceGetAttribute");

    // scratch slots: as many pairs as a block can have
    const Arena::Mark start = scratch.mark();
    int64_t* slot = scratch.take<int64_t>(static_cast<size_t>(n_blocks) + 1);
    block_terms_kernel<<<sms * 8, 256, 0, s>>>(f, blocks.d_docs, blocks.d_bdp, n_blocks, slot);
    cuda_check(cudaGetLastError(), "block_terms_kernel");
    exclusive_scan_i64(slot, slot, n_blocks + 1, s, scratch);
    std::vector<int64_t> h_slot(static_cast<size_t>(n_lists) + 1);
    {
        int64_t* at = scratch.take<int64_t>(h_slot.size());
        gather_i64_kernel<<<std::max(1, (n_lists + 256) / 256), 256, 0, s>>>(
            slot, blocks.d_lbp, n_lists + 1, 0, at, nullptr);
        cuda_check(cudaGetLastError(), "gather_i64_kernel");
        cuda_check(cudaMemcpyAsync(h_slot.data(), at, h_slot.size() * 8, cudaMemcpyDeviceToHost, s),
                   "D2H");
        cuda_check(cudaStreamSynchronize(s), "D2H");
    }
    steps.mark("slots");

    // launch shapes of the tiers
    struct Shape {
        void (*kernel)(SumArgs);
        int warps, cap, sel;
        bool smem_vals;
        size_t smem;
        int grid;
        int64_t groups, spill_cap;
    };
    const int small_cap = std::min(kSmallCap, std::max(f.dim, 1));
    const int mid_cap = std::min(kMidCap, std::max(f.dim, 1));
    Shape shape[kTiers] = {
        {sum_rows_kernel<ESZ>, kRowWarps, kRowCap, 256, true, 0, 0, 0, 0},
        {sum_blocks_kernel<ESZ, 1>, 1, small_cap, 256, true, 0, 0, 0, 0},
        {sum_blocks_kernel<ESZ, kMidWarps>, kMidWarps, mid_cap, 1024, true, 0, 0, 0, 0},
        {sum_blocks_kernel<ESZ, kBigWarps>, kBigWarps, std::max(f.dim, 1), 2048, true, 0, 0, 0, 0},
    };
    int64_t spill = 1;
    for (int t = 0; t < kTiers; ++t) {
        Shape& p = shape[t];
        if (ESZ == 1) p.sel = 0;
        const int per_cta = t == 0 ? kRowWarps : 1;
        const int w = t == 0 ? 0 : words;
        p.smem = per_cta * sum_layout(p.cap, p.sel, w, true).total;
        // static shared memory beside it: under 16 KB for every tier
        if (p.smem + 16 * 1024 > static_cast<size_t>(optin)) {
            p.smem_vals = false;
            p.smem = sum_layout(p.cap, p.sel, w, false).total;
        }
        cuda_check(allow_opt_in_smem(p.kernel), "summary shared memory");
        int per_sm = 0;
        cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, p.kernel, p.warps * 32,
                                                                 p.smem),
                   "summary occupancy");
        p.grid = sms * std::max(1, per_sm);
        p.groups = static_cast<int64_t>(p.grid) * per_cta;
        p.spill_cap = pow2_at_least(p.cap);
        if (ESZ != 1) spill = std::max(spill, p.groups * p.spill_cap);
    }
    uint64_t* spill_keys = scratch.take<uint64_t>(static_cast<size_t>(spill));
    uint32_t* gvals = nullptr;
    uint16_t* gterms = nullptr;
    if (!shape[kTiers - 1].smem_vals) {
        const size_t n = static_cast<size_t>(shape[kTiers - 1].grid) * shape[kTiers - 1].cap;
        gvals = scratch.take<uint32_t>(n);
        gterms = scratch.take<uint16_t>(n);
    }
    // counters: blocks per tier, claims per tier, tied blocks
    constexpr int kCounters = 2 * kTiers + 1;
    unsigned* n_ids = scratch.take<unsigned>(kCounters);
    unsigned* claims = n_ids + kTiers;
    unsigned* n_tied = claims + kTiers;

    Arena keep(s);  // the batches' columns
    std::vector<Piece> pieces;
    size_t cols = 0;
    const int64_t budget = int64_t{1} << 27;  // scratch pairs per batch (1 GB)
    int32_t t0 = 0;
    while (t0 < n_lists) {
        int32_t t1 = t0 + 1;
        while (t1 < n_lists && h_slot[t1 + 1] - h_slot[t0] <= budget) ++t1;
        const int64_t b0 = blocks.lbp[t0], nb = blocks.lbp[t1] - b0;
        const int64_t pairs = h_slot[t1] - h_slot[t0];
        const int32_t nl = t1 - t0;
        if (nb == 0 || pairs == 0) {
            for (int32_t t = t0; t < t1; ++t) ltp.push_back(ltp.back());
            t0 = t1;
            continue;
        }
        const Arena::Mark batch = scratch.mark();
        uint32_t* okey = scratch.take<uint32_t>(static_cast<size_t>(pairs));
        float* oval = scratch.take<float>(static_cast<size_t>(pairs));
        int64_t* kept = scratch.take<int64_t>(static_cast<size_t>(nb) + 1);
        int32_t* ids = scratch.take<int32_t>(static_cast<size_t>(nb) * kTiers);
        int32_t* tied = host != nullptr ? scratch.take<int32_t>(static_cast<size_t>(nb)) : nullptr;
        cuda_check(cudaMemsetAsync(n_ids, 0, kCounters * sizeof(unsigned), s), "memset");
        tier_kernel<<<sms * 8, 256, 0, s>>>(blocks.d_bdp, slot, b0, nb, ids, n_ids, kept);
        cuda_check(cudaGetLastError(), "tier_kernel");
        SumArgs a{};
        a.f = f;
        a.docs = blocks.d_docs;
        a.bdp = blocks.d_bdp;
        a.local = blocks.d_local;
        a.slot = slot;
        a.slot0 = h_slot[t0];
        a.b0 = b0;
        a.alpha = alpha;
        a.keep = kept;
        a.okey = okey;
        a.oval = oval;
        a.tied = tied;
        a.n_tied = n_tied;
        a.spill = spill_keys;
        a.words = words;
        // single rows go first: those that are not ascending join the next tier
        for (int t = 0; t < kTiers; ++t) {
            const Shape& p = shape[t];
            a.ids = ids + static_cast<int64_t>(t) * nb;
            a.n_ids = n_ids + t;
            a.next = claims + t;
            a.retry = ids + nb;
            a.n_retry = n_ids + 1;
            a.cap = p.cap;
            a.sel_cap = p.sel;
            a.spill_cap = p.spill_cap;
            a.gvals = p.smem_vals ? nullptr : gvals;
            a.gterms = p.smem_vals ? nullptr : gterms;
            p.kernel<<<p.grid, p.warps * 32, p.smem, s>>>(a);
            cuda_check(cudaGetLastError(), "block summary kernel");
        }
        steps.mark("summaries");
        if (host != nullptr) {
            unsigned n = 0;
            cuda_check(cudaMemcpyAsync(&n, n_tied, sizeof(n), cudaMemcpyDeviceToHost, s), "D2H");
            cuda_check(cudaStreamSynchronize(s), "D2H");
            if (n > 0) {
                std::vector<int32_t> h_tied(n);
                cuda_check(cudaMemcpyAsync(h_tied.data(), tied, n * sizeof(int32_t),
                                           cudaMemcpyDeviceToHost, s), "D2H");
                cuda_check(cudaStreamSynchronize(s), "D2H");
                settle_ties(*host, blocks, a, nb, std::move(h_tied), s);
            }
            steps.mark("cut ties");
        }
        // packed per list
        exclusive_scan_i64(kept, kept, nb + 1, s, scratch);
        int32_t* list_koff = scratch.take<int32_t>(static_cast<size_t>(nl) + 1);
        gather_i64_kernel<<<std::max(1, (nl + 256) / 256), 256, 0, s>>>(
            kept, blocks.d_lbp + t0, nl + 1, b0, nullptr, list_koff);
        cuda_check(cudaGetLastError(), "gather_i64_kernel");
        int64_t n_kept = 0;
        cuda_check(cudaMemcpyAsync(&n_kept, kept + nb, 8, cudaMemcpyDeviceToHost, s), "D2H");
        cuda_check(cudaStreamSynchronize(s), "D2H");
        uint32_t* tkey = scratch.take<uint32_t>(static_cast<size_t>(n_kept));
        float* tval = scratch.take<float>(static_cast<size_t>(n_kept));
        pack_pairs_kernel<<<sms * 16, 256, 0, s>>>(slot, a.slot0, b0, kept, nb, okey, oval, tkey,
                                                   tval);
        cuda_check(cudaGetLastError(), "pack_pairs_kernel");
        steps.mark("pack");
        pieces.push_back(emit_columns(ESZ, nl, n_kept, tkey, tval, list_koff, cols, s, scratch,
                                      keep, steps, ltp));
        cols += static_cast<size_t>(pieces.back().n_cols);
        scratch.release(batch);
        t0 = t1;
    }
    scratch.release(start);
    join_columns(ESZ, pieces, s, out);
    steps.mark("join");
}

}  // namespace

void summarize_blocks(int esz, const FwdView& f, const BlockSet& blocks, float alpha,
                      const HostCsr* host, cudaStream_t s, Arena& scratch, DevColumns& out,
                      std::vector<int64_t>& ltp,
                      std::vector<std::pair<std::string, double>>* step_times) {
    Steps steps{step_times, s};
    if (esz == 4) summarize_typed<4>(f, blocks, alpha, host, s, scratch, out, ltp, steps);
    else if (esz == 2) summarize_typed<2>(f, blocks, alpha, host, s, scratch, out, ltp, steps);
    else summarize_typed<1>(f, blocks, alpha, host, s, scratch, out, ltp, steps);
}

}  // namespace nsp
