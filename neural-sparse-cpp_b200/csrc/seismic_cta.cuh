// Device code of the SEISMIC search with CTAs per query, shared by the kernel
// of one CTA per query (search_seismic_cta.cu) and that of a thread-block
// cluster per query (search_seismic_cluster.cu): shared-memory layout, row
// scoring, the first list's sort, the query cut, and the heap walk.
#ifndef NSP_SEISMIC_CTA_CUH
#define NSP_SEISMIC_CTA_CUH

#include <cuda_runtime.h>

#include <cfloat>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "nsp_device.h"
#include "search_common.cuh"

namespace nsp {
namespace {

using detail_search::heap_emit;
using detail_search::QueryWeight;
using detail_search::heap_offer;
using detail_search::kFull;
using detail_search::ValT;

constexpr int kSegCap = 128;    // block segments per batch, one CTA per query
constexpr int kSortQueue = 64;  // ranges sorted side by side (two per warp at most)
constexpr size_t kSortQueueBytes = 2 * kSortQueue * 4 + 16;  // both queues and their sizes
constexpr int kSegCapMax = 1024;  // the most any launch asks for (a cluster per query)

// A run of consecutive docs of one block inside a batch.
struct Seg {
    int64_t d0;     // position of the first doc in ix.docs
    int32_t cnt;    // its candidates (with a selector, its member docs)
    int32_t cand0;  // first candidate slot of the batch
    float bs;       // the block's summary score
    int32_t head;   // 1 when the block starts here (its pruning test applies)
    uint32_t best;  // key of its best member score above the heap minimum at the gather (0: none)
    int32_t docs;   // docs in the segment; the cluster kernel's walk sets -1 when it drops it
};

// Order-preserving keys of scores, above 0 (NaN sorts past every number: a
// NaN score passes every `score <= minimum` rejection, as it does there).
__device__ __forceinline__ uint32_t score_key(float v) {
    if (v != v) return 0xffffffffu;
    const uint32_t b = __float_as_uint(v);
    return (b & 0x80000000u) ? ~b : (b | 0x80000000u);
}
__device__ __forceinline__ float key_score(uint32_t k) {
    if (k == 0xffffffffu) return __uint_as_float(0x7fc00000u);
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

struct Ctl {
    int32_t q;
    int32_t nseg;
    int32_t total;
    int32_t next;   // claim counter of the scoring phase
    int32_t nheap;  // heap size when the batch was gathered (warp 0's)
    int32_t pad[3];
};

__host__ __device__ inline size_t a16(size_t x) { return (x + 15) & ~size_t(15); }

struct CtaLayout {
    size_t tbl, qv, qterm, qraw, cuts, hs, hid, cdoc, coff, clen, csc, segs, cseg, sq, wsum, cur,
        uq, total;
};

// Shared-memory layout of one CTA. The four candidate arrays are contiguous
// (16 * batch bytes) and double as the sort-key buffer of the first list; the
// sort's queue takes the end of the segments' place, so that the largest k and
// the longest query that fit depend on the arrays above alone.
__host__ __device__ inline CtaLayout cta_layout(int vsize, int tsize, int dim, int qcap, int k,
                                                int batch, int seg_cap) {
    CtaLayout L;
    size_t o = a16(sizeof(Ctl));
    L.tbl = o;   o += a16(static_cast<size_t>(dim + 1) * tsize);
    L.qv = o;    o += a16(static_cast<size_t>(qcap + 1) * 4);
    L.qterm = o; o += a16(static_cast<size_t>(qcap) * 2);
    L.qraw = o;  o += a16(static_cast<size_t>(qcap) * vsize);
    L.cuts = o;  o += a16(static_cast<size_t>(qcap) * 2);
    L.hs = o;    o += a16(static_cast<size_t>(k) * 4);
    L.hid = o;   o += a16(static_cast<size_t>(k) * 4);
    L.cdoc = o;  o += static_cast<size_t>(batch) * 4;
    L.coff = o;  o += static_cast<size_t>(batch) * 4;
    L.clen = o;  o += static_cast<size_t>(batch) * 4;
    L.csc = o;   o += static_cast<size_t>(batch) * 4;
    L.segs = o;  o += static_cast<size_t>(seg_cap) * sizeof(Seg);
    L.cseg = o;  o += a16(static_cast<size_t>(batch) * 2);
    L.sq = o - kSortQueueBytes;  // (kSegCap segments alone are more)
    L.wsum = o;  o += 32 * 4;
    L.cur = o;   o += 64;  // warp 0's Cursor
    L.uq = o;    o += 2 * 32 * 4;  // counting pass: warp 0's per-lane unique docs, row bytes
    L.total = o;
    return L;
}

// ------------------------------------------------------------ row loads --
// 256-bit loads (sm_100): a lane reads 16 term ids (32 bytes) per step and
// their values (64 bytes fp32, 32 bytes uint16, 16 bytes uint8).
__device__ __forceinline__ void ldg256(const void* p, uint32_t (&r)[8]) {
    asm("ld.global.nc.v8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7])
        : "l"(p));
}

__device__ __forceinline__ uint32_t term_of(const uint32_t (&t)[8], int u) {
    return (u & 1) ? (t[u >> 1] >> 16) : (t[u >> 1] & 0xffffu);
}

// One bulk prefetch of `bytes` (a multiple of 16, 16-byte aligned) into L2
// (the TMA unit fetches it; no registers, no L1 traffic).
__device__ __forceinline__ void prefetch_l2(const void* p, uint32_t bytes) {
    asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(p), "r"(bytes) : "memory");
}

// A candidate row's ids and values from element `from` to the row's end on
// its 64-element boundary. Rows start on 64-element boundaries, so both
// ranges are 16-byte aligned multiples of 16 bytes.
template <typename V>
__device__ __forceinline__ void prefetch_row(const uint16_t* idx_base, const V* val_base,
                                             uint32_t off, uint32_t len, uint32_t from) {
    const uint32_t padded = (len + kRowAlign - 1) & ~static_cast<uint32_t>(kRowAlign - 1);
    if (padded <= from) return;
    const size_t e0 = static_cast<size_t>(off) * kRowAlign + from;
    prefetch_l2(idx_base + e0, (padded - from) * 2u);
    prefetch_l2(val_base + e0, (padded - from) * static_cast<uint32_t>(sizeof(V)));
}

template <typename V>
struct Acc;
template <>
struct Acc<float> {
    using T = float;
};
template <>
struct Acc<uint8_t> {
    using T = int;
};
template <>
struct Acc<uint16_t> {
    using T = long long;
};

// Products of one lane's 16 row elements at ip/vp, `rem` of them real (the
// rest are the row's zero padding, or nothing when rem <= 0).
// fp32: p[u] = w[u] * qv[tbl[t[u]]], the reference's product; with kMask the
// padding gives +0.0.
template <typename TE, bool kMask>
__device__ __forceinline__ void products(const uint16_t* ip, const float* vp, int rem,
                                         const TE* tbl, const float* qv, float (&p)[16]) {
    if (rem <= 0) {
#pragma unroll
        for (int u = 0; u < 16; ++u) p[u] = 0.0f;
        return;
    }
    uint32_t t[8], v0[8], v1[8];
    ldg256(ip, t);
    ldg256(vp, v0);
    ldg256(vp + 8, v1);
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const float q = qv[tbl[term_of(t, u)]];
        const float x = __uint_as_float(u < 8 ? v0[u] : v1[u - 8]);
        p[u] = __fmul_rn(x, q);
        if (kMask && u >= rem) p[u] = 0.0f;
    }
}

// uint8 codes: the sum of code products as int (distance.h:39-47); padding
// codes are 0. (Packing four looked-up codes for __dp4a measured slower: the
// packing waits for all four lookups.)
template <typename TE>
__device__ __forceinline__ int partial(const uint16_t* ip, const uint8_t* vp, int rem,
                                       const TE* tbl) {
    if (rem <= 0) return 0;
    uint32_t t[8];
    ldg256(ip, t);
    const uint4 v = __ldg(reinterpret_cast<const uint4*>(vp));
    const uint32_t w[4] = {v.x, v.y, v.z, v.w};
    int acc = 0;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        const int q = static_cast<int>(tbl[term_of(t, u)]);
        const int x = static_cast<int>((w[u >> 2] >> (8 * (u & 3))) & 0xffu);
        acc += x * q;
    }
    return acc;
}

// kSteps consecutive steps of uint8 codes (elements at ip + s * stride,
// `rem - s * stride` of them real for step s): every step's loads are issued
// before any is used, so a row of up to kSteps steps costs one memory round
// trip.
template <typename TE, int kSteps>
__device__ __forceinline__ int partial_steps(const uint16_t* ip, const uint8_t* vp, int rem,
                                             int stride, const TE* tbl) {
    if (rem <= 0) return 0;
    uint32_t t[kSteps][8];
    uint4 v[kSteps];
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
        v[s] = make_uint4(0u, 0u, 0u, 0u);
        if (s == 0 || rem > s * stride) {
            ldg256(ip + s * stride, t[s]);
            v[s] = __ldg(reinterpret_cast<const uint4*>(vp + s * stride));
        }
    }
    // four independent sums (integer: exact in any order), so the products
    // do not wait on one another
    int acc[4] = {0, 0, 0, 0};
#pragma unroll
    for (int s = 0; s < kSteps; ++s) {
        if (s == 0 || rem > s * stride) {
            const uint32_t w[4] = {v[s].x, v[s].y, v[s].z, v[s].w};
#pragma unroll
            for (int u = 0; u < 16; ++u) {
                const int q = static_cast<int>(tbl[term_of(t[s], u)]);
                // code byte u & 3 of its word, zero-extended (one byte permute)
                const uint32_t x = __byte_perm(w[u >> 2], 0u, 0x4440u | (u & 3));
                acc[u & 3] += static_cast<int>(x) * q;
            }
        }
    }
    return (acc[0] + acc[1]) + (acc[2] + acc[3]);
}

// What a query's table holds per term: the term's rank among the query's
// terms (an index into the query's values), or its code. fp32 values need the
// rank; 16-bit codes take it while a byte holds it, since a table of codes is
// 61 KB for 30,522 terms and leaves room for two CTAs per SM instead of four
// (1,001 queries on 301,000 docs: 8.8 ms with codes, 6.6 ms with ranks).
template <typename V, typename TE>
constexpr bool kRankTable = std::is_same<V, float>::value ||
                            (std::is_same<V, uint16_t>::value && std::is_same<TE, uint8_t>::value);

// uint16 codes: int64 sum (distance.h:49-57). `qv`: the query's codes by
// rank (32-bit words), for a table of ranks.
template <typename TE>
__device__ __forceinline__ long long partial(const uint16_t* ip, const uint16_t* vp, int rem,
                                             const TE* tbl, const float* qv) {
    if (rem <= 0) return 0;
    uint32_t t[8], v[8];
    ldg256(ip, t);
    ldg256(vp, v);
    long long acc = 0;
#pragma unroll
    for (int u = 0; u < 16; ++u) {
        uint32_t q;
        if constexpr (kRankTable<uint16_t, TE>)
            q = reinterpret_cast<const uint32_t*>(qv)[tbl[term_of(t, u)]];
        else
            q = tbl[term_of(t, u)];
        acc += static_cast<long long>(static_cast<unsigned long long>(term_of(v, u)) * q);
    }
    return acc;
}

// fp32: folds the group's products into acc in row order -- lane 0's 16,
// then lane 1's, ... -- one FADD per product, the reference's sequence of
// roundings. Every lane of the warp takes part (the shuffles are warp-wide);
// `acc` is the same on every lane of a group and comes back the same.
template <int kG>
__device__ __forceinline__ float fold(float acc, const float (&p)[16], int gbase) {
    if constexpr (kG == 1) {
#pragma unroll
        for (int u = 0; u < 16; ++u) acc = __fadd_rn(acc, p[u]);
        return acc;
    } else {
        float a = acc;
#pragma unroll
        for (int l = 0; l < kG; ++l) {
            float r = a;
#pragma unroll
            for (int u = 0; u < 16; ++u) r = __fadd_rn(r, p[u]);
            a = __shfl_sync(kFull, r, gbase + l);
        }
        return a;
    }
}

// Integer partial sums of a group, exact in any order.
template <int kG, typename A>
__device__ __forceinline__ A group_sum(A x) {
#pragma unroll
    for (int o = kG / 2; o > 0; o >>= 1) x += __shfl_xor_sync(kFull, x, o);
    return x;
}

__device__ __forceinline__ float finish(float a) { return a; }
__device__ __forceinline__ float finish(int a) { return static_cast<float>(a); }
__device__ __forceinline__ float finish(long long a) { return static_cast<float>(a); }

// Scoring phase. Lanes work in groups of kG (aligned within the warp); a
// group claims one candidate of the batch at a time and walks its row kG*16
// elements per step, lane l of the group taking elements 16l..16l+15 of the
// step, so a step's loads are kG*32 contiguous bytes of ids and the matching
// contiguous values (uint8 rows: two steps per iteration). A group whose row
// ends takes the next candidate at the following iteration.
// kPrefetch: rows are handed to L2 ahead of their turn (not when the caller
// has done so).
template <typename V, typename TE, bool kMask, int kG, bool kPrefetch = true>
__device__ void score_batch(const FwdView& fwd, Ctl* ctl, const TE* tbl, const float* qv,
                            const uint32_t* coff, const uint32_t* clen, float* csc, int total,
                            int lane) {
    using A = typename Acc<V>::T;
    constexpr bool kF32 = std::is_same<V, float>::value;
    // uint8 rows advance kU8Steps steps per iteration (partial_steps)
    constexpr bool kU8 = std::is_same<V, uint8_t>::value;
    constexpr int kU8Steps = 2;
    constexpr int kStep = (kU8 ? 16 * kU8Steps : 16) * kG;
    // rows handed to L2 ahead of their scoring, in claims (3M-doc SQ
    // launch: 16 -> -1.4%, 32 -> -2.0%, 64 -> +0.6%, 128 -> +3.7% in time)
    constexpr int kPrefetchAhead = kPrefetch ? 32 : 0;
    const uint16_t* idx_base = fwd.idx;
    const V* val_base = static_cast<const V*>(fwd.val);
    const int gl = lane & (kG - 1);
    const int gbase = lane - gl;
    int i = -1;  // the group's candidate (the same on every lane of the group)
    const uint16_t* ip = nullptr;
    const V* vp = nullptr;
    int rem = 0;  // row elements from this step on
    A acc = 0;
    bool fin = false;
    for (;;) {
        const bool want = !fin && i < 0;
        const unsigned wm = __ballot_sync(kFull, want && gl == 0);
        if (wm) {
            const int leader = __ffs(wm) - 1;
            int base = 0;
            if (lane == leader) base = atomicAdd(&ctl->next, __popc(wm));
            base = __shfl_sync(kFull, base, leader);
            if (want) {
                const int j = base + __popc(wm & ((1u << gbase) - 1u));
                if (j < total) {
                    i = j;
                    if (kPrefetchAhead > 0 && gl == 0) {
                        // the row a group will claim about one round of
                        // claims from now goes to L2; the first round's own
                        // rows past their first iteration too
                        const int jn = j + kPrefetchAhead;
                        if (jn < total) prefetch_row<V>(idx_base, val_base, coff[jn], clen[jn], 0);
                        if (j < kPrefetchAhead)
                            prefetch_row<V>(idx_base, val_base, coff[j], clen[j], kStep);
                    }
                    const size_t e0 = static_cast<size_t>(coff[j]) * kRowAlign + 16 * gl;
                    ip = idx_base + e0;
                    vp = val_base + e0;
                    rem = static_cast<int>(clen[j]);
                    acc = 0;
                } else {
                    fin = true;
                }
            }
        }
        const bool act = i >= 0;
        if (!__any_sync(kFull, act)) break;
        const int mine = act ? rem - 16 * gl : 0;  // this lane's real elements
        if constexpr (kF32) {
            float p[16];
            products<TE, kMask>(ip, vp, mine, tbl, qv, p);
            acc = fold<kG>(acc, p, gbase);
        } else if constexpr (kU8) {
            acc += group_sum<kG>(partial_steps<TE, kU8Steps>(ip, vp, mine, 16 * kG, tbl));
        } else {
            acc += group_sum<kG>(partial<TE>(ip, vp, mine, tbl, qv));
        }
        if (act) {
            ip += kStep;
            vp += kStep;
            rem -= kStep;
            if (rem <= 0) {
                if (gl == 0) csc[i] = finish(acc);
                i = -1;
            }
        }
    }
}

// Summary scores of list t into bscore[0..nb): hit terms in ascending term
// order, lanes spread over the term's (block, value) run.
template <typename V>
__device__ void list_summaries(const SeismicLaunch& a, int t, int nb, const uint16_t* qterm,
                               const V* qraw, int qn, float* bscore, int lane,
                               uint32_t& bytes) {
    constexpr int vsz = static_cast<int>(sizeof(V));
    // uint8 codes: a block's score is a sum of at most qn products of two
    // codes (<= 255 * 255 each), an integer below 2^24 -- exact in fp32 --
    // while qn * 65025 < 2^24 (the reference sums these integer-valued floats
    // in float as well, inverted_list_clusters.cpp:295-331)
    const bool exact_any_order =
        std::is_same<V, uint8_t>::value && static_cast<long long>(qn) * 65025ll < (1ll << 24);
    for (int b = lane; b < nb; b += 32) bscore[b] = 0.0f;
    __syncwarp();
    const uint2* meta = a.ix.lmeta + static_cast<size_t>(t) * a.ix.words;
    const int64_t colbase = a.ix.ltp[t];
    for (int i0 = 0; i0 < qn; i0 += 32) {
        const int i = i0 + lane;
        bool hit = false;
        int64_t r0 = 0, r1 = 0;
        float qv = 0.0f;
        if (i < qn && qterm[i] < static_cast<uint32_t>(a.fwd.dim)) {
            const uint32_t term = qterm[i];
            const uint2 m = __ldg(meta + (term >> 5));
            const uint32_t bit = 1u << (term & 31);
            if (m.x & bit) {
                const int64_t col = colbase + m.y + __popc(m.x & (bit - 1));
                r0 = __ldg(a.ix.srun + col);
                r1 = __ldg(a.ix.srun + col + 1);
                qv = ValT<V>::f(qraw[i]);
                hit = true;
            }
        }
        bytes += 8u * static_cast<uint32_t>(min(32, qn - i0));
        unsigned hm = __ballot_sync(kFull, hit);
        bytes += 16u * __popc(hm);
        while (hm) {
            const int src = __ffs(hm) - 1;
            hm &= hm - 1;
            const int64_t R0 = __shfl_sync(kFull, r0, src);
            const int64_t R1 = __shfl_sync(kFull, r1, src);
            const float QV = __shfl_sync(kFull, qv, src);
            bytes += static_cast<uint32_t>(R1 - R0) * (2 + vsz);
            const V* sv = static_cast<const V*>(a.ix.sval);
            if (exact_any_order) {
                // integer products and sums below 2^24: every order of the
                // float additions gives the same sum, so the updates need not
                // wait for one another
                for (int64_t e = R0 + lane; e < R1; e += 32) {
                    const int blk = __ldg(a.ix.sblk + e);
                    atomicAdd(bscore + blk, __fmul_rn(QV, ValT<V>::f(__ldg(sv + e))));
                }
            } else {
                for (int64_t e = R0 + lane; e < R1; e += 32) {
                    const int blk = __ldg(a.ix.sblk + e);
                    const float p = __fmul_rn(QV, ValT<V>::f(__ldg(sv + e)));
                    bscore[blk] = __fadd_rn(bscore[blk], p);
                }
                __syncwarp();
            }
        }
    }
}

// ------------------------------------------------ the first list's sort --
// The visiting order of the first list is the reference's std::ranges::sort
// of the block indices by summary score descending (seismic_common.h:105-115):
// equal scores keep the order that unstable sort leaves (ref_ranking.cuh).
// Its partition steps are Hoare's: the k-th element from the left that does
// not come before the pivot is swapped with the k-th from the right that the
// pivot does not come before, as long as they have not met. Which elements
// those are does not depend on the swaps, so a warp finds them with ballots
// and swaps all pairs at once. Ranges are disjoint, so warps take them side
// by side, and ranges of at most 16 elements, which the reference leaves to
// its insertion pass, are stable-sorted by rank. One lane per range took 105
// us for a lone query's 400 blocks and 180 us for 600 (fp32 100k docs, SQ 3M).

// One partition step of a[f, l), l - f > 16, by a warp; returns the cut.
// `stops` has room for l entries.
__device__ int warp_partition(ranking::Blk* a, int f, int l, uint16_t* stops, int lane) {
    const int x = f + 1, y = f + (l - f) / 2, z = l - 1;
    const ranking::Blk vx = a[x], vy = a[y], vz = a[z], vf = a[f];
    int m;
    if (ranking::before(vx, vy)) {
        if (ranking::before(vy, vz)) m = y;
        else m = ranking::before(vx, vz) ? z : x;
    } else if (ranking::before(vx, vz)) {
        m = x;
    } else {
        m = ranking::before(vy, vz) ? z : y;
    }
    const ranking::Blk p = m == x ? vx : (m == y ? vy : vz);
    __syncwarp();
    if (lane == 0) {
        a[f] = p;
        a[m] = vf;
    }
    __syncwarp();
    // at most K pairs are swapped, so the first K + 1 stops from the left and
    // K from the right decide
    const int K = (l - f - 1) / 2;
    uint16_t* ls = stops + f;
    uint16_t* rs = ls + K + 1;
    const unsigned below = (1u << lane) - 1u;
    int nl = 0, nr = 0;
    for (int b = f + 1; b < l && nl <= K; b += 32) {
        const int i = b + lane;
        const bool st = i < l && !ranking::before(a[i], p);
        const unsigned w = __ballot_sync(kFull, st);
        const int at = nl + __popc(w & below);
        if (st && at <= K) ls[at] = static_cast<uint16_t>(i);
        nl += __popc(w);
    }
    for (int b = l - 1; b >= f && nr < K; b -= 32) {
        const int i = b - lane;
        const bool st = i >= f && !ranking::before(p, a[i]);
        const unsigned w = __ballot_sync(kFull, st);
        const int at = nr + __popc(w & below);
        if (st && at < K) rs[at] = static_cast<uint16_t>(i);
        nr += __popc(w);
    }
    nl = min(nl, K + 1);
    nr = min(nr, K);
    __syncwarp();
    int pairs = 0;
    for (int k0 = 0;; k0 += 32) {
        const int k = k0 + lane;
        const bool ok = k < nl && k < nr && ls[k] < rs[k];
        if (ok) {
            const int lo = ls[k], hi = rs[k];
            const ranking::Blk t = a[lo];
            a[lo] = a[hi];
            a[hi] = t;
        }
        const unsigned w = __ballot_sync(kFull, ok);
        pairs += __popc(w);
        if (w != kFull) break;
    }
    // the scan from the left ends at its next stop, or at the last element it
    // swapped to the right
    int cut = pairs < nl ? ls[pairs] : l;
    if (pairs > 0) cut = min(cut, static_cast<int>(rs[pairs - 1]));
    __syncwarp();
    return cut;
}

// a[f, l), at most 16 elements, as the insertion pass leaves it.
__device__ void warp_insertion(ranking::Blk* a, int f, int l, int lane) {
    const int n = l - f;
    if (n < 2) return;
    ranking::Blk v{0.0f, 0};
    if (lane < n) v = a[f + lane];
    if (__any_sync(kFull, v.s != v.s)) {  // NaN scores have no rank
        if (lane == 0) ranking::insertion_range(a, f, l);
        __syncwarp();
        return;
    }
    int r = 0;
    for (int j = 0; j < n; ++j) {
        const float x = __shfl_sync(kFull, v.s, j);
        r += (x > v.s || (x == v.s && j < lane)) ? 1 : 0;
    }
    __syncwarp();
    if (lane < n) a[f + r] = v;
    __syncwarp();
}

// The introsort loop over a[f, l) with depth budget d by a warp, then the
// insertion pass. Lane i holds pending range i (their budgets strictly
// decrease, so at most 2 * 16 wait at once for lists of up to 65,536 blocks).
__device__ void warp_sort_range(ranking::Blk* a, int f, int l, int d, uint16_t* stops, int lane) {
    int pf = 0, pl = 0, pd = 0;
    int sp = 0;
    for (;;) {
        while (l - f > ranking::kSortThreshold && d > 0) {
            --d;
            const int cut = warp_partition(a, f, l, stops, lane);
            if (l - cut > ranking::kSortThreshold && sp < 32) {
                if (lane == sp) {
                    pf = cut;
                    pl = l;
                    pd = d;
                }
                ++sp;
            } else {
                warp_insertion(a, cut, l, lane);
            }
            l = cut;
        }
        if (l - f > ranking::kSortThreshold) {  // the depth budget is spent
            if (lane == 0) ranking::heap_sort_range(a, f, l);
            __syncwarp();
        } else {
            warp_insertion(a, f, l, lane);
        }
        if (sp == 0) return;
        --sp;
        f = __shfl_sync(kFull, pf, sp);
        l = __shfl_sync(kFull, pl, sp);
        d = __shfl_sync(kFull, pd, sp);
    }
}

// All threads: (score, block) pairs into `items`, sorted, block indices into
// order[0..nb). `stops`: scratch of nb entries, which may be `order`.
__device__ void sort_blocks(const float* bscore, int nb, ranking::Blk* items, uint16_t* stops,
                            uint16_t* order, uint32_t* queue, int tid, int lane, int warp,
                            int nwarps) {
    for (int i = tid; i < nb; i += blockDim.x) items[i] = ranking::Blk{__ldcg(bscore + i), i};
    // ranges as first | (last << 16); both queues, then their sizes
    uint32_t* cnt = queue + 2 * kSortQueue;
    if (tid == 0) {
        queue[0] = static_cast<uint32_t>(nb - 1) << 16;
        cnt[0] = 1u;
        cnt[1] = 0u;
    }
    __syncthreads();
    int n = 1, q = 0, d = 2 * ranking::floor_log2(nb);
    // level by level until every warp has a range
    while (n > 0 && n < nwarps && d > 0) {
        --d;
        if (warp < n) {
            const uint32_t r = queue[q * kSortQueue + warp];
            const int f = static_cast<int>(r & 0xffffu), l = static_cast<int>(r >> 16) + 1;
            if (l - f > ranking::kSortThreshold) {
                const int cut = warp_partition(items, f, l, stops, lane);
                const int fs[2] = {f, cut}, es[2] = {cut, l};
#pragma unroll
                for (int u = 0; u < 2; ++u) {
                    if (es[u] - fs[u] > ranking::kSortThreshold) {
                        if (lane == 0)
                            queue[(q ^ 1) * kSortQueue + atomicAdd(cnt + (q ^ 1), 1u)] =
                                static_cast<uint32_t>(fs[u]) |
                                (static_cast<uint32_t>(es[u] - 1) << 16);
                    } else {
                        warp_insertion(items, fs[u], es[u], lane);
                    }
                }
            } else {
                warp_insertion(items, f, l, lane);
            }
        }
        __syncthreads();
        q ^= 1;
        n = static_cast<int>(cnt[q]);
        if (tid == 0) cnt[q ^ 1] = 0u;
        __syncthreads();
    }
    for (int i = warp; i < n; i += nwarps) {
        const uint32_t r = queue[q * kSortQueue + i];
        warp_sort_range(items, static_cast<int>(r & 0xffffu), static_cast<int>(r >> 16) + 1, d,
                        stops, lane);
    }
    __syncthreads();
    for (int i = tid; i < nb; i += blockDim.x) order[i] = static_cast<uint16_t>(items[i].b);
    __syncthreads();
}

// --------------------------------------------------------- the query cut --
// cuts[0..ncut) = positions of the query's ncut largest weights in the order
// of the reference's holder (utils/vector_process.h:18-30). Distinct weights
// come out by value descending, so every thread ranks one; where two of the
// kept weights are equal (or one is NaN) one thread repeats the holder's
// steps -- on (code, position) words for codes, which tie constantly, where
// `room` words hold them. Ranking costs qn loads per thread, so very long
// queries take the one-thread steps at once; a holder of at most 32 codes sits
// in a warp's registers (a lone fp32 query's cut of 10 from 29 terms: 9 us on
// one thread; SQ, 12 from 102: 25 us).
template <typename V>
__device__ void query_cut(uint16_t* cuts, const V* qraw, int qn, int ncut, uint32_t* words,
                          int room, int tid) {
    if constexpr (std::is_same<V, float>::value) {
        bool tie = qn > 1024;
        if (!tie)
            for (int i = tid; i < qn; i += blockDim.x) {
                const float v = qraw[i];
                int r = 0;
                bool eq = v != v;
                for (int j = 0; j < qn; ++j) {
                    const float x = qraw[j];
                    r += x > v ? 1 : 0;
                    eq |= (x == v && j != i) || x != x;
                }
                if (r < ncut) {
                    tie |= eq;
                    if (!eq) cuts[r] = static_cast<uint16_t>(i);
                }
            }
        if (!__syncthreads_or(tie)) return;
        if (tid == 0) ranking::cut_like_reference(cuts, qn, ncut, QueryWeight<V>{qraw});
    } else {
        if (ncut <= 32) {
            if (tid < 32) ranking::warp_cut_like_reference(cuts, qn, ncut, QueryWeight<V>{qraw}, tid);
        } else if (ncut > room) {
            if (tid == 0) ranking::cut_like_reference(cuts, qn, ncut, QueryWeight<V>{qraw});
        } else if (tid == 0) {
            ranking::cut_words_like_reference(words, qn, ncut, qraw);
            for (int i = 0; i < ncut; ++i) cuts[i] = static_cast<uint16_t>(words[i]);
        }
    }
    __syncthreads();
}

// Cursor of warp 0 over one list's visiting order. It lives in shared memory:
// only warp 0 uses it (its lanes write the same values), and held in every
// thread's registers it would cost the scoring loop registers.
struct Cursor {
    int o;            // next position in the visiting order
    bool dead;        // the first list's walk has ended
    bool split;       // a block is part-way through
    int64_t split_d;  // its next doc position
    int split_left;
    float split_bs;
};

// Warp 0: fills the next batch with segments of blocks that pass the pruning
// test against the current heap, taking blocks in the list's visiting order
// `order[0..nb)` (the first list: sorted; later lists: the blocks that passed
// when the list began, in block order). Returns the number of segments;
// `total` receives the number of docs.
__device__ int gather(const SeismicLaunch& a, Cursor& c, bool first, int64_t lb0, int nb,
                      const float* bscore, const uint16_t* order, int n, const float* hs,
                      Seg* segs, int batch, int seg_cap, int& total, int lane) {
    int room = batch;
    int nseg = 0;
    total = 0;
    if (c.split) {
        const int take = min(room, c.split_left);
        if (lane == 0) {
            Seg g;
            g.d0 = c.split_d;
            g.cnt = take;
            g.docs = take;
            g.cand0 = 0;
            g.bs = c.split_bs;
            g.head = 0;
            g.best = 0u;
            segs[0] = g;
        }
        nseg = 1;
        total = take;
        room -= take;
        c.split_d += take;
        c.split_left -= take;
        if (c.split_left == 0) c.split = false;
    }
    const bool full = n == a.k;
    const float hmin = full ? hs[0] : 0.0f;
    while (!c.split && !c.dead && room > 0 && nseg < seg_cap && c.o < nb) {
        const int p = c.o + lane;
        const bool in = p < nb;
        int blk = 0;
        float bs = 0.0f;
        int64_t d0 = 0, d1 = 0;
        if (in) {
            blk = static_cast<int>(order[p]);
            // the block's doc range is loaded with its score, before the test
            bs = __ldcg(bscore + blk);
            d0 = __ldg(a.ix.bdp + lb0 + blk);
            d1 = __ldg(a.ix.bdp + lb0 + blk + 1);
        }
        const bool pass = in && !(full && __fmul_rn(bs, a.heap_factor) < hmin);
        const unsigned inm = __ballot_sync(kFull, in);
        const unsigned pm = __ballot_sync(kFull, pass);
        int lim = __popc(inm);
        bool brk = false;
        if (first) {
            const unsigned fm = inm & ~pm;
            if (fm) {
                lim = __ffs(fm) - 1;
                brk = true;
            }
        }
        const bool cand = pass && lane < lim;
        const int sz = cand ? static_cast<int>(d1 - d0) : 0;
        int incl = sz;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int y = __shfl_up_sync(kFull, incl, o);
            if (lane >= o) incl += y;
        }
        const int excl = incl - sz;
        const unsigned cm = __ballot_sync(kFull, cand);
        const int r = __popc(cm & ((1u << lane) - 1u));
        const bool take = cand && excl < room && nseg + r < seg_cap;
        const unsigned tm = __ballot_sync(kFull, take);
        if (take) {
            Seg g;
            g.d0 = d0;
            g.cnt = min(sz, room - excl);
            g.docs = g.cnt;
            g.cand0 = total + excl;
            g.bs = bs;
            g.head = 1;
            g.best = 0u;
            segs[nseg + r] = g;
        }
        int taken_docs = 0;
        if (tm) {
            const int last = 31 - __clz(tm);
            const int lsz = __shfl_sync(kFull, sz, last);
            const int lexcl = __shfl_sync(kFull, excl, last);
            const int lcnt = min(lsz, room - lexcl);
            const int64_t ld0 = __shfl_sync(kFull, d0, last);
            const float lbs = __shfl_sync(kFull, bs, last);
            taken_docs = lexcl + lcnt;
            if (lcnt < lsz) {
                c.split = true;
                c.split_d = ld0 + lcnt;
                c.split_left = lsz - lcnt;
                c.split_bs = lbs;
            }
        }
        const unsigned nt = cm & ~tm;  // candidates left for the next batch
        if (nt) {
            c.o += __ffs(nt) - 1;
        } else {
            c.o += lim;
            // the failing block ends the first list once the blocks before it
            // (including a block cut short) are done
            if (brk && !c.split) c.dead = true;
        }
        nseg += __popc(tm);
        total += taken_docs;
        room -= taken_docs;
    }
    __syncwarp();
    return nseg;
}

// All threads: the blocks of a later list that pass the pruning test against
// the heap as it stands when the list begins, in block order, into
// order[0..return). The heap minimum only grows, so a block failing now fails
// at its turn too; the walk then visits only these (the reference tests and
// skips every block, seismic_index.cpp:78-86).
__device__ int passing_blocks(const float* bscore, int nb, bool full, float hmin, float hf,
                              uint16_t* order, int* wsum, int tid, int lane, int warp,
                              int nwarps) {
    int base = 0;
    for (int i0 = 0; i0 < nb; i0 += nwarps * 32) {
        const int i = i0 + tid;
        const bool pass = i < nb && !(full && __fmul_rn(__ldcg(bscore + i), hf) < hmin);
        const unsigned m = __ballot_sync(kFull, pass);
        if (lane == 0) wsum[warp] = __popc(m);
        __syncthreads();
        int off = 0, all = 0;
        for (int w = 0; w < nwarps; ++w) {
            const int c = wsum[w];
            off += w < warp ? c : 0;
            all += c;
        }
        if (pass) order[base + off + __popc(m & ((1u << lane) - 1u))] = static_cast<uint16_t>(i);
        base += all;
        __syncthreads();
    }
    return base;
}

// Warp 0 walks a batch's segments in block order as the reference walks its
// blocks (seismic_index.cpp:78-117): each block head is tested against the
// heap as it stands at its turn, then its docs are offered in order. Segments
// whose best score does not pass the heap minimum leave the heap as it is, so
// a run of up to 32 of them sees one minimum and one ballot settles it; the
// others offer their docs. `dead` and `split` are the list cursor's; `n` is
// the heap size. The counters are the warp's.
template <typename V, bool kMark>
__device__ __forceinline__ void walk_batch(const SeismicLaunch& a, Seg* segs, int nseg,
                                           int total, const int32_t* cdoc, const uint32_t* clen,
                                           const float* csc, float* hs, int32_t* hid, int& n,
                                           bool first, bool& dead, bool& split, uint32_t* uq,
                                           uint32_t stamp_value, int lane,
                                           uint32_t& blocks_visited, uint32_t& bytes,
                                           int32_t& docs_scored, int32_t& row_bytes) {
    // Segments [s0, s1) are dropped: marked, or their docs given back by the
    // work counters (segment after segment, their candidates are contiguous:
    // a lone query drops hundreds at once).
    auto drop = [&](int s0, int s1) {
        if constexpr (kMark) {
            for (int t = s0 + lane; t < s1; t += 32) segs[t].docs = -1;
        } else {
            const int c1 = s1 < nseg ? segs[s1].cand0 : total;
            for (int i = segs[s0].cand0 + lane; i < c1; i += 32) {
                if (cdoc[i] >= 0) {
                    --docs_scored;
                    row_bytes -=
                        8 + static_cast<int32_t>(clen[i]) * (2 + static_cast<int>(sizeof(V)));
                }
            }
        }
    };
    // The holder's entries, in registers while they fit a warp and none is NaN.
    float rs = 0.0f;
    int32_t rid = -1;
    bool regs = kMark && a.k <= 32;  // (the one-CTA kernel has no registers to spare)
    if (regs) {
        if (lane < n) {
            rs = hs[lane];
            rid = hid[lane];
        }
        regs = !__any_sync(kFull, lane < n && rs != rs);
    }
    auto spill = [&]() {
        __syncwarp();
        if (lane < n) {
            hs[lane] = rs;
            hid[lane] = rid;
        }
        __syncwarp();
    };
    auto offer = [&](float sc, int32_t d) {
        if (regs && sc != sc) {
            spill();
            regs = false;
        }
        if (!regs) {
            heap_offer(sc, d, hs, hid, n, a.k, lane);
            return;
        }
        if (n >= a.k && sc <= hs[0]) return;
        if (__any_sync(kFull, lane < n && rid == d)) return;
        ranking::warp_heap_add(rs, rid, n, a.k, sc, d, lane);
        if (lane == 0) hs[0] = rs;
        __syncwarp();
    };
    // counting pass: the member docs of a visited block,
    // each counted the first time the query meets it
    auto count_visits = [&](int t) {
        if (a.visit == nullptr) return;
        uint32_t* stamp = a.visit + static_cast<size_t>(blockIdx.x) *
                                        static_cast<size_t>(a.fwd.n_docs);
        const Seg g = segs[t];
        for (int j = lane; j < g.cnt; j += 32) {
            const int i = g.cand0 + j;
            const int32_t d = cdoc[i];
            if (d >= 0 && atomicExch(stamp + d, stamp_value) !=
                              stamp_value) {
                uq[lane] += 1;
                uq[32 + lane] += 8u + clen[i] * (2 + static_cast<int>(sizeof(V)));
            }
        }
    };
    auto end_first_list = [&](int from) {
        drop(from, nseg);
        dead = true;
        split = false;
    };
    bool ended = false;
    for (int s0 = 0; s0 < nseg && !ended; s0 += 32) {
        const bool valid = s0 + lane < nseg;
        int head = 0, cnt = 0, cand0 = 0, docs = 0;
        uint32_t best = 0u;
        float bs = 0.0f;
        if (valid) {
            const Seg g = segs[s0 + lane];
            head = g.head;
            cnt = g.cnt;
            cand0 = g.cand0;
            docs = g.docs;
            best = g.best;
            bs = g.bs;
        }
        const int w = min(32, nseg - s0);
        int pos = 0;
        while (pos < w) {
            const bool full = n == a.k;
            const float hmin = full ? hs[0] : 0.0f;
            // the first segment that may change the heap
            const unsigned sm =
                __ballot_sync(kFull, lane >= pos && best != 0u &&
                                         (!full || !(key_score(best) <= hmin)));
            const int S = sm ? __ffs(sm) - 1 : w;
            const bool fails = head && full &&
                               __fmul_rn(bs, a.heap_factor) < hmin;
            const bool run = lane >= pos && lane < S;
            const unsigned fm = __ballot_sync(kFull, run && fails);
            // the first list ends at its first failing block
            const int upto = (first && fm) ? __ffs(fm) - 1 : S;
            const bool taken = run && lane < upto && !fails;
            const int heads = __popc(__ballot_sync(kFull, taken && head));
            blocks_visited += heads;
            bytes += 16u * heads +
                     4u * __reduce_add_sync(kFull, taken ? docs : 0);
            if (a.visit != nullptr) {
                unsigned tm = __ballot_sync(kFull, taken);
                while (tm) {
                    const int t = __ffs(tm) - 1;
                    tm &= tm - 1;
                    count_visits(s0 + t);
                }
            }
            if (first && fm) {
                end_first_list(s0 + upto);
                ended = true;
                break;
            }
            unsigned dm = fm;
            while (dm) {  // later lists skip failing blocks, run by run
                const int t = __ffs(dm) - 1;
                const unsigned rest = ~(dm >> t);
                const int len = rest ? __ffs(rest) - 1 : 32;
                const int last = min(t + len, 32) - 1;
                dm &= last == 31 ? 0u : ~0u << (last + 1);
                drop(s0 + t, s0 + last + 1);
                if (s0 + last == nseg - 1) split = false;
            }
            pos = upto;
            if (pos == w) break;
            // its test, then its offers
            if (__shfl_sync(kFull, fails ? 1 : 0, pos)) {
                if (first) {
                    end_first_list(s0 + pos);
                    ended = true;
                    break;
                }
                drop(s0 + pos, s0 + pos + 1);
                if (s0 + pos == nseg - 1) split = false;
            } else {
                const int gcnt = __shfl_sync(kFull, cnt, pos);
                const int g0 = __shfl_sync(kFull, cand0, pos);
                if (__shfl_sync(kFull, head, pos)) {
                    ++blocks_visited;
                    bytes += 16;
                }
                bytes += 4u * static_cast<uint32_t>(__shfl_sync(kFull, docs, pos));
                count_visits(s0 + pos);
                for (int b = 0; b < gcnt; b += 128) {
                    // four times 32 docs loaded at once
                    float sc[4];
                    int32_t d[4];
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        const int j = b + 32 * u + lane;
                        d[u] = -1;
                        sc[u] = 0.0f;
                        if (j < gcnt) {
                            d[u] = cdoc[g0 + j];
                            sc[u] = csc[g0 + j];
                        }
                    }
#pragma unroll
                    for (int u = 0; u < 4; ++u) {
                        unsigned m = __ballot_sync(
                            kFull, d[u] >= 0 && (n < a.k || !(sc[u] <= hs[0])));
                        while (m) {
                            const int src = __ffs(m) - 1;
                            m &= m - 1;
                            offer(__shfl_sync(kFull, sc[u], src), __shfl_sync(kFull, d[u], src));
                            // the others against the new minimum
                            m &= __ballot_sync(kFull, n < a.k || !(sc[u] <= hs[0]));
                        }
                    }
                }
            }
            ++pos;
        }
    }
    if (regs) spill();
}

}  // namespace
}  // namespace nsp

#endif  // NSP_SEISMIC_CTA_CUH
