// Cluster assignment of the SEISMIC build for uint8 codes
// (cluster/kmeans_utils.cpp:40-195): every kept doc of a posting list goes to
// the list's centroid of largest dot product, the lowest index on ties.
//
// Code products are integers, and their sums below 2^31 for rows of up to
// 33,025 entries, so a dot product may be summed in any order and split: over
// the corpus's kHot most frequent terms it is a dense contraction on the
// tensor cores (tcgen05.mma kind::i8, uint8 x uint8 into int32 in TMEM), over
// the others it stays sparse. Terms are Zipf-like: two docs of the SPLADE
// shapes share 32 terms on average, all but 0.25 of them among the 1,024 most
// frequent, so the sparse part falls from ~32 products per (doc, centroid)
// pair to a quarter of one, and the dense part's 1,024 multiply-adds per pair
// cost the tensor cores less than the 32 cost the shared-memory pipe.
//
//   hot rows   every doc's codes of the hot terms as a dense row of kHot
//              bytes in global memory (built once per build);
//   a CTA      takes a list at a time; per 128 member docs the A tile (their
//              hot rows, 128 KB) stays in shared memory, the centroids' rows
//              stream through two 32 KB stages of 128 terms x <= 256
//              centroids (cp.async, 128-byte swizzle), one thread issues the
//              MMAs, and the warps move the accumulators to the CTA's scratch
//              rows in global memory (at most 0.5 MB per CTA, mostly in L2);
//   then       a warp per doc adds the sparse products from the list's
//              term-major index of the centroids' other terms (shared-memory
//              integer atomics; a bitmap of the indexed terms spares the
//              lookups of all others) and takes the argmax. The list's own
//              term, which every centroid holds, is a dense array instead of
//              an index run of all centroids.
//
// Lists whose docs are all centroids need none of it.
//
// Measured (SEISMIC-SQ, 200,000 docs, lambda 6000, beta 600: 7.9M docs to
// assign in 5,175 lists): the assignment phase 370 -> 80 ms, this kernel 45 ms
// of it. Per tile of 128 docs, in thousands of cycles: centroid stages and
// MMAs 58 (two stages in flight: bound by the round trips of the centroid
// rows, not by the tensor cores, whose pipe is active 5% of the time),
// accumulators to scratch 17, sparse products and argmax 99 (issue and L2
// latency); 290 per list for its index. No pipe is near its peak (100,000
// docs: issue 49%, L1 data pipe 36%, DRAM 1.9 TB/s, L2 hits 49%): waits for
// memory and barriers are most of the stalls.
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <numeric>
#include <stdexcept>
#include <vector>

#include "seismic_assign_u8.h"
#include "tma.h"

namespace nsp {
namespace {

constexpr unsigned kFull = 0xffffffffu;
constexpr int kHot = 1024;        // frequent terms of the dense part, at most
constexpr int kM = 128;           // member docs per tile
constexpr int kN = 256;           // centroids per accumulator, at most
constexpr int kKBytes = 128;      // terms per stage: one swizzled row
constexpr int kThreads = 1024;
constexpr int kWarps = kThreads / 32;
constexpr int kStageBytes = kN * kKBytes;
constexpr int kHits = 256;        // pieces of index runs listed at once, per warp
static_assert(kWarps * kHits * 8 <= 2 * kStageBytes, "the hits take the stages' place");
constexpr uint32_t kTmemCols = 256;
// The list index's counters take the operands' place while it is built.
constexpr int kMaxDim = (kWarps * kAssignMaxCentroids * 4 + 2 * kStageBytes) / 4;

struct Args {
    FwdView f;
    AssignLists l;
    const uint8_t* hot;          // [n_docs][hot_bytes]
    int hot_bytes;               // a multiple of kKBytes, at most kHot
    const uint32_t* hot_bits;    // bitmap of the hot terms
    int words;
    uint32_t* out_key;
    int32_t* work;               // list counter
    int32_t* err;
    // per-CTA scratch
    int32_t* ends;               // [dim + 1]: where a term's centroid entries end, from [1]
    uint32_t* entry;             // [max_entries]: centroid << 8 | code
    int32_t* member;             // [max_kept]: positions of the docs that are no centroid
    uint8_t* is_centroid;        // [max_kept]
    int32_t* sims;               // [kM][ld]
    int64_t max_entries, max_kept;
    int ld;
};

// ------------------------------------------------------- PTX wrappers --

// 16 bytes to shared memory, zeros when !valid.
__device__ __forceinline__ void copy16(uint32_t dst, const void* src, bool valid) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(dst), "l"(src),
                 "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void copies_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int kLeft>
__device__ __forceinline__ void copies_wait() {
    asm volatile("cp.async.wait_group %0;" ::"n"(kLeft) : "memory");
}
__device__ __forceinline__ void tmem_alloc(uint32_t* slot) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(
                     smem_addr(slot)),
                 "r"(kTmemCols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_free(uint32_t addr) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(addr),
                 "r"(kTmemCols)
                 : "memory");
}

// K-major operand with the 128-byte swizzle: rows of 128 bytes, groups of 8
// rows (1,024 bytes) one after another.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    return static_cast<uint64_t>((addr >> 4) & 0x3fffu) | (1ull << 16) |
           (static_cast<uint64_t>(1024 >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
// uint8 x uint8 -> int32, both K-major, 128 x n.
__device__ __forceinline__ uint32_t instr_desc(int n) {
    return (2u << 4) | (static_cast<uint32_t>(n >> 3) << 17) |
           (static_cast<uint32_t>(kM >> 4) << 24);
}
__device__ __forceinline__ void mma_u8(uint32_t d, uint64_t a, uint64_t b, uint32_t idesc,
                                       bool accumulate) {
    asm volatile(
        "{\n .reg .pred p;\n"
        " setp.ne.b32 p, %4, 0;\n"
        " tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n}" ::"r"(d),
        "l"(a), "l"(b), "r"(idesc), "r"(accumulate ? 1 : 0)
        : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* b) {
    asm volatile(
        "tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(
            smem_addr(b))
        : "memory");
}
__device__ __forceinline__ void tmem_load32(uint32_t addr, uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]),
          "=r"(r[7]), "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]),
          "=r"(r[14]), "=r"(r[15]), "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]),
          "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]), "=r"(r[24]), "=r"(r[25]),
          "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(addr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void store256(int32_t* p, const uint32_t* r) {
    asm volatile("st.global.v8.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8};" ::"l"(p), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}

// Byte offset of 16-byte piece j (of 8) of row r in a swizzled operand.
__device__ __forceinline__ uint32_t swizzled(int r, int j) {
    return static_cast<uint32_t>(r) * kKBytes + (static_cast<uint32_t>(j ^ (r & 7)) << 4);
}

// --------------------------------------------------------------- layout --

struct Layout {
    size_t a, b, hot_bits, cold_bits, cdoc, own, mdoc, total;
};
__host__ __device__ inline Layout smem_layout(int hot_bytes, int words) {
    Layout L;
    size_t o = 0;
    // operands on 1,024-byte boundaries; the A tile later holds the warps'
    // similarity rows
    const size_t a_bytes = static_cast<size_t>(kM) * hot_bytes;
    const size_t rows = static_cast<size_t>(kWarps) * kAssignMaxCentroids * 4;
    L.a = o;         o += a_bytes > rows ? a_bytes : rows;
    L.b = o;         o += 2 * kStageBytes;
    L.hot_bits = o;  o += (static_cast<size_t>(words) * 4 + 15) & ~size_t(15);
    L.cold_bits = o; o += (static_cast<size_t>(words) * 4 + 15) & ~size_t(15);
    L.cdoc = o;      o += kAssignMaxCentroids * 4;
    L.own = o;       o += kAssignMaxCentroids * 4;
    L.mdoc = o;      o += kM * 4;
    L.total = o + 1024;  // slack to align the base
    return L;
}

// One stage of centroid rows: terms [128 kc, 128 kc + 128) of centroids
// [n0, n0 + n).
__device__ __forceinline__ void load_stage(const Args& a, uint32_t stage, const int32_t* cdoc,
                                           int nc, int n0, int n, int kc, int tid) {
    for (int i = tid; i < n * 8; i += kThreads) {
        const int r = i >> 3, j = i & 7;
        const bool valid = n0 + r < nc;
        const int64_t doc = valid ? cdoc[n0 + r] : 0;
        copy16(stage + swizzled(r, j),
               a.hot + doc * a.hot_bytes + kc * kKBytes + 16 * j, valid);
    }
}

__global__ void __launch_bounds__(kThreads, 1) assign_u8_kernel(Args a) {
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t bar[2];  // a stage's MMAs have read it
    __shared__ uint32_t s_tmem;
    __shared__ int32_t s_list, s_members, s_warp[kWarps];
    const uint32_t raw = smem_addr(smem_raw);
    unsigned char* smem = smem_raw + (((raw + 1023u) & ~1023u) - raw);
    const Layout L = smem_layout(a.hot_bytes, a.words);
    const uint32_t smA = smem_addr(smem + L.a), smB = smem_addr(smem + L.b);
    uint32_t* hot_bits = reinterpret_cast<uint32_t*>(smem + L.hot_bits);
    uint32_t* cold_bits = reinterpret_cast<uint32_t*>(smem + L.cold_bits);
    int32_t* cdoc = reinterpret_cast<int32_t*>(smem + L.cdoc);
    int32_t* own = reinterpret_cast<int32_t*>(smem + L.own);  // codes of the list's term
    int32_t* mdoc = reinterpret_cast<int32_t*>(smem + L.mdoc);
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const size_t cta = blockIdx.x;
    int32_t* ends = a.ends + cta * (a.f.dim + 1);
    uint32_t* entry = a.entry + cta * a.max_entries;
    int32_t* member = a.member + cta * a.max_kept;
    uint8_t* isc = a.is_centroid + cta * a.max_kept;
    int32_t* sims_g = a.sims + cta * kM * a.ld;
    const uint8_t* codes = static_cast<const uint8_t*>(a.f.val);

    if (warp == 0) tmem_alloc(&s_tmem);
    if (tid == 0) {
        mbar_init(&bar[0], 1);
        mbar_init(&bar[1], 1);
        fence_mbar_init();
    }
    for (int i = tid; i < a.words; i += kThreads) {
        hot_bits[i] = a.hot_bits[i];
        cold_bits[i] = 0u;
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = s_tmem;
    uint32_t uses0 = 0, uses1 = 0;  // stages issued so far, per buffer
    bool failed = false;

    while (!failed) {
        if (tid == 0) {
            s_list = atomicAdd(a.work, 1);
            s_members = 0;
        }
        __syncthreads();
        const int32_t t = s_list;
        if (t >= a.l.n_lists) break;
        const int64_t kb = a.l.kept_ptr[t];
        const int32_t n = static_cast<int32_t>(a.l.kept_ptr[t + 1] - kb);
        const int32_t nc = static_cast<int32_t>(a.l.cptr[t + 1] - a.l.cptr[t]);
        const int32_t* cp = a.l.cpos + a.l.cptr[t];
        const int32_t* kept = a.l.kept + kb;
        for (int32_t c = tid; c < nc; c += kThreads) {
            a.out_key[kb + cp[c]] = static_cast<uint32_t>(c) * 2u;
            cdoc[c] = kept[cp[c]];
            own[c] = 0;
        }
        if (n <= nc) {  // every doc is a centroid
            __syncthreads();
            continue;
        }
        for (int32_t i = tid; i < n; i += kThreads) isc[i] = 0;
        __syncthreads();
        for (int32_t c = tid; c < nc; c += kThreads) isc[cp[c]] = 1;
        // the centroids' other terms by term, in the operands' place: counts,
        // their exclusive scan, and (below) the scatter, which moves each
        // term's start to its end
        int32_t* at = reinterpret_cast<int32_t*>(smem + L.a);
        for (int i = tid; i < a.f.dim; i += kThreads) at[i] = 0;
        __syncthreads();
        for (int32_t c = warp; c < nc; c += kWarps) {
            const uint2 ri = __ldg(a.f.rowinfo + cdoc[c]);
            const uint16_t* ip = a.f.idx + static_cast<size_t>(ri.x) * kRowAlign;
            for (uint32_t e = lane; e < ri.y; e += 32) {
                const uint32_t term = __ldg(ip + e);
                const uint32_t bit = 1u << (term & 31);
                if ((hot_bits[term >> 5] & bit) || term == static_cast<uint32_t>(t)) continue;
                atomicAdd(&at[term], 1);
                if (!(cold_bits[term >> 5] & bit)) atomicOr(&cold_bits[term >> 5], bit);
            }
        }
        // the docs to assign
        for (int32_t i0 = 0; i0 < n; i0 += kThreads) {
            const int32_t i = i0 + tid;
            const bool is = i < n && !isc[i];
            const unsigned m = __ballot_sync(kFull, is);
            int32_t base = 0;
            if (lane == 0 && m != 0u) base = atomicAdd(&s_members, __popc(m));
            base = __shfl_sync(kFull, base, 0);
            if (is) member[base + __popc(m & ((1u << lane) - 1u))] = i;
        }
        __syncthreads();
        {
            // thread i scans terms [i * per, i * per + per)
            const int per = (a.f.dim + kThreads - 1) / kThreads;
            const int lo = min(a.f.dim, tid * per), hi = min(a.f.dim, lo + per);
            int mine = 0;
            for (int i = lo; i < hi; ++i) mine += at[i];
            int incl = mine;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const int y = __shfl_up_sync(kFull, incl, o);
                if (lane >= o) incl += y;
            }
            if (lane == 31) s_warp[warp] = incl;
            __syncthreads();
            int run = incl - mine;
            for (int w = 0; w < warp; ++w) run += s_warp[w];
            for (int i = lo; i < hi; ++i) {
                const int c = at[i];
                at[i] = run;
                run += c;
            }
        }
        __syncthreads();
        for (int32_t c = warp; c < nc; c += kWarps) {
            const uint2 ri = __ldg(a.f.rowinfo + cdoc[c]);
            const int64_t rb = static_cast<int64_t>(ri.x) * kRowAlign;
            for (uint32_t e = lane; e < ri.y; e += 32) {
                const uint32_t term = __ldg(a.f.idx + rb + e);
                if (hot_bits[term >> 5] & (1u << (term & 31))) continue;
                const uint32_t code = __ldg(codes + rb + e);
                if (term == static_cast<uint32_t>(t)) own[c] = static_cast<int32_t>(code);
                else entry[atomicAdd(&at[term], 1)] = (static_cast<uint32_t>(c) << 8) | code;
            }
        }
        __syncthreads();
        for (int i = tid; i < a.f.dim; i += kThreads) ends[1 + i] = at[i];
        const int32_t members = s_members;
        const int passes = (nc + kN - 1) / kN;
        const int np = ((nc + passes - 1) / passes + 15) & ~15;  // centroids per pass
        const int chunks = a.hot_bytes / kKBytes;
        const int steps = passes * chunks;
        const uint32_t idesc = instr_desc(np);
        __syncthreads();

        for (int32_t m0 = 0; m0 < members && !failed; m0 += kM) {
            const int rows = min(kM, members - m0);
            const bool first_ok = uses0 == 0 || mbar_wait_bounded(&bar[0], (uses0 - 1u) & 1u);
            if (tid < kM) mdoc[tid] = tid < rows ? kept[member[m0 + tid]] : 0;
            __syncthreads();
            // A: the docs' hot rows
            const int pieces = a.hot_bytes / 16;
            for (int i = tid; i < kM * pieces; i += kThreads) {
                const int r = i / pieces, j = i - r * pieces;
                copy16(smA + static_cast<uint32_t>(j >> 3) * (kM * kKBytes) + swizzled(r, j & 7),
                       a.hot + static_cast<int64_t>(mdoc[r]) * a.hot_bytes + 16 * j, r < rows);
            }
            load_stage(a, smB, cdoc, nc, 0, np, 0, tid);
            copies_commit();
            for (int it = 0; it < steps; ++it) {
                const int s = it & 1;
                const int pass = it / chunks, kc = it - pass * chunks;
                bool ok = first_ok;
                if (it + 1 < steps) {
                    // the next stage's buffer is free once the MMAs of the
                    // step before have read it
                    const uint32_t u = s ? uses0 : uses1;
                    if (u > 0) ok &= mbar_wait_bounded(&bar[s ^ 1], (u - 1u) & 1u);
                    const int p1 = (it + 1) / chunks;
                    load_stage(a, smB + (s ^ 1) * kStageBytes, cdoc, nc, p1 * np, np,
                               it + 1 - p1 * chunks, tid);
                    copies_commit();
                    copies_wait<1>();
                } else {
                    copies_wait<0>();
                }
                fence_proxy_async_smem();
                if (__syncthreads_or(!ok)) {
                    failed = true;
                    break;
                }
                if (tid == 0) {
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint32_t ka = smA + static_cast<uint32_t>(kc) * (kM * kKBytes);
                    const uint32_t kbuf = smB + static_cast<uint32_t>(s) * kStageBytes;
#pragma unroll
                    for (int k = 0; k < kKBytes / 32; ++k)
                        mma_u8(tmem, operand_desc(ka + 32 * k), operand_desc(kbuf + 32 * k), idesc,
                               kc > 0 || k > 0);
                    mma_commit(&bar[s]);
                }
                if (s) ++uses1;
                else ++uses0;
                if (kc + 1 < chunks) continue;
                // the pass's accumulators: warp w reads TMEM lanes 32 (w % 4)..
                // and columns 32 (w / 4)..
                ok = mbar_wait_bounded(&bar[s], ((s ? uses1 : uses0) - 1u) & 1u);
                if (__syncthreads_or(!ok)) {
                    failed = true;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const int col = 32 * (warp >> 2);
                if (col < np) {
                    uint32_t r[32];
                    tmem_load32(tmem + (static_cast<uint32_t>(32 * (warp & 3)) << 16) +
                                    static_cast<uint32_t>(col), r);
                    int32_t* out = sims_g + static_cast<size_t>(32 * (warp & 3) + lane) * a.ld +
                                   pass * np + col;
#pragma unroll
                    for (int i = 0; i < 4; ++i)  // np is a multiple of 16
                        if (col + 8 * i < np) store256(out + 8 * i, r + 8 * i);
                }
                asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                __syncthreads();
            }
            if (failed) break;
            // sparse products and argmax, a warp per doc, in the A tile's place
            int32_t* sims = reinterpret_cast<int32_t*>(smem + L.a) + warp * kAssignMaxCentroids;
            uint2* hits = reinterpret_cast<uint2*>(smem + L.b) + warp * kHits;
            // lane i holds the row info of the warp's i-th doc
            uint2 infos = make_uint2(0u, 0u);
            if (lane < kM / kWarps && warp + lane * kWarps < rows)
                infos = __ldg(a.f.rowinfo + mdoc[warp + lane * kWarps]);
            for (int r = warp; r < rows; r += kWarps) {
                // its dense sums, on their way while the row is looked up
                const int32_t* src = sims_g + static_cast<size_t>(r) * a.ld;
                for (int c = lane * 4; c < nc; c += 128) copy16(smem_addr(sims + c), src + c, true);
                copies_commit();
                const int which = (r - warp) / kWarps;
                const int64_t rb =
                    static_cast<int64_t>(__shfl_sync(kFull, infos.x, which)) * kRowAlign;
                const uint32_t len = __shfl_sync(kFull, infos.y, which);
                int own_v = 0;  // the doc's code of the list's term
                int nh = 0;
                bool landed = false;
                // the products of the index runs listed in `hits`: eight
                // lanes per piece, four pieces at once, 16 in flight
                auto apply = [&]() {
                    if (!landed) copies_wait<0>();
                    landed = true;
                    __syncwarp();
                    for (int h0 = 0; h0 < nh; h0 += 16) {
                        uint2 h[4];
                        uint32_t x[4];
#pragma unroll
                        for (int u = 0; u < 4; ++u) {
                            const int i = h0 + 4 * u + (lane >> 3);
                            h[u] = i < nh ? hits[i] : make_uint2(0u, 0u);
                            x[u] = 0u;
                            if ((lane & 7u) < (h[u].y & 0xffffu)) x[u] = entry[h[u].x + (lane & 7)];
                        }
#pragma unroll
                        for (int u = 0; u < 4; ++u)
                            if ((lane & 7u) < (h[u].y & 0xffffu))
                                atomicAdd(&sims[x[u] >> 8], static_cast<int>(h[u].y >> 16) *
                                                                static_cast<int>(x[u] & 0xffu));
                    }
                    __syncwarp();
                    nh = 0;
                };
                for (uint32_t e0 = 0; e0 < len; e0 += 128) {
                    uint32_t term[4], code[4], start[4], cnt[4];
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint32_t e = e0 + 32 * c + lane;
                        term[c] = 0xffffffffu;
                        code[c] = 0u;
                        if (e < len) {
                            term[c] = __ldg(a.f.idx + rb + e);
                            code[c] = __ldg(codes + rb + e);
                        }
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const bool in = term[c] != 0xffffffffu &&
                                        ((cold_bits[term[c] >> 5] >> (term[c] & 31)) & 1u);
                        start[c] = in ? static_cast<uint32_t>(ends[term[c]]) : 0u;
                        cnt[c] = in ? static_cast<uint32_t>(ends[term[c] + 1]) : 0u;
                    }
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        if (term[c] == static_cast<uint32_t>(t)) own_v = static_cast<int>(code[c]);
                        cnt[c] -= start[c];
                        // runs in pieces of up to eight entries
                        for (uint32_t p = 0;; p += 8) {
                            const unsigned m = __ballot_sync(kFull, cnt[c] > p);
                            if (m == 0u) break;
                            if (nh > kHits - 32) apply();
                            if (cnt[c] > p)
                                hits[nh + __popc(m & ((1u << lane) - 1u))] =
                                    make_uint2(start[c] + p, min(cnt[c] - p, 8u) | (code[c] << 16));
                            nh += __popc(m);
                        }
                    }
                }
                apply();
                own_v = __reduce_add_sync(kFull, own_v);
                // strict >, ascending: ties go to the lowest cluster
                int best = 0, bi = -1;
                for (int c = lane; c < nc; c += 32) {
                    const int x = sims[c] + own_v * own[c];
                    if (bi < 0 || x > best) {
                        best = x;
                        bi = c;
                    }
                }
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    const int s2 = __shfl_xor_sync(kFull, best, o);
                    const int i2 = __shfl_xor_sync(kFull, bi, o);
                    if (i2 >= 0 && (bi < 0 || s2 > best || (s2 == best && i2 < bi))) {
                        best = s2;
                        bi = i2;
                    }
                }
                if (lane == 0)
                    a.out_key[kb + member[m0 + r]] = static_cast<uint32_t>(bi) * 2u + 1u;
                __syncwarp();
            }
            __syncthreads();
        }
        for (int i = tid; i < a.words; i += kThreads) cold_bits[i] = 0u;
        __syncthreads();
    }
    if (failed) {
        // the copies in flight end before the CTA does
        copies_wait<0>();
        if (tid == 0) atomicExch(a.err, 1);
    }
    __syncthreads();
    if (warp == 0) tmem_free(tmem);
}

// Hot rows, a warp per doc: the doc's codes of the hot terms at their slots.
// *unsorted = 1 when a row's terms are not strictly ascending.
constexpr int kRowWarps = 8;
__global__ void __launch_bounds__(kRowWarps * 32)
hot_rows_kernel(FwdView f, const uint16_t* slot_of, int hot_bytes, uint8_t* hot, int* unsorted) {
    __shared__ __align__(16) uint8_t row[kRowWarps][kHot];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t nw = static_cast<int64_t>(gridDim.x) * kRowWarps;
    const uint8_t* codes = static_cast<const uint8_t*>(f.val);
    uint4* r4 = reinterpret_cast<uint4*>(row[warp]);
    for (int64_t d = static_cast<int64_t>(blockIdx.x) * kRowWarps + warp; d < f.n_docs; d += nw) {
        for (int i = lane; i < hot_bytes / 16; i += 32) r4[i] = make_uint4(0u, 0u, 0u, 0u);
        __syncwarp();
        const uint2 ri = __ldg(f.rowinfo + d);
        const int64_t rb = static_cast<int64_t>(ri.x) * kRowAlign;
        bool bad = false;
        for (uint32_t e = lane; e < ri.y; e += 32) {
            const uint32_t t = __ldg(f.idx + rb + e);
            bad |= e > 0 && __ldg(f.idx + rb + e - 1) >= t;
            const uint32_t s = __ldg(slot_of + t);
            if (s < static_cast<uint32_t>(hot_bytes)) row[warp][s] = __ldg(codes + rb + e);
        }
        if (__any_sync(kFull, bad) && lane == 0) atomicOr(unsorted, 1);
        __syncwarp();
        uint4* out = reinterpret_cast<uint4*>(hot + d * hot_bytes);
        for (int i = lane; i < hot_bytes / 16; i += 32) out[i] = r4[i];
        __syncwarp();
    }
}

}  // namespace

bool assign_u8(const FwdView& f, const AssignLists& lists, const std::vector<int64_t>& df,
               uint32_t* out_key, cudaStream_t s, Arena& scratch) {
    const int dim = f.dim;
    if (lists.max_nc > kAssignMaxCentroids || f.n_docs == 0 || dim > kMaxDim ||
        lists.max_row > kAssignMaxRowU8)
        return false;
    // the hot terms: as many as the dense rows hold, by document frequency
    size_t free_b = 0, total_b = 0;
    cuda_check(cudaMemGetInfo(&free_b, &total_b), "cudaMemGetInfo");
    int hot_bytes = std::min(kHot, (dim + kKBytes - 1) / kKBytes * kKBytes);
    while (hot_bytes > kKBytes &&
           static_cast<size_t>(f.n_docs) * hot_bytes > free_b / 4)
        hot_bytes -= kKBytes;
    std::vector<int32_t> by_df(static_cast<size_t>(dim));
    std::iota(by_df.begin(), by_df.end(), 0);
    const int n_hot = std::min(dim, hot_bytes);
    std::partial_sort(by_df.begin(), by_df.begin() + n_hot, by_df.end(),
                      [&](int32_t x, int32_t y) { return df[x] != df[y] ? df[x] > df[y] : x < y; });
    // The share of a random pair's products on hot terms: from half on the
    // dense part is worth its multiply-adds. The assignment phase here against
    // the general kernel (100,000 docs, lambda 3000, beta 300, terms Zipf(s)):
    // s = 1.1, share 0.99: 18 against 115 ms; 0.5, 0.65: 39 against 143; 0.3,
    // 0.24: 50 against 178, so the line is on the safe side, and corpora below
    // it, whose terms are close to evenly spread, were not measured further.
    double hot_sq = 0.0, all_sq = 0.0;
    for (int i = 0; i < dim; ++i) {
        const double x = static_cast<double>(df[by_df[i]]);
        all_sq += x * x;
        if (i < n_hot) hot_sq += x * x;
    }
    if (hot_sq < 0.5 * all_sq) return false;
    const int words = (dim + 31) / 32;
    std::vector<uint16_t> slot_of(static_cast<size_t>(dim), 0xffff);
    std::vector<uint32_t> bits(static_cast<size_t>(words), 0u);
    for (int i = 0; i < n_hot; ++i) {
        const int32_t t = by_df[i];
        slot_of[t] = static_cast<uint16_t>(i);
        bits[t >> 5] |= 1u << (t & 31);
    }
    const int sms = device_sm_count();
    const Arena::Mark mark = scratch.mark();
    const uint16_t* d_slot = scratch.put(slot_of.data(), slot_of.size());
    const uint32_t* d_bits = scratch.put(bits.data(), bits.size());
    uint8_t* hot = scratch.take<uint8_t>(static_cast<size_t>(f.n_docs) * hot_bytes);
    int32_t* flags = scratch.take<int32_t>(3);  // unsorted rows, list counter, error
    cuda_check(cudaMemsetAsync(flags, 0, 3 * sizeof(int32_t), s), "memset");
    hot_rows_kernel<<<sms * 8, kRowWarps * 32, 0, s>>>(f, d_slot, hot_bytes, hot, flags);
    cuda_check(cudaGetLastError(), "hot_rows_kernel");
    int32_t unsorted = 0;
    cuda_check(cudaMemcpyAsync(&unsorted, flags, sizeof(unsorted), cudaMemcpyDeviceToHost,
                               s), "D2H");
    cuda_check(cudaStreamSynchronize(s), "sync");
    if (unsorted != 0) {
        scratch.release(mark);
        return false;
    }

    const int ctas = sms;
    const int64_t max_entries = std::max<int64_t>(1, static_cast<int64_t>(lists.max_nc) *
                                                         lists.max_row);
    const int64_t max_kept = std::max<int64_t>(lists.max_kept, 1);
    const size_t n = static_cast<size_t>(ctas);
    int32_t* ends = scratch.take<int32_t>(n * (dim + 1));
    // a pass's centroids are padded to 16, so up to 4 passes fill 1,088 columns
    const int ld = kAssignMaxCentroids + 64;
    cuda_check(cudaMemsetAsync(ends, 0, n * (dim + 1) * sizeof(int32_t), s), "memset");
    Args a{};
    a.f = f;
    a.l = lists;
    a.hot = hot;
    a.hot_bytes = hot_bytes;
    a.hot_bits = d_bits;
    a.words = words;
    a.out_key = out_key;
    a.work = flags + 1;
    a.err = flags + 2;
    a.ends = ends;
    a.entry = scratch.take<uint32_t>(n * max_entries);
    a.member = scratch.take<int32_t>(n * max_kept);
    a.is_centroid = scratch.take<uint8_t>(n * max_kept);
    a.sims = scratch.take<int32_t>(n * kM * ld);
    a.max_entries = max_entries;
    a.max_kept = max_kept;
    a.ld = ld;
    const size_t smem = smem_layout(hot_bytes, words).total;
    cuda_check(allow_opt_in_smem(assign_u8_kernel), "assign shared memory");
    assign_u8_kernel<<<ctas, kThreads, smem, s>>>(a);
    cuda_check(cudaGetLastError(), "assign_u8_kernel");
    int32_t err = 0;
    cuda_check(cudaMemcpyAsync(&err, a.err, sizeof(err), cudaMemcpyDeviceToHost, s), "D2H");
    cuda_check(cudaStreamSynchronize(s), "assign sync");
    scratch.release(mark);
    if (err != 0) throw std::runtime_error("assignment kernel gave up waiting for the tensor core");
    return true;
}

}  // namespace nsp
