// SEISMIC / SEISMIC-SQ search on sm_100a, one CTA per query (kernel
// variants 2-5). A persistent grid steals queries from a global counter; the
// CTA's warps walk the query's blocks together.
//
// Per query (seismic_index.cpp:231-274, seismic_scalar_quantized_index.cpp:
// 307-357):
//   1. the query is scattered into a dense per-term table in shared memory --
//      the reference's dimension-sized dense buffer (seismic_index.cpp:243-
//      246), one byte per term: fp32 queries store the term's rank (0 = not
//      in the query; the rank indexes a table of the query's values, entry 0
//      holding 0), 8-bit queries store the code itself, 16-bit queries the
//      rank while a byte holds it;
//   2. the query cut (utils/vector_process.h:18-30) is a rank selection;
//   3. block summary scores (inverted_list_clusters.cpp:295-331) of up to
//      one list per warp are accumulated at once, each warp hit term by hit
//      term in ascending term order;
//   4. the first list's blocks are sorted by score descending in the order
//      the reference's sort leaves equal scores (seismic_common.h:105-115);
//      later lists keep block order;
//   5. blocks are taken in that order into batches of up to `batch_docs`
//      docs. A block that fails the pruning test (seismic_index.cpp:78-86)
//      against the current heap minimum is skipped (or ends the first list);
//      the heap minimum only grows, so a block that fails now fails at its
//      turn too. Blocks that pass are gathered, their docs scored in
//      parallel, and then -- in block order -- each block is tested again
//      against the heap as it stands when its turn comes, exactly as the
//      reference tests it, and its docs are offered in order. Docs of a block
//      that fails the second test are dropped: the result is the reference's,
//      only some scoring work is speculative;
//   6. a group of kG lanes (1, 2, 4 or 8) scores one doc at a time, 16 row
//      elements per lane per step from 256-bit loads of the padded forward
//      rows, and takes the next doc of the batch as soon as its row ends, so
//      groups stay busy across rows of different lengths. fp32 scores are the
//      reference's sequential sum result += w * dense[t] over the whole row
//      (utils/distance.h:29-37), with the same round-to-nearest products and
//      sums in the same order: bit-identical. The zero padding after a row
//      adds +-0.0, which leaves every sum unchanged unless the query holds a
//      non-finite value, in which case padding elements are masked out. SQ
//      sums are exact integers (distance.h:39-57);
//   7. scores enter a shared-memory top-k in the reference's insertion order;
//      a doc already in the heap is skipped and one scored before and
//      evicted or rejected scores <= the (monotone) heap minimum and is
//      rejected again: the reference's visited set (seismic_index.cpp:104-
//      107) without an O(n_docs) bitmap per query.
#include <cuda_runtime.h>

#include <cfloat>
#include <climits>
#include <cstdint>
#include <type_traits>

#include "nsp_device.h"
#include "search_common.cuh"
#include "seismic_cta.cuh"

namespace nsp {
namespace {

template <typename V, typename TE, int kG>
__global__ void __launch_bounds__(1024, 1) seismic_cta_kernel(SeismicLaunch a) {
    extern __shared__ __align__(16) unsigned char smem[];
    constexpr bool kRank = kRankTable<V, TE>;
    constexpr bool kF32 = std::is_same<V, float>::value;
    constexpr int vsz = static_cast<int>(sizeof(V));
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int nwarps = blockDim.x >> 5;
    const int dim = a.fwd.dim;
    const int batch = a.batch_docs;
    const CtaLayout L =
        cta_layout(vsz, static_cast<int>(sizeof(TE)), dim, a.qcap, a.k, batch, a.seg_cap);
    Ctl* ctl = reinterpret_cast<Ctl*>(smem);
    TE* tbl = reinterpret_cast<TE*>(smem + L.tbl);
    float* qv = reinterpret_cast<float*>(smem + L.qv);
    uint16_t* qterm = reinterpret_cast<uint16_t*>(smem + L.qterm);
    V* qraw = reinterpret_cast<V*>(smem + L.qraw);
    uint16_t* cuts = reinterpret_cast<uint16_t*>(smem + L.cuts);
    float* hs = reinterpret_cast<float*>(smem + L.hs);
    int32_t* hid = reinterpret_cast<int32_t*>(smem + L.hid);
    int32_t* cdoc = reinterpret_cast<int32_t*>(smem + L.cdoc);
    uint32_t* coff = reinterpret_cast<uint32_t*>(smem + L.coff);
    uint32_t* clen = reinterpret_cast<uint32_t*>(smem + L.clen);
    float* csc = reinterpret_cast<float*>(smem + L.csc);
    Seg* segs = reinterpret_cast<Seg*>(smem + L.segs);
    uint16_t* cseg = reinterpret_cast<uint16_t*>(smem + L.cseg);  // each candidate's segment
    int* wsum = reinterpret_cast<int*>(smem + L.wsum);

    const int maxb = a.ix.max_blocks;
    float* bscore_cta = a.bscore + static_cast<size_t>(blockIdx.x) * nwarps * maxb;
    uint16_t* order = a.order + static_cast<size_t>(blockIdx.x) * a.order_stride;
    unsigned long long* keys_g =
        a.sortkeys != nullptr ? a.sortkeys + static_cast<size_t>(blockIdx.x) * a.sort_stride
                              : nullptr;

    for (int i = tid; i <= dim; i += blockDim.x) tbl[i] = 0;
    if (tid == 0) qv[0] = 0.0f;

    const unsigned cid = blockIdx.x, ncl = gridDim.x;  // this CTA's query slot, and the slots

    int iter = 0;
    for (;;) {
        if (tid == 0) {
            int q;
            if (a.work_counter != nullptr) {
                q = atomicAdd(a.work_counter, 1);
                if (a.qorder != nullptr && q < a.q.n) q = a.qorder[q];
            } else
                q = a.first_query + static_cast<int>(cid) + iter * static_cast<int>(ncl);
            ctl->q = q;
            ctl->nheap = 0;  // the query's heap starts empty
        }
        ++iter;
        __syncthreads();
        const int q = ctl->q;
        if (q >= a.q.n) break;

        const uint64_t* sel = a.sel_q != nullptr ? a.sel_q[q] : a.sel_bits;
        // 1. scatter the query
        const int32_t qs = a.q.indptr[q];
        int qn = a.q.indptr[q + 1] - qs;
        // the caller's max_nnz was wrong, or the row lies past the query
        // arrays: padding, and the error is reported
        if (qn > a.qcap || qn < 0 || qs < 0 || (a.nnz_cap >= 0 && qs + qn > a.nnz_cap)) {
            if (tid == 0 && a.err != nullptr) atomicExch(a.err, 3);
            qn = 0;
        }
        bool bad = false;
        for (int i = tid; i < qn; i += blockDim.x) {
            const uint32_t t = a.q.idx[qs + i];
            const V v = static_cast<const V*>(a.q.val)[qs + i];
            qterm[i] = static_cast<uint16_t>(t);
            qraw[i] = v;
            if (t < static_cast<uint32_t>(dim)) {
                if constexpr (kRank) {
                    tbl[t] = static_cast<TE>(i + 1);
                } else {
                    tbl[t] = static_cast<TE>(v);
                }
            }
            if constexpr (kF32) {
                qv[i + 1] = v;
                bad |= !isfinite(v);
            } else if constexpr (kRank) {
                reinterpret_cast<uint32_t*>(qv)[i + 1] = v;
            }
        }
        const bool nonfinite = __syncthreads_or(bad) != 0;

        // 2. query cut (utils/vector_process.h:18-30): the query's order when
        // cut >= nnz, else the reference's TopKHolder over (value, position)
        int ncut;
        if (a.cut >= qn) {
            ncut = qn;
            for (int i = tid; i < qn; i += blockDim.x) cuts[i] = qterm[i];
        } else {
            ncut = a.cut;
            query_cut<V>(cuts, qraw, qn, ncut, reinterpret_cast<uint32_t*>(smem + L.cdoc),
                         static_cast<int>((L.wsum - L.cdoc) / 4), tid);
            for (int i = tid; i < ncut; i += blockDim.x) cuts[i] = qterm[cuts[i]];
        }
        __syncthreads();

        // counting pass: this CTA's stamps, and warp 0's per-lane counts
        uint32_t* uq = reinterpret_cast<uint32_t*>(smem + L.uq);
        if (a.visit != nullptr && warp == 0) {
            uq[lane] = 0;
            uq[32 + lane] = 0;
        }
        int n = 0;  // heap size (warp 0)
        bool first = true;
        // Counters of this query (32 bits: a query reads far less than 4 GB).
        // docs_scored / row_bytes: every thread adds the member docs of each
        // batch it checks after scoring; warp 0 takes back those of segments
        // the second test drops, so a thread's value may be negative.
        uint32_t blocks_visited = 0, bytes = 0, lists = 0;
        int32_t docs_scored = 0, row_bytes = 0;
        for (int c = 0; c < ncut; ++c) {
            // 3. summary scores of the next nwarps lists, one warp per list
            if (c % nwarps == 0) {
                const int cw = c + warp;
                if (cw < ncut) {
                    const int tw = cuts[cw];
                    if (tw < a.ix.n_lists) {
                        const int nbw = static_cast<int>(a.ix.lbp[tw + 1] - a.ix.lbp[tw]);
                        if (nbw > 0)
                            list_summaries<V>(a, tw, nbw, qterm, qraw, qn,
                                              bscore_cta + static_cast<size_t>(warp) * maxb,
                                              lane, bytes);
                    }
                }
                __syncthreads();
            }
            const int t = cuts[c];
            if (t >= a.ix.n_lists) continue;  // seismic_index.cpp:254-256
            const int64_t lb0 = a.ix.lbp[t];
            const int nb = static_cast<int>(a.ix.lbp[t + 1] - lb0);
            if (nb > 0) {
                ++lists;
                const float* bscore = bscore_cta + static_cast<size_t>(c % nwarps) * maxb;
                // 4. visiting order: the first list's blocks sorted; a later
                // list's blocks that can still pass, in block order
                int nbv = nb;
                if (first) {
                    // in the batch arrays' place where they are large enough
                    const size_t room = L.sq - L.cdoc;
                    const size_t pairs = static_cast<size_t>(nb) * sizeof(ranking::Blk);
                    ranking::Blk* items = reinterpret_cast<ranking::Blk*>(
                        pairs <= room ? reinterpret_cast<unsigned long long*>(cdoc) : keys_g);
                    if (items == nullptr) {  // the host sizes sortkeys; never taken
                        if (tid == 0) atomicExch(a.err, 2);
                        break;
                    }
                    uint16_t* stops = pairs + static_cast<size_t>(nb) * 2 <= room
                                          ? reinterpret_cast<uint16_t*>(smem + L.cdoc + pairs)
                                          : order;
                    sort_blocks(bscore, nb, items, stops, order,
                                reinterpret_cast<uint32_t*>(smem + L.sq), tid, lane, warp, nwarps);
                } else {
                    const int nh = ctl->nheap;
                    nbv = passing_blocks(bscore, nb, nh == a.k, nh == a.k ? hs[0] : 0.0f,
                                         a.heap_factor, order, wsum, tid, lane, warp, nwarps);
                }
                // 5. batches
                Cursor& cur = *reinterpret_cast<Cursor*>(smem + L.cur);
                if (warp == 0) {
                    cur.o = 0;
                    cur.dead = false;
                    cur.split = false;
                    cur.split_d = 0;
                    cur.split_left = 0;
                    cur.split_bs = 0.0f;
                }
                for (;;) {
                    if (warp == 0) {
                        int total = 0;
                        const int nseg = gather(a, cur, first, lb0, nbv, bscore, order, n, hs,
                                                segs, batch, a.seg_cap, total, lane);
                        if (lane == 0) {
                            ctl->nseg = nseg;
                            ctl->total = total;
                            ctl->next = 0;
                            ctl->nheap = n;
                        }
                    }
                    __syncthreads();
                    const int nseg = ctl->nseg;
                    int total = ctl->total;
                    if (nseg == 0) break;
                    if (total > 0) {
                        // candidates: doc ids and row info of every segment's docs
                        // (with a selector: of its members, in order)
                        int members = 0;
                        for (int i0 = 0; i0 < total; i0 += blockDim.x) {
                            const int i = i0 + tid;
                            bool member = i < total;
                            int32_t d = 0;
                            int lo = 0, at = i;
                            uint2 ri = make_uint2(0u, 0u);
                            if (member) {
                                int hi = nseg - 1;
                                while (lo < hi) {
                                    const int mid = (lo + hi + 1) >> 1;
                                    if (segs[mid].cand0 <= i)
                                        lo = mid;
                                    else
                                        hi = mid - 1;
                                }
                                const Seg& g = segs[lo];
                                const int64_t pj = g.d0 + (i - g.cand0);
                                d = __ldg(a.ix.docs + pj);
                                // row info stored with the posting, else looked up
                                ri = a.ix.drow != nullptr ? __ldg(a.ix.drow + pj)
                                                          : __ldg(a.fwd.rowinfo + d);
                                if (sel != nullptr)
                                    member = (__ldg(sel + (d >> 6)) >> (d & 63)) & 1ull;
                            }
                            if (sel != nullptr) {
                                const unsigned m = __ballot_sync(kFull, member);
                                if (lane == 0) wsum[warp] = __popc(m);
                                __syncthreads();
                                at = members + __popc(m & ((1u << lane) - 1u));
                                for (int w = 0; w < nwarps; ++w) {
                                    const int c = wsum[w];
                                    at += w < warp ? c : 0;
                                    members += c;
                                }
                                __syncthreads();
                            }
                            if (member) {
                                cdoc[at] = d;
                                coff[at] = ri.x;
                                clen[at] = ri.y;
                                cseg[at] = static_cast<uint16_t>(lo);
                            }
                        }
                        __syncthreads();
                        if (sel != nullptr) {
                            total = members;
                            // the segments' members among the candidates
                            for (int t = tid; t < nseg; t += blockDim.x) {
                                int bound[2];
#pragma unroll
                                for (int u = 0; u < 2; ++u) {
                                    int lo = 0, hi = total;
                                    while (lo < hi) {
                                        const int mid = (lo + hi) >> 1;
                                        if (cseg[mid] < t + u) lo = mid + 1;
                                        else hi = mid;
                                    }
                                    bound[u] = lo;
                                }
                                segs[t].cand0 = bound[0];
                                segs[t].cnt = bound[1] - bound[0];
                            }
                            __syncthreads();
                        }
                        // 6. scores
                        if (kF32 && nonfinite)
                            score_batch<V, TE, true, kG>(a.fwd, ctl, tbl, qv, coff, clen, csc,
                                                         total, lane);
                        else
                            score_batch<V, TE, false, kG>(a.fwd, ctl, tbl, qv, coff, clen,
                                                          csc, total, lane);
                        __syncthreads();
                    }
                    // 7. second pruning test and heap offers, in block order.
                    // (a) All threads: a doc can still enter the heap only if
                    // it is a member scoring above the heap minimum as it
                    // stood when the batch was gathered (the minimum only
                    // grows); segments take the best score of such docs.
                    {
                        const int nh = ctl->nheap;
                        const float hmin0 = nh == a.k ? hs[0] : 0.0f;
                        for (int i = tid; i < total; i += blockDim.x) {
                            ++docs_scored;
                            row_bytes += 8 + static_cast<int32_t>(clen[i]) * (2 + vsz);
                            if (nh < a.k || !(csc[i] <= hmin0))
                                atomicMax(&segs[cseg[i]].best, score_key(csc[i]));
                        }
                        __syncthreads();
                    }
                    // (b) Warp 0 walks the segments.
                    if (warp == 0)
                        walk_batch<V, false>(a, segs, nseg, total, cdoc, clen, csc, hs, hid, n, first,
                                      cur.dead, cur.split, uq, static_cast<uint32_t>(iter), lane,
                                      blocks_visited, bytes, docs_scored, row_bytes);
                }
            }
            first = false;  // seismic_index.cpp:261
        }

        // results, padded with (-1.0, -1); SQ scores decoded
        // (seismic_scalar_quantized_index.cpp:345-355)
        if (warp == 0) {
            heap_emit(hs, hid, n, a.k, a.decode_scale, a.out_d + static_cast<size_t>(q) * a.k,
                      a.out_l + static_cast<size_t>(q) * a.k, lane);
            if (a.done != nullptr) {
                // every lane's results reach memory (mapped host memory
                // included) before the flag does
                __threadfence_system();
                __syncwarp();
                if (lane == 0) *reinterpret_cast<volatile int32_t*>(a.done + q) = 1;
            }
        }
        if (a.stats != nullptr) {
            // per warp: its threads' doc counts and row bytes, plus its
            // summary bytes (the same on every lane) and, for warp 0, the
            // block counts
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                row_bytes += __shfl_xor_sync(kFull, row_bytes, o);
                docs_scored += __shfl_xor_sync(kFull, docs_scored, o);
            }
            if (lane == 0) {
                if (warp == 0) {
                    atomicAdd(a.stats + kStatBlocksVisited,
                              static_cast<unsigned long long>(blocks_visited));
                    atomicAdd(a.stats + kStatListsProbed, static_cast<unsigned long long>(lists));
                }
                // a warp's net counts can be negative: widened with their sign,
                // they add up modulo 2^64 to the exact total
                atomicAdd(a.stats + kStatDocsScored,
                          static_cast<unsigned long long>(static_cast<long long>(docs_scored)));
                atomicAdd(a.stats + kStatBytes,
                          static_cast<unsigned long long>(bytes) +
                              static_cast<unsigned long long>(static_cast<long long>(row_bytes)));
                atomicAdd(a.stats + kStatRowBytes,
                          static_cast<unsigned long long>(static_cast<long long>(row_bytes)));
            }
            if (a.visit != nullptr && warp == 0) {
                uint32_t ud = uq[lane], ub = uq[32 + lane];
#pragma unroll
                for (int o = 16; o > 0; o >>= 1) {
                    ud += __shfl_xor_sync(kFull, ud, o);
                    ub += __shfl_xor_sync(kFull, ub, o);
                }
                if (lane == 0) {
                    atomicAdd(a.stats + kStatUniqueDocs, static_cast<unsigned long long>(ud));
                    atomicAdd(a.stats + kStatUniqueRowBytes, static_cast<unsigned long long>(ub));
                }
            }
        }
        // restore the all-zero table for the next query
        __syncthreads();
        for (int i = tid; i < qn; i += blockDim.x) {
            const uint32_t t = qterm[i];
            if (t < static_cast<uint32_t>(dim)) tbl[t] = 0;
        }
    }
}

template <typename V, typename TE>
size_t smem_typed(int dim, int qcap, int k, int batch, int seg_cap) {
    return cta_layout(static_cast<int>(sizeof(V)), static_cast<int>(sizeof(TE)), dim, qcap, k,
                      batch, seg_cap)
        .total;
}

template <typename V, typename TE, int kG>
int max_blocks_cta_g(int threads, size_t smem) {
    if (allow_opt_in_smem(seismic_cta_kernel<V, TE, kG>) != cudaSuccess)
        return 0;
    return resident_blocks(seismic_cta_kernel<V, TE, kG>, threads, smem);
}

template <typename V, typename TE>
int max_blocks_cta_typed(int group, int threads, size_t smem) {
    if (group == 8) return max_blocks_cta_g<V, TE, 8>(threads, smem);
    if (group == 4) return max_blocks_cta_g<V, TE, 4>(threads, smem);
    if (group == 2) return max_blocks_cta_g<V, TE, 2>(threads, smem);
    return max_blocks_cta_g<V, TE, 1>(threads, smem);
}

template <typename V, typename TE, int kG>
cudaError_t launch_cta_g(const SeismicLaunch& a, int warps, int blocks, size_t smem,
                         cudaStream_t s) {
    cudaError_t e = allow_opt_in_smem(seismic_cta_kernel<V, TE, kG>);
    if (e != cudaSuccess) return e;
    seismic_cta_kernel<V, TE, kG><<<blocks, warps * 32, smem, s>>>(a);
    return cudaGetLastError();
}

template <typename V, typename TE>
cudaError_t launch_cta_typed(const SeismicLaunch& a, int warps, int blocks, cudaStream_t s) {
    const size_t smem = smem_typed<V, TE>(a.fwd.dim, a.qcap, a.k, a.batch_docs, a.seg_cap);
    if (a.group_lanes == 8) return launch_cta_g<V, TE, 8>(a, warps, blocks, smem, s);
    if (a.group_lanes == 4) return launch_cta_g<V, TE, 4>(a, warps, blocks, smem, s);
    if (a.group_lanes == 2) return launch_cta_g<V, TE, 2>(a, warps, blocks, smem, s);
    return launch_cta_g<V, TE, 1>(a, warps, blocks, smem, s);
}

}  // namespace

// Claim order of a batched launch: queries by row length, longest first (a
// counting sort over lengths clamped to 255, one CTA).
__global__ void __launch_bounds__(1024) order_by_length_kernel(const int32_t* indptr, int32_t n,
                                                               int32_t* order) {
    __shared__ int32_t bin[256];
    for (int i = threadIdx.x; i < 256; i += blockDim.x) bin[i] = 0;
    __syncthreads();
    auto key = [&](int32_t i) {
        const int32_t len = indptr[i + 1] - indptr[i];
        return 255 - (len < 0 ? 0 : (len > 255 ? 255 : len));
    };
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) atomicAdd(&bin[key(i)], 1);
    __syncthreads();
    if (threadIdx.x == 0) {
        int32_t run = 0;
        for (int b = 0; b < 256; ++b) {
            const int32_t c = bin[b];
            bin[b] = run;
            run += c;
        }
    }
    __syncthreads();
    for (int32_t i = threadIdx.x; i < n; i += blockDim.x) order[atomicAdd(&bin[key(i)], 1)] = i;
}

// Table entries: fp32 and 16-bit queries hold ranks, one byte while the query
// has at most 255 terms; else two bytes (fp32: ranks, 16-bit: codes). 8-bit
// queries hold their codes.
static bool wide_table(int val_kind, int qcap) {
    return (val_kind == kU16 || val_kind == kF32) && qcap > 255;
}

size_t seismic_cta_smem(int val_kind, int dim, int qcap, int k, int batch, int seg_cap) {
    if (val_kind == kF32)
        return wide_table(val_kind, qcap)
                   ? smem_typed<float, uint16_t>(dim, qcap, k, batch, seg_cap)
                   : smem_typed<float, uint8_t>(dim, qcap, k, batch, seg_cap);
    if (val_kind == kU8) return smem_typed<uint8_t, uint8_t>(dim, qcap, k, batch, seg_cap);
    return wide_table(val_kind, qcap)
               ? smem_typed<uint16_t, uint16_t>(dim, qcap, k, batch, seg_cap)
               : smem_typed<uint16_t, uint8_t>(dim, qcap, k, batch, seg_cap);
}

int seismic_cta_seg_cap(int cluster) { return cluster > 1 ? kSegCapMax : kSegCap; }

int seismic_cta_max_blocks_per_sm(int val_kind, int qcap, int group, int warps, size_t smem) {
    const int th = warps * 32;
    if (val_kind == kF32)
        return wide_table(val_kind, qcap)
                   ? max_blocks_cta_typed<float, uint16_t>(group, th, smem)
                   : max_blocks_cta_typed<float, uint8_t>(group, th, smem);
    if (val_kind == kU8) return max_blocks_cta_typed<uint8_t, uint8_t>(group, th, smem);
    return wide_table(val_kind, qcap) ? max_blocks_cta_typed<uint16_t, uint16_t>(group, th, smem)
                                      : max_blocks_cta_typed<uint16_t, uint8_t>(group, th, smem);
}

cudaError_t launch_seismic_cta(int val_kind, const SeismicLaunch& launch, int warps, int blocks,
                               cudaStream_t s) {
    SeismicLaunch a = launch;
    // A device that cannot place a cluster that large runs smaller ones or one
    // CTA per query (same results): the same grid walks the same queries, and
    // what is left over of it finds none.
    for (; a.cluster > 1; a.cluster /= 2) {
        bool placed = false;
        const cudaError_t e = launch_seismic_cluster(
            val_kind, a, warps, blocks,
            seismic_cta_smem(val_kind, a.fwd.dim, a.qcap, a.k, a.batch_docs, a.seg_cap), placed, s);
        if (e != cudaSuccess || placed) return e;
    }
    if (val_kind == kF32)
        return wide_table(val_kind, a.qcap) ? launch_cta_typed<float, uint16_t>(a, warps, blocks, s)
                                            : launch_cta_typed<float, uint8_t>(a, warps, blocks, s);
    if (val_kind == kU8) return launch_cta_typed<uint8_t, uint8_t>(a, warps, blocks, s);
    return wide_table(val_kind, a.qcap) ? launch_cta_typed<uint16_t, uint16_t>(a, warps, blocks, s)
                                        : launch_cta_typed<uint16_t, uint8_t>(a, warps, blocks, s);
}

cudaError_t launch_order_by_length(const int32_t* indptr, int32_t n, int32_t* order,
                                   cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    order_by_length_kernel<<<1, 1024, 0, s>>>(indptr, n, order);
    return cudaGetLastError();
}

}  // namespace nsp
