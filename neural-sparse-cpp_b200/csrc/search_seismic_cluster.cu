// SEISMIC / SEISMIC-SQ search on sm_100a, a thread-block cluster of 2-16 CTAs
// per query: launches of so few queries that one CTA each would leave the GPU
// idle (a lone query, small batches). The results are those of the kernel of
// one CTA per query (search_seismic_cta.cu describes the search); here every
// phase is spread to shorten the query:
//
//   1. every CTA keeps the query's table and ranks its cut;
//   2. summary scores: a CTA takes a whole list at a time, its hit terms' runs
//      staged in shared memory and applied in ascending term order;
//   3. rank 0 sorts the first list's blocks with all its warps;
//   4. the first list is one walk; all later lists whose summaries are known
//      are one more, their passing blocks one after another in list and block
//      order. A block that fails the pruning test now fails at its turn too,
//      and the walk tests each block again at its turn, so batches may span
//      lists: a lone query takes a few batches instead of one or more per
//      list (a batch costs three cluster barriers and its longest row);
//   5. rank 0 gathers a batch with all its threads; every CTA copies the
//      batch's segments, looks up and scores its share of the docs (rows are
//      handed to L2 whole while they are listed) and writes doc ids, lengths,
//      segments and scores into rank 0's arrays; rank 0's first warp walks.
//
// Control words: rank 0 writes a batch's size into every CTA before a cluster
// barrier (kNextLists: summaries of the next lists; kQueryDone), so all CTAs
// pass the same barriers in the same order and nothing spins. Between two
// writes of one word lies at least one barrier that its readers arrive at
// after their read, for queries without lists too.
//
// Measured, one query per call (whole calls): fp32, 100,000 docs 431 -> 275 us,
// SQ, 3M docs 689 -> 385 us, against the same cluster with rank 0 doing 2-4
// and the others only scoring. A query's share of the row scoring (45-110 us)
// runs at the rate its SMs reach in a full launch, so 16 CTAs are taken where
// at most a few queries run; what is left is the walk (55-70 us) and the
// barriers around each batch.
#include <cooperative_groups.h>

#include "seismic_cta.cuh"

namespace nsp {
namespace {

namespace cg = cooperative_groups;

constexpr int kNextLists = -2;
constexpr int kQueryDone = -1;
constexpr int kGroup = 8;      // lanes per scored doc
constexpr int kApplyWarps = 8;  // warps that apply a list's runs
constexpr int kHitWindow = 256;  // query terms looked up in a list at once

__device__ __forceinline__ void cluster_sync() { cg::this_cluster().sync(); }

// The leader writes a control word into every other CTA of its cluster.
__device__ __forceinline__ void push_to_cluster(int32_t* field, int32_t v) {
    cg::cluster_group cl = cg::this_cluster();
    for (unsigned r = 1; r < cl.num_blocks(); ++r) *cl.map_shared_rank(field, r) = v;
}

// A hit term of a list: its summary entries, where they are staged, and the
// query's value.
struct Hit {
    int64_t r0;
    int32_t len;
    float q;
    int32_t at;
    int32_t pad;
};

struct Shared {
    int32_t scan[2][32];  // per-warp sums
    int32_t taken_docs, next, cut_at;
    int32_t hits;
    Cursor cur;
};

// Exclusive prefix of v over the CTA and its total.
__device__ __forceinline__ int block_scan(int v, int32_t* sums, int lane, int warp, int nwarps,
                                          int& total) {
    int incl = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const int y = __shfl_up_sync(kFull, incl, o);
        if (lane >= o) incl += y;
    }
    __syncthreads();
    if (lane == 31) sums[warp] = incl;
    __syncthreads();
    int before = incl - v;
    total = 0;
    for (int w = 0; w < nwarps; ++w) {
        const int x = sums[w];
        before += w < warp ? x : 0;
        total += x;
    }
    return before;
}

// Summary scores of list t into out[0..nb) (global), by the whole CTA
// (inverted_list_clusters.cpp:295-331): the hit terms are looked up a thread
// each, their runs copied to shared memory a warp each -- so a list costs a
// few memory round trips, not some per term -- and then applied in ascending
// term order, a thread per entry (a term's entries are of distinct blocks)
// and a barrier between terms. `mem`: `room` bytes of shared memory.
template <typename V>
__device__ void list_summaries_cta(const SeismicLaunch& a, int t, int nb, const uint16_t* qterm,
                                   const V* qraw, int qn, float* out, unsigned char* mem,
                                   size_t room, Shared& sh, int tid, int lane, int warp,
                                   int nwarps, uint32_t& bytes) {
    const int NT = blockDim.x;
    const int window = min(kHitWindow, NT);
    Hit* hits = reinterpret_cast<Hit*>(mem);
    mem += kHitWindow * sizeof(Hit);
    room -= kHitWindow * sizeof(Hit);
    // sums in shared memory where half the room holds them, else in `out`
    const bool in_smem = static_cast<size_t>(nb) * 4 <= room / 2;
    float* bs = in_smem ? reinterpret_cast<float*>(mem) : out;
    if (in_smem) {
        mem += a16(static_cast<size_t>(nb) * 4);
        room -= a16(static_cast<size_t>(nb) * 4);
    }
    // staged entries: values, then block ids
    const int cap = static_cast<int>(room / (sizeof(V) + 2)) & ~15;
    V* eval = reinterpret_cast<V*>(mem);
    uint16_t* eblk = reinterpret_cast<uint16_t*>(mem + static_cast<size_t>(cap) * sizeof(V));
    // uint8 codes: integer sums below 2^24, exact in any order
    const bool ints = std::is_same<V, uint8_t>::value && static_cast<long long>(qn) * 65025ll < (1ll << 24);
    int* is = reinterpret_cast<int*>(bs);
    // (+0.0f and 0 are the same bits)
    for (int b = tid; b < nb; b += NT) bs[b] = 0.0f;
    const uint2* meta = a.ix.lmeta + static_cast<size_t>(t) * a.ix.words;
    const int64_t colbase = a.ix.ltp[t];
    const V* sv = static_cast<const V*>(a.ix.sval);
    for (int i0 = 0; i0 < qn; i0 += window) {
        const int i = i0 + tid;
        bool hit = false;
        Hit h{0, 0, 0.0f, 0, 0};
        if (tid < window && i < qn && qterm[i] < static_cast<uint32_t>(a.fwd.dim)) {
            const uint32_t term = qterm[i];
            const uint2 m = __ldg(meta + (term >> 5));
            const uint32_t bit = 1u << (term & 31);
            if (m.x & bit) {
                const int64_t col = colbase + m.y + __popc(m.x & (bit - 1));
                h.r0 = __ldg(a.ix.srun + col);
                h.len = static_cast<int32_t>(__ldg(a.ix.srun + col + 1) - h.r0);
                h.q = ValT<V>::f(qraw[i]);
                hit = true;
            }
        }
        int nh = 0, entries = 0;
        const int rank = block_scan(hit ? 1 : 0, sh.scan[0], lane, warp, nwarps, nh);
        h.at = block_scan(hit ? h.len : 0, sh.scan[1], lane, warp, nwarps, entries);
        if (hit) hits[rank] = h;
        __syncthreads();
        if (tid == 0)
            bytes += 8u * static_cast<uint32_t>(min(window, qn - i0)) + 16u * nh +
                     static_cast<uint32_t>(entries) * (2 + static_cast<int>(sizeof(V)));
        if (ints) {  // a warp per term
            for (int j = warp; j < nh; j += nwarps) {
                const Hit x = hits[j];
                const int q = static_cast<int>(x.q);
#pragma unroll 4
                for (int e = lane; e < x.len; e += 32)
                    atomicAdd(&is[__ldg(a.ix.sblk + x.r0 + e)],
                              q * static_cast<int>(__ldg(sv + x.r0 + e)));
            }
            __syncthreads();
            continue;
        }
        // as many terms at a time as their entries fit; a longer run is
        // applied from global memory
        for (int h0 = 0; h0 < nh;) {
            const int base = hits[h0].at;
            int h1 = h0;
            while (h1 < nh && hits[h1].at + hits[h1].len - base <= cap) ++h1;
            for (int j = h0 + warp; j < h1; j += nwarps) {
                const Hit x = hits[j];
#pragma unroll 4
                for (int e = lane; e < x.len; e += 32) {
                    eblk[x.at - base + e] = __ldg(a.ix.sblk + x.r0 + e);
                    eval[x.at - base + e] = __ldg(sv + x.r0 + e);
                }
            }
            __syncthreads();
            // runs are a few hundred entries: the first warps apply them, with
            // a barrier of their own
            const int aw = min(kApplyWarps, nwarps);
            if (warp < aw) {
                for (int j = h0; j < h1; ++j) {
                    const int at = hits[j].at - base, len = hits[j].len;
                    const float q = hits[j].q;
                    for (int e = tid; e < len; e += aw * 32) {
                        const int b = eblk[at + e];
                        bs[b] = __fadd_rn(bs[b], __fmul_rn(q, ValT<V>::f(eval[at + e])));
                    }
                    asm volatile("bar.sync 1, %0;" ::"r"(aw * 32) : "memory");
                }
            }
            __syncthreads();
            if (h1 == h0) {
                const Hit x = hits[h0];
                for (int e = tid; e < x.len; e += NT) {
                    const int b = __ldg(a.ix.sblk + x.r0 + e);
                    bs[b] = __fadd_rn(bs[b], __fmul_rn(x.q, ValT<V>::f(__ldg(sv + x.r0 + e))));
                }
                __syncthreads();
                ++h1;
            }
            h0 = h1;
        }
    }
    __syncthreads();
    if (ints) {
        for (int b = tid; b < nb; b += NT) out[b] = static_cast<float>(is[b]);
    } else if (in_smem) {
        for (int b = tid; b < nb; b += NT) out[b] = bs[b];
    }
    __syncthreads();
}

// All of the leader's threads: fills the next batch with segments of blocks
// that pass the pruning test against the current heap, from position cur.o of
// `vis` (list slot << 16 | block) on, as `gather` does by one warp. Returns
// the number of segments; `total` receives the number of docs.
__device__ int gather_cta(const SeismicLaunch& a, Shared& sh, bool first, const uint32_t* vis,
                          int nv, const float* bscore, int maxb, const int64_t* slot_lb0, bool full,
                          float hmin, Seg* segs, int batch, int seg_cap, int& total, int tid,
                          int lane, int warp, int nwarps) {
    Cursor& c = sh.cur;
    const int NT = blockDim.x;
    int room = batch, nseg = 0;
    total = 0;
    int o = c.o;
    bool split = c.split, dead = c.dead;
    if (split) {
        const int take = min(room, c.split_left);
        const int64_t d0 = c.split_d;
        const float bs = c.split_bs;
        split = take < c.split_left;
        __syncthreads();
        if (tid == 0) {
            segs[0] = Seg{d0, take, 0, bs, 0, 0u, take};
            c.split_d = d0 + take;
            c.split_left -= take;
            c.split = split;
        }
        nseg = 1;
        total = take;
        room -= take;
    }
    while (!split && !dead && room > 0 && nseg < seg_cap && o < nv) {
        const int p = o + tid;
        const bool in = p < nv;
        int64_t d0 = 0, d1 = 0;
        float bs = 0.0f;
        if (in) {
            const uint32_t x = vis[p];
            const int slot = static_cast<int>(x >> 16), blk = static_cast<int>(x & 0xffffu);
            bs = __ldcg(bscore + static_cast<size_t>(slot) * maxb + blk);
            const int64_t g = slot_lb0[slot] + blk;
            d0 = __ldg(a.ix.bdp + g);
            d1 = __ldg(a.ix.bdp + g + 1);
        }
        const bool pass = in && !(full && __fmul_rn(bs, a.heap_factor) < hmin);
        // the first list ends at its first failing block
        const int window = min(NT, nv - o);
        int lim = window;
        if (first) {
            if (tid == 0) sh.cut_at = window;
            __syncthreads();
            const unsigned fm = __ballot_sync(kFull, in && !pass);
            if (lane == 0 && fm) atomicMin(&sh.cut_at, warp * 32 + __ffs(fm) - 1);
            __syncthreads();
            lim = sh.cut_at;
        }
        const bool cand = pass && tid < lim;
        const int sz = cand ? static_cast<int>(d1 - d0) : 0;
        int docs = 0, cands = 0;
        const int excl = block_scan(sz, sh.scan[0], lane, warp, nwarps, docs);
        const int r = block_scan(cand ? 1 : 0, sh.scan[1], lane, warp, nwarps, cands);
        const bool take = cand && excl < room && nseg + r < seg_cap;
        if (tid == 0) {
            sh.taken_docs = 0;
            sh.next = -1;
        }
        const int nt = __syncthreads_count(take);  // a prefix of the candidates
        if (take) {
            const int cnt = min(sz, room - excl);
            segs[nseg + r] = Seg{d0, cnt, total + excl, bs, 1, 0u, cnt};
            if (r == nt - 1) {
                sh.taken_docs = excl + cnt;
                if (cnt < sz) {
                    c.split = true;
                    c.split_d = d0 + cnt;
                    c.split_left = sz - cnt;
                    c.split_bs = bs;
                }
            }
        } else if (cand && r == nt) {
            sh.next = tid;
        }
        __syncthreads();
        split = c.split;
        if (sh.next >= 0) {
            o += sh.next;
        } else {
            o += lim;
            if (lim < window && !split) dead = true;
        }
        nseg += nt;
        total += sh.taken_docs;
        room -= sh.taken_docs;
        __syncthreads();
    }
    __syncthreads();
    if (tid == 0) {
        c.o = o;
        c.dead = dead;
    }
    __syncthreads();
    return nseg;
}

// This CTA's share of a batch: candidates [i0, i1), looked up from the
// segments (copied into `segs` before), scored, and written to the leader's
// arrays.
template <typename V, typename TE, bool kMask>
__device__ void score_share(const SeismicLaunch& a, const uint64_t* sel, Ctl* ctl, const TE* tbl,
                            const float* qv, int32_t* cdoc, uint32_t* coff, uint32_t* clen,
                            float* csc, uint16_t* cseg, const Seg* segs, int nseg, int i0, int i1,
                            int tid, int lane) {
    cg::cluster_group cl = cg::this_cluster();
    const int NT = blockDim.x;
    for (int i = i0 + tid; i < i1; i += NT) {
        int lo = 0, hi = nseg - 1;
        while (lo < hi) {
            const int mid = (lo + hi + 1) >> 1;
            if (segs[mid].cand0 <= i) lo = mid;
            else hi = mid - 1;
        }
        const int64_t pj = segs[lo].d0 + (i - segs[lo].cand0);
        const int32_t d = __ldg(a.ix.docs + pj);
        uint2 ri = a.ix.drow != nullptr ? __ldg(a.ix.drow + pj) : __ldg(a.fwd.rowinfo + d);
        bool member = true;
        if (sel != nullptr) member = (__ldg(sel + (d >> 6)) >> (d & 63)) & 1ull;
        const int j = i - i0;
        if (!member) ri = make_uint2(0u, 0u);
        else prefetch_row<V>(a.fwd.idx, static_cast<const V*>(a.fwd.val), ri.x, ri.y, 0);
        cdoc[j] = member ? d : -1;
        coff[j] = ri.x;
        clen[j] = ri.y;
        cseg[j] = static_cast<uint16_t>(lo);
    }
    if (tid == 0) ctl->next = 0;
    __syncthreads();
    score_batch<V, TE, kMask, kGroup, false>(a.fwd, ctl, tbl, qv, coff, clen, csc, i1 - i0, lane);
    __syncthreads();
    if (cl.block_rank() == 0) return;  // its share starts at candidate 0
    int32_t* rdoc = cl.map_shared_rank(cdoc, 0);
    uint32_t* rlen = cl.map_shared_rank(clen, 0);
    float* rsc = cl.map_shared_rank(csc, 0);
    uint16_t* rseg = cl.map_shared_rank(cseg, 0);
    for (int i = i0 + tid; i < i1; i += NT) {
        const int j = i - i0;
        rdoc[i] = cdoc[j];
        rlen[i] = clen[j];
        rsc[i] = csc[j];
        rseg[i] = cseg[j];
    }
}

template <typename V, typename TE>
__global__ void __launch_bounds__(1024, 1) seismic_cluster_kernel(SeismicLaunch a) {
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ Shared sh;
    __shared__ int64_t slot_lb0[32];
    __shared__ int32_t slot_nb[32];
    constexpr bool kRank = kRankTable<V, TE>;
    constexpr bool kF32 = std::is_same<V, float>::value;
    constexpr int vsz = static_cast<int>(sizeof(V));
    cg::cluster_group cl = cg::this_cluster();
    const int rank = static_cast<int>(cl.block_rank()), ncl = static_cast<int>(cl.num_blocks());
    const int tid = threadIdx.x;
    const int lane = tid & 31;
    const int warp = tid >> 5;
    const int NT = blockDim.x;
    const int nwarps = NT >> 5;
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
    uint16_t* cseg = reinterpret_cast<uint16_t*>(smem + L.cseg);
    const size_t room = L.wsum - L.cdoc;  // the batch arrays, free between batches

    // Scratch of the cluster: the leader's block scores (a slot per list of a
    // group), and in the next CTA's share the visiting order.
    const int maxb = a.ix.max_blocks;
    const unsigned lead = blockIdx.x - static_cast<unsigned>(rank);
    float* bscore = a.bscore + static_cast<size_t>(lead) * nwarps * maxb;
    uint32_t* vis = reinterpret_cast<uint32_t*>(bscore + static_cast<size_t>(nwarps) * maxb);
    uint16_t* order = a.order + static_cast<size_t>(lead) * a.order_stride;
    unsigned long long* keys_g =
        a.sortkeys != nullptr ? a.sortkeys + static_cast<size_t>(lead) * a.sort_stride : nullptr;
    const unsigned cid = blockIdx.x / static_cast<unsigned>(ncl);
    const unsigned slots = gridDim.x / static_cast<unsigned>(ncl);

    for (int i = tid; i <= dim; i += NT) tbl[i] = 0;
    if (tid == 0) qv[0] = 0.0f;
    // every CTA of the cluster runs before any touches another's memory
    __syncthreads();
    cluster_sync();

    for (int iter = 0;; ++iter) {
        if (rank == 0 && tid == 0) {
            int q;
            if (a.work_counter != nullptr) {
                q = atomicAdd(a.work_counter, 1);
                if (a.qorder != nullptr && q < a.q.n) q = a.qorder[q];
            } else {
                q = a.first_query + static_cast<int>(cid) + iter * static_cast<int>(slots);
            }
            ctl->q = q;
            ctl->nheap = 0;  // the query's heap starts empty
            push_to_cluster(&ctl->q, q);
        }
        __syncthreads();
        cluster_sync();
        const int q = ctl->q;
        if (q >= a.q.n) break;
        const uint64_t* sel = a.sel_q != nullptr ? a.sel_q[q] : a.sel_bits;
        // 1. scatter the query
        const int32_t qs = a.q.indptr[q];
        int qn = a.q.indptr[q + 1] - qs;
        // the caller's max_nnz was wrong, or the row lies past the query
        // arrays: padding, and the error is reported
        if (qn > a.qcap || qn < 0 || qs < 0 || (a.nnz_cap >= 0 && qs + qn > a.nnz_cap)) {
            if (rank == 0 && tid == 0 && a.err != nullptr) atomicExch(a.err, 3);
            qn = 0;
        }
        bool bad = false;
        for (int i = tid; i < qn; i += NT) {
            const uint32_t t = a.q.idx[qs + i];
            const V v = static_cast<const V*>(a.q.val)[qs + i];
            qterm[i] = static_cast<uint16_t>(t);
            qraw[i] = v;
            if (t < static_cast<uint32_t>(dim)) {
                if constexpr (kRank) tbl[t] = static_cast<TE>(i + 1);
                else tbl[t] = static_cast<TE>(v);
            }
            if constexpr (kF32) {
                qv[i + 1] = v;
                bad |= !isfinite(v);
            } else if constexpr (kRank) {
                reinterpret_cast<uint32_t*>(qv)[i + 1] = v;
            }
        }
        const bool nonfinite = __syncthreads_or(bad) != 0;
        // 2. query cut (utils/vector_process.h:18-30)
        int ncut;
        if (a.cut >= qn) {
            ncut = qn;
            for (int i = tid; i < qn; i += NT) cuts[i] = qterm[i];
        } else {
            ncut = a.cut;
            query_cut<V>(cuts, qraw, qn, ncut, reinterpret_cast<uint32_t*>(smem + L.cdoc),
                         static_cast<int>(room / 4), tid);
            for (int i = tid; i < ncut; i += NT) cuts[i] = qterm[cuts[i]];
        }
        __syncthreads();

        int n = 0;  // heap size (the leader's warp 0)
        bool first = true;
        uint32_t blocks_visited = 0, bytes = 0, lists = 0;
        int32_t docs_scored = 0, row_bytes = 0;
        for (int c0 = 0; c0 < ncut; c0 += nwarps) {
            // 3. summary scores of the next lists, a CTA per list: the leader
            // takes the group's first, the others the rest
            const int ng = min(nwarps, ncut - c0);
            if (tid < ng) {
                const int t = cuts[c0 + tid];
                int64_t lb0 = 0;
                int nb = -1;  // no such list (seismic_index.cpp:254-256)
                if (t < a.ix.n_lists) {
                    lb0 = a.ix.lbp[t];
                    nb = static_cast<int>(a.ix.lbp[t + 1] - lb0);
                }
                slot_lb0[tid] = lb0;
                slot_nb[tid] = nb;
            }
            __syncthreads();
            for (int s = 0; s < ng; ++s)
                if (slot_nb[s] > 0 && (s == 0 ? 0 : 1 + (s - 1) % (ncl - 1)) == rank)
                    list_summaries_cta<V>(a, cuts[c0 + s], slot_nb[s], qterm, qraw, qn,
                                          bscore + static_cast<size_t>(s) * maxb, smem + L.cdoc,
                                          room, sh, tid, lane, warp, nwarps, bytes);
            __syncthreads();
            cluster_sync();
            // 4.-5. the group's first list if it is the query's first, then the
            // rest as one
            if (rank == 0) {
                int s = 0;
                while (s < ng) {
                    int nv = 0;
                    if (first) {
                        const int nb = slot_nb[s];
                        if (nb < 0) {
                            ++s;
                            continue;
                        }
                        if (nb == 0) {
                            first = false;
                            ++s;
                            continue;
                        }
                        ++lists;
                        const size_t pairs = static_cast<size_t>(nb) * sizeof(ranking::Blk);
                        const size_t sort_room = L.sq - L.cdoc;
                        ranking::Blk* items = reinterpret_cast<ranking::Blk*>(
                            pairs <= sort_room ? reinterpret_cast<unsigned long long*>(cdoc) : keys_g);
                        if (items == nullptr) {  // the host sizes sortkeys; never taken
                            if (tid == 0) atomicExch(a.err, 2);
                            break;
                        }
                        uint16_t* stops = pairs + static_cast<size_t>(nb) * 2 <= sort_room
                                              ? reinterpret_cast<uint16_t*>(smem + L.cdoc + pairs)
                                              : order;
                        sort_blocks(bscore + static_cast<size_t>(s) * maxb, nb, items, stops, order,
                                    reinterpret_cast<uint32_t*>(smem + L.sq), tid, lane, warp,
                                    nwarps);
                        for (int i = tid; i < nb; i += NT)
                            vis[i] = (static_cast<uint32_t>(s) << 16) | order[i];
                        nv = nb;
                    } else {
                        // blocks of the lists from s on that pass the test now,
                        // a warp per list
                        const bool full = ctl->nheap == a.k;
                        const float hmin = full ? hs[0] : 0.0f;
                        const int nb = s + warp < ng ? slot_nb[s + warp] : 0;
                        const float* bs = bscore + static_cast<size_t>(s + warp) * maxb;
                        auto passes = [&](int i) {
                            return i < nb && !(full && __fmul_rn(__ldcg(bs + i), a.heap_factor) < hmin);
                        };
                        int mine = 0;
                        for (int i = 0; i < nb; i += 32)
                            mine += __popc(__ballot_sync(kFull, passes(i + lane)));
                        int at = block_scan(lane == 0 ? mine : 0, sh.scan[0], lane, warp, nwarps, nv);
                        at = __shfl_sync(kFull, at, 0);
                        for (int i = 0; i < nb; i += 32) {
                            const bool ok = passes(i + lane);
                            const unsigned m = __ballot_sync(kFull, ok);
                            if (ok)
                                vis[at + __popc(m & ((1u << lane) - 1u))] =
                                    (static_cast<uint32_t>(s + warp) << 16) |
                                    static_cast<uint32_t>(i + lane);
                            at += __popc(m);
                        }
                        for (int u = s; u < ng; ++u) lists += slot_nb[u] > 0 ? 1 : 0;
                    }
                    if (tid == 0) sh.cur = Cursor{};
                    __syncthreads();
                    for (;;) {
                        int total = 0;
                        const int nh = ctl->nheap;
                        const float hmin0 = nh == a.k ? hs[0] : 0.0f;
                        const int nseg = gather_cta(a, sh, first, vis, nv, bscore, maxb, slot_lb0,
                                                    nh == a.k, hmin0, segs, batch, a.seg_cap, total,
                                                    tid, lane, warp, nwarps);
                        if (nseg == 0) break;
                        if (total > 0) {
                            if (tid == 0) {
                                ctl->nseg = nseg;
                                push_to_cluster(&ctl->nseg, nseg);
                                push_to_cluster(&ctl->total, total);
                            }
                            __syncthreads();
                            cluster_sync();
                            // (the others copy the segments)
                            const int per = (total + ncl - 1) / ncl;
                            const int i1 = min(total, per);
                            if (kF32 && nonfinite)
                                score_share<V, TE, true>(a, sel, ctl, tbl, qv, cdoc, coff, clen, csc,
                                                         cseg, segs, nseg, 0, i1, tid, lane);
                            else
                                score_share<V, TE, false>(a, sel, ctl, tbl, qv, cdoc, coff, clen,
                                                          csc, cseg, segs, nseg, 0, i1, tid, lane);
                            cluster_sync();
                        }
                        // segments take the best score of docs above the heap
                        // minimum as it stood at the gather
                        for (int i = tid; i < total; i += NT)
                            if (cdoc[i] >= 0 && (nh < a.k || !(csc[i] <= hmin0)))
                                atomicMax(&segs[cseg[i]].best, score_key(csc[i]));
                        __syncthreads();
                        if (warp == 0) {
                            walk_batch<V, true>(a, segs, nseg, total, cdoc, clen, csc, hs, hid, n, first,
                                          sh.cur.dead, sh.cur.split, nullptr, 0u, lane,
                                          blocks_visited, bytes, docs_scored, row_bytes);
                            if (lane == 0) ctl->nheap = n;
                        }
                        __syncthreads();
                        // the work counters: docs of segments the walk took
                        for (int i = tid; i < total; i += NT) {
                            if (cdoc[i] >= 0 && segs[cseg[i]].docs >= 0) {
                                ++docs_scored;
                                row_bytes += 8 + static_cast<int32_t>(clen[i]) * (2 + vsz);
                            }
                        }
                        __syncthreads();
                    }
                    if (first) {
                        first = false;
                        ++s;
                    } else {
                        s = ng;
                    }
                }
                if (tid == 0)
                    push_to_cluster(&ctl->total, c0 + nwarps < ncut ? kNextLists : kQueryDone);
                __syncthreads();
                cluster_sync();
            } else {
                for (;;) {
                    cluster_sync();
                    const int total = ctl->total;
                    if (total < 0) break;
                    const int nseg = ctl->nseg;
                    const uint4* src = reinterpret_cast<const uint4*>(cl.map_shared_rank(segs, 0));
                    uint4* dst = reinterpret_cast<uint4*>(segs);
                    const int pieces = nseg * static_cast<int>(sizeof(Seg) / 16);
                    for (int i = tid; i < pieces; i += NT) dst[i] = src[i];
                    __syncthreads();
                    const int per = (total + ncl - 1) / ncl;
                    const int i0 = min(total, rank * per), i1 = min(total, i0 + per);
                    if (kF32 && nonfinite)
                        score_share<V, TE, true>(a, sel, ctl, tbl, qv, cdoc, coff, clen, csc, cseg,
                                                 segs, nseg, i0, i1, tid, lane);
                    else
                        score_share<V, TE, false>(a, sel, ctl, tbl, qv, cdoc, coff, clen, csc, cseg,
                                                  segs, nseg, i0, i1, tid, lane);
                    cluster_sync();
                }
            }
        }
        // A query of no lists passed none of the barriers above: without this
        // one the leader could write the next query's number over the one
        // that another CTA's threads are still about to read.
        if (ncut == 0) cluster_sync();
        // results, padded with (-1.0, -1); SQ scores decoded
        // (seismic_scalar_quantized_index.cpp:345-355)
        if (rank == 0 && warp == 0) {
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
            // summary bytes are thread 0's; the block counts and walked bytes
            // are the same on every lane of the leader's warp 0
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                row_bytes += __shfl_xor_sync(kFull, row_bytes, o);
                docs_scored += __shfl_xor_sync(kFull, docs_scored, o);
            }
            if (lane == 0) {
                if (rank == 0 && warp == 0) {
                    atomicAdd(a.stats + kStatBlocksVisited,
                              static_cast<unsigned long long>(blocks_visited));
                    atomicAdd(a.stats + kStatListsProbed, static_cast<unsigned long long>(lists));
                }
                if (warp == 0)
                    atomicAdd(a.stats + kStatBytes, static_cast<unsigned long long>(bytes));
                if (rank == 0) {
                    // a warp's net counts can be negative: widened with their
                    // sign, they add up modulo 2^64 to the exact total
                    atomicAdd(a.stats + kStatDocsScored,
                              static_cast<unsigned long long>(static_cast<long long>(docs_scored)));
                    const auto rb =
                        static_cast<unsigned long long>(static_cast<long long>(row_bytes));
                    atomicAdd(a.stats + kStatBytes, rb);
                    atomicAdd(a.stats + kStatRowBytes, rb);
                }
            }
        }
        // restore the all-zero table for the next query
        __syncthreads();
        for (int i = tid; i < qn; i += NT) {
            const uint32_t t = qterm[i];
            if (t < static_cast<uint32_t>(dim)) tbl[t] = 0;
        }
    }
}

template <typename V, typename TE>
cudaError_t launch_typed(const SeismicLaunch& a, int warps, int blocks, size_t smem, bool& placed,
                         cudaStream_t s) {
    auto* f = seismic_cluster_kernel<V, TE>;
    placed = false;
    cudaError_t e = allow_opt_in_smem(f);
    if (e != cudaSuccess) return e;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(static_cast<unsigned>(blocks));
    cfg.blockDim = dim3(static_cast<unsigned>(warps * 32));
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = static_cast<unsigned>(a.cluster);
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    static thread_local Memo<LaunchKey, bool, 16> known;  // whether it can be placed
    LaunchKey k;
    k.f = reinterpret_cast<const void*>(f);
    k.threads = warps * 32;
    k.cluster = a.cluster;
    k.smem = smem;
    e = cudaGetDevice(&k.dev);
    if (e != cudaSuccess) return e;
    const bool* fits = known.find(k);
    if (fits == nullptr) {
        bool ok = true;
        if (a.cluster > 8)  // past the portable size
            ok = cudaFuncSetAttribute(f, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) ==
                 cudaSuccess;
        int clusters = 0;
        ok = ok && cudaOccupancyMaxActiveClusters(&clusters, f, &cfg) == cudaSuccess && clusters > 0;
        if (!ok) (void)cudaGetLastError();
        known.put(k, ok);
        fits = known.find(k);
    }
    if (!*fits) return cudaSuccess;
    placed = true;
    return cudaLaunchKernelEx(&cfg, f, a);
}

}  // namespace

cudaError_t launch_seismic_cluster(int val_kind, const SeismicLaunch& a, int warps, int blocks,
                                   size_t smem, bool& placed, cudaStream_t s) {
    if (val_kind == kF32)
        return a.qcap > 255 ? launch_typed<float, uint16_t>(a, warps, blocks, smem, placed, s)
                            : launch_typed<float, uint8_t>(a, warps, blocks, smem, placed, s);
    if (val_kind == kU8) return launch_typed<uint8_t, uint8_t>(a, warps, blocks, smem, placed, s);
    return a.qcap > 255 ? launch_typed<uint16_t, uint16_t>(a, warps, blocks, smem, placed, s)
                        : launch_typed<uint16_t, uint8_t>(a, warps, blocks, smem, placed, s);
}

}  // namespace nsp
