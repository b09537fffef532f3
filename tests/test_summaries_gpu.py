"""Block summaries of the device build against a sequential restatement
(cluster/inverted_list_clusters.cpp:37-124) at the sizes where the kernels
change: single rows of up to 512 entries, blocks of up to 1,024 and 8,192
distinct terms, larger ones, and a vocabulary whose table exceeds shared
memory; rows that are unsorted or repeat a term; cuts that keep a few pairs,
all of them, or split a level of equal codes."""

import numpy as np
import pytest

import nsparse
import oracle as O
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


def corpus(dim, lengths, order, seed):
    """Rows of the given lengths; every row holds term 0, so its list's one
    block spans them all, and other lists hold every smaller subset."""
    g = np.random.default_rng(seed)
    terms = []
    for n in lengths:
        if order == "repeat":
            t = np.concatenate([[0], g.integers(0, dim, n - 1)])
        else:
            t = np.concatenate([[0], 1 + g.permutation(dim - 1)[:n - 1]])
            t = np.sort(t) if order == "ascending" else g.permutation(t)
        terms.append(t)
    indptr = np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32)
    values = g.lognormal(0.0, 0.8, int(indptr[-1])).astype(np.float32)
    return synth.Csr(dim, indptr, np.concatenate(terms).astype(np.uint16), values)


def summary(docs, values, block, alpha):
    """(terms, values) of a block, by value descending, then term ascending."""
    best = np.full(docs.dim, -1.0, np.float32)
    increments = []
    for d in block:
        for e in range(docs.indptr[d], docs.indptr[d + 1]):
            t, v = docs.indices[e], values[e]
            if best[t] < 0:
                best[t] = max(np.float32(0), v)
                increments.append(best[t])
            elif v > best[t]:
                increments.append(v - best[t])
                best[t] = v
    mass = np.add.accumulate(np.array(increments, np.float32))[-1]
    terms = np.nonzero(best >= 0)[0]
    terms = terms[np.lexsort((terms, -best[terms]))]
    reached = np.add.accumulate(best[terms]) / mass >= np.float32(alpha)
    n = int(np.argmax(reached)) + 1 if reached.any() else len(terms)
    return terms[:n], best[terms[:n]]


@pytest.mark.parametrize("dim,lengths,order,alpha", [
    (600, [1, 31, 32, 33, 511, 512, 513], "ascending", 0.4),
    (600, [1, 255, 256, 257, 511, 512], "ascending", 1.5),
    (3000, [500, 524, 40], "ascending", 0.4),
    (2100, [1023, 1024, 1025, 7], "shuffled", 1.0),
    (9000, [4000, 8191, 8192, 8193, 300], "ascending", 0.05),
    (30522, [257, 256, 255] * 12, "ascending", 0.4),
    (65535, [12000, 30000, 40], "ascending", 0.02),
    (400, [700, 50, 3], "repeat", 0.4),
])
@pytest.mark.parametrize("kind", ["fp32", "sq8", "sq16"])
def test_block_summaries(tmp_path, dim, lengths, order, alpha, kind):
    docs = corpus(dim, lengths, order, seed=dim)
    lists = f"lambda=0|beta=1|alpha={alpha}|seed=3"
    vmin, vmax = 0.0, float(docs.values.max())
    values = docs.values
    if kind == "fp32":
        spec = f"seismic,{lists}"
    else:
        bits = int(kind[2:])
        top = np.float32(2 ** bits - 1)
        scale = top / (np.float32(vmax) - np.float32(vmin))
        values = np.floor(np.clip((docs.values - np.float32(vmin)) * scale, 0, top)
                          + np.float32(0.5)).astype(np.float32)
        spec = f"seismic_sq,quantizer={bits}bit|vmin={vmin!r}|vmax={vmax!r}|{lists}"
    idx = nsparse.index_factory(dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    path = str(tmp_path / "s.idx")
    nsparse.write_index(idx, path)
    known = {}
    checked = 0
    for lst in O.read_index_file(path)["lists"]:
        if len(lst["docs"]) == 0:
            continue
        block = tuple(int(d) for d in lst["docs"])  # one block per list
        if block not in known:
            known[block] = summary(docs, values, block, alpha)
        want_t, want_v = known[block]
        col = np.repeat(np.arange(len(lst["term_ids"])), np.diff(lst["term_ptr"]))
        got_t = lst["term_ids"][col]
        got_v = lst["csc_value"].astype(np.float32)
        order_ = np.argsort(want_t)
        np.testing.assert_array_equal(got_t, want_t[order_])
        np.testing.assert_array_equal(got_v, want_v[order_])
        checked += 1
    assert checked > 0
