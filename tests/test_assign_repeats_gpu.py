"""Cluster assignment of rows that repeat a term (cluster/kmeans_utils.cpp:
40-195): every entry of a doc meets every entry of a centroid that holds its
term, in the doc's order and, for one term, the centroid's. Terms that most
centroids hold, and hold several times, are the ones a dense row or a
side-by-side update would lose. fp32 sums are rounded product by product;
sums of codes are exact integers."""

import numpy as np
import pytest

import nsparse
import oracle as O
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


def corpus(dim, n, nnz, seed):
    g = np.random.default_rng(seed)
    weight = 1.0 / np.arange(1, dim + 1)
    rows = [g.choice(dim, nnz, p=weight / weight.sum()) for _ in range(n)]
    indptr = np.arange(0, n * nnz + 1, nnz, dtype=np.int32)
    codes = g.integers(1, 256, n * nnz).astype(np.float32)
    codes[0], codes[1] = 0.0, 255.0
    return synth.Csr(dim, indptr, np.concatenate(rows).astype(np.uint16), codes)


def similarity(docs, values, d, centroids, held):
    """Sums of doc d with every centroid, in the reference's order. `held[c]`:
    term -> the centroid's values of it, in row order."""
    out = np.zeros(len(centroids), values.dtype)
    for e in range(docs.indptr[d], docs.indptr[d + 1]):
        for i, c in enumerate(centroids):
            for w in held[c].get(int(docs.indices[e]), ()):
                out[i] += values[e] * w
    return out


@pytest.mark.parametrize("kind", ["fp32", "sq8", "sq16"])
@pytest.mark.parametrize("dim,n,nnz,beta", [
    (12, 60, 40, 7),      # a term several times within 32 entries
    (300, 120, 45, 33),   # runs of more than 32 entries
    (40, 50, 150, 16),    # rows of more than 128 entries
    (300, 400, 20, 150),  # runs of more than 128 entries
])
def test_repeated_terms(tmp_path, kind, dim, n, nnz, beta):
    docs = corpus(dim, n, nnz, seed=dim + nnz)
    lists = f"lambda=0|beta={beta}|alpha=0.1|seed=5"
    spec = f"seismic,{lists}" if kind == "fp32" else \
        f"seismic_sq,quantizer={kind[2:]}bit|vmin=0.0|vmax={2 ** int(kind[2:]) - 1}.0|{lists}"
    values = docs.values if kind == "fp32" else docs.values.astype(np.int64)
    idx = nsparse.index_factory(dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    path = str(tmp_path / "r.idx")
    nsparse.write_index(idx, path)
    held = {}
    for c in range(docs.n):
        h = held[c] = {}
        for e in range(docs.indptr[c], docs.indptr[c + 1]):
            h.setdefault(int(docs.indices[e]), []).append(values[e])
    moved = 0
    for t, lst in enumerate(O.read_index_file(path)["lists"]):
        off, members = lst["offsets"], lst["docs"]
        if t > 3 and t % 17:
            continue
        if len(members) == 0 or len(off) - 1 == len(members):
            continue
        blocks = [members[off[b]:off[b + 1]] for b in range(len(off) - 1)]
        centroids = [int(b[0]) for b in blocks]  # a block begins with its centroid
        for b, block in enumerate(blocks):
            for d in block[1:3]:
                assert np.argmax(similarity(docs, values, int(d), centroids, held)) == b
                moved += 1
    assert moved > 0
