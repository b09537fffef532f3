"""Cluster assignment of uint8 codes on the tensor cores against exact integer
dot products (cluster/kmeans_utils.cpp:40-195): every doc of a posting list in
the block of the centroid of largest product, the lowest block on ties. Sizes
at the edges of the kernel's tiles: lists of one doc more than centroids, of
128 and 129 member docs, centroid counts around 16 and 256, a vocabulary below
and above the 1,024 terms of the dense part, and inputs that stay with the
general kernel (evenly spread terms, unsorted rows, more than 1,024 centroids).
"""

import numpy as np
import pytest

import nsparse
import oracle as O
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


def corpus(dim, n, nnz, kind, seed):
    g = np.random.default_rng(seed)
    weight = 1.0 / np.arange(1, dim + 1) if kind != "even" else np.ones(dim)
    weight /= weight.sum()
    rows = []
    for _ in range(n):
        t = np.unique(np.concatenate([[0], g.choice(dim, nnz, p=weight)]))
        rows.append(g.permutation(t) if kind == "shuffled" else t)
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    codes = g.integers(0, 256, int(indptr[-1])).astype(np.float32)
    codes[0], codes[1] = 0.0, 255.0
    return synth.Csr(dim, indptr, np.concatenate(rows).astype(np.uint16), codes)


@pytest.mark.parametrize("dim,n,nnz,beta,kind", [
    (100, 18, 20, 17, "zipf"),
    (1000, 144, 40, 16, "zipf"),
    (1025, 145, 40, 16, "zipf"),
    (3000, 600, 60, 255, "zipf"),
    (3000, 600, 60, 257, "zipf"),
    (5000, 1300, 50, 1024, "zipf"),
    (5000, 1300, 50, 1025, "zipf"),
    (6000, 300, 50, 20, "even"),
    (2000, 300, 50, 20, "shuffled"),
    (40000, 300, 300, 33, "zipf"),
])
def test_assignment_matches_integer_products(tmp_path, dim, n, nnz, beta, kind):
    docs = corpus(dim, n, nnz, kind, seed=dim + n)
    spec = (f"seismic_sq,quantizer=8bit|vmin=0.0|vmax=255.0|"
            f"lambda=0|beta={beta}|alpha=0.1|seed=5")
    idx = nsparse.index_factory(dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    path = str(tmp_path / "a.idx")
    nsparse.write_index(idx, path)
    dense = np.zeros((docs.n, dim), np.int64)
    rows = np.repeat(np.arange(docs.n), np.diff(docs.indptr))
    dense[rows, docs.indices] = docs.values.astype(np.int64)
    product = (dense.astype(np.float64) @ dense.T.astype(np.float64)).astype(np.int64)
    moved = 0
    for lst in O.read_index_file(path)["lists"]:
        off, members = lst["offsets"], lst["docs"]
        if len(members) == 0 or len(off) - 1 == len(members):
            continue
        blocks = [members[off[b]:off[b + 1]] for b in range(len(off) - 1)]
        centroids = np.array([b[0] for b in blocks])  # a block begins with its centroid
        for b, block in enumerate(blocks):
            for d in block[1:]:
                assert np.argmax(product[d, centroids]) == b
                moved += 1
    assert moved > 0
