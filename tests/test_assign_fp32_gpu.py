"""Cluster assignment of fp32 values (cluster/kmeans_utils.cpp:40-195) against
products rounded and summed in fp32 in the doc's term order: every doc of a
posting list in the block of the centroid of largest sum, the lowest block on
ties, exactly. Sizes at the edges of the kernel: centroid counts around a
multiple of 4 and of 128, more frequent terms than it keeps as dense rows, room
for few rows, sums that do not fit in shared memory, sums that overflow.
"""

import numpy as np
import pytest

import nsparse
import oracle as O
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim,n,nnz,beta,kind", [
    (60, 18, 20, 17, "zipf"),
    (200, 150, 120, 16, "zipf"),
    (200, 150, 120, 33, "shuffled"),
    (3000, 600, 60, 127, "zipf"),
    (3000, 600, 60, 129, "zipf"),
    (900, 1300, 40, 1201, "zipf"),
    (900, 1700, 40, 1400, "zipf"),
    (400, 200, 80, 20, "huge"),
])
def test_assignment_matches_fp32_sums(tmp_path, dim, n, nnz, beta, kind):
    g = np.random.default_rng(dim + n + beta)
    weight = 1.0 / np.arange(1, dim + 1)
    weight /= weight.sum()
    rows = []
    for _ in range(n):
        t = np.unique(np.concatenate([[0], g.choice(dim, nnz, p=weight)]))
        rows.append(g.permutation(t) if kind == "shuffled" else t)
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    values = g.uniform(0.01, 3.0, int(indptr[-1])).astype(np.float32)
    if kind == "huge":
        values *= np.float32(1e19)
    docs = synth.Csr(dim, indptr, np.concatenate(rows).astype(np.uint16), values)
    idx = nsparse.index_factory(dim, f"seismic,lambda=0|beta={beta}|alpha=0.1|seed=5")
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    path = str(tmp_path / "a.idx")
    nsparse.write_index(idx, path)
    dense = np.zeros((dim, docs.n), np.float32)
    dense[docs.indices, np.repeat(np.arange(docs.n), np.diff(docs.indptr))] = docs.values
    moved = 0
    for t, lst in enumerate(O.read_index_file(path)["lists"]):
        off, members = lst["offsets"], lst["docs"]
        if len(members) == 0 or len(off) - 1 == len(members) or (t >= 40 and t % 16):
            continue
        blocks = [members[off[b]:off[b + 1]] for b in range(len(off) - 1)]
        centroids = np.array([b[0] for b in blocks])  # a block begins with its centroid
        for b, block in enumerate(blocks):
            for d in block[1:9]:
                sums = np.zeros(len(centroids), np.float32)
                with np.errstate(over="ignore"):
                    for e in range(docs.indptr[d], docs.indptr[d + 1]):
                        sums += docs.values[e] * dense[docs.indices[e], centroids]
                assert np.argmax(sums) == b
                moved += 1
    assert moved > 0
