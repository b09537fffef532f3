"""Cluster assignment of uint8 codes where a dot product passes 2^31: rows that
share more than 33,025 terms at the largest codes. Every doc goes to the
centroid of the largest exact product, whether the frequent terms hold most of
the products (the tensor-core path otherwise) or not."""

import numpy as np
import pytest

import nsparse
import oracle as O
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dim", [40000, 60000])
@pytest.mark.parametrize("n_long,n_short", [(9, 12), (9, 600)])
def test_products_past_31_bits(tmp_path, dim, n_long, n_short):
    g = np.random.default_rng(dim + n_short)
    rows = [np.sort(g.permutation(38000)[:36000]) for _ in range(n_long)]
    rows += [np.sort(g.permutation(700)[:300]) for _ in range(n_short)]
    rows = [rows[i] for i in g.permutation(len(rows))]
    rows = [np.union1d([0], r) for r in rows]  # term 0's list holds every doc
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    codes = g.integers(253, 256, int(indptr[-1])).astype(np.float32)
    codes[0], codes[1] = 0.0, 255.0
    docs = synth.Csr(dim, indptr, np.concatenate(rows).astype(np.uint16), codes)
    spec = f"seismic_sq,quantizer=8bit|vmin=0.0|vmax=255.0|lambda=0|beta={len(rows) // 3}|" \
        "alpha=0.01|seed=5"
    idx = nsparse.index_factory(dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    path = str(tmp_path / "l.idx")
    nsparse.write_index(idx, path)
    dense = np.zeros((docs.n, dim))
    dense[np.repeat(np.arange(docs.n), np.diff(indptr)), docs.indices] = codes
    product = dense @ dense.T  # integers below 2^53
    assert product.max() > 2.0 ** 31
    lst = O.read_index_file(path)["lists"][0]
    off, members = lst["offsets"], lst["docs"]
    blocks = [members[off[b]:off[b + 1]] for b in range(len(off) - 1)]
    centroids = np.array([b[0] for b in blocks])  # a block begins with its centroid
    passed = 0
    for b, block in enumerate(blocks):
        for d in block[1:]:
            assert np.argmax(product[d, centroids]) == b
            passed += product[d, centroids].max() > 2.0 ** 31
    assert passed > 0
