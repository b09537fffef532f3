"""Exact search where its launch changes shape, against the oracle: doc counts
around a chunk part and a chunk, query counts that split a chunk 16 ways down
to not at all, terms held by most docs (dense rows) between rare ones, equal
scores across the k-th place, fewer eligible docs than k, and more query terms
than are located at once."""

import numpy as np
import pytest

import nsparse
import oracle as O
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


def corpus(n, seed, tied):
    g = np.random.default_rng(seed)
    dim = 700
    share = np.where(np.arange(dim) % 9 == 4, 0.6, 0.02)  # every ninth term is frequent
    rows = [np.nonzero(g.random(dim) < share)[0] for _ in range(n)]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    values = np.ones(int(indptr[-1])) if tied else g.lognormal(0.0, 0.8, int(indptr[-1]))
    return synth.Csr(dim, indptr, np.concatenate(rows).astype(np.uint16),
                     values.astype(np.float32))


def queries(n, nnz, tied, seed):
    g = np.random.default_rng(seed)
    rows = [np.sort(g.permutation(700)[:nnz]) for _ in range(n)]
    values = np.ones(n * nnz) if tied else g.lognormal(0.0, 0.8, n * nnz)
    return synth.Csr(700, np.arange(0, n * nnz + 1, nnz, dtype=np.int32),
                     np.concatenate(rows).astype(np.uint16), values.astype(np.float32))


@pytest.mark.parametrize("n_docs", [3, 704, 705, 11264, 11265])
@pytest.mark.parametrize("nq,nnz", [(1, 300), (9, 20), (700, 6)])
@pytest.mark.parametrize("k", [1, 100, 128])
@pytest.mark.parametrize("tied", [False, True])
def test_matches_oracle(n_docs, nq, nnz, k, tied):
    docs, qs = corpus(n_docs, n_docs, tied), queries(nq, nnz, tied, nq)
    for mode, kind in enumerate(("brutal", "inverted")):
        idx = nsparse.index_factory(docs.dim, kind)
        idx.add(docs.n, docs.indptr, docs.indices, docs.values)
        if kind == "inverted":
            idx.build()
        D, L = idx.search(qs.n, qs.indptr, qs.indices, qs.values, k)
        Do, Lo = O.exact_search(docs, qs, k, mode)
        np.testing.assert_array_equal(L, Lo)
        np.testing.assert_array_equal(D, Do)
