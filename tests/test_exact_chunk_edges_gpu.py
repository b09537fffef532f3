"""Exact search at the edges of the parts and chunks that its launch divides the
docs into -- 720 and 11,520 docs on a B200, a lone query's chunk in 16 parts --
against the oracle."""

import numpy as np
import pytest

import nsparse
import oracle as O
from test_exact_split_gpu import corpus, queries

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n_docs", [720, 721, 11519, 11520, 11521, 23041])
@pytest.mark.parametrize("nq,nnz", [(1, 300), (20, 20), (700, 6)])
@pytest.mark.parametrize("k", [1, 128])
def test_matches_oracle(n_docs, nq, nnz, k):
    docs, qs = corpus(n_docs, n_docs, False), queries(nq, nnz, False, nq)
    for mode, kind in enumerate(("brutal", "inverted")):
        idx = nsparse.index_factory(docs.dim, kind)
        idx.add(docs.n, docs.indptr, docs.indices, docs.values)
        if kind == "inverted":
            idx.build()
        D, L = idx.search(qs.n, qs.indptr, qs.indices, qs.values, k)
        Do, Lo = O.exact_search(docs, qs, k, mode)
        np.testing.assert_array_equal(L, Lo)
        np.testing.assert_array_equal(D, Do)
