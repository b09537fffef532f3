"""Exact search over docs whose scores are NaN or infinite -- such values
stored, or finite products that overflow: a query's row does not depend on how
many queries it is searched with, though a few are spread over more CTAs."""

import numpy as np
import pytest

import nsparse

pytestmark = pytest.mark.gpu

DIM, DOCS, TERMS = 60, 12000, 6


def corpus(kind):
    g = np.random.default_rng(71)
    terms = np.sort(np.argsort(g.random((DOCS, DIM)), axis=1)[:, :TERMS], axis=1)
    values = g.lognormal(0.0, 0.8, (DOCS, TERMS)).astype(np.float32)
    odd = np.arange(DOCS) % 3 == 1
    if kind == "nan":
        values[odd, 2] = np.nan
    elif kind == "inf":
        values[odd, 1], values[odd, 4] = np.inf, -np.inf
    else:
        values[odd, 1], values[odd, 4] = 3e38, -3e38
    return (np.arange(0, DOCS * TERMS + 1, TERMS, dtype=np.int32),
            terms.astype(np.uint16).ravel(), values.ravel())


@pytest.mark.parametrize("index", ["brutal", "inverted"])
@pytest.mark.parametrize("kind", ["nan", "inf", "overflow"])
@pytest.mark.parametrize("k", [3, 40])
def test_rows_do_not_depend_on_the_batch(index, kind, k):
    idx = nsparse.index_factory(DIM, index)
    idx.add(DOCS, *corpus(kind))
    if index == "inverted":
        idx.build()
    n, nnz = 700, 50  # 700: a CTA per chunk of docs
    g = np.random.default_rng(72)
    indptr = np.arange(0, n * nnz + 1, nnz, dtype=np.int32)
    terms = np.concatenate([np.sort(g.permutation(DIM)[:nnz]) for _ in range(n)]).astype(np.uint16)
    values = g.uniform(1.5, 4.0, n * nnz).astype(np.float32)
    want_d, want_l = idx.search(n, indptr, terms, values, k)
    for few in (1, 9, 80):
        d, labels = idx.search(few, indptr[:few + 1], terms, values, k)
        np.testing.assert_array_equal(labels, want_l[:few])
        np.testing.assert_array_equal(d, want_d[:few])
