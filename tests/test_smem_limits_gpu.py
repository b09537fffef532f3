"""The largest k whose holder fits a CTA's shared memory beside the smallest
candidate batch: accepted, with the rows of a small k; four more are refused."""

import numpy as np
import pytest
import torch

import nsparse
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu

DIM, DOCS = 30522, 300


def a16(n):
    return (n + 15) // 16 * 16


def largest_k(nnz, segments):
    """fp32 queries of up to 255 terms: control words, a byte per term, the
    query's values, terms, raw values and cut, a batch of 32 candidates with
    their segments, warp sums, cursor and counters; 8 bytes per result."""
    optin = torch.cuda.get_device_properties(0).shared_memory_per_block_optin
    rest = (32 + a16(DIM + 1) + a16(4 * (nnz + 1)) + 2 * a16(2 * nnz) + a16(4 * nnz) + 32 * 16
            + segments * 32 + a16(32 * 2) + 128 + 64 + 256)
    return (optin - rest) // 2 // 16 * 4


def index():
    docs = synth.docs_config0(DOCS, seed=61)
    assert docs.dim == DIM
    idx = nsparse.index_factory(DIM, "seismic,lambda=0|beta=20|alpha=0.9|seed=7")
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    return idx


def test_one_cta_takes_the_largest_k():
    idx = index()
    qs = synth.queries_config0(1, seed=62)
    nnz = int(qs.indptr[1])
    p = nsparse.SeismicSearchParameters(nnz, 1.0)
    p.set_split(1)
    want_d, want_l = idx.search(1, qs.indptr, qs.indices, qs.values, DOCS, p)
    k = largest_k(nnz, 128)
    d, labels = idx.search(1, qs.indptr, qs.indices, qs.values, k, p)
    np.testing.assert_array_equal(labels[0, :DOCS], want_l[0])
    np.testing.assert_array_equal(d[0, :DOCS], want_d[0])
    assert (labels[0, DOCS:] == -1).all()
    with pytest.raises(ValueError):
        idx.search(1, qs.indptr, qs.indices, qs.values, k + 4, p)
