"""Filtered and mid-size launches of the CTA-per-query kernel against the
warp-per-query kernel: selectors holding no doc, a few, half and all of them
(a batch keeps only its members), query counts that change the CTA's width,
and 16-bit queries at the longest length a byte of rank holds and past it."""

import numpy as np
import pytest

import nsparse
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["fp32", "sq16"])
def built(request):
    docs = synth.docs_config0(3000, seed=31)
    lists = "lambda=600|beta=40|alpha=0.4|seed=7"
    spec = f"seismic,{lists}" if request.param == "fp32" else \
        f"seismic_sq,quantizer=16bit|vmin=0.0|vmax=40.0|{lists}"
    idx = nsparse.index_factory(docs.dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    return docs, idx


@pytest.mark.parametrize("share", [None, 0.0, 0.003, 0.5, 1.0])
@pytest.mark.parametrize("n,nnz,k", [(5, 255, 10), (5, 256, 10), (160, 20, 33), (310, 20, 100),
                                     (700, 12, 10)])
def test_rows_equal_the_warp_kernel(built, share, n, nnz, k):
    docs, idx = built
    g = np.random.default_rng(n + nnz)
    rows = [np.sort(g.permutation(2000)[:nnz]) for _ in range(n)]
    indptr = np.arange(0, n * nnz + 1, nnz, dtype=np.int32)
    values = g.lognormal(0.0, 0.8, n * nnz).astype(np.float32)
    terms = np.concatenate(rows).astype(np.uint16)
    got = []
    for variant in (0, 4):
        p = nsparse.SeismicSearchParameters(8, 0.9)
        p.set_kernel(variant)
        p.set_split(1)
        if share is not None:
            member = np.random.default_rng(3).random(docs.n // 64 * 64 + 64) < share
            p.set_id_selector(nsparse.BitmapIDSelector(
                docs.n, np.packbits(member, bitorder="little").view(np.uint64)))
        got.append(idx.search(n, indptr, terms, values, k, p))
    np.testing.assert_array_equal(got[0][1], got[1][1])
    np.testing.assert_array_equal(got[0][0], got[1][0])
