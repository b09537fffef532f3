"""A thread-block cluster per query against one CTA per query: identical rows
on lists whose blocks and runs do not fit the kernel's shared-memory stages,
queries longer than a lookup window, more cut lists than warps, batches that
split blocks and span lists, holders on both sides of a warp, filters, empty
and non-finite queries."""

import numpy as np
import pytest

import nsparse
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module", params=["fp32", "sq8", "sq16"])
def built(request):
    docs = synth.docs_config0(4000, seed=21)
    lists = "lambda=0|beta=900|alpha=0.5|seed=7"
    spec = f"seismic,{lists}" if request.param == "fp32" else \
        f"seismic_sq,quantizer={request.param[2:]}bit|vmin=0.0|vmax=9.0|{lists}"
    idx = nsparse.index_factory(docs.dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    return request.param, docs, idx


@pytest.mark.parametrize("split", [2, 4, 8, 0])
@pytest.mark.parametrize("nnz,cut,k,warps,batch,filtered", [
    (29, 10, 10, 0, 0, False),
    (300, 40, 32, 0, 0, False),      # more cut lists than warps, two lookup windows
    (60, 12, 33, 2, 32, False),      # blocks split over tiny batches
    (29, 10, 100, 8, 64, True),
    (3, 10, 1, 0, 0, False),
])
def test_cluster_rows_equal_one_cta(built, split, nnz, cut, k, warps, batch, filtered):
    kind, docs, idx = built
    g = np.random.default_rng(nnz + k)
    weight = 1.0 / np.arange(1, docs.dim + 1)
    rows = [np.unique(g.choice(docs.dim, nnz, p=weight / weight.sum())) for _ in range(4)]
    rows[2] = rows[2][:0]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    values = g.lognormal(0.0, 0.8, int(indptr[-1])).astype(np.float32)
    if kind == "fp32" and not filtered:
        values[indptr[3]] = np.inf
    got = []
    for s in (1, split):
        p = nsparse.SeismicSearchParameters(cut, 0.9)
        p.set_split(s)
        p.set_kernel(4, batch)
        p.set_engine(warps_per_block=warps)
        if filtered:
            member = np.random.default_rng(5).random(docs.n // 64 * 64 + 64) < 0.3
            p.set_id_selector(nsparse.BitmapIDSelector(
                docs.n, np.packbits(member, bitorder="little").view(np.uint64)))
        got.append(idx.search(4, indptr, np.concatenate(rows).astype(np.uint16), values, k, p))
    np.testing.assert_array_equal(got[0][1], got[1][1])
    np.testing.assert_array_equal(got[0][0].view(np.int32), got[1][0].view(np.int32))
