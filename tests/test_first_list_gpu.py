"""The first list's visiting order and the query cut of the CTA-per-query
kernel against the warp-per-query kernel, which takes the reference's sort and
holder steps on one thread per range: identical rows, labels and scores, on
indexes whose block scores and query weights tie, for lists around the sort's
switch points (16 blocks; a queue of ranges per warp; more blocks than the
shared-memory buffers hold) and cuts that keep none, some and all terms."""

import numpy as np
import pytest

import nsparse
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu


def coarse(c, step):
    values = (np.floor(c.values / step) + 1) * step
    return synth.Csr(c.dim, c.indptr, c.indices, values.astype(np.float32))


@pytest.mark.parametrize("beta", [16, 17, 700, 1400])
@pytest.mark.parametrize("kind", ["fp32", "sq8"])
def test_ties_match_the_warp_kernel(kind, beta):
    docs = coarse(synth.docs_config0(2500, seed=11), 1.0)
    qs = coarse(synth.queries_config0(20, seed=12), 1.0)
    lists = f"lambda=0|beta={beta}|alpha=0.3|seed=7"
    spec = f"seismic,{lists}" if kind == "fp32" else \
        f"seismic_sq,quantizer=8bit|vmin=0.0|vmax=40.0|{lists}"
    idx = nsparse.index_factory(docs.dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    for cut, hf, k, n in ((1, 0.9, 10, 20), (7, 0.8, 100, 20), (200, 1.0, 10, 3)):
        got = []
        for variant in (0, 4):
            p = nsparse.SeismicSearchParameters(cut, hf)
            p.set_kernel(variant)
            got.append(idx.search(n, qs.indptr[:n + 1], qs.indices, qs.values, k, p))
        np.testing.assert_array_equal(got[0][1], got[1][1])
        np.testing.assert_array_equal(got[0][0], got[1][0])
