"""The query cut against the oracle: codes and values that tie heavily, cuts
around the 32 terms that a warp holds in registers, past them, and past the
words that shared memory holds beside a small batch; fp32 queries of more terms
than are ranked by all threads. One CTA, a cluster and a warp per query."""

import numpy as np
import pytest

import nsparse
from helpers import oracle_seismic_from_file, sq_codes
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu

VMAX = 9.0


@pytest.fixture(scope="module", params=["fp32", "sq8", "sq16"])
def built(request, tmp_path_factory):
    docs = synth.docs_config0(1500, seed=81)
    lists = "lambda=100|beta=10|alpha=0.5|seed=7"
    bits = 0 if request.param == "fp32" else int(request.param[2:])
    spec = f"seismic,{lists}" if bits == 0 else \
        f"seismic_sq,quantizer={bits}bit|vmin=0.0|vmax={VMAX}|{lists}"
    idx = nsparse.index_factory(docs.dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    path = str(tmp_path_factory.mktemp("cut") / "c.idx")
    nsparse.write_index(idx, path)
    return bits, docs, idx, path


@pytest.mark.parametrize("nnz,levels,cut", [
    (200, 4, 31), (200, 4, 32), (200, 4, 33), (250, 2, 100), (250, 1000, 33),
    (1400, 3, 1200),   # a holder past the words beside a small batch
    (1025, 5, 20), (1025, 5, 300), (1025, 100000, 300), (1024, 5, 300),
])
def test_matches_oracle(built, nnz, levels, cut):
    bits, docs, idx, path = built
    g = np.random.default_rng(nnz + levels + cut)
    n = 6
    frequent = np.argsort(-np.bincount(docs.indices, minlength=docs.dim))[:3000]
    rows = [np.sort(g.choice(frequent, nnz, replace=False)) for _ in range(n)]
    values = ((1 + g.integers(0, levels, n * nnz)) * (VMAX / (levels + 1))).astype(np.float32)
    qs = synth.Csr(docs.dim, np.arange(0, n * nnz + 1, nnz, dtype=np.int32),
                   np.concatenate(rows).astype(np.uint16), values)
    codes = None if bits == 0 else sq_codes(0.0, VMAX, values, bits)
    _, want = oracle_seismic_from_file(path, qs, 10, cut, 0.9, codes=codes)
    for variant, split in ((4, 1), (4, 8), (0, 0)):
        p = nsparse.SeismicSearchParameters(cut, 0.9)
        p.set_kernel(variant, 32 if variant == 4 and split == 1 else 0)
        p.set_split(split)
        _, labels = idx.search(n, qs.indptr, qs.indices, qs.values, 10, p)
        np.testing.assert_array_equal(labels, want)
