"""Queries without terms among others in launches where every cluster of CTAs
takes several queries: the leader hands its cluster the next query's number
while the others may still be reading the empty one's, unless a barrier lies
between. Rows equal those of one CTA per query, over many launches; rows past
the caller's bound, which the kernel treats as empty, included."""

import numpy as np
import pytest
import torch

import nsparse
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu

DOCS = synth.docs_config0(3000, seed=41)
LISTS = "lambda=600|beta=40|alpha=0.4|seed=7"


def build(kind):
    spec = f"seismic,{LISTS}" if kind == "fp32" else \
        f"seismic_sq,quantizer={kind[2:]}bit|vmin=0.0|vmax=40.0|{LISTS}"
    idx = nsparse.index_factory(DOCS.dim, spec)
    idx.add(DOCS.n, DOCS.indptr, DOCS.indices, DOCS.values)
    idx.build()
    return idx


def with_empty_rows(n, every):
    """n queries; only every `every`-th holds terms."""
    full = synth.queries_config0(n, seed=43)
    keep = np.arange(n) % every == 0
    lengths = np.where(keep, np.diff(full.indptr), 0)
    rows = [slice(full.indptr[i], full.indptr[i + 1]) for i in range(n) if keep[i]]
    return (np.concatenate([[0], np.cumsum(lengths)]).astype(np.int32),
            np.concatenate([full.indices[r] for r in rows]),
            np.concatenate([full.values[r] for r in rows]))


@pytest.mark.parametrize("kind", ["fp32", "sq8", "sq16"])
@pytest.mark.parametrize("every", [2, 7, 400])
def test_rows_equal_one_cta(kind, every):
    idx = build(kind)
    n = 400
    indptr, terms, values = with_empty_rows(n, every)
    got = {}
    for split in (1, 2, 4, 8):
        p = nsparse.SeismicSearchParameters(8, 0.9)
        p.set_split(split)
        for _ in range(10):
            d, labels = idx.search(n, indptr, terms, values, 10, p)
            if split == 1:
                got = (d, labels)
            np.testing.assert_array_equal(labels, got[1])
            np.testing.assert_array_equal(d, got[0])


def test_rows_past_the_bound_are_padding():
    idx = build("fp32")
    n, bound = 300, 12
    qs = synth.queries_config0(n, seed=44)
    lengths = np.diff(qs.indptr)
    assert (lengths > bound).any() and (lengths <= bound).any()
    dev = torch.device("cuda")
    ip = torch.from_numpy(qs.indptr).to(dev)
    ix = torch.from_numpy(qs.indices.view(np.int16)).to(dev)
    v = torch.from_numpy(qs.values).to(dev)
    out = {}
    for split in (1, 8):
        p = nsparse.SeismicSearchParameters(8, 0.9)
        p.set_split(split)
        d = torch.zeros((n, 10), dtype=torch.float32, device=dev)
        labels = torch.zeros((n, 10), dtype=torch.int32, device=dev)
        idx.search(1, qs.indptr[:2], qs.indices, qs.values, 10, p)  # resident
        torch.cuda.synchronize()
        for _ in range(10):
            idx.search_device(n, ip.data_ptr(), ix.data_ptr(), v.data_ptr(), bound, 10,
                              d.data_ptr(), labels.data_ptr(), p,
                              torch.cuda.current_stream().cuda_stream)
            torch.cuda.synchronize()
        out[split] = (d.cpu().numpy(), labels.cpu().numpy())
    np.testing.assert_array_equal(out[8][1], out[1][1])
    np.testing.assert_array_equal(out[8][0], out[1][0])
    assert (out[1][1][lengths > bound] == -1).all()
