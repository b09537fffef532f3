"""CTAs per query where the cluster does not fit: one the caller asks for is
refused, the engine's own choice -- its rule's or the autotuner's -- shrinks,
in shared memory (a k too large for the cluster's segments) and in the fixed
scratch of the no-allocation search (a list of very many blocks)."""

import ctypes

import numpy as np
import pytest
import torch

import nsparse
from nsparse_b200 import synth
from test_smem_limits_gpu import index, largest_k

pytestmark = pytest.mark.gpu

_P = ctypes.c_void_p
_noalloc = nsparse._L.nsp_index_search_device_noalloc
_noalloc.restype = ctypes.c_int
_noalloc.argtypes = [_P, ctypes.c_int32, _P, _P, _P, ctypes.c_int32, ctypes.c_int32, ctypes.c_int,
                     _P, _P, _P, _P, _P]


def test_shared_memory():
    idx = index()
    qs = synth.queries_config0(1, seed=62)
    nnz = int(qs.indptr[1])
    args = (1, qs.indptr, qs.indices, qs.values)
    p = nsparse.SeismicSearchParameters(nnz, 1.0)
    want_d, want_l = idx.search(*args, 300, p)
    k = largest_k(nnz, 1024)
    for split, kk in ((8, k), (2, k), (1, k + 4), (0, k + 4)):
        p.set_split(split)
        d, labels = idx.search(*args, kk, p)
        np.testing.assert_array_equal(labels[0, :300], want_l[0])
        np.testing.assert_array_equal(d[0, :300], want_d[0])
    for split in (2, 8):
        p.set_split(split)
        with pytest.raises(ValueError):
            idx.search(*args, k + 4, p)
    p.set_split(0)
    c = idx.autotune(*args, 10, p)
    assert c["ctas_per_query"] in (1, 2, 4, 8)
    _, labels = idx.search(*args, k + 4, p)
    np.testing.assert_array_equal(labels[0, :300], want_l[0])


def test_fixed_scratch():
    # A list of more than 16,200 blocks: 16 CTAs' block scores, visiting orders
    # and sort keys pass 32 MiB, those of 8 do not up to twice that.
    docs = synth.docs_config0(22000, seed=3)
    blocks = int(np.bincount(docs.indices, minlength=docs.dim).max())
    assert 16200 < blocks < 26000
    qs = synth.queries_config0(16, seed=64)
    idx = nsparse.index_factory(docs.dim, "seismic,lambda=22000|beta=22000|alpha=0.4|seed=7")
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    p = nsparse.SeismicSearchParameters(8, 0.9)
    want_d, want_l = idx.search(qs.n, qs.indptr, qs.indices, qs.values, 10, p)
    dev = torch.device("cuda")
    ip = torch.from_numpy(qs.indptr).to(dev)
    ix = torch.from_numpy(qs.indices.view(np.int16)).to(dev)
    v = torch.from_numpy(qs.values).to(dev)
    longest = int(np.diff(qs.indptr).max())
    for tuned in (False, True):
        if tuned:
            idx.autotune(qs.n, qs.indptr, qs.indices, qs.values, 10, p)
        for n in (1, 4, 16):
            d = torch.zeros((n, 10), dtype=torch.float32, device=dev)
            labels = torch.zeros((n, 10), dtype=torch.int32, device=dev)
            status = torch.full((1,), -5, dtype=torch.int32, device=dev)
            torch.cuda.synchronize()
            rc = _noalloc(idx._h, n, ip.data_ptr(), ix.data_ptr(), v.data_ptr(),
                          int(qs.indptr[n]), longest, 10, d.data_ptr(), labels.data_ptr(), p._h,
                          torch.cuda.current_stream().cuda_stream, status.data_ptr())
            assert rc == 0, nsparse._L.nsp_last_error().decode()
            torch.cuda.synchronize()
            assert int(status.item()) == 0
            np.testing.assert_array_equal(labels.cpu().numpy(), want_l[:n])
            np.testing.assert_array_equal(d.cpu().numpy(), want_d[:n])
