"""Two indexes of different vocabularies built side by side on two host threads:
what a kernel may use of a function's settings (shared memory above all) is
process-wide, so one build must not lower it under the other. Every build
writes the file that the same build alone writes."""

import threading

import numpy as np
import pytest

import nsparse
from nsparse_b200 import synth

pytestmark = pytest.mark.gpu

SIZES = {"large": (30522, 1500, 80), "small": (500, 120, 12)}
ROUNDS = 40


def corpus(size):
    dim, n, nnz = SIZES[size]
    g = np.random.default_rng(dim)
    weight = 1.0 / np.arange(1, dim + 1)
    rows = [np.unique(g.choice(dim, nnz, p=weight / weight.sum())) for _ in range(n)]
    indptr = np.concatenate([[0], np.cumsum([len(r) for r in rows])]).astype(np.int32)
    values = g.uniform(0.01, 9.0, int(indptr[-1])).astype(np.float32)
    return synth.Csr(dim, indptr, np.concatenate(rows).astype(np.uint16), values)


def built_file(docs, kind, path):
    lists = "lambda=0|beta=20|alpha=0.4|seed=7"
    spec = f"seismic,{lists}" if kind == "fp32" else \
        f"seismic_sq,quantizer={kind[2:]}bit|vmin=0.0|vmax=9.0|{lists}"
    idx = nsparse.index_factory(docs.dim, spec)
    idx.add(docs.n, docs.indptr, docs.indices, docs.values)
    idx.build()
    nsparse.write_index(idx, str(path))
    return path.read_bytes()


@pytest.mark.parametrize("kind", ["fp32", "sq8", "sq16"])
def test_side_by_side_builds_equal_builds_alone(tmp_path, kind):
    docs = {size: corpus(size) for size in SIZES}
    want = {size: built_file(docs[size], kind, tmp_path / size) for size in SIZES}
    failures = []
    large_done = threading.Event()

    def work(size):
        try:
            i = 0
            while i < ROUNDS if size == "large" else not large_done.is_set():
                if built_file(docs[size], kind, tmp_path / f"{size}.t") != want[size]:
                    failures.append((size, i, "file differs"))
                i += 1
        except Exception as e:
            failures.append((size, i, repr(e)))
        finally:
            if size == "large":
                large_done.set()

    threads = [threading.Thread(target=work, args=(size,)) for size in SIZES]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures, failures
