"""Performance cases of the sparse-retrieval engine.

Each case is work a program has the engine do through its public Python API:
one query, a batch or a burst of requests against a resident index, a
device-resident step, or an index built from a corpus and searched for the
first time. The corpora and queries are the seeded synthetic ones of
``nsparse_b200.synth`` (the shape of MS MARCO SPLADE vectors), with the index
parameters and sizes of ``bench.py`` and the tests.

In a search case the index is what the program keeps: it is built from one
corpus of the case's size and held while cases and seeds share it; the seed
draws the queries and the filter. In a build case the seed draws the corpus.
"""

import gc
import math
import os
import sys

import numpy as np
import torch

_PY = os.path.join(os.path.abspath(sys.path[0] or "."), "neural-sparse-cpp_b200", "python")
if not os.path.isdir(_PY):
    _PY = os.path.abspath(os.path.join("neural-sparse-cpp_b200", "python"))
if _PY not in sys.path:
    sys.path.insert(0, _PY)

import nsparse  # noqa: E402
from nsparse_b200 import synth  # noqa: E402

CORPUS_SEED = 7
DIM = synth.VOCAB


def listed():
    return [
        # An interactive program: one short query at a time against a small
        # index; the call's latency.
        dict(name="one_fp32_100k", op="search", index="fp32", docs=100_000, lam=4000, beta=400,
             queries=1, shape="short", k=10, cut=10, hf=0.8, select=0),
        # Offline retrieval (fp32): the whole query set in one host call.
        dict(name="batch_fp32_1m", op="search", index="fp32", docs=1_000_000, lam=4000, beta=400,
             queries=10_000, shape="short", k=10, cut=10, hf=0.8, select=0),
        # A re-ranking stage: an odd batch of queries restricted to a tenth of
        # the docs by a bitmap, 100 results each.
        dict(name="filtered_fp32_1m", op="search", index="fp32", docs=1_000_000, lam=4000,
             beta=400, queries=333, shape="short", k=100, cut=10, hf=0.9, select=10),
        # The latency of a lone long query on a large quantized index.
        dict(name="one_sq8_3m", op="search", index="sq8", docs=3_000_000, lam=6000, beta=600,
             queries=1, shape="long", k=10, cut=12, hf=0.9, select=0),
        # The serving loop: requests that have piled up, k 10 or 100, 30% of
        # them filtered, worked off in continuous batches.
        dict(name="serve_sq8_3m", op="serve", index="sq8", docs=3_000_000, lam=6000, beta=600,
             queries=2_000, shape="long", k=100, cut=12, hf=0.9, select=30),
        # Throughput: device-resident queries, one captured step per batch.
        dict(name="step_sq8_3m", op="step", index="sq8", docs=3_000_000, lam=6000, beta=600,
             queries=16_384, shape="long", k=10, cut=12, hf=0.9, select=0),
        # 16-bit codes, an ordinary odd batch.
        dict(name="batch_sq16_301k", op="search", index="sq16", docs=301_000, lam=3000, beta=300,
             queries=1_001, shape="long", k=20, cut=12, hf=0.9, select=0),
        # Exact search: a batch for ground truth, and a few queries with a
        # selector against posting lists.
        dict(name="exact_100k", op="search", index="brutal", docs=100_000, lam=0, beta=0,
             queries=1_000, shape="short", k=10, cut=0, hf=0.0, select=0),
        dict(name="exact_few_300k", op="search", index="inverted", docs=300_001, lam=0, beta=0,
             queries=7, shape="short", k=100, cut=0, hf=0.0, select=10),
        # An index rebuilt from its vectors and searched for the first time.
        dict(name="build_fp32_80k", op="build", index="fp32", docs=80_000, lam=4000, beta=400,
             queries=100, shape="short", k=100, cut=10, hf=1.0, select=0),
        dict(name="build_sq8_200k", op="build", index="sq8", docs=200_000, lam=6000, beta=600,
             queries=100, shape="long", k=100, cut=12, hf=1.0, select=0),
        # A small shard, as an ingest job flushes them.
        dict(name="build_sq8_20k", op="build", index="sq8", docs=20_011, lam=1000, beta=100,
             queries=10, shape="long", k=10, cut=12, hf=1.0, select=0),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["search", "search", "search", "exact", "exact", "build", "build", "serve",
                     "step"])
    if op == "exact":
        return dict(op="search", index=rng.choice(["brutal", "inverted"]),
                    docs=_log_int(rng, 5_000, 300_000), lam=0, beta=0,
                    queries=_log_int(rng, 1, 1_000), shape="short",
                    k=rng.choice([1, 10, 33, 100]), cut=0, hf=0.0, select=rng.choice([0, 0, 10]))
    if op == "build":
        index = rng.choice(["fp32", "sq8", "sq16"])
        docs = _log_int(rng, 10_000, 200_000 if index == "sq8" else 80_000)
    else:
        index = rng.choice(["fp32", "sq8", "sq8", "sq16"])
        docs = _log_int(rng, 20_000, 600_000)
    queries = {"search": _log_int(rng, 1, 8_000), "serve": _log_int(rng, 20, 2_000),
               "step": _log_int(rng, 64, 8_192), "build": _log_int(rng, 10, 200)}[op]
    lam = rng.choice([400, 1000, 2500, 4000, 6000])
    return dict(op=op, index=index, docs=docs, lam=lam, beta=lam // rng.choice([8, 10, 20]),
                queries=queries, shape=rng.choice(["short", "long"]),
                k=rng.choice([5, 10, 20, 100]), cut=rng.choice([3, 8, 10, 12]),
                hf=rng.choice([0.7, 0.8, 0.9, 0.95, 1.0]),
                select=0 if op in ("build", "step") else rng.choice([0, 0, 10, 30]))


# ------------------------------------------------------------- inputs --

def _corpus(case, seed):
    make = synth.docs_config2 if case["index"] in ("sq8", "sq16") else synth.docs_config0
    return make(case["docs"], seed=seed)


def _queries(case, seed):
    make = synth.queries_config2 if case["shape"] == "long" else synth.queries_config0
    return make(case["queries"], seed=1_000 + seed)


def _description(case, docs):
    index = case["index"]
    if index in ("brutal", "inverted"):
        return index
    lists = f"lambda={case['lam']}|beta={case['beta']}|alpha=0.4|seed=7"
    if index == "fp32":
        return f"seismic,{lists}"
    vmin, vmax = float(docs.values.min()), float(docs.values.max())
    bits = "16bit" if index == "sq16" else "8bit"
    return f"seismic_sq,quantizer={bits}|vmin={vmin!r}|vmax={vmax!r}|{lists}"


def _build(case, docs):
    index = nsparse.index_factory(DIM, _description(case, docs))
    index.add(docs.n, docs.indptr, docs.indices, docs.values)
    if case["index"] != "brutal":
        index.build()
    return index


_kept = {"key": None, "index": None}  # the resident index, shared by the cases that use it


def _resident(case):
    key = tuple(case[f] for f in ("index", "docs", "lam", "beta"))
    if _kept["key"] != key:
        _kept.update(key=None, index=None)
        gc.collect()
        index = _build(case, _corpus(case, CORPUS_SEED))
        _kept.update(key=key, index=index)
    return _kept["index"]


def _parameters(case):
    if case["index"] in ("brutal", "inverted"):
        return nsparse.SearchParameters()
    return nsparse.SeismicSearchParameters(case["cut"], case["hf"])


def _tenth(case, seed):
    """A bitmap over the docs with a random tenth of them set."""
    n = case["docs"]
    member = np.random.default_rng(2_000 + seed).random((n + 64) // 64 * 64) < 0.1
    member[n:] = False
    return np.packbits(member, bitorder="little").view(np.uint64)


def prepare(case, seed):
    q = _queries(case, seed)
    state = {"case": case, "queries": q, "params": _parameters(case)}
    if case["op"] == "build":
        state["docs"] = _corpus(case, seed)
        return state
    index = state["index"] = _resident(case)
    if case["op"] == "search":
        if case["select"]:
            state["params"].set_id_selector(
                nsparse.BitmapIDSelector(case["docs"], _tenth(case, seed)))
    elif case["op"] == "serve":
        rng = np.random.default_rng(3_000 + seed)
        server = state["server"] = nsparse.Server(index)
        some = server.add_filter(_tenth(case, seed))
        state["k_per"] = np.where(rng.random(q.n) < 0.5, min(10, case["k"]),
                                  case["k"]).astype(np.int32)
        state["k_per"][0] = case["k"]
        state["filters"] = np.where(rng.random(q.n) * 100 < case["select"], some,
                                    -1).astype(np.int32)
        state["arrival"] = np.zeros(q.n)
    else:
        dev = torch.device("cuda")
        b = state["buffers"] = {
            "indptr": torch.from_numpy(q.indptr).to(dev),
            "indices": torch.from_numpy(q.indices.view(np.int16)).to(dev),
            "values": torch.from_numpy(q.values).to(dev),
            "distances": torch.empty((q.n, case["k"]), dtype=torch.float32, device=dev),
            "labels": torch.empty((q.n, case["k"]), dtype=torch.int32, device=dev)}
        torch.cuda.synchronize()
        state["graph"] = nsparse.SearchGraph(
            index, q.n, q.nnz, int(np.diff(q.indptr).max()), case["k"], state["params"],
            {name: t.data_ptr() for name, t in b.items()})
    return state


def run(state):
    case, q, params = state["case"], state["queries"], state["params"]
    if case["op"] == "step":
        state["graph"].launch()
        return state["buffers"]["distances"], state["buffers"]["labels"]
    if case["op"] == "serve":
        d, labels, _ = state["server"].replay(
            q.indptr, q.indices, q.values, state["k_per"], state["arrival"], cut=case["cut"],
            heap_factor=case["hf"], filter_per=state["filters"])
        # a row's slots past its own k are not written
        past = np.arange(d.shape[1])[None, :] >= state["k_per"][:, None]
        d[past] = -1.0
        labels[past] = -1
        return d, labels
    index = _build(case, state["docs"]) if case["op"] == "build" else state["index"]
    return index.search(q.n, q.indptr, q.indices, q.values, case["k"], params)


# --------------------------------------------------------------- work --

_MEAN_NNZ = {"short": (128.0, 29.0), "long": (139.0, 102.5)}  # of the docs, of the queries


def _mean_list(docs, nnz, cap):
    """Posting list length, cap applied, of a term as it is met in a query
    (terms drawn Zipf(1.1)); and the total kept postings."""
    p = np.arange(1, DIM + 1, dtype=np.float64) ** -1.1
    p /= p.sum()
    length = docs * -np.expm1(-nnz * 2.0 * p)
    length *= docs * nnz / length.sum()
    kept = np.minimum(length, cap) if cap > 0 else length
    return float((p * kept).sum()), float(kept.sum())


def work(case):
    esz = {"sq8": 1, "sq16": 2}.get(case["index"], 4)
    doc_nnz = 139.0 if case["index"] in ("sq8", "sq16") else 128.0
    q_nnz = _MEAN_NNZ[case["shape"]][1]
    n, docs, k = case["queries"], case["docs"], case["k"]
    io = n * (4 + q_nnz * 6 + k * 8)
    if case["index"] in ("brutal", "inverted"):
        # every posting of the query's terms, once per query
        postings = n * q_nnz * _mean_list(docs, doc_nnz, 0)[0]
        return {"bytes": io + min(postings, docs * doc_nnz) * 8, "flops": 2.0 * postings}
    met, kept = _mean_list(docs, doc_nnz, case["lam"])
    # the docs of the cut lists' blocks, about three quarters of which pass
    # the pruning tests; each query reads its own
    scored = 0.75 * min(case["cut"], q_nnz) * met
    search = {"bytes": io + n * scored * (12 + doc_nnz * (2 + esz)),
              "flops": 2.0 * n * scored * doc_nnz}
    if case["op"] != "build":
        return search
    # the vectors in, and per kept posting its doc's row for the assignment
    # to one of the list's centroids and for its block's summary
    return {"bytes": search["bytes"] + docs * doc_nnz * 6 + 2 * kept * doc_nnz * (2 + esz),
            "flops": search["flops"] + 2.0 * kept * doc_nnz}


# -------------------------------------------------------------- exact --

def exact(case, seed):
    """Exact indexes: the k largest dot products in 64 bits. A SEISMIC search's
    results depend on its pruned walk, which has no value without the index."""
    if case["index"] not in ("brutal", "inverted"):
        return None
    docs, q = _corpus(case, CORPUS_SEED), _queries(case, seed)
    dev = torch.device("cuda" if torch.cuda.is_available() else "cpu")
    rows = torch.sparse_csr_tensor(torch.from_numpy(docs.indptr.astype(np.int64)),
                                   torch.from_numpy(docs.indices.astype(np.int64)),
                                   torch.from_numpy(docs.values.astype(np.float64)),
                                   size=(docs.n, DIM)).to(dev)
    member = None
    if case["select"] and case["index"] == "inverted":  # brute force takes no selector
        bits = np.unpackbits(_tenth(case, seed).view(np.uint8), bitorder="little")[:docs.n]
        member = torch.from_numpy(bits.astype(bool)).to(dev)
    out = np.full((q.n, case["k"]), -1.0)
    for lo in range(0, q.n, 128):
        part = q.rows(lo, min(q.n, lo + 128))
        dense = np.zeros((DIM, part.n))
        for i in range(part.n):
            s, e = part.indptr[i], part.indptr[i + 1]
            dense[part.indices[s:e], i] = part.values[s:e]
        scores = rows @ torch.from_numpy(dense).to(dev)
        if case["index"] == "inverted":
            # a doc without a common term is not in any of the query's lists
            scores[scores <= 0] = -1.0
        if member is not None:
            scores[~member] = -1.0
        top = torch.topk(scores, min(case["k"], docs.n), dim=0).values.T
        out[lo:lo + part.n, :top.shape[1]] = top.cpu().numpy()
    return out, None
