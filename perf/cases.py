"""The work a user has this framework do, as cases that can be timed.

Four kinds, all through the public `ANN` object:

  search    `ANN.search` of a query batch over an index that is already built
  build     `ANN(vectors=...)`: the graph of a vector set, from the circulant or the tensor-core start graph
  load      `ANN(vectors=..., beams=...)`: a saved graph comes back without its distances
  clusters  `ANN.clusters()` and `ANN.cluster_labels(...)`: every indexed vector is searched, close ones are grouped

`listed()` holds fixed cases from the smallest call to the largest, `draw(rng)` gives others of the same ranges.
"""
import math
import os
import sys

import torch

# the package lives in a folder whose name is no identifier; the working folder is the repository's root
_PACKAGES = os.path.abspath("vectorlink-gpu_b200")
if _PACKAGES not in sys.path:
    sys.path.insert(0, _PACKAGES)

from vectorlink_gpu import ANN  # noqa: E402

PVC = 4                # parallel_visit_count: its default, which no configuration of this repository changes
EXCLUDE = 5            # exclude_factor: likewise
EXACT_DIMS = (64, 96, 128, 256, 384, 512, 768, 1024)


def _search(name, n, dim, metric, rows, degree, factor, seeds=1, entry=0):
    return {"name": name, "kind": "search", "n": n, "dim": dim, "metric": metric, "rows": rows, "degree": degree,
            "factor": factor, "seeds": seeds, "entry": entry}


def _build(name, n, dim, metric, degree, factor, init, loops):
    return {"name": name, "kind": "build", "n": n, "dim": dim, "metric": metric, "degree": degree, "factor": factor,
            "init": init, "loops": loops}


def listed():
    return [
        # one question typed by one person: nothing hides the latency of the search or of the calls around it
        _search("search_1", 200_000, 128, "l2", 1, 32, 2),
        # the handful of questions of one retrieval request over text embeddings, wide beam
        _search("search_16_embedding", 100_000, 768, "cosine", 16, 64, 2),
        # a served micro-batch with the keyword defaults of ANN and rows that no exact-fit layout matches
        _search("search_301_ragged", 60_013, 50, "cosine", 301, 24, 3),
        # a served batch over deep-learning descriptors, keyword defaults
        _search("search_1000", 500_000, 96, "cosine", 1_000, 24, 3),
        # a batch whose starting points come from the tensor-core scan of a sample of the index
        _search("search_2500_entry", 200_000, 256, "cosine", 2_500, 32, 2, entry=32_768),
        # offline evaluation: ten thousand queries against a million vectors, widened seed scan
        _search("search_10000", 1_000_000, 128, "l2", 10_000, 32, 2, seeds=30),
        # the index of one document collection or of one test: launches and host work count
        _build("build_2000", 2_000, 64, "cosine", 16, 2, "circulant", 3),
        # the reference's schedule on an ordinary set
        _build("build_150k_circulant", 150_000, 128, "l2", 32, 2, "circulant", 3),
        # embeddings from the tensor-core start graph, a row count that no tile divides
        _build("build_60k_embedding", 60_007, 768, "cosine", 64, 2, "knn_tile", 1),
        # the largest single call: a million rows from the tensor-core start graph
        _build("build_1M_tile", 1_000_000, 128, "l2", 32, 2, "knn_tile", 1),
        # a saved index is opened again and its link lengths are computed
        {"name": "load_1M", "kind": "load", "n": 1_000_000, "dim": 128, "metric": "l2", "degree": 32},
        # groups of near-duplicates among all indexed vectors
        {"name": "clusters_30k", "kind": "clusters", "n": 30_000, "dim": 96, "metric": "cosine", "degree": 24, "factor": 3},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _dim(rng):
    pick = rng.random()
    if pick < 0.4:
        return rng.choice(EXACT_DIMS)
    d = _log_int(rng, 24, 1024)
    return d if pick > 0.7 else max(24, d // 4 * 4)


def draw(rng):
    """One more case: sizes over the logarithm of their range, cut down where the whole would cost more than the
    largest listed case of its kind."""
    kind = rng.choice(("search",) * 5 + ("build",) * 3 + ("load", "clusters"))
    dim = _dim(rng)
    metric = rng.choice(("cosine", "l2"))
    degree, factor = rng.choice(((16, 2), (24, 3), (32, 2), (64, 2)))
    if kind == "search":
        n = min(_log_int(rng, 2_000, 500_000), 60_000_000 // dim)
        if dim % 4:
            n = min(n, 60_013)      # building such an index takes long, and `prepare` has to be quick
        rows = _log_int(rng, 1, 10_000)
        seeds, entry = rng.choice(((1, 0), (1, 0), (8, 0), (30, 0), (1, 32_768)))
        rows = max(1, min(rows, int(1e11 / (_evaluations(degree, factor, degree) * (4 * dim + 12)))))
        return {"kind": kind, "n": n, "dim": dim, "metric": metric, "rows": rows, "degree": degree, "factor": factor,
                "seeds": seeds, "entry": entry}
    if kind == "build":
        init, loops = rng.choice((("circulant", 3), ("knn_tile", 1)))
        n = _log_int(rng, 1_000, 150_000)
        n = max(1_000, min(n, int(5e12 / (loops * _evaluations(degree, factor, 3 * degree) * (4 * dim + 12)))))
        if dim % 4:
            n = min(n, 20_011)
        return {"kind": kind, "n": n, "dim": dim, "metric": metric, "degree": degree, "factor": factor, "init": init,
                "loops": loops}
    if kind == "load":
        n = min(_log_int(rng, 10_000, 1_000_000), 128_000_000 // dim)
        return {"kind": kind, "n": n, "dim": dim, "metric": metric, "degree": degree}
    n = _log_int(rng, 2_000, 30_000)
    n = max(1_000, min(n, int(2.5e11 / (_evaluations(degree, factor, degree) * (4 * dim + 12)))))
    if dim % 4:
        n = min(n, 10_007)
    return {"kind": kind, "n": n, "dim": dim, "metric": metric, "degree": degree, "factor": factor}


def _evaluations(degree, factor, width):
    """Neighbours that one row's budgeted search looks at: visits times list width."""
    visits = EXCLUDE * factor * degree
    return (visits // PVC + 1) * PVC * width


def _vectors(case, count, which, seed):
    """Rows of a Gaussian mixture: integer-valued descriptors for "l2", unit vectors for "cosine".  `which` numbers
    independent draws around the same centres (0 the indexed rows, 1 the queries).  A centre has 1,500 rows or more,
    as in the mixtures that the benchmark builds from."""
    dim = case["dim"]
    centres_n = max(1, min(256, case["n"] // 1_500))
    g = torch.Generator(device="cuda")
    g.manual_seed(1_000_003 * seed + 17)
    if case["metric"] == "l2":
        centres = torch.rand((centres_n, dim), generator=g, device="cuda") * 255.0
        noise = 20.0
    else:
        centres = torch.nn.functional.normalize(torch.randn((centres_n, dim), generator=g, device="cuda"), dim=1)
        noise = 1.0 / math.sqrt(dim)
    g.manual_seed(1_000_003 * seed + 101 + which)
    own = torch.randint(0, centres_n, (count,), generator=g, device="cuda")
    rows = torch.randn((count, dim), generator=g, device="cuda").mul_(noise).add_(centres[own])
    if case["metric"] == "l2":
        return rows.round_().clamp_(0.0, 255.0)
    return torch.nn.functional.normalize(rows, dim=1)


def _keywords(case):
    return {"beam_size": case["degree"], "visit_queue_factor": case["factor"], "recall_search_queue_factor": case["factor"],
            "metric": case["metric"]}


def prepare(case, seed):
    vectors = _vectors(case, case["n"], 0, seed)
    state = {"case": case, "vectors": vectors}
    kind = case["kind"]
    if kind in ("search", "clusters"):
        more = {}
        if kind == "search":
            more = {"search_seed_factor": case["seeds"], "search_entry_sample": case["entry"]}
            state["queries"] = _vectors(case, case["rows"], 1, seed)
        # the index that such a program holds; its build is timed by the cases of that kind
        state["index"] = ANN(vectors=vectors, init="knn_tile", optimization_loops=1, **_keywords(case), **more)
        if kind == "clusters":
            # links shorter than the usual distance to the 4th neighbour
            state["threshold"] = float(state["index"].distances[:, 3].median())
    elif kind == "load":
        # the lists that a build leaves: neighbours by distance are scattered over the whole set
        g = torch.Generator(device="cuda")
        g.manual_seed(1_000_003 * seed + 211)
        state["beams"] = torch.randint(0, case["n"], (case["n"], case["degree"]), generator=g, device="cuda",
                                       dtype=torch.int32)
    return state


def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "search":
        queue = state["index"].search(state["queries"])
        return queue.indices, queue.distances
    if kind == "build":
        index = ANN(vectors=state["vectors"], init=case["init"], optimization_loops=case["loops"], **_keywords(case))
        return index.beams, index.distances
    if kind == "load":
        index = ANN(vectors=state["vectors"], beams=state["beams"], beam_size=case["degree"], metric=case["metric"])
        return index.distances
    queues = state["index"].clusters()
    labels = state["index"].cluster_labels(state["threshold"], queues)
    return queues.indices, queues.distances, labels


#: Of the neighbours that a search looks at on a graph of near neighbours, about this share are ones it has not met
#: before: the rest need no row and no arithmetic.
DISTINCT = 0.2


def _search_work(rows, n, dim, degree, width, factor, out_cols):
    """Bytes and operations of searching `rows` rows: each query and result once, the rows and lists met once, but no
    more of the index than there is."""
    met = DISTINCT * _evaluations(degree, factor, width)
    visits = EXCLUDE * factor * degree
    index = min(n * (4.0 * dim + 4.0 * width), rows * (met * 4.0 * dim + visits * 4.0 * width))
    return rows * 4.0 * dim + rows * out_cols * 8.0 + index, rows * met * 3.0 * dim


def work(case):
    n, dim, degree, kind = case["n"], case["dim"], case["degree"], case["kind"]
    if kind == "load":
        # every neighbour's row is fetched: the lists are scattered and a set this size does not stay on the chip
        pairs = float(n) * degree
        return {"bytes": n * 4.0 * dim + pairs * 8.0 + (pairs * 4.0 * dim if n * 4.0 * dim > 100e6 else 0.0),
                "flops": pairs * 3.0 * dim}
    queue = case["factor"] * degree
    if kind == "search":
        b, f = _search_work(case["rows"], n, dim, degree, degree, case["factor"], queue + max(queue, PVC * degree))
        if case["entry"]:
            f += 2.0 * case["rows"] * min(n, case["entry"]) * dim
        return {"bytes": b, "flops": f}
    if kind == "clusters":
        b, f = _search_work(n, n, dim, degree, degree, case["factor"], queue + max(queue, PVC * degree))
        return {"bytes": b + n * 4.0, "flops": f}
    # one round is the least that a build can need
    b, f = _search_work(n, n, dim, degree, 3 * degree, case["factor"], degree)
    if case["init"] == "knn_tile":
        return {"bytes": b, "flops": 2.0 * n * n * dim + f}
    return {"bytes": b, "flops": f / DISTINCT}      # neighbours in the circulant graph hardly repeat


def tolerance(case):
    """Distances are sums in a fixed order and ties are broken by id, so searches, loads and builds from the circulant
    graph give the same bits whatever computes them.  The tensor-core start graph picks its candidates by bf16 scores:
    there the last candidate of a list may be another one."""
    if case["kind"] == "build" and case["init"] == "knn_tile":
        return {"rel": 1e-5, "max": 1e-2, "differ": 1e-3}
    return "exact"


def exact(case, seed):
    """A load's distances in 64 bits.  What a search or a build returns depends on which rows it visits, so it has no
    value apart from the search itself; its distances are the same sums as a load's."""
    if case["kind"] != "load":
        return None
    state = prepare(case, seed)
    vectors, beams = state["vectors"], state["beams"]
    out = torch.empty(beams.shape, dtype=torch.float64, device="cuda")
    step = max(1, 20_000_000 // (case["degree"] * case["dim"]))
    for lo in range(0, case["n"], step):
        rows = vectors[lo:lo + step].double().unsqueeze(1)
        near = vectors[beams[lo:lo + step].long()].double()
        if case["metric"] == "cosine":
            out[lo:lo + step] = ((1.0 - (rows * near).sum(2)) * 0.5).clamp(0.0, 1.0)
        else:
            out[lo:lo + step] = ((rows - near) ** 2).sum(2)
    return out
