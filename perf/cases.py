"""The calls whose time is watched, over the range of sizes they are made with.

Every case is one public entry point as a program uses it: the graph (or
corpus) is loaded beforehand and kept, the call is made with a root, a batch
of roots or a list of queries, and its results come back as the entry point
returns them.  Inputs are drawn on the GPU from the seed: R-MAT graphs
(0.57 / 0.19 / 0.19) and Erdos-Renyi graphs with shuffled ids and weights 1 to
128, and a Zipf corpus, as the benchmark's generators draw them; records carry
the duplicates and self-loops that edge files carry.
"""
import ctypes
import math

import numpy as np
import torch

import la3_gb300 as la3


def _rmat(nodes, edges, kind="rmat"):
    return {"nodes": nodes, "edges": edges, "graph": kind}


def listed():
    return [
        # one small graph queried on its own: latency and launches count
        {"name": "bfs_rmat_4k", "app": "bfs", "parents": True, **_rmat(1 << 12, 8 << 12)},
        # the benchmark's BFS, hop counts only
        {"name": "bfs_rmat_4m", "app": "bfs", "parents": False, **_rmat(1 << 22, 16 << 22)},
        # a caller that owns all device memory: CSR in, device arrays out
        {"name": "bfs_device_rmat_200k", "app": "bfs_device", **_rmat(200_003, 3_200_048)},
        # the benchmark's SSSP, distances to the host
        {"name": "sssp_rmat_4m", "app": "sssp", **_rmat(1 << 22, 16 << 22)},
        # the benchmark's connected components, labels to the host
        {"name": "cc_rmat_4m", "app": "cc", **_rmat(1 << 22, 16 << 22)},
        # the benchmark's triangle count, total and per-vertex counts
        {"name": "tc_rmat_1m", "app": "tc", **_rmat(1 << 20, 16 << 20)},
        # the FP64 PageRank configuration (20 iterations, reference summation order)
        {"name": "pagerank_f64_rmat_64k", "app": "pagerank", "dtype": "f64", "tiled": False, "iters": 20,
         **_rmat(1 << 16, 16 << 16)},
        # the FP32 form on a large graph, until it has settled
        {"name": "pagerank_f32_rmat_4m", "app": "pagerank", "dtype": "f32", "tiled": False, "iters": 50,
         **_rmat(1 << 22, 16 << 22)},
        # many-source sweeps (distance sketches, centrality samples)
        {"name": "bfs_batch_rmat_256k", "app": "bfs_batch", "roots": 64, **_rmat(1 << 18, 16 << 18)},
        {"name": "sssp_batch_er_50k", "app": "sssp_batch", "roots": 64, **_rmat(50_021, 800_336, "er")},
        # a file of search queries answered one after another, top 10 each
        {"name": "bm25_500k_docs", "app": "bm25", "docs": 500_000, "terms": 62_500, "doc_terms": 50, "queries": 16,
         "k": 10},
        # loading a weighted directed edge list that is in host memory
        {"name": "load_rmat_1m", "app": "load", **_rmat(1 << 20, 16 << 20)},
    ]


def draw(rng):
    def size(lo, hi):
        return int(round(2.0 ** rng.uniform(math.log2(lo), math.log2(hi))))

    def graph(lo, hi):
        n = size(lo, hi)
        return _rmat(n, n * rng.choice((8, 12, 16)) + rng.randrange(8), rng.choice(("rmat", "rmat", "er")))

    app = rng.choice(("bfs", "bfs_device", "sssp", "cc", "tc", "pagerank", "pagerank", "bfs_batch", "sssp_batch", "bm25",
                      "load"))
    if app == "bfs":
        return {"app": app, "parents": rng.random() < 0.5, **graph(1 << 10, 1 << 22)}
    if app == "bfs_device":
        return {"app": app, **graph(1 << 10, 1 << 20)}
    if app in ("sssp", "cc"):
        return {"app": app, **graph(1 << 12, 1 << 22)}
    if app == "tc":
        return {"app": app, **graph(1 << 12, 1 << 20)}
    if app == "pagerank":
        dtype = rng.choice(("f64", "f64", "f32"))
        return {"app": app, "dtype": dtype, "tiled": dtype == "f32" and rng.random() < 0.5,
                "iters": rng.choice((10, 20, 50)), **graph(1 << 12, 1 << 20 if dtype == "f64" else 1 << 22)}
    if app == "bfs_batch":
        return {"app": app, "roots": rng.choice((16, 64, 100, 256)), **graph(1 << 12, 1 << 18)}
    if app == "sssp_batch":
        return {"app": app, "roots": rng.choice((16, 64, 100)), **graph(1 << 12, 1 << 16)}
    if app == "bm25":
        docs = size(10_000, 500_000)
        return {"app": app, "docs": docs, "terms": max(2000, docs // 8), "doc_terms": rng.choice((30, 50)),
                "queries": rng.choice((4, 16)), "k": rng.choice((10, 10, 50))}
    return {"app": app, **graph(1 << 12, 1 << 20)}


# -- inputs ---------------------------------------------------------------------


def _generator(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed) & 0x7FFFFFFFFFFF)


def _edges(case, seed):
    """Edge list on the GPU: ids 1..nodes, int64 src / dst, int64 weights 1..128."""
    g = _generator(seed)
    n, m = case["nodes"], case["edges"]

    if case["graph"] == "er":
        src = torch.randint(1, n + 1, (m,), generator=g, device="cuda")
        dst = torch.randint(1, n + 1, (m,), generator=g, device="cuda")
    else:
        scale = max(1, math.ceil(math.log2(n)))
        src = torch.zeros(m, dtype=torch.int32, device="cuda")
        dst = torch.zeros(m, dtype=torch.int32, device="cuda")
        for _ in range(scale):
            r = torch.rand(m, generator=g, device="cuda")
            down = r >= 0.76
            src.mul_(2).add_(down)
            dst.mul_(2).add_(((r >= 0.57) & ~down) | (r >= 0.95))
        shuffle = torch.randperm(n, generator=g, device="cuda") + 1
        src, dst = shuffle[(src.long() * n) >> scale], shuffle[(dst.long() * n) >> scale]
    w = torch.randint(1, 129, (m,), generator=g, device="cuda")
    return src, dst, w


def _records(case, seed, weighted):
    src, dst, w = _edges(case, seed)
    cols = [src, dst, w] if weighted else [src, dst]
    return torch.stack([c.to(torch.int32) for c in cols], 1).cpu().numpy().view(np.uint32)


def _file_records(case, seed):
    """The records of a weighted edge file: `edges` different edges and, among
    them, a 32nd as many again with another weight (the first one counts)."""
    n, m = case["nodes"], case["edges"]
    src, dst, _ = _edges({**case, "edges": 2 * m}, seed)
    g = _generator(seed + 1)
    pairs = torch.unique((src * (n + 1) + dst)[src != dst])
    pairs = pairs[torch.randperm(len(pairs), generator=g, device="cuda")[:m]]
    if len(pairs) < m:
        raise ValueError("too few different edges for %r" % (case,))
    pairs = torch.cat([pairs, pairs[torch.randint(0, m, (m // 32,), generator=g, device="cuda")]])
    pairs = pairs[torch.randperm(len(pairs), generator=g, device="cuda")]
    w = torch.randint(1, 129, (len(pairs),), generator=g, device="cuda")
    return torch.stack([pairs // (n + 1), pairs % (n + 1), w], 1).to(torch.int32).cpu().numpy().view(np.uint32)


FLAGS = {"bfs": 0, "cc": 0, "bfs_batch": 0, "sssp": la3.DIRECTED | la3.WEIGHTED,
         "sssp_batch": la3.DIRECTED | la3.WEIGHTED, "tc": la3.DIRECTED | la3.ACYCLIC, "pagerank": la3.DIRECTED}


def _roots(graph, seed, count):
    """Vertices with out-edges (regular ones): a root elsewhere reaches nothing."""
    _, ids = graph.positions()
    at = np.random.RandomState(seed & 0x7FFFFFFF).randint(0, graph.info.nregular, count)
    return ids[at]


def _hashed(n):
    """The hashed id of every vertex id 0..n (the order BFS parents are chosen in)."""
    ids = torch.arange(n + 1, device="cuda")
    height = n // 128
    return torch.where(ids >= height * 128, ids, ids // 128 + (ids % 128) * height)


def _device_csr(case, seed):
    src, dst, _ = _edges(case, seed)
    slots = case["nodes"] + 1
    key = _hashed(case["nodes"])
    keep = src != dst
    src, dst = src[keep], dst[keep]
    pairs = torch.unique(torch.cat([src * slots + key[dst], dst * slots + key[src]]))
    id_of_key = torch.empty_like(key)
    id_of_key[key] = torch.arange(slots, device="cuda")
    rows, cols = pairs // slots, id_of_key[pairs % slots]
    ptr = torch.zeros(slots + 1, dtype=torch.int64, device="cuda")
    ptr[1:] = torch.bincount(rows, minlength=slots).cumsum(0)
    return ptr.to(torch.int32), cols.to(torch.int32), key.to(torch.int32), int(rows[len(rows) // 3])


def _corpus(case, seed):
    """(doc, term, tf) postings on the GPU, no (doc, term) twice, and the queries' term ids (1-based)."""
    g = _generator(seed)
    docs, terms, mean = case["docs"], case["terms"], case["doc_terms"]
    lengths = torch.randint(mean // 2, mean // 2 + mean + 1, (docs,), generator=g, device="cuda")
    doc = torch.repeat_interleave(torch.arange(docs, device="cuda"), lengths)
    p = torch.arange(1, terms + 1, device="cuda", dtype=torch.float64) ** -1.1
    cdf = (p / p.sum()).cumsum(0)
    name = torch.randperm(terms, generator=g, device="cuda")

    def zipf(count):
        u = torch.rand(count, generator=g, device="cuda", dtype=torch.float64)
        return name[torch.searchsorted(cdf, u).clamp_(max=terms - 1)]

    pairs = torch.unique(doc * terms + zipf(len(doc)))
    doc, term = pairs // terms, pairs % terms
    # terms in nearly every document are thinned to below 0.9 of them
    df = torch.bincount(term, minlength=terms)
    cap = 0.9 * docs
    chance = torch.where(df >= cap, 0.95 * cap / df.clamp(min=1).double(), 1.0)
    keep = torch.rand(len(term), generator=g, device="cuda", dtype=torch.float64) < chance[term]
    doc, term = doc[keep], term[keep]
    tf = 1 + (-torch.log2(torch.rand(len(doc), generator=g, device="cuda").clamp_(min=1e-6))).long().clamp_(max=6)
    asked = zipf(8 * case["queries"]).cpu().numpy().reshape(case["queries"], 8)
    sizes = np.random.RandomState(seed & 0x7FFFFFFF).randint(2, 9, case["queries"])
    queries = [sorted(set(int(t) + 1 for t in row[:k])) for row, k in zip(asked, sizes)]
    return doc + 1, term + 1, tf, queries


def prepare(case, seed):
    app = case["app"]
    if app == "bfs_device":
        ptr, col, key, root = _device_csr(case, seed)
        slots = case["nodes"] + 1
        return {"case": case, "ptr": ptr, "col": col, "key": key, "root": root,
                "hops": torch.empty(slots, dtype=torch.uint8, device="cuda"),
                "parent": torch.empty(slots, dtype=torch.int32, device="cuda")}
    if app == "bm25":
        doc, term, tf, queries = _corpus(case, seed)
        records = torch.stack([doc, term, tf], 1).to(torch.int32).cpu().numpy().view(np.uint32)
        graph = la3.Graph.from_records(records, case["docs"], la3.BIPARTITE | la3.WEIGHTED, case["terms"])
        return {"case": case, "index": la3.BM25(graph), "queries": [[case["docs"] + t for t in q] for q in queries]}
    if app == "load":
        return {"case": case, "records": _file_records(case, seed)}
    flags = FLAGS[app]
    graph = la3.Graph.from_records(_records(case, seed, bool(flags & la3.WEIGHTED)), case["nodes"], flags)
    state = {"case": case, "graph": graph}
    if app in ("bfs", "sssp"):
        state["root"] = int(_roots(graph, seed, 1)[0])
    elif app in ("bfs_batch", "sssp_batch"):
        state["roots"] = _roots(graph, seed, case["roots"])
    return state


# -- one pass -------------------------------------------------------------------


class _DeviceArray:
    """A graph's device array as torch sees it; keeps the graph alive."""

    def __init__(self, graph, address, count):
        self.graph = graph
        self.__cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (address, False), "version": 2}


def _load(case, records):
    graph = la3.Graph.from_records(records, case["nodes"], la3.DIRECTED | la3.WEIGHTED)
    view = la3.N.DeviceGraph()
    la3.N.check(la3.N.lib().la3g_graph_device_view(graph._h, ctypes.byref(view)))
    pos, ids = graph.positions()
    arrays = [torch.as_tensor(_DeviceArray(graph, a, c), device="cuda")
              for a, c in ((view.row_ptr, view.nslots + 1), (view.col, view.nentries), (view.weight, view.nentries))]
    return _whole(pos), _whole(ids), arrays


def _whole(a):
    """uint32 ids, labels and distances as int32 (the same bytes; none here passes 2^31)."""
    return a.view(np.int32)


def run(state):
    case = state["case"]
    app = case["app"]
    if app == "bfs":
        hops, parent, _ = la3.bfs(state["graph"], state["root"], want_parent=case["parents"])
        return hops, _whole(parent) if case["parents"] else None
    if app == "bfs_device":
        stats = la3.Stats()
        la3.N.check(la3.N.lib().la3g_bfs_noalloc(
            state["ptr"].data_ptr(), state["col"].data_ptr(), state["key"].data_ptr(), case["nodes"] + 1, state["root"],
            state["hops"].data_ptr(), state["parent"].data_ptr(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream), ctypes.byref(stats)))
        return state["hops"], state["parent"]
    if app == "sssp":
        return _whole(la3.sssp(state["graph"], state["root"])[0])
    if app == "cc":
        return _whole(la3.cc(state["graph"])[0])
    if app == "tc":
        total, counts, _ = la3.tc(state["graph"])
        return total, _whole(counts)
    if app == "pagerank" and case["dtype"] == "f64":
        rank, degree, _ = la3.pagerank(state["graph"], case["iters"])
        return rank, _whole(degree)
    if app == "pagerank":
        rank, _, _ = la3.pagerank_f32(state["graph"], case["iters"], tiled=case["tiled"])
        return rank
    if app == "bfs_batch":
        return la3.bfs_batch(state["graph"], state["roots"])[0]
    if app == "sssp_batch":
        return _whole(la3.sssp_batch(state["graph"], state["roots"])[0])
    if app == "bm25":
        found = [state["index"].query(q, case["k"]) for q in state["queries"]]
        return [(_whole(ids), scores) for ids, scores, _, _ in found]
    return _load(case, state["records"])


def work(case):
    """Bytes and operations one pass cannot do without (edges and outputs
    counted as drawn; a few per cent of them are duplicates)."""
    app = case["app"]
    if app == "bm25":
        # 5 terms a query; a Zipf 1.1 term drawn by its own frequency is in about a fifth of the documents
        postings = case["queries"] * 5 * 0.2 * case["docs"]
        return {"bytes": 12.0 * postings, "flops": 5.0 * postings}
    n, m = case["nodes"], case["edges"]
    if app == "bfs":
        # row offsets and one neighbour of every vertex, then the outputs
        return {"bytes": 8.0 * n + (5.0 if case["parents"] else 1.0) * n, "flops": 0.0}
    if app == "bfs_device":
        return {"bytes": 13.0 * n, "flops": 0.0}
    if app == "sssp":
        return {"bytes": 8.0 * m + 8.0 * n, "flops": 0.0}
    if app == "cc":
        return {"bytes": 8.0 * n + 4.0 * n, "flops": 0.0}
    if app == "tc":
        # the edges, and the closing list of each
        return {"bytes": 12.0 * m + 8.0 * n, "flops": 0.0}
    if app == "pagerank":
        b = 8 if case["dtype"] == "f64" else 4
        return {"bytes": float(case["iters"]) * (4 * m + (4 + 3 * b) * n) + 12 * n, "flops": float(case["iters"]) * (m + 3 * n)}
    if app == "bfs_batch":
        words = -(-case["roots"] // 64)
        return {"bytes": 8.0 * m + 16.0 * words * n + 1.0 * case["roots"] * n, "flops": 0.0}
    if app == "sssp_batch":
        return {"bytes": 8.0 * m + 8.0 * case["roots"] * n, "flops": 0.0}
    return {"bytes": 12.0 * m + 8.0 * m + 12.0 * n, "flops": 0.0}


# -- the same in 64 bits --------------------------------------------------------


def _exact_pagerank(case, seed):
    n, alpha = case["nodes"], 0.15
    src, dst, _ = _edges(case, seed)
    keep = src != dst
    pairs = torch.unique(src[keep] * (n + 1) + dst[keep])
    src, dst = pairs // (n + 1), pairs % (n + 1)
    degree = torch.bincount(src, minlength=n + 1).double()
    rank = torch.full((n + 1,), alpha, dtype=torch.float64, device="cuda")

    def step(r):
        x = torch.where(degree > 0, r / degree.clamp(min=1), 0.0)
        return alpha + (1 - alpha) * torch.zeros_like(r).index_add_(0, dst, x[src])

    for _ in range(case["iters"]):
        rank = step(rank)
    # vertices without out-edges take one more step, from the final ranks
    rank = torch.where(degree > 0, rank, step(rank))
    return rank.cpu().numpy()


def _exact_bm25(case, seed):
    doc, term, tf, queries = _corpus(case, seed)
    docs, terms = case["docs"], case["terms"]
    df = torch.bincount(term, minlength=terms + 1).double()
    idf = torch.log10((docs - df + 0.5) / (df + 0.5))
    length = torch.zeros(docs + 1, dtype=torch.float64, device="cuda").index_add_(0, doc, tf.double())
    # the token count takes every vertex's value, the terms' truncated idf among them
    tokens = length.sum() + torch.where((df > 0) & (idf > 0), idf.floor(), 0.0).sum()
    k = 1.2 * (0.25 + 0.75 * length / (tokens / docs))
    answers = []
    for q in queries:
        score = torch.zeros(docs + 1, dtype=torch.float64, device="cuda")
        seen = torch.zeros(docs + 1, dtype=torch.bool, device="cuda")
        for t in q:
            at = torch.nonzero(term == t).squeeze(1)
            d, f = doc[at], tf[at].double()
            score[d] += f * 2.2 / (f + k[d]) * idf[t]
            seen[d] = True
        best = score[seen].sort(descending=True).values[: case["k"]]
        answers.append((None, best.cpu().numpy()))
    return answers


def exact(case, seed):
    if case["app"] == "pagerank":
        rank = _exact_pagerank(case, seed)
        return (rank, None) if case["dtype"] == "f64" else rank
    if case["app"] == "bm25":
        return _exact_bm25(case, seed)
    return None
