"""Calls during which a device allocation fails: each of the call's allocations in
turn, on a graph on which nothing was called yet.  The call returns LA3G_ENOMEM
(or does without), and so does a second one; made again with memory there, it
returns what it returns on a graph that never saw the failure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENOMEM = 4


def _same(a, b):
    return all(x == y if isinstance(x, int) else np.array_equal(x, y) for x, y in zip(a, b, strict=True))


def _each(L, make, call, same=_same):
    """Returns how many allocations the call makes."""
    fail = L.N.lib().la3g_fail_allocation
    want = call(make())
    for n in range(200):
        g = make()
        done = False
        for again in (False, True):
            fail(n)
            try:
                got = call(g)
            except L.N.LA3GError as e:
                assert e.status == ENOMEM, e
                assert fail(-1) < 0
            else:
                done |= fail(-1) >= 0 and not again
                assert same(got, want), n
        assert same(call(g), want), n
        if done:
            return n
    raise AssertionError("too many allocations")


@pytest.fixture(scope="module")
def records():
    rng = np.random.default_rng(2)
    n = 3000
    rec = rng.integers(1, n + 1, (9 * n, 3)).astype(np.uint32)
    rec[:700, 1] = 5  # a row that SSSP's pull and PageRank cut up
    rec[:1500, 0] = rng.permutation(n)[:1500] + 1
    zero = rec.copy()
    zero[0, :2] = 0, 9
    return n, rec, zero


@pytest.mark.parametrize("case", ["bfs", "cc", "cc_zero", "sssp", "tc", "pagerank", "pagerank_f32", "bfs_batch", "sssp_batch",
                                  "sssp_batch_huge"])
def test_graph_calls(gpu, records, case):
    L = gpu
    n, rec, zero = records
    pairs = np.ascontiguousarray(rec[:, :2])
    roots = np.arange(1, 130, dtype=np.uint32)
    graph = {
        "bfs": (pairs, 0), "bfs_batch": (pairs, 0), "cc": (pairs, 0), "cc_zero": (np.ascontiguousarray(zero[:, :2]), 0),
        "tc": (pairs, L.DIRECTED | L.ACYCLIC), "pagerank": (pairs, L.DIRECTED), "pagerank_f32": (pairs, L.DIRECTED),
    }.get(case, (rec, L.DIRECTED | L.WEIGHTED))
    if case == "sssp_batch_huge":  # weights that make the batch run its roots one by one
        graph = rec * np.array([1, 1, 1 << 19], np.uint32), graph[1]
        roots = roots[:3]
    call = {
        "bfs": lambda g: L.bfs(g, 7)[:2], "cc": lambda g: L.cc(g)[:1], "cc_zero": lambda g: L.cc(g)[:1],
        "sssp": lambda g: L.sssp(g, 7)[:1], "tc": lambda g: L.tc(g)[:2], "pagerank": lambda g: L.pagerank(g, 3)[:2],
        "pagerank_f32": lambda g: L.pagerank_f32(g, 3)[:1], "bfs_batch": lambda g: L.bfs_batch(g, roots)[:1],
    }.get(case, lambda g: L.sssp_batch(g, roots)[:1])
    assert _each(L, lambda: L.Graph.from_records(graph[0], n, graph[1]), call) > 0


def test_tiled_pagerank(gpu, records):
    """Its rows are FP32 sums in any order: of at most 1024 positive numbers each,
    1023 x 2^-24 of relative difference, three iterations (and the long rows', in
    fixed order) below 2e-4."""
    L = gpu
    n, rec, _ = records
    calls = _each(L, lambda: L.Graph.from_records(np.ascontiguousarray(rec[:, :2]), n, L.DIRECTED),
                  lambda g: [L.pagerank_f32(g, 3, tiled=True)[0]], lambda a, b: np.allclose(a[0], b[0], rtol=2e-4, atol=0))
    assert calls > 0


def test_growing_batches(gpu, records):
    """A batch that cannot get larger buffers leaves the ones that smaller batches use."""
    L = gpu
    n, rec, _ = records
    few, many = np.arange(1, 20, dtype=np.uint32), np.arange(1, 300, dtype=np.uint32)
    fail = L.N.lib().la3g_fail_allocation
    for flags, data, call in ((0, np.ascontiguousarray(rec[:, :2]), L.bfs_batch),
                              (L.DIRECTED | L.WEIGHTED, rec, L.sssp_batch)):
        ref = L.Graph.from_records(data, n, flags)
        want = {len(r): call(ref, r)[0] for r in (few, many)}
        for k in range(200):
            g = L.Graph.from_records(data, n, flags)
            call(g, few)
            fail(k)
            try:
                assert np.array_equal(call(g, many)[0], want[len(many)])
            except L.N.LA3GError as e:
                assert e.status == ENOMEM
            done = fail(-1) >= 0
            for r in (few, many, few):
                assert np.array_equal(call(g, r)[0], want[len(r)]), (k, len(r))
            if done:
                break


@pytest.mark.parametrize("app", ["bm25", "lm"])
def test_queries(gpu, app):
    L = gpu
    rng = np.random.default_rng(4)
    docs, terms = 500, 150
    rec = np.stack([rng.integers(1, docs + 1, 6000), rng.integers(1, terms + 1, 6000), rng.integers(1, 9, 6000)], 1)
    rec = rec.astype(np.uint32)
    longer = docs + 1 + rng.permutation(terms)[:90]  # above the terms that go by value
    make = L.BM25 if app == "bm25" else L.LM

    def call(g):
        q = make(g)
        return [x for t in (longer[:3], longer, longer[:3]) for x in q.query(t, 10)[:2]]

    assert _each(L, lambda: L.Graph.from_records(rec, docs, L.BIPARTITE | L.WEIGHTED, terms), call) > 0


@pytest.mark.parametrize("weighted", [False, True])
def test_push_view(gpu, records, weighted):
    """The push CSR: built on demand, whole or not at all."""
    import ctypes as C

    import torch
    L = gpu
    n, rec, _ = records
    data = rec if weighted else np.ascontiguousarray(rec[:, :2])

    def array(address, count):
        class A:
            __cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (address, False), "version": 2}
        return torch.as_tensor(A(), device="cuda").cpu().numpy()

    def call(g):
        ptr, row = C.c_void_p(), C.c_void_p()
        L.N.check(L.N.lib().la3g_graph_push_view(g._h, C.byref(ptr), C.byref(row)))
        assert ptr.value and row.value
        return array(ptr.value, g.nslots + 1), array(row.value, g.info.nentries)

    make = lambda: L.Graph.from_records(data, n, L.DIRECTED | (L.WEIGHTED if weighted else 0))
    assert _each(L, make, call) > 0


def test_loads(gpu, records):
    L = gpu
    n, rec, _ = records
    fail = L.N.lib().la3g_fail_allocation
    for flags in (0, L.DIRECTED | L.WEIGHTED):
        data = rec if flags else np.ascontiguousarray(rec[:, :2])
        want = L.Graph.from_records(data, n, flags).positions()
        for k in range(50):
            fail(k)
            try:
                got = L.Graph.from_records(data, n, flags)
            except L.N.LA3GError as e:
                assert e.status == ENOMEM
            else:
                break
            finally:
                left = fail(-1)
        assert k and left >= 0 and _same(got.positions(), want)
