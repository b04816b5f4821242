"""Grid-barrier waits of the single-root BFS and SSSP: whatever the limit, a call
either says that a wait ran out or returns the whole result, and the next call
on the same graph is right again."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ETIMEOUT = 6


@pytest.mark.parametrize("app", ["bfs", "sssp"])
@pytest.mark.parametrize("scale", [12, 16])
def test_runs_out_or_is_whole(gpu, app, scale):
    L = gpu
    g = L.Graph.from_edges(L.EdgeList.rmat(scale, 8, seed=5, weighted=app == "sssp", wseed=2),
                           0 if app == "bfs" else L.DIRECTED | L.WEIGHTED)
    run = (lambda r: L.bfs(g, r)[:2]) if app == "bfs" else (lambda r: L.sssp(g, r)[:1])
    roots = g.positions()[1][[0, g.info.nregular // 3, g.info.nregular - 1]].tolist()  # each reaches other vertices first
    want = [run(r) for r in roots]
    ran_out = whole = 0
    for polls in list(range(0, 130)) + list(range(130, 2000, 31)):
        g.set_wait_limit(polls)
        for r, x in zip(roots, want):
            try:
                got = run(r)
            except L.N.LA3GError as e:
                assert e.status == ETIMEOUT, e
                ran_out += 1
            else:
                assert all(np.array_equal(a, b) for a, b in zip(got, x)), (polls, r)
                whole += 1
    assert ran_out and whole
    g.set_wait_limit()
    assert all(np.array_equal(a, b) for r, x in zip(roots, want) for a, b in zip(run(r), x))


def test_runs_out_in_the_last_level(gpu):
    """A clique reached in one level, and a hub that its vertices do not reach:
    the last level looks at all of the hub's neighbours, in the first block,
    while the others wait.  The first block must not go on alone."""
    L = gpu
    k, b, hub = 512, 1 << 20, 128  # the smallest hashed id with edges
    clique = np.arange(1000, 1000 + k, dtype=np.uint32)
    leaves = np.arange(2000, 2000 + b, dtype=np.uint32)
    i, j = np.triu_indices(k, 1)
    rec = np.concatenate([np.stack([clique[i], clique[j]], 1), np.stack([np.full(k, 1, np.uint32), clique], 1),
                          np.stack([np.full(b, hub, np.uint32), leaves], 1)])
    g = L.Graph.from_records(rec, 2000 + b, 0)
    hops = np.full(g.nslots, 255, np.uint8)
    hops[1], hops[clique] = 0, 1
    far = np.full(g.nslots, 255, np.uint8)
    far[hub], far[leaves], far[2000] = 1, 2, 0
    for polls in (50_000, -1, 50_000):
        g.set_wait_limit()
        assert np.array_equal(L.bfs(g, 2000)[0], far)
        g.set_wait_limit(polls)
        if polls < 0:
            assert np.array_equal(L.bfs(g, 1)[0], hops)
            continue
        with pytest.raises(L.N.LA3GError) as e:
            L.bfs(g, 1)
        assert e.value.status == ETIMEOUT


def test_long_sink_is_waited_for(gpu):
    """One lane walks the in-edges of a sink (seconds): slow, but an answer."""
    L = gpu
    m = (1 << 24) - 1
    i = np.arange(2, m + 2, dtype=np.uint32)
    rec = np.full((3 * m, 3), 7, np.uint32)
    rec[:m, 0], rec[:m, 1] = 1, i
    rec[m: 2 * m, 0], rec[m: 2 * m, 1] = i, 1  # regular vertices: their distances are looked up
    rec[2 * m:, 0], rec[2 * m:, 1] = i, m + 2
    g = L.Graph.from_records(rec, m + 2, L.DIRECTED | L.WEIGHTED)
    want = np.full(m + 3, 7, np.uint32)
    want[[0, 1, m + 2]] = 0x7FFFFFFF, 0, 14
    assert np.array_equal(L.sssp(g, 1)[0], want)


def test_long_unreached_hub_is_waited_for(gpu):
    """One lane looks through all neighbours of a hub that the root does not reach."""
    L = gpu
    k, m, b = 64, 98_304, 36 << 20
    mid = np.arange(2, 2 + k, dtype=np.uint32)
    leaf = np.arange(2 + k, 2 + k + m, dtype=np.uint32)
    hub = 2 + k + m
    rec = np.concatenate([np.stack([np.full(k, 1, np.uint32), mid], 1), np.stack([np.repeat(mid, m), np.tile(leaf, k)], 1),
                          np.stack([np.full(b, hub, np.uint32), np.arange(hub + 1, hub + 1 + b, dtype=np.uint32)], 1)])
    g = L.Graph.from_records(rec, hub + b, 0)
    want = np.full(g.nslots, 255, np.uint8)
    want[1], want[mid], want[leaf] = 0, 1, 2
    hops, _, st = L.bfs(g, 1, want_parent=False)
    assert st.pull_iterations > 0 and np.array_equal(hops, want)
