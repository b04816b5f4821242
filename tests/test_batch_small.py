"""Batches with more roots than the graph has vertices: every root's row equals
the single-root call's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 2, 10, 39])
@pytest.mark.parametrize("nroots", [1, 65, 256, 1024])
def test_more_roots_than_vertices(gpu, n, nroots):
    L = gpu
    rng = np.random.default_rng(n)
    rec = rng.integers(1, n + 1, (3 * n, 3)).astype(np.uint32)
    roots = rng.integers(0, n + 3, nroots).astype(np.uint32)
    g = L.Graph.from_records(rec[:, :2].copy(), n, 0)
    one = {r: L.bfs(g, int(r), want_parent=False)[0] for r in np.unique(roots)}
    assert np.array_equal(L.bfs_batch(g, roots)[0], np.stack([one[r] for r in roots]))
    g = L.Graph.from_records(rec, n, L.DIRECTED | L.WEIGHTED)
    one = {r: L.sssp(g, int(r))[0] for r in np.unique(roots)}
    assert np.array_equal(L.sssp_batch(g, roots)[0], np.stack([one[r] for r in roots]))
