"""Connected components on the shapes that the compressions, the link rounds
and the giant component's sample treat differently, against the oracle: chains
in position order (longer than one compression walks), paths in id and in
random order, many small components, two large ones, a dense one with a fringe,
stars, sizes from one edge up."""
import numpy as np
import pytest

from test_zz_no_alloc import bucket_hash

pytestmark = pytest.mark.gpu


def _path(ids):
    return np.stack([ids[:-1], ids[1:]], 1)


def _graph(kind, n, rng):
    ids = np.arange(1, n + 1)
    if kind == "chain":  # neighbours in position order: every row hooks under the one before
        return _path(ids[np.argsort(bucket_hash(ids, n))])
    if kind == "path":
        return _path(ids)
    if kind == "shuffled":
        return _path(rng.permutation(ids))
    if kind == "pairs":
        p = rng.permutation(ids)
        return np.stack([p[0::2][: n // 2], p[1::2][: n // 2]], 1)
    if kind == "halves":  # two components of the same size, dense
        half = n // 2
        a = rng.integers(1, half + 1, (6 * n, 2))
        a[::2] += half
        return a
    if kind == "fringe":  # a dense component, paths hanging off it, a component aside
        core = rng.integers(1, n // 2 + 1, (6 * n, 2))
        return np.concatenate([core, _path(ids[n // 3: 3 * n // 4]), _path(ids[4 * n // 5:])])
    return np.stack([np.full(n - 1, n // 2 + 1), np.delete(ids, n // 2)], 1)  # star


@pytest.mark.parametrize("kind", ["chain", "path", "shuffled", "pairs", "halves", "fringe", "star"])
@pytest.mark.parametrize("n", [2, 130, 1100, 3000])
def test_components(gpu, oracle, tmp_path, kind, n):
    rec = _graph(kind, n, np.random.default_rng(n)).astype(np.uint32)
    p = tmp_path / "g.bin"
    rec.tofile(p)
    lab, _ = gpu.cc(gpu.Graph.load_undirected(p, n))
    olab, _ = oracle.OracleGraph(p, n, 0).cc()
    assert np.array_equal(lab, olab)
