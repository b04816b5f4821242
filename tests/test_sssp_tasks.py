"""SSSP's pull steps where a hundred warps work on one row and lower its distance
while others read it, against the oracle, run several times."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("weights", ["falling", "random"])
def test_shared_rows(gpu, oracle, tmp_path, weights):
    rng = np.random.default_rng(41)
    n, rows = 60_000, 3
    pool = np.arange(10, n + 1)
    rec = [np.stack([np.full(len(pool), 1), pool], 1)]  # the root reaches every column at once
    rec += [np.stack([rng.permutation(pool), np.full(len(pool), 2 + r)], 1) for r in range(rows)]
    rec.append(np.stack([np.repeat(np.arange(2, 2 + rows), 50), rng.choice(pool, 50 * rows)], 1))
    rec.append(np.stack([pool, np.roll(pool, 1)], 1))
    rec = np.concatenate(rec)
    w = rng.integers(1, 1 << 16, len(rec))
    if weights == "falling":  # a column's message and its edges' weights in opposite order: the minimum lies anywhere
        w = np.where(rec[:, 0] == 1, rec[:, 1], np.where(rec[:, 1] < 10, 2 * n - rec[:, 0] - rng.integers(0, 900, len(rec)), w))
    rec = np.concatenate([rec, w[:, None]], 1).astype(np.uint32)
    p = tmp_path / "g.bin"
    rec.tofile(p)
    g = gpu.Graph.load_directed(p, n, weighted=True)
    for root in (1, 2, 500):
        od, oit = oracle.OracleGraph(p, n, oracle.DIRECTED | oracle.WEIGHTED).sssp(root)
        for _ in range(5):
            d, st = gpu.sssp(g, root)
            assert np.array_equal(d, od) and st.iterations == oit, root
