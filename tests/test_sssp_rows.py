"""SSSP's pull steps against the oracle: rows around the lengths that change
form (a lane group's step, the long rows' tasks), weights that are equal,
spread, wider than the bits the rows are ordered by and near the largest a
pull takes, and graphs whose frontier makes it pull at once."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 3, 4, 15, 16, 17, 31, 33, 63, 64, 65, 127, 128, 129, 255, 256, 257, 511, 512, 513, 769, 1025, 3000]


@pytest.mark.parametrize("weights", ["ones", "small", "zero", "wide", "huge", "over"])
def test_rows(gpu, oracle, tmp_path, weights):
    rng = np.random.default_rng(23)
    n = 9000
    targets = np.arange(2, len(LENGTHS) + 2)
    pool = np.arange(100, n + 1)
    rec = [np.stack([np.full(len(pool[::2]), 1), pool[::2]], 1)]  # the root reaches half of the columns at once
    rec += [np.stack([rng.choice(pool, k, replace=False), np.full(k, t)], 1) for t, k in zip(targets, LENGTHS)]
    rec.append(np.stack([np.repeat(targets, 4), rng.choice(pool, 4 * len(targets))], 1))
    rec.append(rng.integers(1, n + 1, (6 * n, 2)))
    rec = np.concatenate(rec)
    m = len(rec)
    w = {"ones": np.ones(m), "small": rng.integers(1, 129, m), "zero": rng.integers(0, 3, m),
         "wide": rng.integers(1, 200_000, m), "huge": rng.integers(1, (1 << 31) - 5, m),
         "over": rng.integers(1, 1 << 32, m)}[weights]
    rec = np.concatenate([rec, w.astype(np.int64)[:, None]], 1).astype(np.uint32)
    rec = rec[rng.permutation(m)]
    p = tmp_path / "g.bin"
    rec.tofile(p)
    g = gpu.Graph.load_directed(p, n, weighted=True)
    og = oracle.OracleGraph(p, n, oracle.DIRECTED | oracle.WEIGHTED)
    for root in (1, 2, 24, 100, 5000, 0, n + 3):
        d, st = gpu.sssp(g, root)
        od, oit = og.sssp(root)
        assert np.array_equal(d, od) and st.iterations == oit, root
