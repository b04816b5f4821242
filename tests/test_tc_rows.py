"""Triangle counts against the oracle where a row changes form: every length
of row and of suffix up to past the longest that a table holds (close ranks:
bitmaps), and long rows whose ranks are far apart (hash tables)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("shape", ["clique", "spread"])
def test_rows(gpu, oracle, tmp_path, shape):
    rng = np.random.default_rng(31)
    if shape == "clique":
        n = 5000
        ids = rng.permutation(n)[:2080] + 1  # rows of 0 .. 2079, ids and ranks in different orders
        a, b = np.triu_indices(len(ids), 1)
        rec = np.concatenate([np.stack([ids[a], ids[b]], 1), rng.integers(1, n + 1, (8 * n, 2))])
    else:
        n = 60_000  # equal degrees: a row of up to 192 reaches almost all ranks
        ids = rng.permutation(n) + 1
        rec = np.concatenate([np.stack([ids, ids[(np.arange(n) + 299 * j) % n]], 1) for j in range(1, 97)])
    flip = rng.random(len(rec)) < 0.5
    rec[flip] = rec[flip][:, ::-1]
    p = tmp_path / "g.bin"
    rec[rng.permutation(len(rec))].astype(np.uint32).tofile(p)
    total, per, _ = gpu.tc(gpu.Graph.load_directed(p, n, remove_cycles=True))
    ototal, oper = oracle.OracleGraph(p, n, oracle.DIRECTED | oracle.ACYCLIC).tc()
    assert total == ototal and np.array_equal(per, oper)
