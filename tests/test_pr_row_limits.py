"""PageRank on either side of the row count (2^15) at which the limit for a lane's
rows goes from 64 to 256 entries, with rows around both limits: FP64 bit for
bit against the oracle; FP32 against FP64.  An FP32 row adds at most 1024 / 4
numbers in a chain and two more to join the chains, 258 x 2^-24 of relative
error; six iterations, each with two more roundings: below 1.2e-4.  The tiled
form adds a row's numbers in one chain: four times that."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [2, 3, 31, 32, 33, 63, 64, 65, 66, 100, 127, 128, 129, 200, 255, 256, 257, 258, 300, 511, 777, 1023, 1024]


@pytest.mark.parametrize("nrows", [32_767, 32_768, 32_769, 40_000])
def test_row_limits(gpu, oracle, tmp_path, nrows):
    rng = np.random.default_rng(nrows)
    sources = 3000
    n = nrows + sources
    rows = np.arange(1, nrows + 1)
    pool = np.arange(1, n + 1)
    long = np.concatenate([rng.permutation(rows)[: 3 * len(LENGTHS)]])
    rec = [np.stack([rng.choice(pool[pool != t], k, replace=False), np.full(k, t)], 1) for t, k in zip(long, 3 * LENGTHS)]
    rest = np.setdiff1d(rows, long)
    rec.append(np.stack([rng.integers(nrows + 1, n + 1, len(rest)), rest], 1))  # each row has an entry
    rec.append(np.stack([rng.integers(1, nrows + 1, 2 * nrows), rng.choice(rest, 2 * nrows)], 1))
    rec.append(np.stack([pool[nrows:], rng.choice(rest, sources)], 1))
    rec = np.concatenate(rec).astype(np.uint32)
    rec = rec[rng.permutation(len(rec))]
    rec.tofile(tmp_path / "g.bin")
    g = gpu.Graph.load_directed(tmp_path / "g.bin", n)
    assert g.info.nregular + g.info.nsink == nrows and g.info.nregular > 1000 and g.info.nsink > 1000
    rank, deg, _ = gpu.pagerank(g, 6)
    orank, odeg = oracle.OracleGraph(tmp_path / "g.bin", n, oracle.DIRECTED).pagerank(6)
    assert np.array_equal(deg, odeg)
    assert np.array_equal(rank.view(np.uint64), orank.view(np.uint64))
    for tiled in (False, True):
        assert np.allclose(gpu.pagerank_f32(g, 6, tiled=tiled)[0], orank, rtol=1.2e-4 if not tiled else 4 * 1.2e-4, atol=0)
