"""FP64 PageRank's parallel row sums against the oracle's sequential ones, bit
for bit, on rows around the lengths where the kernel changes form and around
its chunk sizes.  Columns have out-degrees of very different size (1, powers
of two, odd numbers), so a row's values span many binades, arrive in any
order and tie often."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

LENGTHS = [1, 2, 7, 63, 64, 65, 66, 127, 255, 256, 257, 300, 511, 513, 1000, 1023, 1024, 1025, 1026, 2047, 2048, 2049,
           2051, 4096, 4097, 9001]


@pytest.mark.parametrize("degrees", ["ones", "powers", "mixed"])
@pytest.mark.parametrize("sinks", [False, True])
def test_row_sums_bit_exact(gpu, oracle, tmp_path, degrees, sinks):
    rng = np.random.default_rng(17)
    n = 16000
    targets = np.arange(1, len(LENGTHS) + 1)
    pool = np.arange(100, n + 1)
    rec = [np.stack([rng.choice(pool, k, replace=False), np.full(k, t)], 1) for t, k in zip(targets, LENGTHS)]
    # more out-edges for the columns, to give them their degrees
    extra = {"ones": np.zeros(len(pool), int), "powers": 2 ** rng.integers(0, 7, len(pool)),
             "mixed": rng.integers(0, 40, len(pool)) ** 2 // 8}[degrees]
    src = np.repeat(pool, extra)
    rec.append(np.stack([src, rng.integers(100, n + 1, len(src))], 1))
    if not sinks:  # the long rows point back: regular rows, their ranks feed the next iteration
        rec.append(np.stack([np.repeat(targets, 3), rng.choice(pool, 3 * len(targets))], 1))
    rec = np.concatenate(rec).astype(np.uint32)
    rec = rec[rng.permutation(len(rec))]
    p = tmp_path / "g.bin"
    rec.tofile(p)
    rank, deg, _ = gpu.pagerank(gpu.Graph.load_directed(p, n), 6)
    orank, odeg = oracle.OracleGraph(p, n, oracle.DIRECTED).pagerank(6)
    assert np.array_equal(deg, odeg)
    assert np.array_equal(rank.view(np.uint64), orank.view(np.uint64))
