"""The query kernel of BM25 and LM against the oracle: corpora around the
chunk sizes (one block, several, several chunks to a block), documents that
tie in whole chunks (so that a top-k selection lists more keys than it has room
for), terms above the number handled at a time, repeated and unordered terms,
k up to the largest."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _corpus(rng, docs, terms, ties):
    if ties:  # term 1 in every document with the same tf, term 2 in every other
        d = np.arange(1, docs + 1)
        rec = [np.stack([d, np.full(docs, 1), np.full(docs, 3)], 1), np.stack([d[::2], np.full(len(d[::2]), 2), np.full(len(d[::2]), 1)], 1)]
        t = rng.integers(3, terms + 1, docs)
        rec.append(np.stack([d, t, np.full(docs, 2)], 1))
    else:
        m = docs * 8
        t = np.minimum((terms * rng.random(m) ** 3).astype(np.int64), terms - 1) + 1
        rec = [np.stack([rng.integers(1, docs + 1, m), t, rng.integers(1, 9, m)], 1)]
    rec = np.concatenate(rec)
    return rec[rng.permutation(len(rec))].astype(np.uint32)


@pytest.mark.parametrize("app", ["bm25", "lm"])
@pytest.mark.parametrize("docs,terms,ties", [(5, 3, False), (900, 124, False), (1024, 200, True), (3000, 150, True),
                                             (20_000, 500, False), (700_000, 90, True)])
def test_queries(gpu, oracle, tmp_path, app, docs, terms, ties):
    rng = np.random.default_rng(docs)
    p = tmp_path / "c.bin"
    _corpus(rng, docs, terms, ties).tofile(p)
    g = gpu.Graph.load_bipartite(p, docs, terms)
    og = oracle.OracleGraph(p, docs, oracle.BIPARTITE | oracle.WEIGHTED, nright=terms)
    b, ob = (gpu.BM25(g), oracle.OracleBM25(og)) if app == "bm25" else (gpu.LM(g), oracle.OracleLM(og))
    some = [int(docs + 1 + t) for t in rng.permutation(terms)]
    for q, k in ((some[:1], 1), (some[:4], 10), ([docs + 1], 64), ([docs + 2, docs + 1], 64), (some[:8] + some[:3], 33),
                 (some[:64], 64), (some[:65], 64), (some + some[:5] + [1, 2], 10), ([3, 1], 7), (some[:2], 0)):
        ids, sc, (alls, act), _ = b.query(q, k, full=True)
        oids, osc, oscores, oact = ob.query(q, k)
        assert ids.tolist() == oids.tolist() and np.array_equal(sc, osc), (q[:9], k)
        assert np.array_equal(act, oact) and np.array_equal(alls.view(np.uint32), oscores.view(np.uint32)), (q[:9], k)
