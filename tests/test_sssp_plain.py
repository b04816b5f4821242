"""SSSP without its ordered copy of the in-edges: where the memory for it is not
there, and in a server, whose budget has not counted it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _graph(weights):
    rng = np.random.default_rng(6)
    n = 6000
    rec = [np.stack([np.full(n // 2, 1), np.arange(2, n + 1, 2)[: n // 2]], 1)]  # the root reaches half at once: pulls follow
    rec += [np.stack([rng.choice(np.arange(50, n + 1), k, replace=False), np.full(k, 2 + i)], 1)
            for i, k in enumerate((1, 15, 16, 17, 255, 256, 257, 513, 3000))]
    rec += [rng.integers(1, n + 1, (9 * n, 2))]
    rec = np.concatenate(rec)
    m = len(rec)
    w = {"small": rng.integers(1, 129, m), "zero": rng.integers(0, 3, m), "wide": rng.integers(1, 1 << 20, m),
         "over": rng.integers(1, 1 << 32, m)}[weights]
    return n, np.concatenate([rec, w[:, None]], 1).astype(np.uint32)


@pytest.mark.parametrize("weights", ["small", "zero", "wide", "over"])
def test_without_memory(gpu, oracle, tmp_path, weights):
    L = gpu
    n, rec = _graph(weights)
    rec.tofile(tmp_path / "g.bin")
    og = oracle.OracleGraph(tmp_path / "g.bin", n, oracle.DIRECTED | oracle.WEIGHTED)
    roots = (1, 2, 10, 999, 0)
    want = {r: og.sssp(r) for r in roots}
    fail = L.N.lib().la3g_fail_allocation
    went_without = 0
    for k in range(60):
        g = L.Graph.from_records(rec, n, L.DIRECTED | L.WEIGHTED)
        fail(k)
        try:
            L.sssp(g, 1)
        except L.N.LA3GError as e:
            assert e.status == 4 and fail(-1) < 0  # LA3G_ENOMEM, before the copy
            continue
        if fail(-1) >= 0:
            break
        went_without += 1
        for r in roots:
            d, st = L.sssp(g, r)
            assert np.array_equal(d, want[r][0]) and st.iterations == want[r][1], (k, r)
    assert went_without >= 3  # the columns' slots, the entries, the sorts' memory


@pytest.mark.parametrize("before", [False, True])
def test_server_orders_nothing(gpu, before):
    L = gpu
    n, rec = _graph("small")
    want = {r: L.sssp(L.Graph.from_records(rec, n, L.DIRECTED | L.WEIGHTED), r)[0] for r in (1, 5, 77)}
    g = L.Graph.from_records(rec, n, L.DIRECTED | L.WEIGHTED)
    if before:
        L.sssp(g, 1)
    S = L.Server(1 << 32)
    gid = S.add_graph(g)
    S.set_solo(16, 16)
    held = g._info().device_bytes
    for r, d in want.items():
        assert np.array_equal(S.poll(S.submit_sssp(gid, r))[1][0], d)
    grown = g._info().device_bytes - held
    S.free()
    assert grown == 0 if before else grown < 60 * g.nslots < 8 * g.info.nentries
