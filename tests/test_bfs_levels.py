"""The one-kernel BFS at the places where its levels change form, against the
oracle, in both its entry points: roots and vertices with as many edges as a
small / hub vertex may have and one more, hubs found top-down and bottom-up,
switches in both directions, more levels than a byte of hops holds (where hop
counts wrap and vertices are visited again), sizes around a bitmap word."""
import ctypes as C

import numpy as np
import pytest

from test_zz_no_alloc import bucket_hash, csr_by_key

pytestmark = pytest.mark.gpu


def _star(centre, leaves):
    return [np.stack([np.full(len(leaves), centre), leaves], 1)]


def _path(ids):
    return [np.stack([ids[:-1], ids[1:]], 1)]


def _graph(kind, rng):
    if kind.startswith("star"):  # a centre with exactly that many edges, and one chord
        k = int(kind[4:])
        return k + 1, _star(1, np.arange(2, k + 2)) + [np.array([[2, min(3, k + 1)]])], [1, 2, k + 1]
    if kind == "hubs":  # three hubs in a row, each with leaves of its own, and a tail
        a = _star(1, np.arange(10, 700)) + _star(2, np.arange(700, 2900)) + _star(3, np.arange(2900, 3400))
        return 3500, a + [np.array([[1, 2], [2, 3], [3, 4], [4, 5], [3399, 3450]])], [1, 5, 10, 3450, 3500]
    if kind == "words":  # 33 vertices, dense
        return 33, [rng.integers(1, 34, (120, 2))], [1, 32, 33]
    if kind == "sparse":  # long thin components, some dense parts
        return 5000, [rng.integers(1, 5001, (6000, 2)), rng.integers(1, 60, (900, 2))], [1, 7, 2500, 4999]
    if kind == "deep":  # a path past the last hop a byte holds, a dense part at its end, a cycle back
        ids = np.arange(1, 600)
        blob = np.arange(600, 1800)
        dense = blob[rng.integers(0, len(blob), (9000, 2))]
        return 1800, _path(ids) + [dense, np.array([[599, 600], [598, 610], [256, 700]])], [1, 2, 599, 700, 1799]
    if kind == "deep_hub":  # a hub exactly at the depths where hops wrap
        ids = np.arange(1, 300)
        return 3000, _path(ids) + _star(254, np.arange(300, 1000)) + _star(255, np.arange(1000, 1700)) + _star(
            257, np.arange(1700, 2500)) + [np.array([[300, 1000], [1001, 1700]])], [1, 2, 3, 299]
    raise ValueError(kind)


@pytest.mark.parametrize("kind", ["star1", "star511", "star512", "star513", "star1024", "star1025", "star5000", "hubs",
                                  "words", "sparse", "deep", "deep_hub"])
def test_levels(gpu, oracle, tmp_path, kind):
    import torch
    rng = np.random.default_rng(5)
    n, rec, roots = _graph(kind, rng)
    rec = np.concatenate(rec).astype(np.uint32)
    p = tmp_path / "g.bin"
    rec.tofile(p)
    g = gpu.Graph.load_undirected(p, n)
    og = oracle.OracleGraph(p, n, 0)
    key = bucket_hash(np.arange(n + 1), n)
    ptr, col = csr_by_key(rec[:, 0], rec[:, 1], n + 1, key)
    dev = [torch.from_numpy(a.view(np.int32)).cuda() for a in (ptr, col, key)]
    hops = torch.empty(n + 1, dtype=torch.uint8, device="cuda")
    parent = torch.empty(n + 1, dtype=torch.int32, device="cuda")
    for root in roots + [0, n + 7]:
        h, par, st = gpu.bfs(g, root)
        oh, opar, oit = og.bfs(root)
        assert np.array_equal(h, oh) and np.array_equal(par, opar) and st.iterations == oit, root
        only, _, _ = gpu.bfs(g, root, want_parent=False)
        assert np.array_equal(only, oh), root
        st = gpu.Stats()
        gpu.N.check(gpu.N.lib().la3g_bfs_noalloc(*(t.data_ptr() for t in dev), n + 1, root, hops.data_ptr(), parent.data_ptr(),
                                                 C.c_void_p(torch.cuda.current_stream().cuda_stream), C.byref(st)))
        assert np.array_equal(hops.cpu().numpy(), oh) and np.array_equal(parent.cpu().numpy().view(np.uint32), opar), root
        assert st.iterations == oit, root


@pytest.mark.parametrize("n", [32766, 32767, 32768, 32769])
def test_small_outputs(gpu, oracle, tmp_path, n):
    """Outputs written to host memory by the kernel, up to a size, else copied."""
    rec = np.random.default_rng(9).integers(1, n + 1, (3 * n, 2)).astype(np.uint32)
    p = tmp_path / "g.bin"
    rec.tofile(p)
    g = gpu.Graph.load_undirected(p, n)
    og = oracle.OracleGraph(p, n, 0)
    for root in (1, 0, n, n + 9, int(rec[0, 0])):
        oh, op, _ = og.bfs(root)
        for want in ((True, True), (True, False), (False, True)):
            hops, parent, _ = gpu.bfs(g, root, *want)
            assert hops is None or np.array_equal(hops, oh)
            assert parent is None or np.array_equal(parent, op)
