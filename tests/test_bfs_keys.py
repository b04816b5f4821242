"""la3g_bfs_noalloc with keys up to the largest a uint32 holds, against a numpy
restatement of the BFS rules: the parent is the largest key among a vertex's
neighbours in the frontier, whatever the keys are."""
import ctypes as C

import numpy as np
import pytest

from test_zz_no_alloc import csr_by_key

pytestmark = pytest.mark.gpu


def _bfs(ptr, col, key, root):
    n = len(key)
    row = np.repeat(np.arange(n), np.diff(ptr.astype(np.int64)))
    hops, parent = np.full(n, 255, np.uint8), np.zeros(n, np.uint32)
    hops[root] = 0
    front, it = np.arange(n) == root, 0
    while front.any():
        at = front[col] & (hops[row] == 255)
        best = np.full(n, -1, np.int64)
        np.maximum.at(best, row[at], key[col[at]].astype(np.int64))
        front = best >= 0
        hops[front], parent[front] = (it + 1) & 255, best[front]
        it += 1
    return hops, parent


@pytest.mark.parametrize("kind", ["pair", "dense", "sparse", "path"])
@pytest.mark.parametrize("order", ["down", "up", "shuffled"])
def test_largest_keys(gpu, kind, order):
    import torch
    rng = np.random.default_rng(3)
    n = {"pair": 2, "dense": 60, "sparse": 3000, "path": 700}[kind]
    if kind in ("pair", "path"):
        src, dst = np.arange(n - 1), np.arange(1, n)
    else:
        src, dst = rng.integers(0, n, (2, 400 if kind == "dense" else 5000))
    top = np.uint32(0xFFFFFFFF) - np.arange(n, dtype=np.uint32)
    key = {"down": top, "up": top[::-1].copy(), "shuffled": top[rng.permutation(n)]}[order]
    ptr, col = csr_by_key(src, dst, n, key)
    dev = [torch.from_numpy(a.view(np.int32)).cuda() for a in (ptr, col, key)]
    hops = torch.empty(n, dtype=torch.uint8, device="cuda")
    parent = torch.empty(n, dtype=torch.int32, device="cuda")
    for root in sorted({0, 1, n // 2, n - 1, int(np.argmax(key))}):
        gpu.N.check(gpu.N.lib().la3g_bfs_noalloc(*(t.data_ptr() for t in dev), n, root, hops.data_ptr(), parent.data_ptr(),
                                                 C.c_void_p(torch.cuda.current_stream().cuda_stream), None))
        h, p = _bfs(ptr, col, key, root)
        assert np.array_equal(hops.cpu().numpy(), h), root
        assert np.array_equal(parent.cpu().numpy().view(np.uint32), p), root
