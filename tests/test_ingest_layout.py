"""The device matrix of a load (positions, pull CSR, weights, push CSR) against
a numpy restatement of the load rules, over every kind of load, with
duplicates (the first record's weight counts), self-loops, vertices of every
class and empty inputs."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIRECTED, REVERSE, ACYCLIC, BIPARTITE, WEIGHTED = 1, 2, 4, 8, 16


def _device(address, count):
    import torch

    class A:
        __cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (address, False), "version": 2}

    return torch.as_tensor(A(), device="cuda").cpu().numpy() if count else np.empty(0, np.int32)


def _hash(ids, n, flags):
    ids = np.asarray(ids, np.int64)
    height = n // 128
    if flags & BIPARTITE:
        return ids
    return np.where(ids >= height * 128, ids, ids // 128 + (ids % 128) * height)


def _expect(rec, n, flags, nleft):
    """(id_of_pos, nreg, nsink, nsrc, rows, cols, weights) in the pull order."""
    entries = {}
    for r in rec.tolist():
        row, col, w = r[0], r[1], r[2] if flags & WEIGHTED else 0
        if flags & BIPARTITE:
            col += nleft
        if row == col:
            continue
        if flags & DIRECTED and not flags & REVERSE:
            row, col = col, row
        if flags & ACYCLIC and (col < row if flags & REVERSE else col > row):
            row, col = col, row
        entries.setdefault((row, col), w)
        if not flags & DIRECTED:
            entries.setdefault((col, row), w)
    rows, cols = {r for r, _ in entries}, {c for _, c in entries}
    ids = np.arange(n + 1)
    cls = np.array([0 if i in rows and i in cols else 1 if i in rows else 2 if i in cols else 3 for i in ids])
    order = np.lexsort((_hash(ids, n, flags), cls))
    pos = np.empty(n + 1, np.int64)
    pos[order] = ids
    count = [int((cls == k).sum()) for k in range(3)]
    nrows = count[0] + count[1]
    pulls = sorted((pos[r], pos[c] - nrows if pos[c] >= nrows else pos[c] + count[2], pos[c], w)
                   for (r, c), w in entries.items())
    return order, count, [(r, c, w) for r, _, c, w in pulls]


def _ptr(keys, n):
    return np.searchsorted(np.asarray(keys, np.int64), np.arange(n + 2))


@pytest.mark.parametrize("flags", [0, WEIGHTED, DIRECTED, DIRECTED | WEIGHTED, DIRECTED | REVERSE, DIRECTED | ACYCLIC,
                                   DIRECTED | REVERSE | ACYCLIC, BIPARTITE | WEIGHTED, BIPARTITE | DIRECTED | WEIGHTED])
@pytest.mark.parametrize("n,m", [(1, 3), (7, 0), (127, 40), (128, 900), (129, 5), (1000, 700), (1000, 9000)])
def test_layout(gpu, flags, n, m):
    rng = np.random.default_rng(n + m + flags)
    nright = max(1, n // 3) if flags & BIPARTITE else 0
    lo = 0 if not flags & BIPARTITE else 1
    src = rng.integers(lo, n + 1, m)
    dst = rng.integers(lo, (nright if nright else n) + 1, m)
    src = np.where(rng.random(m) < 0.3, src // 2, src).clip(lo)
    rec = np.stack([src, dst, rng.integers(1, 1 << 32, m)][: 3 if flags & WEIGHTED else 2], 1).astype(np.uint32)
    g = gpu.Graph.from_records(rec, n, flags, nright)
    order, count, pulls = _expect(rec.astype(np.int64), n + nright, flags, n)
    slots = n + nright + 1
    i = g.info
    assert (i.nslots, i.nregular, i.nsink, i.nsource, i.nentries) == (slots, *count, len(pulls))
    pos, ids = g.positions()
    assert np.array_equal(ids, order) and np.array_equal(pos[ids], np.arange(slots))
    v = gpu.N.DeviceGraph()
    gpu.N.check(gpu.N.lib().la3g_graph_device_view(g._h, C.byref(v)))
    rows, cols, ws = (np.array(x, np.int64) for x in zip(*pulls)) if pulls else (np.empty(0, np.int64),) * 3
    assert np.array_equal(_device(v.row_ptr, slots + 1), _ptr(rows, slots - 1))
    assert np.array_equal(_device(v.col, len(cols)), cols)
    if flags & WEIGHTED:
        assert np.array_equal(_device(v.weight, len(ws)).view(np.uint32), ws)
    out_ptr, out_row = C.c_void_p(), C.c_void_p()
    gpu.N.check(gpu.N.lib().la3g_graph_push_view(g._h, C.byref(out_ptr), C.byref(out_row)))
    at = np.lexsort((rows, cols)) if flags & DIRECTED else np.arange(len(rows))
    assert np.array_equal(_device(out_ptr.value, slots + 1), _ptr((cols if flags & DIRECTED else rows)[at], slots - 1))
    assert np.array_equal(_device(out_row.value, len(rows)), (rows if flags & DIRECTED else cols)[at])
