"""Device memory that batches keep on a graph: that of the largest batch, in
whatever order the sizes come, and nothing that grows from call to call."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _device_bytes(L, g):
    info = L.N.GraphInfo()
    L.N.check(L.N.lib().la3g_graph_info_get(g._h, C.byref(info)))
    return info.device_bytes


@pytest.mark.parametrize("app", ["bfs", "sssp"])
def test_growing_batches_replace_their_buffers(gpu, app):
    L = gpu
    n = 5000
    rec = np.random.default_rng(8).integers(1, n + 1, (8 * n, 3)).astype(np.uint32)
    flags = 0 if app == "bfs" else L.DIRECTED | L.WEIGHTED
    call = L.bfs_batch if app == "bfs" else L.sssp_batch
    sizes = [3, 20, 64, 65, 130, 250]

    def kept(order):
        g = L.Graph.from_records(np.ascontiguousarray(rec[:, : 3 if flags else 2]), n, flags)
        out = []
        for k in order:
            call(g, np.arange(1, k + 1, dtype=np.uint32))
            out.append(_device_bytes(L, g))
        return out

    once = kept(sizes[-1:])[0]
    assert kept(sizes)[-1] == once
    assert kept([sizes[-1]] + sizes) == [once] * (len(sizes) + 1)
