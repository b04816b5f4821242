"""Triangle counts asked for by several threads at once, each on a graph of its
own, the first of the process among them."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_threads(gpu):
    L = gpu
    n = 2000
    # a clique's rows and suffixes need every kernel, the row sort in shared memory too
    ids = np.arange(1, 1400)
    a, b = np.triu_indices(len(ids), 1)
    rec = np.stack([ids[a], ids[b]], 1).astype(np.uint32)
    m = len(ids)
    want = m * (m - 1) * (m - 2) // 6
    got = [None] * 6

    def work(i):
        got[i] = [L.tc(L.Graph.from_records(rec, n, L.DIRECTED | L.ACYCLIC))[0] for _ in range(3)]

    threads = [threading.Thread(target=work, args=(i,)) for i in range(len(got))]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert got == [[want] * 3] * len(got)
