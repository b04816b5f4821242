"""Calls during which a device allocation fails: each of the call's allocations in
turn, on a graph on which nothing was called yet.  The call returns LA3G_ENOMEM
(or does without), and so does a second one; made again with memory there, it
returns what it returns on a graph that never saw the failure."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

ENOMEM = 4


def _same(a, b):
    return all(x == y if isinstance(x, int) else np.array_equal(x, y) for x, y in zip(a, b, strict=True))


def _each(L, make, call):
    """Returns how many allocations the call makes."""
    fail = L.N.lib().la3g_fail_allocation
    want = call(make())
    for n in range(200):
        g = make()
        done = False
        for again in (False, True):
            fail(n)
            try:
                got = call(g)
            except L.N.LA3GError as e:
                assert e.status == ENOMEM, e
                assert fail(-1) < 0
            else:
                done |= fail(-1) >= 0 and not again
                assert _same(got, want), n
        assert _same(call(g), want), n
        if done:
            return n
    raise AssertionError("too many allocations")


@pytest.fixture(scope="module")
def records():
    rng = np.random.default_rng(2)
    n = 3000
    rec = rng.integers(1, n + 1, (9 * n, 3)).astype(np.uint32)
    rec[:700, 1] = 5  # a row that SSSP's pull and PageRank cut up
    rec[:1500, 0] = rng.permutation(n)[:1500] + 1
    zero = rec.copy()
    zero[0, :2] = 0, 9
    return n, rec, zero


@pytest.mark.parametrize("weighted", [False, True])
def test_push_view(gpu, records, weighted):
    """The push CSR: built on demand, whole or not at all."""
    import ctypes as C

    import torch
    L = gpu
    n, rec, _ = records
    data = rec if weighted else np.ascontiguousarray(rec[:, :2])

    def array(address, count):
        class A:
            __cuda_array_interface__ = {"shape": (count,), "typestr": "<i4", "data": (address, False), "version": 2}
        return torch.as_tensor(A(), device="cuda").cpu().numpy()

    def call(g):
        ptr, row = C.c_void_p(), C.c_void_p()
        L.N.check(L.N.lib().la3g_graph_push_view(g._h, C.byref(ptr), C.byref(row)))
        assert ptr.value and row.value
        return array(ptr.value, g.nslots + 1), array(row.value, g.info.nentries)

    make = lambda: L.Graph.from_records(data, n, L.DIRECTED | (L.WEIGHTED if weighted else 0))
    assert _each(L, make, call) > 0


def test_loads(gpu, records):
    L = gpu
    n, rec, _ = records
    fail = L.N.lib().la3g_fail_allocation
    for flags in (0, L.DIRECTED | L.WEIGHTED):
        data = rec if flags else np.ascontiguousarray(rec[:, :2])
        want = L.Graph.from_records(data, n, flags).positions()
        for k in range(50):
            fail(k)
            try:
                got = L.Graph.from_records(data, n, flags)
            except L.N.LA3GError as e:
                assert e.status == ENOMEM
            else:
                break
            finally:
                left = fail(-1)
        assert k and left >= 0 and _same(got.positions(), want)
