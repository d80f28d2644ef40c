"""Large host arrays: the edge list goes up through the pinned ring and the
links come back into untouched pages; sizes around the ring's slots."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _edges(m, seed):
    rng = np.random.default_rng(seed)
    n = 4096
    key = rng.permutation(n * n)[:m + n]
    key = key[key // n != key % n][:m]
    return n, (key // n).astype(np.int32), (key % n).astype(np.int32), rng.uniform(1, 2, len(key))


def _check(n, src, dst, w):
    from relaxmap_b200 import Graph
    with Graph.from_edges(src, dst, w, n=n) as g:
        off, gdst, gw, _ = g.links()
    order = np.argsort(src.astype(np.int64) * n + dst)
    assert np.array_equal(np.repeat(np.arange(n), np.diff(off)), src[order])
    assert np.array_equal(gdst, dst[order]) and np.array_equal(gw, w[order])


@pytest.mark.parametrize("m", [(1 << 18) - 1, 1 << 20, (1 << 20) + 1, (1 << 22) + 12345, 1 << 23])
def test_links_round_trip(built_lib, m):
    from relaxmap_b200 import release_device_cache
    _check(*_edges(m, m))
    release_device_cache()  # the ring goes and comes back
    _check(*_edges(m, m + 1))


def test_two_threads(built_lib):
    """Two handles created at once: one takes the ring, the other copies without it."""
    _check(*_edges(1 << 23, 1))  # the ring exists
    errors = []

    def work(seed):
        try:
            for k in range(3):
                _check(*_edges((1 << 21) + seed, 10 * seed + k))
        except Exception as e:  # handed to the main thread
            errors.append(e)
    t = [threading.Thread(target=work, args=(s,)) for s in (1, 2)]
    for x in t:
        x.start()
    for x in t:
        x.join()
    assert not errors


@pytest.mark.parametrize("touched", ["none", "half", "all", "last"])
def test_results_into_pages_of_an_array(built_lib, touched):
    """The gradient written to a mapping of which no page, half of the pages, every page or only the last one has
    been touched, from an address inside a page, equals the one written to pinned memory."""
    import mmap
    import torch
    from relaxmap_b200 import Graph
    n, src, dst, w = _edges(1 << 20, 5)
    part = (np.arange(n) // 64).astype(np.int32)
    with Graph.from_edges(src, dst, w, n=n) as g:
        want = torch.empty(g.n_links, dtype=torch.float64).pin_memory().numpy()
        g.adjoint_backward(part, out=want)
        m = mmap.mmap(-1, 8 * g.n_links + 4096)
        out = np.frombuffer(m, dtype=np.float64, count=g.n_links, offset=2008)
        k = {"none": (0, 0), "half": (0, len(out) // 2), "all": (0, len(out)), "last": (len(out) - 1, len(out))}[touched]
        out[k[0]:k[1]] = 1.0
        g.adjoint_backward(part, out=out)
    assert np.array_equal(out, want)
