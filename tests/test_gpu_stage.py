"""The stage of sweeps as one launch against the same stage as separate
kernels (per-sweep printing selects those): same decisions, exact integer
sums, so partitions, code lengths and sweep counts are equal bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# one unit on each side of every bound between two ways of evaluating a unit
DEGREES = [1, 7, 8, 9, 16, 17, 32, 33, 128, 129, 512, 513, 1024, 1025, 4095, 4096]


def _graph(n, seed, degrees=(), mean=6, weighted=False, top=None):
    """A random graph whose first nodes have the given numbers of links (half out, half in)."""
    rng = np.random.default_rng(seed)
    src, dst = [], []
    for u, d in enumerate(degrees):
        others = rng.permutation(np.arange(len(degrees), n))[:d]
        out = d // 2
        src += [np.full(out, u), others[out:]]
        dst += [others[:out], np.full(d - out, u)]
    m = mean * n
    lo = len(degrees)
    a = rng.integers(lo, n, m)
    b = np.where(rng.random(m) < 0.7, lo + (a - lo) // 40 * 40 + rng.integers(0, 40, m), rng.integers(lo, n, m))
    src.append(a)
    dst.append(np.minimum(b, n - 1))
    src, dst = np.concatenate(src), np.concatenate(dst)
    key = np.unique(src[src != dst] * np.int64(n) + dst[src != dst])
    w = rng.uniform(1, 10, len(key)) if weighted else None
    return key // n, key % n, w


@pytest.mark.parametrize("prior", [1, 0])
@pytest.mark.parametrize("nsub", [1, 4, 32])
@pytest.mark.parametrize("case", ["pair", "small", "weighted", "degrees", "wide"])
def test_one_launch_equals_kernels(built_lib, case, nsub, prior, capfd):
    from relaxmap_b200 import Graph
    if case == "pair":
        n, (src, dst, w) = 2, (np.array([0]), np.array([1]), None)
    elif case == "small":
        n = 333
        src, dst, w = _graph(n, 1)
    elif case == "weighted":
        n = 4001
        src, dst, w = _graph(n, 2, weighted=True, mean=14)
    elif case == "degrees":
        n = 6000
        src, dst, w = _graph(n, 3, DEGREES, weighted=True)
    else:  # more units than warps: teams take units in turn
        n = 90001
        src, dst, w = _graph(n, 4, DEGREES * 3, mean=9)
    opts = dict(seed=7, prior=prior, sub_batches=nsub, max_iter=4)
    with Graph.from_edges(src, dst, w, n=n) as g:
        one = g.optimize(**opts)
        s1 = g.profile()["sweeps"]
        kernels = g.optimize(verbose=2, **opts)
        s2 = g.profile()["sweeps"]
    capfd.readouterr()
    assert s2 - s1 == s1
    assert one["L"] == kernels["L"]
    assert np.array_equal(one["steps_bits"], kernels["steps_bits"])
    assert np.array_equal(one["part"], kernels["part"])
