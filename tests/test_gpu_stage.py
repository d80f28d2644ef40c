"""Stages and conversions as one launch.

The stage of sweeps as one launch against the same stage as separate
kernels (per-sweep printing selects those): same decisions, exact integer
sums, so partitions, code lengths and sweep counts are equal bit for bit.
The conversion to super-nodes: link sums equal to the exact integer sums of
the members' links, on groups around every bound between two team sizes."""
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


@pytest.mark.parametrize("links", [1, 255, 256, 257, 1023, 1024, 1025, 4095, 4096, 4097, 8193, 16383, 16384, 16385])
def test_conversion_of_a_group_of(built_lib, links):
    """One module with the given number of links to other modules, all of them distinct, among small ones."""
    from relaxmap_b200 import Graph
    members, others = 48, 17000
    n = members + others
    rng = np.random.default_rng(links)
    to = members + rng.permutation(others)[:links]
    src = np.concatenate([np.arange(links) % members, np.arange(members), members + np.arange(others)])
    dst = np.concatenate([to, (np.arange(members) + 1) % members, members + (np.arange(others) * 7 + 3) % others])
    keep = src != dst
    src, dst = src[keep], dst[keep]
    part = np.concatenate([np.zeros(members), members + np.arange(others) // 2 * 2]) if links % 2 else \
        np.concatenate([np.zeros(members), members + np.arange(others)])
    part = part.astype(np.int32)
    with Graph.from_edges(src, dst, rng.uniform(1, 3, len(src)), n=n) as g:
        off, gdst, _, _ = g.links()
        f = g.initiate()["f"]
        c = g.coarsen_engine(part)
    fx = np.rint(f * 2.0 ** 62).astype(np.int64)
    group = c["sn_of_mod"][part].astype(np.int64)
    a, b = np.repeat(group, np.diff(off)), group[gdst]
    cross = a != b
    key, at = np.unique(a[cross] * c["n_sn"] + b[cross], return_inverse=True)
    want = np.zeros(len(key), dtype=np.int64)
    np.add.at(want, at, fx[cross])
    assert c["n_sn"] == len(np.unique(part)) and len(c["out_dst"]) == len(key)
    rows = np.repeat(np.arange(c["n_sn"], dtype=np.int64), np.diff(c["out_off"]))
    got = rows * c["n_sn"] + c["out_dst"]
    order = np.argsort(got)
    assert np.array_equal(got[order], key) and np.array_equal(c["out_fx"][order], want)
    cols = np.repeat(np.arange(c["n_sn"], dtype=np.int64), np.diff(c["in_off"]))
    got = c["in_src"].astype(np.int64) * c["n_sn"] + cols
    order = np.argsort(got)
    assert np.array_equal(got[order], key) and np.array_equal(c["in_fx"][order], want)


@pytest.mark.parametrize("links", [4095, 4096, 4097, 8192, 8193, 20000])
def test_links_inside_modules_of_rows_of(built_lib, links):
    """Rows of the given number of out- and of in-links (on either side of the bound and of a chunk's end), part of
    them inside the row's module; row 0 has links of its own module only, row 1 none, row 2 about half."""
    from relaxmap_b200 import Graph
    n = 24001
    rng = np.random.default_rng(links)
    src, dst = [np.arange(3, n)], [3 + (np.arange(3, n) * 7 + 5) % (n - 3)]
    for u in range(3):
        for a, b in ((src, dst), (dst, src)):
            a.append(np.full(links, u))
            b.append(3 + rng.permutation(n - 3)[:links])
    src, dst = np.concatenate(src), np.concatenate(dst)
    key = np.unique((src * np.int64(n) + dst)[src != dst])
    src, dst = key // n, key % n
    for mine in (0, 1, 2):
        part = np.where(rng.random(n) < 0.5, 0, 5).astype(np.int32) if mine == 2 else np.zeros(n, dtype=np.int32)
        part[:3] = 0
        part[1] = 9 if mine == 1 else 0
        with Graph.from_edges(src, dst, rng.uniform(1, 3, len(src)), n=n) as g:
            off, gdst, _, _ = g.links()
            f = g.initiate()["f"]
            c = g.sub_level(part)
        fx = np.rint(f * 2.0 ** 62).astype(np.int64)
        row = np.repeat(np.arange(n, dtype=np.int64), np.diff(off))
        keep = part[row] == part[gdst]
        key = row[keep] * n + gdst[keep]
        order = np.argsort(key)
        rows = np.repeat(np.arange(n, dtype=np.int64), np.diff(c["out_off"]))
        got = rows * n + c["out_dst"]
        at = np.argsort(got)
        assert np.array_equal(got[at], key[order]) and np.array_equal(c["out_fx"][at], fx[keep][order])
        cols = np.repeat(np.arange(n, dtype=np.int64), np.diff(c["in_off"]))
        got = c["in_src"].astype(np.int64) * n + cols
        at = np.argsort(got)
        assert np.array_equal(got[at], key[order]) and np.array_equal(c["in_fx"][at], fx[keep][order])
        want = np.zeros(n, dtype=np.int64)
        np.add.at(want, row[keep], fx[keep])
        assert np.array_equal(c["out_sum"], want)


def _mix32(x):
    x = x.astype(np.uint32)
    for shift, mul in ((16, 0x7feb352d), (15, 0x846ca68b)):
        x ^= x >> np.uint32(shift)
        x *= np.uint32(mul)
    return x ^ (x >> np.uint32(16))


@pytest.mark.parametrize("modules,links", [(1, 4500), (1, 16000), (40, 5000)])
def test_conversion_of_groups_whose_ids_share_a_hash(built_lib, modules, links):
    """Modules whose links lead to super-nodes that one of the conversion's rounds (4 up to 8192 links, 8 above)
    takes all of: more of them per warp than its list holds, so the launch is dropped and the separate kernels
    give the sums. With as many links to any ids the one launch is kept."""
    from relaxmap_b200 import Graph
    n, size, rounds = 1 << 18, 16, 4 if links <= 8192 else 8
    members = modules * size
    assert links / 16 > 256  # distinct ids over the 16 warps of a block, in one round
    rng = np.random.default_rng(links)
    part = np.arange(n, dtype=np.int32)
    part[:members] -= part[:members] % size
    group = np.searchsorted(np.unique(part), part)
    ids = np.arange(members, n)
    same = ids[(_mix32(group[ids] ^ 0x5bd1e995) >> np.uint32(7)) % rounds == 1]
    launches = {}
    for name, pool in (("same", same), ("any", ids)):
        to = np.concatenate([rng.permutation(pool)[:links] for _ in range(modules)])
        src = np.concatenate([m * size + np.arange(links) % size for m in range(modules)])
        with Graph.from_edges(src, to, rng.uniform(1, 3, len(src)), n=n) as g:
            off, gdst, _, _ = g.links()
            f = g.initiate()["f"]
            before = g.profile()["kernel_launches"]
            c = g.coarsen_engine(part)
            launches[name] = g.profile()["kernel_launches"] - before
        a, b = np.repeat(group, np.diff(off)), group[gdst]
        key = a * np.int64(c["n_sn"]) + b
        order = np.argsort(key)  # every link leads to a super-node of its own
        want = np.rint(f * 2.0 ** 62).astype(np.int64)[order]
        rows = np.repeat(np.arange(c["n_sn"], dtype=np.int64), np.diff(c["out_off"])) * c["n_sn"] + c["out_dst"]
        at = np.argsort(rows)
        assert np.array_equal(rows[at], key[order]) and np.array_equal(c["out_fx"][at], want)
        cols = c["in_src"].astype(np.int64) * c["n_sn"] + np.repeat(np.arange(c["n_sn"]), np.diff(c["in_off"]))
        at = np.argsort(cols)
        assert np.array_equal(cols[at], key[order]) and np.array_equal(c["in_fx"][at], want)
    assert launches["same"] >= launches["any"] + 10
