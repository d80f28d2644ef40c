"""Batched multi-graph x multi-attempt optimisation (rmx_batch_*).

Checked per graph against the single-graph path: the code length returned for
each graph is the code length of the returned partition computed from scratch
on that graph alone (1e-10 relative: fixed-point module sums against FP64),
which also checks the per-component flows of the disjoint union; a batch of
one graph and one attempt is exactly rmx_optimize; quality of the best of 4
attempts is within 0.5% of the single-graph optimiser."""
import numpy as np
import pytest

from conftest import GOLDEN

pytestmark = pytest.mark.gpu


def _graphs():
    from relaxmap_b200 import synth
    gs = []
    for k, spec in enumerate(synth.batched_graphs(6, seed=3, n_range=(200, 3000))):
        g = synth.batched_graph(spec)
        gs.append((g.n, g.src, g.dst, g.w))
    # a graph without links and one with dangling nodes and weights
    gs.append((5, np.zeros(0, np.int32), np.zeros(0, np.int32), None))
    rng = np.random.default_rng(0)
    s = rng.integers(0, 300, 2000).astype(np.int32)
    d = rng.integers(0, 300, 2000).astype(np.int32)
    keep = s % 7 != 0
    gs.append((300, s[keep], d[keep], rng.uniform(1, 5, keep.sum())))
    return gs


def _single_L(g, part):
    from relaxmap_b200 import Graph
    with Graph.from_edges(g[1], g[2], g[3], n=g[0]) as G:
        return G.codelength(part)


def _check_part(part, n, nm):
    assert len(part) == n
    assert part.min() == 0 and part.max() == nm - 1
    # first-appearance numbering
    first = []
    seen = set()
    for m in part.tolist():
        if m not in seen:
            seen.add(m)
            first.append(m)
    assert first == list(range(nm))


@pytest.mark.parametrize("waves", ["one", "many"])
def test_batch_matches_single_graph_code_lengths(built_lib, waves):
    from relaxmap_b200 import Batch
    gs = _graphs()
    with Batch(gs) as B:
        if waves == "many":
            B.set_wave(20_000, 10_000)
        r = B.optimize(seed=1, attempts=4)
        info = B.info()
    assert info["instances"] == 4 * len(gs)
    assert (info["waves"] > 1) == (waves == "many")
    for k, g in enumerate(gs):
        part = r["part"][k]
        _check_part(part, g[0], r["n_modules"][k])
        L = _single_L(g, part)
        assert abs(L - r["L"][k]) <= 1e-10 * abs(L), (k, L, r["L"][k])
        assert 0 <= r["best_attempt"][k] < 4


def test_batch_quality_against_single_optimiser(built_lib):
    from relaxmap_b200 import Batch, Graph
    gs = _graphs()[:6]
    with Batch(gs) as B:
        r = B.optimize(seed=1, attempts=4)
    for k, g in enumerate(gs):
        with Graph.from_edges(g[1], g[2], g[3], n=g[0]) as G:
            single = np.median([G.optimize(seed=s)["L"] for s in (1, 2, 3)])
        assert r["L"][k] <= 1.005 * single, (k, r["L"][k], single)


def test_batch_of_one_is_rmx_optimize(built_lib):
    from relaxmap_b200 import Batch, Graph, parse_file
    pf = parse_file(GOLDEN / "directNet_1k_sm_mu_03.txt")
    g = (pf["n"], pf["src"], pf["dst"], pf["w"])
    with Batch([g]) as B:
        r = B.optimize(seed=5, attempts=1)
    with Graph.from_edges(g[1], g[2], g[3], n=g[0]) as G:
        s = G.optimize(seed=5)
    assert r["L"][0] == s["L"]
    # same modules up to renumbering
    a, b = r["part"][0], np.asarray(s["part"])
    pairs = set(zip(a.tolist(), b.tolist()))
    assert len(pairs) == len(set(a.tolist())) == len(set(b.tolist()))


def test_batch_rejects_bad_input(built_lib):
    from relaxmap_b200 import Batch, RmxError
    with pytest.raises(RmxError):
        Batch([(3, np.array([0, 3], np.int32), np.array([1, 2], np.int32), None)])
    with pytest.raises(RmxError):
        Batch([(0, np.zeros(0, np.int32), np.zeros(0, np.int32), None)])


def test_batch_captured_loops_match_host_loops(built_lib, capfd):
    """A batch wave (a union of graph-attempt instances) runs its stage loops
    as captured while graphs from its first run; with per-sweep printing
    (verbose 2) the same loops are driven from the host. Same partitions, code
    lengths and best attempts."""
    from relaxmap_b200 import Batch
    gs = _graphs()
    with Batch(gs) as B:
        a = B.optimize(seed=2, attempts=3)
        b = B.optimize(seed=2, attempts=3, verbose=2)
    capfd.readouterr()  # the host loop's per-sweep lines
    np.testing.assert_array_equal(a["L"], b["L"])
    np.testing.assert_array_equal(a["best_attempt"], b["best_attempt"])
    for pa, pb in zip(a["part"], b["part"]):
        np.testing.assert_array_equal(pa, pb)


@pytest.mark.parametrize("attempts", [1, 3])
def test_union_flow_of_uneven_graphs(built_lib, attempts):
    """Graphs whose sizes leave part of a row group, of a block and of a warp's run over, with and
    without dangling nodes: each returned code length is the single-graph one of its partition."""
    from relaxmap_b200 import Batch, Graph
    rng = np.random.default_rng(3)
    graphs = []
    for n in (2, 3, 31, 33, 255, 256, 257, 2049, 6001):
        m = 5 * n
        src, dst = rng.integers(0, max(1, n - n // 7), m), rng.integers(0, n, m)
        src[0], dst[0] = 0, n - 1
        key = np.unique((src * np.int64(n) + dst)[src != dst])
        graphs.append((n, (key // n).astype(np.int32), (key % n).astype(np.int32), rng.uniform(1, 5, len(key))))
    with Batch(graphs) as b:
        r = b.optimize(seed=3, attempts=attempts)
    for (n, src, dst, w), part, L in zip(graphs, r["part"], r["L"]):
        with Graph.from_edges(src, dst, w, n=n) as g:
            assert abs(g.codelength(part) - L) <= 1e-10


@pytest.fixture
def every_unit_a_hub():
    """Every unit of more than 32 links in the hub bin: levels that have one take the separate kernels and their
    captured loops, as levels of large networks do."""
    from relaxmap_b200 import get_tuning, set_tuning
    before = get_tuning()
    set_tuning(warp_max_degree=32, mid_max_degree=32, block_max_degree=32, large_max_degree=32)
    yield
    set_tuning(**before)


def test_union_of_many_nodes_and_few_links(built_lib, every_unit_a_hub):
    """Two graphs of 920,000 nodes, most of them without links, whose conversions by the separate kernels take
    nearly all of the union's scratch memory, which one graph's conversions would."""
    from relaxmap_b200 import Batch
    n, linked = 920_000, 5000
    gs = []
    for seed in (1, 2):
        rng = np.random.default_rng(seed)
        s = rng.integers(0, linked, 5 * linked)
        d = np.where(rng.random(len(s)) < 0.8, s // 25 * 25 + rng.integers(0, 25, len(s)), rng.integers(0, linked, len(s)))
        s, d = np.concatenate([s, np.zeros(40, np.int64)]), np.concatenate([d, np.arange(1, 41)])
        key = np.unique((s * n + d)[s != d])
        gs.append((n, (key // n).astype(np.int32), (key % n).astype(np.int32), None))
    with Batch(gs) as B:
        r = B.optimize(seed=1, threshold=1e-9)
    for g, part, L in zip(gs, r["part"], r["L"]):
        assert abs(_single_L(g, part) - L) <= 1e-10 * L


def _launches():
    from relaxmap_b200 import Graph
    with Graph.from_edges(np.array([0]), np.array([1]), None, n=2) as G:
        return G.profile()["kernel_launches"]


def _batch_run(gs, **opts):
    from relaxmap_b200 import Batch
    with Batch(gs) as B:
        before = _launches()
        r = B.optimize(**opts)
        return r, _launches() - before


def _assert_same(a, b):
    np.testing.assert_array_equal(a["L"], b["L"])
    np.testing.assert_array_equal(a["best_attempt"], b["best_attempt"])
    for pa, pb in zip(a["part"], b["part"]):
        np.testing.assert_array_equal(pa, pb)


@pytest.mark.parametrize("prior", [1, 0])
def test_captured_loops_of_a_union_match_host_loops(built_lib, every_unit_a_hub, capfd, prior):
    """Levels with hub units run their stages and the coarse-tune sub-problems as captured while graphs, every
    instance under its own stop rule; per-sweep printing drives the same loops from the host. The captured sweep
    launches the kernel of every bin, the host loop those of bins with units: more launches show the graph ran."""
    gs = _graphs()
    a, captured = _batch_run(gs, seed=2, attempts=3, prior=prior)
    b, host = _batch_run(gs, seed=2, attempts=3, prior=prior, verbose=2)
    capfd.readouterr()
    assert captured > host
    _assert_same(a, b)


@pytest.mark.parametrize("prior", [1, 0])
def test_conversions_of_a_union_with_stopped_instances(built_lib, capfd, prior):
    """The separate kernels' conversions leave out the links of instances that have stopped, the one-launch
    conversion sums them all: same partitions, code lengths and best attempts, over graphs from 200 to 6000 nodes
    that stop after different numbers of supersteps."""
    from relaxmap_b200 import get_tuning, set_tuning, synth
    gs = _graphs()
    for k, spec in enumerate(synth.batched_graphs(5, seed=8, n_range=(2000, 6000), mu_range=(0.1, 0.6))):
        g = synth.batched_graph(spec)
        gs.append((g.n, g.src, g.dst, g.w))
    a, one = _batch_run(gs, seed=4, attempts=3, prior=prior)
    before = get_tuning()
    set_tuning(warp_max_degree=32, mid_max_degree=32, block_max_degree=32, large_max_degree=32)
    try:
        b, many = _batch_run(gs, seed=4, attempts=3, prior=prior)
    finally:
        set_tuning(**before)
    assert many > 10 * one
    _assert_same(a, b)


@pytest.mark.parametrize("graphs,below,bound", [(1, 13, 10 << 20), (2, 21, 1 << 25)])
def test_union_around_the_bounds_of_the_one_launch_stage(built_lib, capfd, graphs, below, bound):
    """Copies of one graph have their stages run as one launch up to 10 * 2^20 links, unions of several up to 2^25;
    one attempt more and they run as captured while graphs, with far more launches: the same result as the host
    loops on either side."""
    from relaxmap_b200 import synth
    gs = []
    for seed in range(graphs):
        g = synth.planted_partition(40_000, 20, 400, 20, 500, 0.3, seed=5 + seed, weights="uniform")
        gs.append((g.n, g.src, g.dst, g.w))
    links = sum(len(g[1]) for g in gs)
    assert below * links <= bound < (below + 1) * links
    launches = []
    for attempts in (below, below + 1):
        a, n = _batch_run(gs, seed=6, attempts=attempts, max_iter=3)
        b, _ = _batch_run(gs, seed=6, attempts=attempts, max_iter=3, verbose=2)
        launches.append(n)
        _assert_same(a, b)
        for g, part, L in zip(gs, a["part"], a["L"]):
            assert abs(_single_L(g, part) - L) <= 1e-10 * L
    capfd.readouterr()
    assert launches[1] > launches[0] + 200


def test_union_of_large_graphs_with_one_attempt(built_lib):
    """Every copy of the union is canonical: the build's scratch, with the input and the copies' links in it, is the
    union's largest."""
    n, m = 400_000, 9_000_000  # hardly an edge twice
    gs = []
    for seed in (1, 2):
        rng = np.random.default_rng(seed)
        s, d = rng.integers(0, n, m), rng.integers(0, n, m)
        near = rng.random(m) < 0.7
        d[near] = s[near] // 1000 * 1000 + rng.integers(0, 1000, int(near.sum()))
        gs.append((n, s.astype(np.int32), d.astype(np.int32), None))
    r, _ = _batch_run(gs, seed=1, attempts=1, max_iter=1)
    for g, part, L in zip(gs, r["part"], r["L"]):
        assert abs(_single_L(g, part) - L) <= 1e-10 * L
