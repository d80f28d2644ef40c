"""Stationary flow, edge flows and the initial code length on the GPU against
the reference (golden vectors) and the oracle (larger seeded graphs)."""
import numpy as np
import pytest

from conftest import FIXTURES, GOLDEN, golden

pytestmark = pytest.mark.gpu


def rel_l1(a, b):
    return np.abs(a - b).sum() / max(np.abs(b).sum(), 1e-300)


@pytest.mark.parametrize("name", FIXTURES)
def test_flows_match_reference(built_lib, name):
    from relaxmap_b200 import Graph
    g = golden(name)
    with Graph.from_file(GOLDEN / name) as G:
        off, dst, w, tw = G.links()
        np.testing.assert_array_equal(off, g["off"])
        np.testing.assert_array_equal(dst, g["dst"])
        keep = (g["map_w"] > 0) & (g["map_src"] != g["map_dst"])
        np.testing.assert_array_equal(w, g["map_w"][keep])
        np.testing.assert_array_equal(tw, g["tw"])
        r = G.initiate()
    assert rel_l1(r["p"], g["p"]) <= 1e-12          # flow within 1e-12 relative L1
    assert rel_l1(r["f"], g["f"]) <= 1e-12
    assert rel_l1(r["exit"], g["exit"]) <= 1e-12
    np.testing.assert_array_equal(r["dangling"], g["dangling"])
    assert abs(r["L0"] - float(g["L0"])) <= 1e-10
    assert 50 <= r["iters"] <= 200


@pytest.mark.parametrize("weights", [None, "uniform", "lognormal"])
def test_flows_synthetic_vs_oracle(built_lib, oracle_mod, weights):
    from relaxmap_b200 import Graph, synth
    O = oracle_mod
    sg = synth.planted_partition(5000, 12, 300, 10, 200, 0.35, seed=3, weights=weights)
    # some dangling nodes: drop every out-link of 3% of the nodes
    rng = np.random.default_rng(0)
    dead = rng.random(sg.n) < 0.03
    keep = ~dead[sg.src]
    src, dst = sg.src[keep], sg.dst[keep]
    w = None if sg.w is None else sg.w[keep]
    prep = O.prepare(O.from_edges(sg.n, src, dst, w))
    st = O.initiate(prep)
    with Graph.from_edges(src, dst, w, n=sg.n) as G:
        r = G.initiate()
    assert rel_l1(r["p"], st["p"]) <= 1e-12
    assert rel_l1(r["f"], st["f"]) <= 1e-12
    assert abs(r["L0"] - st["L0"]) <= 1e-10


def test_node_weights_teleport(built_lib, oracle_mod, tmp_path):
    """Pajek node weights set non-uniform teleportation (FileIO.cpp:114-120)."""
    from relaxmap_b200 import Graph
    O = oracle_mod
    rng = np.random.default_rng(5)
    n = 300
    src = rng.integers(0, n, 3000)
    dst = rng.integers(0, n, 3000)
    nw = rng.uniform(0.1, 5.0, n)
    path = tmp_path / "g.net"
    with open(path, "w") as f:
        f.write(f"*Vertices {n}\n")
        for i in range(n):
            f.write(f'{i + 1} "v{i}" {nw[i]!r}\n')
        f.write("*Arcs\n")
        for a, b in zip(src, dst):
            f.write(f"{a + 1} {b + 1} 1.5\n")
    prep = O.load(path)
    st = O.initiate(prep)
    with Graph.from_file(path) as G:
        _, _, _, tw = G.links()
        np.testing.assert_array_equal(tw, prep.tw)
        r = G.initiate()
    assert rel_l1(r["p"], st["p"]) <= 1e-12
    assert abs(r["L0"] - st["L0"]) <= 1e-10


def test_reset_flow_recomputes_the_same_flow(built_lib):
    """rmx_reset_flow: the next initiate recomputes p and the edge flows from
    the raw weights; they equal the first computation bit for bit, and so do
    the partitions that follow."""
    from relaxmap_b200 import Graph
    with Graph.from_file(GOLDEN / "directNet_1k_sm_mu_03.txt") as G:
        a = G.initiate()
        ra = G.optimize(seed=3)
        for _ in range(2):
            G.reset_flow()
            b = G.initiate()
            np.testing.assert_array_equal(a["p"], b["p"])
            np.testing.assert_array_equal(a["f"], b["f"])
            assert a["L0"] == b["L0"]
        G.reset_flow()
        rb = G.optimize(seed=3)
        assert ra["L"] == rb["L"]
        np.testing.assert_array_equal(ra["part"], rb["part"])


def test_flow_with_in_degree_hubs(built_lib, oracle_mod):
    """R-MAT in-degree hubs (rows of more than 64 lane steps) are pulled in
    256-link chunks by whole warps: the flow still matches the oracle's
    one-thread steady state to 1e-12 relative L1."""
    from relaxmap_b200 import Graph, synth
    O = oracle_mod
    g = synth.rmat(14, 16, seed=42)
    indeg = np.bincount(g.dst, minlength=g.n)
    assert indeg.max() > 512  # the chunked path is exercised
    st = O.initiate(O.prepare(O.from_edges(g.n, g.src, g.dst)))
    with Graph.from_edges(g.src, g.dst, None, n=g.n) as G:
        got = G.initiate()
    assert got["iters"] == st["iters"]
    assert np.abs(got["p"] - st["p"]).sum() / np.abs(st["p"]).sum() <= 1e-12


def test_flow_gathered_copy(built_lib, oracle_mod):
    """A flow vector above 96 MB (2^24 nodes) of which half the nodes have no
    out-link: the pull gathers from the compact copy of the out-linked nodes'
    flows. The flow matches a restatement of the same iteration (as many
    sweeps) with scipy's sparse product and numpy's pairwise sums to 1e-12
    relative L1, and the oracle's one-thread steady state on the library's own
    prepared links to 1e-9. At this size the oracle's serial FP64 sums of
    millions of terms (the reference's loop) are themselves off (at 2^22 nodes
    its flow differs from the same iteration with exactly rounded sums by
    8.6e-12, the pairwise one by 2e-17), and its L1 change never falls to the
    1e-15 stop threshold, so it runs the 200-sweep cap where the GPU stops
    at the rule's 50."""
    import scipy.sparse as sparse
    from relaxmap_b200 import Graph
    O = oracle_mod
    n, m = 1 << 24, 12_000_000
    rng = np.random.default_rng(21)
    src = rng.integers(0, n // 2, m)
    dst = rng.integers(0, n, m)
    with Graph.from_edges(src, dst, None, n=n) as G:
        off, dst_k, w, tw = G.links()
        got = G.initiate()
    st = O.initiate(O.Prepared(n, off, dst_k, w, tw))
    assert 50 <= got["iters"] <= st["iters"]
    # the reference's iteration (Module.cpp:340-469) with scipy's product
    s = np.repeat(np.arange(n), np.diff(off))
    outw = np.bincount(s, weights=w, minlength=n)
    dang = outw == 0
    W = sparse.csr_matrix((w / outw[s], (dst_k, s)), shape=(n, n))
    x = np.full(n, 1.0 / n)
    for _ in range(got["iters"]):
        y = (0.15 + 0.85 * x[dang].sum()) * tw + 0.85 * (W @ x)
        x = y / y.sum()
    assert rel_l1(got["p"], x) <= 1e-12
    assert rel_l1(got["p"], st["p"]) <= 1e-9  # measured 1.1e-10: the oracle's own rounding
    assert rel_l1(got["f"], st["f"]) <= 1e-9


def test_flow_with_weighted_out_degree_hubs(built_lib, oracle_mod):
    """Rows of more than 256 out-links are normalised, turned into edge flows
    and summed into singleton exits by a whole warp (the reference sums them
    in link order, so the last bits of a weighted hub row's sum may differ):
    flows, edge flows and exits stay within 1e-12 relative L1 of the oracle,
    and the initial code length within 1e-10."""
    from relaxmap_b200 import Graph
    O = oracle_mod
    rng = np.random.default_rng(21)
    n = 20000
    src = [rng.integers(0, n, 6 * n)]
    dst = [rng.integers(0, n, 6 * n)]
    for hub, deg in ((0, 9000), (1, 3000), (2, 700), (3, 300)):
        src.append(np.full(deg, hub))
        dst.append(rng.choice(n, deg, replace=False))
    src, dst = np.concatenate(src), np.concatenate(dst)
    w = rng.lognormal(0.0, 1.0, len(src))
    prep = O.prepare(O.from_edges(n, src, dst, w))
    st = O.initiate(prep)
    assert np.diff(prep.off).max() > 256
    with Graph.from_edges(src, dst, w, n=n) as G:
        got = G.initiate()
    rel = lambda a, b: np.abs(a - b).sum() / np.abs(b).sum()  # noqa: E731
    assert abs(got["iters"] - st["iters"]) <= 1
    assert rel(got["p"], st["p"]) <= 1e-12
    assert rel(got["f"], st["f"]) <= 1e-12
    assert rel(got["exit"], st["exit"]) <= 1e-12
    assert abs(got["L0"] - st["L0"]) <= 1e-10


def _flow_error(O, src, dst, w, n):
    from relaxmap_b200 import Graph
    st = O.initiate(O.prepare(O.from_edges(n, src, dst, w)))
    with Graph.from_edges(src, dst, w, n=n) as G:
        r = G.initiate()
    return rel_l1(r["p"], st["p"])


@pytest.mark.parametrize("n,deg", [(2, 1), (255, 3), (256, 9), (257, 20), (1000, 40), (4096, 20), (4097, 20),
                                   (8192, 7), (8193, 7)])
def test_small_graph_flow(built_lib, oracle_mod, n, deg):
    """Sizes around the bounds of the one-cluster form of the power iteration (virtual blocks of
    256 threads, 128 of them, 8192 nodes); dangling nodes among them."""
    rng = np.random.default_rng(n)
    src, dst = rng.integers(0, max(1, n - n // 10), n * deg), rng.integers(0, n, n * deg)
    src[0], dst[0] = 0, n - 1
    key = np.unique((src * np.int64(n) + dst)[src != dst])
    src, dst = (key // n).astype(np.int32), (key % n).astype(np.int32)
    assert _flow_error(oracle_mod, src, dst, rng.uniform(1, 10, len(src)), n) <= 1e-12


@pytest.mark.parametrize("hub", [256, 257, 2999])
def test_small_graph_flow_with_hub(built_lib, oracle_mod, hub):
    """In-degrees on both sides of the bound (64 steps of 4 lanes) above which a small graph goes to
    the grid form and its chunked rows."""
    n = 3000
    rng = np.random.default_rng(hub)
    m = 6 * n
    src = np.concatenate([np.arange(1, hub + 1), rng.integers(0, n, m)])
    dst = np.concatenate([np.zeros(hub, dtype=np.int64), rng.integers(1, n, m)])
    key = np.unique((src * np.int64(n) + dst)[src != dst])
    src, dst = (key // n).astype(np.int32), (key % n).astype(np.int32)
    assert _flow_error(oracle_mod, src, dst, None, n) <= 1e-12


@pytest.mark.parametrize("n,deg", [(4096, 12), (4097, 12), (5000, 2), (5100, 2), (3000, 22), (3100, 22),
                                   (16384, 6), (16385, 6), (18432, 6), (18433, 6)])
def test_flow_around_the_bounds_of_its_forms(built_lib, oracle_mod, n, deg):
    """Either side of the bounds of the one-cluster form: four virtual blocks for each of its blocks, and the cost
    of nodes and links above that; 256 partial sums, one per thread of a block, and 257; 288, the most that the grid form adds from shared
    memory, and 289."""
    rng = np.random.default_rng(n + deg)
    src, dst = rng.integers(0, n - n // 10, n * deg), rng.integers(0, n, n * deg)
    src[0], dst[0] = 0, n - 1
    key = np.unique((src * np.int64(n) + dst)[src != dst])
    src, dst = (key // n).astype(np.int32), (key % n).astype(np.int32)
    assert _flow_error(oracle_mod, src, dst, rng.uniform(1, 10, len(src)), n) <= 1e-12
