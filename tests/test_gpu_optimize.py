"""The whole optimiser on the GPU: known answers, quality against the
reference's median over 8 seeds, exact code-length bookkeeping, determinism."""
import numpy as np
import pytest

from conftest import GOLDEN, golden

pytestmark = pytest.mark.gpu


def test_flow_known_answer(built_lib):
    from relaxmap_b200 import Graph
    with Graph.from_file(GOLDEN / "flow.net") as G:
        r = G.optimize(seed=1)
    assert round(r["L_bits"], 5) == 3.32773
    assert r["n_modules"] == 4
    groups = {}
    for v, m in enumerate(r["part"]):
        groups.setdefault(m, []).append(v)
    assert sorted(groups.values()) == [[0, 1, 2, 3], [4, 5, 6, 7], [8, 9, 10, 11], [12, 13, 14, 15]]


@pytest.mark.parametrize("name", ["directNet_1k_sm_mu_03.txt", "small_planted.txt", "flow.txt"])
@pytest.mark.parametrize("prior", [1, 0])
def test_quality_vs_reference_median(built_lib, name, prior):
    """Final code length within 0.5% of the reference's median over 8 seeds."""
    from relaxmap_b200 import Graph
    g = golden(name)
    ref_median = float(np.median(g["final_L_computed_bits"]))
    Ls = []
    with Graph.from_file(GOLDEN / name) as G:
        for seed in range(1, 9):
            r = G.optimize(seed=seed, prior=prior)
            # the running code length equals a from-scratch FP64 recompute
            assert abs(r["L"] - G.codelength(r["part"])) <= 1e-10
            Ls.append(r["L_bits"])
    assert np.median(Ls) <= ref_median * 1.005, (np.median(Ls), ref_median)


QUALITY = {
    "rmat14": lambda synth: synth.rmat(14, 16, seed=42),
    "planted20k_mid": lambda synth: synth.config_mid(seed=42, n=20_000),
    "planted20k_adjoint": lambda synth: synth.config_adjoint(seed=42, n=20_000),
}


@pytest.mark.parametrize("name", sorted(QUALITY))
def test_quality_larger_graphs(built_lib, name):
    """The R-MAT, mid and adjoint shapes at ~20K nodes (the same seeded
    generators): median over 8 seeds within 0.5% of the reference's median over
    8 seeds (tests/golden/quality.ref.npz, made by make_golden.py)."""
    from relaxmap_b200 import Graph, synth
    ref_median = float(np.median(np.load(GOLDEN / "quality.ref.npz")[name]))
    g = QUALITY[name](synth)
    Ls = []
    with Graph.from_edges(g.src, g.dst, g.w, n=g.n) as G:
        for seed in range(1, 9):
            r = G.optimize(seed=seed)
            assert abs(r["L"] - G.codelength(r["part"])) <= 1e-10
            Ls.append(r["L_bits"])
    assert np.median(Ls) <= ref_median * 1.005, (np.median(Ls), ref_median)


def test_deterministic_per_seed(built_lib):
    from relaxmap_b200 import Graph
    with Graph.from_file(GOLDEN / "small_planted.txt") as G:
        a = G.optimize(seed=5)
        b = G.optimize(seed=5)
    np.testing.assert_array_equal(a["part"], b["part"])
    assert a["L"] == b["L"]


def test_attempts_keep_best(built_lib):
    from relaxmap_b200 import Graph
    with Graph.from_file(GOLDEN / "directNet_1k_sm_mu_03.txt") as G:
        singles = [G.optimize(seed=s)["L"] for s in (3, 4, 5)]
        best = G.optimize(seed=3, attempts=3)["L"]
    assert best == min(singles)


def test_synthetic_vs_oracle_codelength(built_lib, oracle_mod):
    from relaxmap_b200 import Graph, synth
    O = oracle_mod
    sg = synth.planted_partition(20000, 15, 500, 20, 400, 0.3, seed=7, weights="uniform")
    prep = O.prepare(O.from_edges(sg.n, sg.src, sg.dst, sg.w))
    st = O.initiate(prep)
    with Graph.from_edges(sg.src, sg.dst, sg.w, n=sg.n) as G:
        r = G.optimize(seed=1)
    assert abs(r["L"] - O.codelength(prep, st, r["part"])) <= 1e-10
    # the planted partition is a good solution; the optimiser must match or beat it
    L_planted = O.codelength(prep, st, sg.community)
    assert r["L"] <= L_planted * 1.005


@pytest.mark.parametrize("prior", [1, 0])
def test_captured_stage_loops_match_host_loops(built_lib, prior):
    """From a handle's second run on, every stage loop of sweeps runs as one
    CUDA graph: a while node whose body is one sweep followed by the stop rule
    evaluated on the device. The first run, and runs with profiling on, drive
    the loop from the host. Both give the same partition, code length,
    per-superstep code lengths and number of sweeps."""
    from relaxmap_b200 import Graph, synth
    g = synth.config_mid(seed=9, n=20_000)
    with Graph.from_edges(g.src, g.dst, g.w, n=g.n) as G:
        G.set_profiling(True)  # host-driven loops, direct launches
        ref = G.optimize(seed=4, prior=prior)
        ref_sweeps = G.profile()["sweeps"]
        G.set_profiling(False)
        for _ in range(2):  # the first captures the stage graphs, the second replays them
            s0 = G.profile()["sweeps"]
            r = G.optimize(seed=4, prior=prior)
            np.testing.assert_array_equal(r["part"], ref["part"])
            assert r["L"] == ref["L"]
            np.testing.assert_array_equal(r["steps_bits"], ref["steps_bits"])
            assert G.profile()["sweeps"] - s0 == ref_sweeps


def hub_network():
    """30,000 nodes, three of them with 5000 links: its node levels run as separate kernels."""
    n, hubs = 30_000, 3
    rng = np.random.default_rng(5)
    a = rng.integers(hubs, n, 10 * n)
    b = np.where(rng.random(len(a)) < 0.7, hubs + (a - hubs) // 40 * 40 + rng.integers(0, 40, len(a)),
                 rng.integers(hubs, n, len(a)))
    src, dst = [a], [np.minimum(b, n - 1)]
    for u in range(hubs):  # out- and in-links, 5000 in all
        other = hubs + rng.permutation(n - hubs)[:5000]
        src += [np.full(2500, u), other[2500:]]
        dst += [other[:2500], np.full(2500, u)]
    src, dst = np.concatenate(src), np.concatenate(dst)
    key = np.unique((src * n + dst)[src != dst])
    return n, key // n, key % n, rng.uniform(1, 5, len(key))


@pytest.mark.parametrize("prior", [1, 0])
def test_captured_stage_loops_of_levels_with_hubs(built_lib, prior, capfd):
    """The node levels of this network have units of more than 4096 links, so their stages run as captured while
    graphs from the handle's second run on; the first run, and one with per-sweep printing, drive them from the
    host. Same partition, code length, per-superstep code lengths and number of sweeps. A captured sweep launches
    the kernel of every bin, the first run's those of bins with units: more launches show that graphs ran."""
    from relaxmap_b200 import Graph
    n, src, dst, w = hub_network()
    runs = []
    with Graph.from_edges(src, dst, w, n=n) as G:
        for verbose in (0, 0, 0, 2):
            before = G.profile()
            r = G.optimize(seed=4, prior=prior, verbose=verbose)
            after = G.profile()
            r["sweeps"] = after["sweeps"] - before["sweeps"]
            r["launches"] = after["kernel_launches"] - before["kernel_launches"]
            runs.append(r)
    capfd.readouterr()
    for r in runs[1:]:
        np.testing.assert_array_equal(r["part"], runs[0]["part"])
        assert r["L"] == runs[0]["L"] and r["sweeps"] == runs[0]["sweeps"]
        np.testing.assert_array_equal(r["steps_bits"], runs[0]["steps_bits"])
    assert runs[1]["launches"] == runs[2]["launches"] > runs[0]["launches"]
