"""Performance cases: the calls a user of the library makes, over the range of sizes they are made at.

listed()            the named cases
draw(rng)           one more case of the same ranges
prepare(case, seed) a user's inputs (host arrays, device tensors) and the handle kept between calls
run(state)          one pass through the public entry points, and its outputs
work(case)          compulsory bytes and operations of one pass: inputs read once, outputs written once
exact(case, seed)   the outputs that are computed numbers, in plain FP64 torch
"""
from __future__ import annotations

import math

import numpy as np
import torch

from relaxmap_b200 import Batch, Graph
from relaxmap_b200._lib import steady_state_noalloc

DEV = "cuda"
TAU = 0.15


# ---------------------------------------------------------------- the cases


def _planted(name, op, n, deg, kmax, cmin, cmax, mu, weights, **more):
    return {"name": name, "op": op, "graph": "planted", "n": n, "deg": float(deg), "kmax": kmax, "cmin": cmin,
            "cmax": cmax, "mu": mu, "weights": weights, **more}


def _rmat(name, op, scale, weights="none", **more):
    return {"name": name, "op": op, "graph": "rmat", "n": 1 << scale, "scale": scale, "deg": 16.0,
            "weights": weights, **more}


def listed():
    return [
        # the smallest optimiser run: an unweighted LFR-style network of 1000 nodes (the small configuration)
        _planted("optimize 1k", "optimize", 1000, 20, 50, 10, 50, 0.3, "none", prior=True, attempts=1),
        # an ordinary network in normal mode (every sweep takes every unit)
        _planted("optimize 20k normal", "optimize", 20011, 11, 110, 10, 200, 0.45, "none", prior=False, attempts=1),
        # an ordinary weighted network in prior mode
        _planted("optimize 150k", "optimize", 150001, 20, 1000, 20, 1000, 0.4, "uniform", prior=True, attempts=1),
        # the mid configuration: a million nodes, 20 million weighted links
        _planted("optimize 1m", "optimize", 1000000, 20, 1000, 20, 1000, 0.4, "uniform", prior=True, attempts=1),
        # a skewed network of the R-MAT family, as the CPU baseline's sample
        _rmat("optimize rmat18", "optimize", 18, prior=True, attempts=1),
        # the largest R-MAT network of which three handles fit one device
        _rmat("optimize rmat23", "optimize", 23, prior=True, attempts=1),
        # a program that meets a network once: host edge list in, best of three attempts out, handle closed
        _planted("once 60k", "once", 60013, 14, 400, 10, 500, 0.35, "lognormal", prior=True, attempts=3,
                 node_weights=True),
        # the graph build alone, from a host edge list with duplicate pairs and self-links, and the kept links back
        _rmat("build rmat19", "build", 19, "uniform"),
        # the stationary flow on a caller's own device arrays: one small network, and a large one
        _planted("flow 3k", "flow", 3001, 9, 90, 10, 100, 0.3, "none"),
        _planted("flow 700k", "flow", 700001, 20, 1000, 20, 1000, 0.3, "lognormal"),
        # the code length of a fixed partition and its gradient by every link weight (the adjoint configuration's shape)
        _planted("gradient 250k", "gradient", 250007, 20, 1000, 20, 1000, 0.3, "lognormal", tau=TAU),
        # many small networks optimised together, several attempts each (the batched configuration's ranges)
        {"name": "batch 40x4", "op": "batch", "graph": "many", "count": 40, "nmin": 200, "nmax": 20000, "attempts": 4},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["optimize", "optimize", "optimize", "rmat", "rmat", "once", "build", "flow", "flow",
                       "gradient", "batch"])
    mu = round(rng.uniform(0.1, 0.6), 3)
    deg = round(rng.uniform(5, 24), 2)
    weights = rng.choice(["none", "uniform", "lognormal"])

    def planted(op, n, **more):
        kmax = max(2, min(1000, n // 2, int(10 * deg) if rng.random() < 0.5 else 1000))
        cmin = rng.randint(8, 20)
        cmax = max(cmin + 1, min(1000, n // 4))
        c = _planted("", op, n, deg, kmax, cmin, cmax, mu, weights, **more)
        del c["name"]
        return c

    def rmat(op, scale, w):
        # edge factors around the configurations' 16
        c = _rmat("", op, scale, w, **({} if op == "build" else {"prior": rng.random() < 0.7, "attempts": 1}))
        c["deg"] = round(rng.uniform(6, 16), 2)
        del c["name"]
        return c

    if kind == "optimize":
        return planted("optimize", _log(rng, 500, 800000), prior=rng.random() < 0.7, attempts=rng.choice([1, 1, 2]))
    if kind == "rmat":
        return rmat("optimize", rng.randint(12, 22), "none")
    if kind == "once":
        return planted("once", _log(rng, 500, 200000), prior=rng.random() < 0.7, attempts=rng.randint(1, 4),
                       node_weights=rng.random() < 0.5)
    if kind == "build":
        return rmat("build", rng.randint(12, 20), weights)
    if kind == "flow":
        return planted("flow", _log(rng, 500, 1 << 20))
    if kind == "gradient":
        return planted("gradient", _log(rng, 2000, 400000), tau=round(rng.uniform(0.1, 0.3), 3))
    return {"op": "batch", "graph": "many", "count": rng.randint(4, 60), "nmin": 200,
            "nmax": _log(rng, 1000, 20000), "attempts": rng.randint(1, 4)}


# ---------------------------------------------------------------- inputs (drawn on the device, handed over on the host)


def _powerlaw_low(mean, kmax):
    """The lower end of a power law of exponent 2 up to kmax with the given mean."""
    lo, hi = 1e-3, float(kmax)
    for _ in range(100):
        a = 0.5 * (lo + hi)
        m = a * kmax * math.log(kmax / a) / (kmax - a) if a < kmax else kmax
        lo, hi = (a, hi) if m < mean else (lo, a)
    return lo


def _draw_planted(gen, n, deg, kmax, cmin, cmax, mu):
    """LFR-style: power-law out-degrees (exponent 2), community sizes power law (1) in [cmin, cmax], a share mu of
    the links anywhere; no self-links, no duplicate pairs. int64 (src, dst) on the device and the communities."""
    def rnd(k):
        return torch.rand(k, generator=gen, device=DEV, dtype=torch.float64)
    sizes = torch.round(cmin * (cmax / cmin) ** rnd(max(4, 3 * n // cmin + 8))).long()
    ends = torch.cumsum(sizes, 0)
    ends = torch.clamp(ends[: int((ends < n).sum()) + 1], max=n)
    start = torch.cat([torch.zeros(1, dtype=torch.long, device=DEV), ends[:-1]])
    place = torch.randperm(n, generator=gen, device=DEV)  # node at each place; communities are runs of places
    comm_at = torch.searchsorted(ends, torch.arange(n, device=DEV), right=True)
    comm = torch.empty_like(comm_at)
    comm[place] = comm_at
    lo = _powerlaw_low(deg, kmax)
    k = torch.clamp(torch.round(lo / (1.0 - rnd(n) * (1.0 - lo / kmax))).long(), 1, kmax)
    src = torch.repeat_interleave(torch.arange(n, device=DEV), k)
    c = comm[src]
    inside = rnd(src.numel()) >= mu
    u = rnd(src.numel())
    size = ends - start
    near = place[start[c] + torch.clamp((u * size[c]).long(), max=n).minimum(size[c] - 1)]
    far = torch.clamp((u * n).long(), max=n - 1)
    dst = torch.where(inside, near, far)
    key = torch.unique((src * n + dst)[src != dst])
    # the same number of links for every seed: surplus pairs dropped at random, missing ones drawn anywhere
    want = _planted_links(n, deg)
    while key.numel() < want:
        more = (rnd(2 * (want - key.numel()) + 8) * n * n).long()
        key = torch.unique(torch.cat([key, more[more // n != more % n]]))
    if key.numel() > want:
        key = torch.sort(key[torch.randperm(key.numel(), generator=gen, device=DEV)[:want]]).values
    return key // n, key % n, comm


def _planted_links(n, deg):
    return int(0.95 * n * min(deg, n / 8))


def _draw_rmat(gen, scale, m):
    """R-MAT (0.57, 0.19, 0.19, 0.05), ids permuted, self-links and duplicate pairs removed."""
    n = 1 << scale
    keys = []
    for s0 in range(0, m, 1 << 25):
        k = min(1 << 25, m - s0)
        u = torch.zeros(k, dtype=torch.int64, device=DEV)
        v = torch.zeros(k, dtype=torch.int64, device=DEV)
        for lvl in range(scale):
            r = torch.rand(k, generator=gen, device=DEV)
            u |= (r >= 0.76).long() << lvl
            v |= (((r >= 0.57) & (r < 0.76)) | (r >= 0.95)).long() << lvl
        keys.append(torch.unique((u * n + v)[u != v]))
    key = torch.unique(torch.cat(keys))
    perm = torch.randperm(n, generator=gen, device=DEV)
    return perm[key // n], perm[key % n]


def _rmat_pairs(case):
    return int(0.6 * case["deg"] * case["n"])


def _draw_weights(gen, m, kind):
    if kind == "uniform":
        return 1.0 + 9.0 * torch.rand(m, generator=gen, device=DEV, dtype=torch.float64)
    if kind == "lognormal":
        return torch.exp(torch.randn(m, generator=gen, device=DEV, dtype=torch.float64))
    return None


def _draw_graph(case, seed):
    """(src, dst, weights or None, communities or None) on the device."""
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed) * 7919 + 17)
    comm = None
    if case["graph"] == "planted":
        src, dst, comm = _draw_planted(gen, case["n"], case["deg"], case["kmax"], case["cmin"], case["cmax"],
                                       case["mu"])
    else:
        src, dst = _draw_rmat(gen, case["scale"], int(case["deg"] * case["n"]))
        if case["op"] == "build":
            # as a raw edge list: shuffled, an eighth of the pairs given twice, a few self-links; the number of
            # distinct pairs is the same for every seed
            n, kept = case["n"], _rmat_pairs(case)
            pick = torch.randperm(src.numel(), generator=gen, device=DEV)[:kept]
            again = pick[: kept // 8]
            own = torch.randint(n, (n // 64,), generator=gen, device=DEV)
            src, dst = torch.cat([src[pick], src[again], own]), torch.cat([dst[pick], dst[again], own])
            mix = torch.randperm(src.numel(), generator=gen, device=DEV)
            src, dst = src[mix], dst[mix]
    return src, dst, _draw_weights(gen, src.numel(), case["weights"]), comm


def _host_edges(case, seed):
    src, dst, w, comm = _draw_graph(case, seed)
    host = {"n": case["n"], "src": src.int().cpu().numpy(), "dst": dst.int().cpu().numpy(),
            "w": None if w is None else w.cpu().numpy(), "node_w": None}
    if case.get("node_weights"):
        host["node_w"] = np.random.default_rng(seed).uniform(0.5, 4.0, case["n"])
    return host, comm


def _in_links(src, dst, w, n):
    """The in-links as CSC with row-normalised weights, and the dangling nodes."""
    if w is None:
        w = torch.ones(src.numel(), dtype=torch.float64, device=DEV)
    out = torch.segment_reduce(w, "sum", lengths=torch.bincount(src, minlength=n))
    order = torch.argsort(dst * n + src)
    off = torch.zeros(n + 1, dtype=torch.int64, device=DEV)
    off[1:] = torch.cumsum(torch.bincount(dst, minlength=n), 0)
    return off, src[order].int(), (w / out[src])[order], (torch.bincount(src, minlength=n) == 0).to(torch.uint8)


def prepare(case, seed):
    op = case["op"]
    st = {"op": op, "seed": int(seed) % 100000 + 1}
    if op == "batch":
        st["batch"] = Batch(_many(case, seed))
        st["opts"] = {"attempts": case["attempts"], "seed": st["seed"]}
        return st
    if op == "flow":
        n = case["n"]
        src, dst, w, _ = _draw_graph(case, seed)
        st["off"], st["src"], st["w"], st["dangling"] = _in_links(src, dst, w, n)
        st["tw"] = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
        st["p"] = torch.zeros(n, dtype=torch.float64, device=DEV)
        st["iters"] = torch.zeros(1, dtype=torch.int32, device=DEV)
        return st
    host, comm = _host_edges(case, seed)
    if op in ("optimize", "once"):
        st["opts"] = {"seed": st["seed"], "prior": int(case["prior"]), "attempts": case["attempts"]}
    if op in ("once", "build"):
        st["edges"] = host
        return st
    st["graph"] = Graph.from_edges(host["src"], host["dst"], host["w"], n=host["n"])
    if op == "gradient":
        st["part"] = comm.int().cpu().numpy()
        st["tau"] = case["tau"]
    return st


def _many(case, seed):
    """Graphs of the batched configuration's ranges: nodes (the same for every seed), mean degree and mixing
    uniform, one draw per graph."""
    rng = np.random.default_rng(int(seed))
    sizes = np.random.default_rng(case["count"]).integers(case["nmin"], case["nmax"] + 1, case["count"])
    graphs = []
    for n in sizes.tolist():
        deg, mu = float(rng.uniform(5, 30)), float(rng.uniform(0.1, 0.6))
        gen = torch.Generator(device=DEV)
        gen.manual_seed(int(rng.integers(1 << 40)))
        src, dst, _c = _draw_planted(gen, n, deg, max(2, min(n // 2, int(10 * deg))), 10, 200, mu)
        graphs.append((n, src.int().cpu().numpy(), dst.int().cpu().numpy(), None))
    return graphs


# ---------------------------------------------------------------- one pass


def _whole(r):
    """An optimiser result with its list of supersteps, whose length varies, in an array of fixed length."""
    steps = np.zeros(64)
    k = min(64, len(r["steps_bits"]))
    steps[:k] = r["steps_bits"][:k]
    return {"part": r["part"], "L": r["L"], "n_modules": r["n_modules"], "steps_bits": steps}


def run(st):
    op = st["op"]
    if op == "optimize":  # a resident graph: flow, all supersteps, the partition back
        st["graph"].reset_flow()
        return _whole(st["graph"].optimize(**st["opts"]))
    if op == "once":
        e = st["edges"]
        with Graph.from_edges(e["src"], e["dst"], e["w"], n=e["n"], node_w=e["node_w"]) as g:
            return _whole(g.optimize(**st["opts"]))
    if op == "build":
        e = st["edges"]
        with Graph.from_edges(e["src"], e["dst"], e["w"], n=e["n"], node_w=e["node_w"]) as g:
            off, dst, w, tw = g.links()
            return {"off": off, "dst": dst, "w": w, "tw": tw, "self": g.n_self}
    if op == "flow":
        steady_state_noalloc(st["p"].numel(), st["src"].numel(), st["off"].data_ptr(), st["src"].data_ptr(),
                             st["w"].data_ptr(), st["tw"].data_ptr(), st["dangling"].data_ptr(), st["p"].data_ptr(),
                             iters_ptr=st["iters"].data_ptr(), stream_ptr=torch.cuda.current_stream().cuda_stream)
        return {"p": st["p"]}
    if op == "gradient":
        return st["graph"].adjoint_backward(st["part"], st["tau"])
    return st["batch"].optimize(**st["opts"])


def work(case):
    if case["op"] == "batch":
        n = case["count"] * 0.5 * (case["nmin"] + case["nmax"])
        e = 17.5 * n * 0.9
        return {"bytes": 8 * e + 4 * n, "flops": 40 * e * case["attempts"]}
    n = case["n"]
    if case["graph"] == "planted":
        e = _planted_links(n, case["deg"])
    else:
        e = _rmat_pairs(case) if case["op"] == "build" else int(0.95 * case["deg"] * n)
    wide = 0 if case["weights"] == "none" else 8
    if case["op"] == "flow":  # off, src, w, teleport, dangling in; p out
        return {"bytes": 12 * e + 25 * n, "flops": 2 * 50 * e}
    if case["op"] == "build":  # src, dst, w in; off, dst, w, tw out
        return {"bytes": (8 + wide) * (e + e // 8 + n // 64) + 12 * e + 16 * n, "flops": 0.0}
    if case["op"] == "gradient":  # links and partition in; a derivative per link out
        return {"bytes": 20 * e + 12 * n, "flops": 4 * 50 * e}
    # links in, modules out; one evaluation of every link's module per attempt at the least
    return {"bytes": (8 + wide) * e + 4 * n, "flops": (2 * 50 + 40 * case["attempts"]) * e}


# ---------------------------------------------------------------- the same in plain FP64


def _pull(src, dst, w, n):
    """x -> sum over links a -> b of w_ab x_a, at b."""
    m = torch.sparse_coo_tensor(torch.stack([dst, src]), w, (n, n)).coalesce().to_sparse_csr()
    return lambda x: (m @ x.unsqueeze(1)).squeeze(1)


def _stationary(pull, tw, dang, tau):
    """p = (1-tau) W^T p + (tau + (1-tau) d.p) tw, iterated well past FP64 rounding."""
    p = tw.clone()
    for _ in range(400):
        q = (1 - tau) * pull(p) + (tau + (1 - tau) * p[dang].sum()) * tw
        q = q / q.sum()
        done = float((q - p).abs().sum()) < 1e-16
        p = q
        if done:
            break
    return p


def _plogp(x):
    return torch.where(x > 0, x * torch.log(torch.where(x > 0, x, torch.ones_like(x))), torch.zeros_like(x))


def _exact_build(case, seed):
    host, _ = _host_edges(case, seed)
    n = host["n"]
    key = host["src"].astype(np.int64) * n + host["dst"]
    order = np.argsort(key, kind="stable")
    w = np.ones(len(key)) if host["w"] is None else host["w"]
    k, at = np.unique(key[order], return_index=True)
    s = np.add.reduceat(w[order], at)
    keep = (k // n != k % n) & (s > 0)
    off = np.zeros(n + 1, dtype=np.int64)
    np.cumsum(np.bincount(k[keep] // n, minlength=n), out=off[1:])
    return {"off": off, "dst": (k[keep] % n).astype(np.int32), "w": s[keep], "tw": np.full(n, 1.0 / n),
            "self": int(((k // n == k % n) & (s > 0)).sum())}


def _exact_gradient(case, seed):
    """Code length and its derivatives by automatic differentiation of the closed form in p, with the stationary
    flow's own derivative from the transposed system."""
    n, tau = case["n"], case["tau"]
    src, dst, w, comm = _draw_graph(case, seed)  # already in (src, dst) order, no duplicates
    tw = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
    if w is None:
        w = torch.ones(src.numel(), dtype=torch.float64, device=DEV)
    rows = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, src, w)
    dang = rows == 0
    wn0 = w / rows[src]
    p0 = _stationary(_pull(src, dst, wn0, n), tw, dang, tau)
    p = p0.clone().requires_grad_()
    wn = wn0.clone().requires_grad_()
    t = torch.tensor(tau, dtype=torch.float64, device=DEV, requires_grad=True)

    def per_module(x, at):
        return torch.zeros(n, dtype=torch.float64, device=DEV).index_add(0, at, x)
    crossing = (comm[src] != comm[dst]).double()
    out = per_module(p[src] * wn * crossing, comm[src])
    P, T, D = per_module(p, comm), per_module(tw, comm), per_module(p * dang.double(), comm)
    q = t * (1 - T) * P + (1 - t) * (out + (1 - T) * D)
    length = _plogp(q.sum()) - 2 * _plogp(q).sum() + _plogp(q + P).sum() - _plogp(p).sum()
    c, gw, gt = torch.autograd.grad(length, [p, wn, t])
    # lambda = c + (1-t)(W lambda + d (tw . lambda)) with tw . lambda = p.c / t
    push = _pull(dst, src, wn0, n)
    target = (p0 * c).sum() / tau
    lam = c + (target - (tw * c).sum())
    for _ in range(500):
        new = c + (1 - tau) * (push(lam) + dang.double() * target)
        new = new + (target - (tw * new).sum())
        done = float((new - lam).abs().sum()) <= 1e-16 * float(new.abs().sum())
        lam = new
        if done:
            break
    g = gw + (1 - tau) * p0[src] * lam[dst]
    mean = torch.zeros(n, dtype=torch.float64, device=DEV).index_add_(0, src, wn0 * g)
    dt = gt + ((lam * tw).sum() - (lam * p0).sum()) / (1 - tau)
    return {"dL_dw": (g - mean[src]) / rows[src], "dL_dtau": float(dt), "L": float(length)}


def exact(case, seed):
    if case["op"] == "flow":
        src, dst, w, _ = _draw_graph(case, seed)
        n = case["n"]
        off, s, wn, dang = _in_links(src, dst, w, n)
        to = torch.repeat_interleave(torch.arange(n, device=DEV), off[1:] - off[:-1])
        tw = torch.full((n,), 1.0 / n, dtype=torch.float64, device=DEV)
        return {"p": _stationary(_pull(s.long(), to, wn, n), tw, dang.bool(), TAU)}
    if case["op"] == "build":
        return _exact_build(case, seed)
    if case["op"] == "gradient":
        return _exact_gradient(case, seed)
    return None  # a partition: its code length has no value without it
