"""Performance cases of the k-NN-graph path, through the package's public entry
points: `build_graph` in its forms, `build_graph_batched`, `build_graph_stream`
and queries of a built `Index`.

`listed()` names the cases, `draw(rng)` gives another of the same ranges,
`prepare(case, seed)` makes what a program holds before the call, `run(state)`
is one call, `work(case)` what it cannot do without and `exact(case, seed)` the
exact k nearest neighbours' distances in 64 bits where that is quick (the trees
find most of them: a missed neighbour leaves a slightly larger distance).

Inputs have the shapes and distributions of `drpt_b200.synth`, drawn on the GPU
from the seed alone.
"""
from __future__ import annotations

import math

import numpy as np
import torch

from drpt_b200 import build_graph, build_graph_batched, build_graph_stream, build_index

SEED = 12345  # of the projections, as in bench.py

# the largest listed amount of leaf work (flops of the pairs), which no drawn case exceeds
_MOST = 2.0 * 500_000 * 32 * 2048 * 960


def listed() -> list[dict]:
    return [
        # The main workload: a million 128-dim descriptors (SIFT-like), one graph.
        dict(name="mixed-1m-128", kind="build", mode="mixed", data="clustered", n=1_000_000, d=128,
             trees=6, nn=10, leaf=1024),
        # The smallest dataset of the batch workload built on its own: launches and latency.
        dict(name="mixed-2k-96", kind="build", mode="mixed", data="batch", n=2_003, d=96, trees=8,
             nn=16, leaf=512),
        # 60,000 x 784 byte images (MNIST-shaped), Gaussian projection.
        dict(name="u8-60k-784", kind="build", mode="mixed", data="images", n=60_000, d=784,
             trees=12, nn=10, leaf=1024),
        # The same images with the integer sign projection, an odd number of them.
        dict(name="u8-sign-31k-784", kind="build", mode="mixed", data="images", n=31_337, d=784,
             trees=12, nn=10, leaf=1024, projection="sign"),
        # Wide vectors (GIST-like), E4M3 leaf tiles, nn 20, large leaves, many trees.
        dict(name="fp8-500k-960", kind="build", mode="mixed", data="anisotropic", n=500_000, d=960,
             trees=32, nn=20, leaf=2048, precision="fp8"),
        # Many uneven datasets in one call.
        dict(name="batch-64x96", kind="batch", sets=64, lo=2_000, hi=200_000, d=96, trees=8, nn=16,
             leaf=512),
        # The reference's own method and parameters, bit for bit.
        dict(name="exact-131k-128", kind="build", mode="exact", data="broad", n=131_072, d=128,
             trees=16, nn=10),
        # The FP32 form of the whole-leaf method on the CUDA cores.
        dict(name="gram-262k-128", kind="build", mode="fp32_gram", data="clustered", n=262_144,
             d=128, trees=6, nn=10, leaf=1024),
        # Vectors on a low-dimensional manifold (embeddings), half of the trees learned.
        dict(name="learned-250k-256", kind="build", mode="mixed", data="manifold", n=250_000,
             d=256, trees=16, nn=10, leaf=1024, learned=8, iters=3),
        # Serving: one query against a built index, and a large block of queries.
        dict(name="query-1", kind="query", n=262_144, d=128, trees=6, nn=10, leaf=1024, nq=1),
        dict(name="query-50k", kind="query", n=262_144, d=128, trees=6, nn=10, leaf=1024,
             nq=50_000),
        # Datasets that lie in host memory, one call for several, copies and builds overlapped.
        dict(name="stream-3x131k-128", kind="stream", jobs=3, n=131_071, d=128, trees=6, nn=10,
             leaf=1024),
    ]


def _log(rng, lo, hi) -> int:
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng) -> dict:
    """A case of the listed ranges: sizes spread over their logarithms, mostly odd."""
    while True:
        kind = rng.choice(["mixed", "mixed", "images", "wide", "batch", "exact", "gram", "learned",
                           "query", "query", "stream"])
        if kind == "mixed":
            nn = rng.choice([5, 10, 16, 20])
            c = dict(kind="build", mode="mixed", data=rng.choice(["clustered", "batch"]),
                     n=_log(rng, 2_000, 1_000_000), d=4 * _log(rng, 8, 64), trees=rng.randint(2, 12),
                     nn=nn, leaf=rng.choice([256, 512, 1024]))
        elif kind == "images":
            c = dict(kind="build", mode="mixed", data="images", n=_log(rng, 8_000, 80_000),
                     d=rng.choice([784, 784, 1024, 512]), trees=rng.randint(4, 12), nn=10,
                     leaf=rng.choice([512, 1024]), projection=rng.choice(["gaussian", "sign"]))
        elif kind == "wide":
            c = dict(kind="build", mode="mixed", data="anisotropic", n=_log(rng, 20_000, 400_000),
                     d=4 * rng.randint(96, 250), trees=rng.randint(4, 24), nn=rng.choice([10, 20]),
                     leaf=rng.choice([1024, 2048]), precision=rng.choice(["bf16", "fp8"]))
        elif kind == "batch":
            c = dict(kind="batch", sets=_log(rng, 3, 100), lo=2_000, hi=_log(rng, 10_000, 200_000),
                     d=4 * rng.randint(16, 32), trees=rng.randint(4, 8), nn=rng.choice([10, 16]),
                     leaf=rng.choice([256, 512, 1024]))
        elif kind == "exact":
            c = dict(kind="build", mode="exact", data="broad", n=_log(rng, 60_000, 262_144),
                     d=_log(rng, 32, 256), trees=rng.randint(4, 16), nn=10)
        elif kind == "gram":
            c = dict(kind="build", mode="fp32_gram", data="clustered", n=_log(rng, 20_000, 400_000),
                     d=8 * _log(rng, 8, 64), trees=rng.randint(2, 8), nn=rng.choice([10, 20]),
                     leaf=rng.choice([512, 1024]))
        elif kind == "learned":
            trees = rng.randint(4, 16)
            c = dict(kind="build", mode="mixed", data="manifold", n=_log(rng, 50_000, 400_000),
                     d=4 * rng.randint(24, 64), trees=trees, nn=10, leaf=1024,
                     learned=rng.randint(1, trees // 2), iters=3)
        elif kind == "query":
            c = dict(kind="query", n=_log(rng, 20_000, 400_000), d=4 * _log(rng, 8, 64),
                     trees=rng.randint(2, 8), nn=rng.choice([1, 10, 20]), leaf=1024,
                     nq=_log(rng, 1, 60_000))
        else:
            c = dict(kind="stream", jobs=rng.randint(2, 4), n=_log(rng, 10_000, 150_000),
                     d=4 * rng.randint(8, 32), trees=rng.randint(2, 8), nn=10,
                     leaf=rng.choice([512, 1024]))
        if work(c)["flops"] <= _MOST:
            return c


# ------------------------------------------------------------------ inputs
def _gen(seed: int) -> torch.Generator:
    return torch.Generator(device="cuda").manual_seed(int(seed) + 1)


def _mix(g, n: int, d: int, k: int, lo: float, hi: float, sigma: float, clip=None) -> torch.Tensor:
    """A mixture of k Gaussians, centres uniform in [lo, hi]^d."""
    x = torch.randn(n, d, generator=g, device="cuda") * sigma
    c = torch.rand(k, d, generator=g, device="cuda") * (hi - lo) + lo
    x += c[torch.randint(k, (n,), generator=g, device="cuda")]
    return x.clamp_(*clip) if clip else x


def _rows(data: str, n: int, d: int, g) -> torch.Tensor:
    if data == "clustered":  # about a thousand points a cluster
        return _mix(g, n, d, max(2, n // 1000), 0.0, 200.0, 12.0, (0.0, 255.0))
    if data == "broad":  # clusters that overlap: no global leaf is empty or tiny
        return _mix(g, n, d, max(2, n // 1000), 0.0, 200.0, 60.0)
    if data == "batch":
        return _mix(g, n, d, 100, -10.0, 10.0, 1.0)
    if data == "anisotropic":
        k = max(2, n // 4000)
        c = torch.rand(k, d, generator=g, device="cuda")
        s = torch.rand(k, d, generator=g, device="cuda") * 0.29 + 0.01
        w = torch.randint(k, (n,), generator=g, device="cuda")
        x = torch.randn(n, d, generator=g, device="cuda")
        for i in range(0, n, 1 << 16):
            j = slice(i, i + (1 << 16))
            x[j] = (x[j] * s[w[j]] + c[w[j]]).clamp_(0.0, 1.0)
        return x
    if data == "images":  # ten centres, four fifths of each one's pixels dark
        c = (torch.randn(10, d, generator=g, device="cuda") * 60.0 + 128.0).clamp_(0, 255)
        lit = torch.rand(10, d, generator=g, device="cuda") >= 0.8
        w = torch.randint(10, (n,), generator=g, device="cuda")
        x = torch.randn(n, d, generator=g, device="cuda") * 20.0 + (c * lit)[w]
        return (x.round_().clamp_(0, 255) * lit[w]).to(torch.uint8)
    if data == "manifold":
        a = torch.randn(16, d, generator=g, device="cuda")
        b = torch.randn(d, generator=g, device="cuda")
        x = torch.randn(n, d, generator=g, device="cuda") * 0.05
        z = torch.randn(n, 16, generator=g, device="cuda")
        for k in range(16):  # z @ a, one rank at a time: the same bits everywhere
            b = b + z[:, k:k + 1] * a[k] if k else b + z[:, :1] * a[0]
        return x + torch.tanh(b) * 4.0
    raise ValueError(data)


def _sizes(case: dict) -> np.ndarray:
    """Sizes of a batch's datasets, log-uniform: part of the case, not of the seed."""
    r = np.random.default_rng(case["sets"] * 1_000_003 + case["hi"])
    return np.exp(r.uniform(np.log(case["lo"]), np.log(case["hi"]), case["sets"])).astype(np.int64)


def _inputs(case: dict, seed: int):
    g = _gen(seed)
    if case["kind"] == "build":
        return _rows(case["data"], case["n"], case["d"], g)
    if case["kind"] == "batch":
        return torch.cat([_rows("batch", int(m), case["d"], g) for m in _sizes(case)])
    if case["kind"] == "query":
        x = _rows("clustered", case["n"] + case["nq"], case["d"], g)
        return x[:case["n"]].clone(), x[case["n"]:].clone()
    return [_rows("clustered", case["n"], case["d"], g) for _ in range(case["jobs"])]


def _options(case: dict) -> dict:
    o = dict(mode=case["mode"])
    for key, name in (("leaf", "leaf_size"), ("precision", "precision"),
                      ("projection", "projection"), ("learned", "learned_trees"),
                      ("iters", "learn_iters")):
        if key in case:
            o[name] = case[key]
    return o


def prepare(case: dict, seed: int) -> dict:
    x = _inputs(case, seed)
    kind = case["kind"]
    if kind == "build":
        return dict(case=case, x=x, options=_options(case))
    if kind == "batch":
        return dict(case=case, x=x, offsets=np.concatenate([[0], np.cumsum(_sizes(case))]))
    if kind == "query":
        index = build_index(x[0], case["trees"], case["nn"], SEED, leaf_size=case["leaf"])[0]
        return dict(case=case, index=index, q=x[1])
    n, nn = case["n"], case["nn"]  # pinned, so that the copies can overlap the builds
    return dict(case=case, x=[r.cpu().pin_memory().numpy() for r in x],
                outs=[(torch.empty((n, nn), dtype=torch.int32).pin_memory().numpy(),
                       torch.empty((n, nn), dtype=torch.float32).pin_memory().numpy())
                      for _ in x])


def run(state: dict):
    case = state["case"]
    if case["kind"] == "build":
        idx, dist, _ = build_graph(state["x"], case["trees"], case["nn"], SEED,
                                   **state["options"])
    elif case["kind"] == "batch":
        idx, dist, _ = build_graph_batched(state["x"], state["offsets"], case["trees"], case["nn"],
                                           SEED, leaf_size=case["leaf"])
    elif case["kind"] == "query":
        idx, dist = state["index"].query(state["q"], case["nn"])
    else:
        outs, _ = build_graph_stream(state["x"], case["trees"], case["nn"], SEED,
                                     leaf_size=case["leaf"], outs=state["outs"])
        return [dict(idx=i, dist=d) for i, d in outs]
    return dict(idx=idx, dist=dist)


# ------------------------------------------------------------------ work
def _points(case: dict) -> int:
    return {"batch": lambda: int(_sizes(case).sum()), "stream": lambda: case["jobs"] * case["n"],
            "query": lambda: case["nq"]}.get(case["kind"], lambda: case["n"])()


def _leaf(case: dict) -> float:
    """Points of a leaf: halved from n until at most the asked size."""
    n = case["n"] if case["kind"] != "batch" else float(np.mean(_sizes(case)))
    if case.get("mode") == "exact":  # the reference's depths: global, then local by the leaf size
        n = n / 2 ** (int(int(math.log2(n) - 2) * 0.6) - 1)
        return n / 2 ** max(1, int(math.log2(n) - math.log2(case["nn"]) - 2))
    while n > case["leaf"]:
        n /= 2
    return n


def work(case: dict) -> dict:
    """Bytes: each input row read once, each list written once (a query reads the rows of its
    leaves, at most all).  Flops: a multiply and an add per dimension and pair of a leaf."""
    m, d, leaf = _points(case), case["d"], _leaf(case)
    pairs = m * case["trees"] * leaf
    esz = 1 if case.get("data") == "images" else 4
    rows = m + min(case["n"], pairs) if case["kind"] == "query" else m
    return {"bytes": rows * d * esz + m * case["nn"] * 8, "flops": 2.0 * pairs * d}


# ------------------------------------------------------------------ exact
def _nearest(x: torch.Tensor, q: torch.Tensor, k: int, own: bool) -> torch.Tensor:
    """Distances of the k nearest rows of x to each row of q in 64 bits; `own`: q is x, and a row
    is not its own neighbour."""
    x, q = x.double(), q.double()
    sq, out = (x * x).sum(1), []
    step = max(1, min(4096, (1 << 28) // len(x)))
    for i in range(0, len(q), step):
        b = q[i:i + step]
        d2 = (b * b).sum(1)[:, None] + sq[None] - 2.0 * (b @ x.T)
        if own:
            d2[torch.arange(len(b)), torch.arange(i, i + len(b))] = math.inf
        near = torch.topk(d2, min(k + 4, len(x) - 1), dim=1, largest=False).indices
        e = torch.stack([(x[near[:, j]] - b).square().sum(1) for j in range(near.shape[1])], 1)
        out.append(e.sqrt().sort(1).values[:, :k])
    return torch.cat(out)


def exact(case: dict, seed: int):
    """The exact neighbours' distances.  None for the graph of a method that only samples its
    leaves (the reference's positional split) and where all pairs would take too long."""
    kind, k = case["kind"], case["nn"]
    pairs = {"query": lambda: case["nq"] * case["n"],
             "batch": lambda: int((_sizes(case).astype(float) ** 2).sum()),
             "stream": lambda: case["jobs"] * case["n"] ** 2}.get(kind, lambda: case["n"] ** 2)()
    if case.get("mode") == "exact" or pairs * max(case["d"], 256) > 8e12:
        return None
    x = _inputs(case, seed)
    if kind == "build":
        return dict(idx=None, dist=_nearest(x, x, k, True))
    if kind == "query":
        return dict(idx=None, dist=_nearest(x[0], x[1], k, False))
    if kind == "batch":
        parts = torch.split(x, [int(m) for m in _sizes(case)])
        return dict(idx=None, dist=torch.cat([_nearest(p, p, k, True) for p in parts]))
    return [dict(idx=None, dist=_nearest(r, r, k, True)) for r in x]
