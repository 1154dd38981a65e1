"""Performance cases of the exact epsilon-join: what a user's program asks of the public entry points.

Each case is a dict of plain values; ``prepare`` makes its inputs and threshold on the GPU from a
seed, ``run`` is one call a user makes, ``work`` is what that call cannot do without.  The point set
of a case is one draw of its distribution; the seed gives every dimension a sign and a place and
every row a place, which moves all values and ids but, distances being the same, keeps the number of
result pairs, so that outputs of all seeds have one shape.  Kinds:

* ``mixture``  R-S join of two Gaussian-mixture samples (clustered embeddings), device or host rows
* ``factor``   joins of L2-normalised rows of a rank-32 factor model (dense embeddings: no pruning)
* ``uniform``  self-join (i < j) of U[0,1)^d rows, the classic grid-join benchmark
* ``planar``   self-join of clustered 2-D points with many neighbours, as a neighbour table
* ``int14``    exact join of quantised rows with near-duplicates (two int8 limbs per element)
* ``batch``    many independent ragged R-S joins in one call

The thresholds are quantiles of sampled FP64 distances that give a target number of neighbours per
row, as in ``tensorjoin_variants_b200.workloads``, whose five configurations these cases follow.
All results are row numbers, which every path computes exactly, so there is no rounded output whose
64-bit value ``exact`` could give.
"""
from __future__ import annotations

import math

import torch

import tensorjoin_variants_b200 as tj
from tensorjoin_variants_b200 import workloads

DIMS = {"all": (8, 32, 128), "low": (8, 32), "high": (32, 128)}


def listed():
    return [
        # one query batch against a small table: the smallest single call, latency only
        dict(name="join_small", kind="mixture", n_r=311, n_s=256, d=8, clusters=8, degree=16, screen="bf16",
             host=False),
        # an ordinary small join of odd shape with the default screen
        dict(name="join_odd", kind="mixture", n_r=5003, n_s=3217, d=65, clusters=8, degree=16, screen="bf16",
             host=False),
        # host rows in, host ids out, as a script that holds its data in pinned memory calls it
        dict(name="join_host", kind="mixture", n_r=90007, n_s=131071, d=33, clusters=64, degree=16,
             screen="fp16x3", host=True),
        # clustered embeddings at full size (1M x 1M, 64-d mixture)
        dict(name="mixture64", kind="mixture", n_r=1_000_000, n_s=1_000_000, d=64, clusters=64, degree=16,
             screen="bf16x3", host=False),
        # the plain exact self-join of the grid-join papers (20,000 x 16)
        dict(name="uniform16", kind="uniform", n=20_000, d=16, degree=32, screen="plain"),
        # low dimension, hundreds of neighbours per point, neighbour-table output (the 100,000-point 2-D set)
        dict(name="planar_table", kind="planar", n=100_000, degree=280, screen="plain"),
        # canonical directed self-join of 60,000 x 512 descriptors with ~64 neighbours
        dict(name="directed512", kind="factor", n=60_000, d=512, mode="directed", degree=64, screen="fp16"),
        # dense embeddings at full size (500k x 500k, d = 512)
        dict(name="factor512", kind="factor", n=500_000, d=512, mode="rs", degree=8, screen="bf16"),
        # quantised rows of odd width, directed output
        dict(name="int14_odd", kind="int14", n=50_021, d=100, mode="directed", degree=24),
        # quantised near-duplicate search at full size (2M x 128)
        dict(name="int14x128", kind="int14", n=2_000_000, d=128, mode="upper", degree=24),
        # a few dozen small joins in one call
        dict(name="batch_small", kind="batch", joins=64, lo=256, hi=4096, dims="all", degree=16, screen="bf16x3"),
        # a large ragged batch (half of the 4,096-join configuration: three of it fit the card at once)
        dict(name="batch_ragged", kind="batch", joins=2048, lo=256, hi=65536, dims="all", degree=16,
             screen="bf16x3"),
    ]


def _log_int(rng, lo, hi):
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["mixture", "mixture", "mixture", "factor", "uniform", "planar", "int14", "batch"])
    if kind == "mixture":
        while True:
            n_r, n_s, d = _log_int(rng, 256, 1_000_000), _log_int(rng, 256, 1_000_000), _log_int(rng, 8, 130)
            clusters = 8 if max(n_r, n_s) <= 65536 else 64
            if n_r * n_s // clusters * d <= 10 ** 12:
                return dict(kind=kind, n_r=n_r, n_s=n_s, d=d, clusters=clusters, degree=rng.randint(4, 32),
                            screen=rng.choice(["bf16", "fp16", "bf16x3", "fp16x3", "plain"]),
                            host=rng.random() < 0.25)
    if kind == "factor":
        while True:
            n, d = _log_int(rng, 3000, 400_000), rng.randint(200, 784)
            if n * n * d <= 64 * 10 ** 12:
                return dict(kind=kind, n=n, d=d, mode=rng.choice(["rs", "directed"]), degree=rng.randint(8, 64),
                            screen=rng.choice(["bf16", "fp16"]))
    if kind == "uniform":
        return dict(kind=kind, n=_log_int(rng, 2000, 100_000), d=rng.randint(6, 24), degree=rng.randint(8, 48),
                    screen=rng.choice(["plain", "bf16x3"]))
    if kind == "planar":
        return dict(kind=kind, n=_log_int(rng, 5000, 100_000), degree=rng.randint(16, 280),
                    screen=rng.choice(["plain", "bf16x3"]))
    if kind == "int14":
        while True:
            n, d = _log_int(rng, 4000, 1_500_000), rng.randint(32, 256)
            if n * n * (1 if d <= 128 else 3) <= 2_000_000 ** 2:
                return dict(kind=kind, n=n, d=d, mode=rng.choice(["upper", "directed"]), degree=rng.randint(4, 32))
    return dict(kind="batch", joins=_log_int(rng, 16, 1024), lo=256, hi=_log_int(rng, 2048, 65536),
                dims=rng.choice(sorted(DIMS)), degree=rng.randint(8, 24), screen=rng.choice(["bf16x3", "bf16"]))


def _threshold(R, S, degree, g):
    """Squared distance that leaves ~``degree`` neighbours per row: a quantile of sampled distances."""
    n_s = S.shape[0]
    q = min(1.0, degree / n_s)
    count = min(1 << 22, max(1 << 18, 1 << int(math.ceil(math.log2(64 / q)))))
    step = max(1, (1 << 27) // R.shape[1])
    d2 = []
    for o in range(0, count, step):
        m = min(step, count - o)
        i = torch.randint(0, R.shape[0], (m,), generator=g, device="cuda")
        j = torch.randint(0, n_s, (m,), generator=g, device="cuda")
        if R is S:
            j = torch.where(j == i, (j + 1) % n_s, j)
        d2.append((R[i].double() - S[j].double()).square_().sum(1))
    d2 = torch.cat(d2).sort().values
    k = min(count - 2, int(q * count))
    t = float(d2[k] + d2[k + 1]) / 2   # between two sampled distances: no sampled pair is a tie
    return t if R.dtype == torch.float32 else math.floor(t)


def _mixture(n, centres, std, g):
    label = torch.randint(0, centres.shape[0], (n,), generator=g, device="cuda")
    x = torch.randn((n, centres.shape[1]), generator=g, device="cuda")
    return x.mul_(std).add_(centres[label])


def _factor(n, W, noise, g):
    x = torch.randn((n, W.shape[0]), generator=g, device="cuda") @ W
    x += noise * torch.randn(x.shape, generator=g, device="cuda")
    return torch.nn.functional.normalize(x, dim=1)


def _moved(sides, seed):
    """The sides with their dimensions reordered and reflected (alike) and their rows reordered."""
    g = torch.Generator("cuda").manual_seed(seed)
    d = sides[0].shape[1]
    place = torch.randperm(d, generator=g, device="cuda")
    flip = torch.randint(0, 2, (d,), generator=g, device="cuda", dtype=torch.int16)
    out = []
    for X in sides:
        X = X[torch.randperm(X.shape[0], generator=g, device="cuda")][:, place]
        # int14: -1 - x, which keeps [-8192, 8191]
        X = X ^ -flip if X.dtype == torch.int16 else X.mul_((1 - 2 * flip).float())
        out.append(X.contiguous())
    return out


def _prepare_batch(case, seed):
    joins, rows = workloads.ragged4096_device(joins=case["joins"], lo=case["lo"], hi=case["hi"],
                                              dims=DIMS[case["dims"]], degree=case["degree"], seed=17)
    g = torch.Generator("cuda").manual_seed(seed)
    for k in range(0, len(rows), 2):   # one dimension's R and S rows, each the joins' rows back to back
        d = rows[k].shape[1]
        flip = 1 - 2 * torch.randint(0, 2, (d,), generator=g, device="cuda").float()
        place = torch.randperm(d, generator=g, device="cuda")
        of_d = [q for q, (R, _, _) in enumerate(joins) if R.shape[1] == d]
        for side in (0, 1):
            sizes = torch.tensor([joins[q][side].shape[0] for q in of_d], device="cuda")
            owner = torch.repeat_interleave(torch.arange(len(of_d), device="cuda"), sizes)
            order = (owner + torch.rand(owner.shape, generator=g, device="cuda", dtype=torch.float64)).argsort()
            rows[k + side].copy_(rows[k + side][order][:, place] * flip)   # the joins are views of it
    return dict(kind="batch", joins=joins, screen=case["screen"])


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        return _prepare_batch(case, seed)
    g = torch.Generator("cuda").manual_seed(17)
    mode, screen = case.get("mode", "rs"), case.get("screen", "int8limb")
    if kind == "mixture":
        centres = torch.rand((case["clusters"], case["d"]), generator=g, device="cuda")
        sides = [_mixture(n, centres, 0.05, g) for n in (case["n_r"], case["n_s"])]
    elif kind == "factor":
        W = torch.randn((32, case["d"]), generator=g, device="cuda") / math.sqrt(32)
        sides = [_factor(case["n"], W, 0.1, g) for _ in range(2 if mode == "rs" else 1)]
    elif kind == "int14":
        n, d = case["n"], case["d"]
        X = torch.randint(-8192, 8192, (n, d), generator=g, device="cuda", dtype=torch.int16)
        m = n // 10   # a tenth of the rows are near-duplicates of other rows
        dst = torch.randperm(n, generator=g, device="cuda")[:m]
        src = torch.randint(0, n, (m,), generator=g, device="cuda")
        jitter = torch.randint(-1, 2, (m, d), generator=g, device="cuda", dtype=torch.int16)
        X[dst] = (X[src] + jitter).clamp_(-8192, 8191)
        sides = [X]
    elif kind == "planar":
        lo, size = torch.tensor([0.0, -90.0], device="cuda"), torch.tensor([360.0, 180.0], device="cuda")
        centres = lo + size * torch.rand((64, 2), generator=g, device="cuda")
        sides, mode = [_mixture(case["n"], centres, 8.0, g)], "table"
    else:
        sides, mode = [torch.rand((case["n"], case["d"]), generator=g, device="cuda")], "upper"
    T = _threshold(sides[0], sides[-1], case["degree"], g)
    sides = _moved(sides, seed)
    if case.get("host"):
        sides = [X.cpu().pin_memory() for X in sides]
    return dict(kind=mode, R=sides[0], S=sides[-1], T=T, screen=screen)


def run(state):
    kind = state["kind"]
    if kind == "batch":
        res = tj.join_batched_result(state["joins"], screen=state["screen"])
        i, j = res.pairs()
        return i, j, torch.tensor(res.offsets())
    if kind == "rs":
        return tj.join(state["R"], state["S"], eps2=state["T"], screen=state["screen"])
    if kind == "table":
        return tj.join_result(state["R"], None, eps2=state["T"], mode="directed",
                              screen=state["screen"]).neighbor_table()
    return tj.self_join(state["R"], eps2=state["T"], mode=kind, screen=state["screen"])


def work(case):
    """Bytes: rows read once, ids written once (two int64 per pair; a neighbour table holds one).
    Operations: two per element of every distance that no bound on groups of rows can rule out --
    pairs of one cluster in a mixture, all pairs of dense rows, the result's own pairs in the plane."""
    kind = case["kind"]
    if kind == "batch":
        lo, hi, nj = case["lo"], case["hi"], case["joins"]
        mean = (hi - lo) / math.log(hi / lo)   # of a log-uniform size
        d = sum(DIMS[case["dims"]]) / len(DIMS[case["dims"]])
        return {"bytes": nj * mean * (8 * d + 16 * case["degree"]), "flops": nj * mean * mean / 8 * 2 * d}
    if kind == "mixture":
        n_r, n_s, d = case["n_r"], case["n_s"], case["d"]
        return {"bytes": 4 * d * (n_r + n_s) + 16 * case["degree"] * n_r,
                "flops": 2 * d * n_r * n_s / case["clusters"]}
    if kind == "planar":
        pairs = case["n"] * case["degree"]
        return {"bytes": 8 * case["n"] + 8 * pairs, "flops": 4 * pairs / 2}
    n, d, deg = case["n"], case["d"], case["degree"]
    if kind == "factor" and case["mode"] == "rs":
        return {"bytes": 8 * d * n + 16 * deg * n, "flops": 2 * d * n * n}
    out = 16 * deg * n if case.get("mode") == "directed" else 8 * deg * n   # i < j: half the pairs
    return {"bytes": (2 if kind == "int14" else 4) * d * n + out, "flops": d * n * n}
