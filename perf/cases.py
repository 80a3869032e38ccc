"""Performance cases of the UMAP fit path: what a program that uses the package calls.

A program has its points' exact kNN lists in hand (the path takes them as input), calls
`Umap.fit` and reads the embedding; or stops at `learn_manifold`; or fits many small datasets
at once; or starts a large fit from the learned warm start; and it gets the kNN lists from
`knn_bruteforce`.  Sizes are those of the benchmark workloads, the tests and the usual calls
around them: 500 to 2,000,000 points in memory-resident fits, a DRAM-bound one above 4,000,000,
5 to 128 neighbours, 2 to 10 embedding dimensions, host (numpy) and device (CUDA) inputs.

Fits start from the data's principal components with a small learning rate, as a program does
that wants a layout which stays near them and hardly changes from run to run: the epochs race
by design (Hogwild), and from a random start at learning rate 1 two runs share nothing but
their statistics.  The rate scales the moves only; an epoch does the same work at every rate.
Their embeddings have no 64-bit value; the graph and the kNN do.  Inputs come from the seed
alone, made on the GPU.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "umap-rs_b200"))
import umap_b200 as ub  # noqa: E402
from umap_b200 import workloads  # noqa: E402

DEFAULTS = {"k": 15, "dim": 32, "clusters": 10, "components": 2, "epochs": 0, "rate": 0.01, "host": False}


def _case(name, kind, **kw):
    c = {**DEFAULTS, "kind": kind, **kw}
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # one small dataset (a batch of documents, a per-user set): latency and launches
        _case("fit_500", "fit", n=500, rate=0.006, host=True),
        # an ordinary notebook dataset, the 10,000-point mixture of the parity tests
        _case("fit_10k", "fit", n=10_000, epochs=200),
        # an image or single-cell dataset of MNIST's size, ragged, arrays on the host
        _case("fit_70k", "fit", n=69_997, host=True),
        # an embedding in 5-D, the usual step before density clustering
        _case("fit_20k_5d", "fit", n=20_000, components=5, rate=0.05),
        # the benchmark's 2,000,000-point fit: the largest L2-resident embedding in use
        _case("fit_2m", "fit", n=2_000_000, dim=64, clusters=50, epochs=500, rate=0.002),
        # a fit whose embedding does not stay in L2: the noisy swiss roll above 4,000,000 points
        _case("fit_roll_5m", "fit_roll", n=5_000_001, dim=3, rate=0.005),
        # the graph alone, wider neighbourhoods, every array of it read back
        _case("manifold_30k_k30", "manifold", n=30_011, k=30),
        # 64 independent sets of 3-D positions, uneven sizes, in one call
        _case("batch_64", "batch", n=64, lo=500, hi=20_000, dim=3, k=10, clusters=5, epochs=200),
        # kNN of a notebook dataset held on the host
        _case("knn_10k", "knn", n=10_000, host=True),
        # kNN of MNIST's shape and value distribution
        _case("knn_70k_784", "knn", n=70_000, dim=784),
        # long lists (n_neighbors = 100) over 50 principal components
        _case("knn_20k_k100", "knn", n=20_003, dim=50, k=100),
        # the learned warm start: subsample fit, network training, prediction, short fit
        _case("warm_1m", "warm", n=1_000_000, dim=64, clusters=50, sub=50_000, epochs=100, rate=0.003),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "fit", "fit_roll", "manifold", "batch", "knn", "knn", "warm"])
    host = rng.random() < 0.4
    if kind == "fit":
        comp = rng.choice([2, 2, 2, 3, 5, 8, 10])
        n = _log_int(rng, 300, 1_000_000 if comp <= 3 else 100_000)
        return _case("", kind, n=n, k=rng.randint(8, 30 if n > 200_000 else 50), dim=rng.choice([16, 32, 50, 64]),
                     clusters=rng.randint(3, 50), components=comp, epochs=rng.choice([0, 100, 200, 300]),
                     rate=0.002 if n > 100_000 else 0.01 if n > 2_000 else 0.006, host=host)
    if kind == "fit_roll":
        return _case("", kind, n=rng.randint(4_000_001, 5_000_001), k=rng.randint(8, 15), dim=3,
                     epochs=rng.choice([50, 100, 200]), rate=0.005)
    if kind == "manifold":
        return _case("", kind, n=_log_int(rng, 300, 100_000), k=rng.randint(5, 60), dim=rng.choice([16, 32, 64]),
                     clusters=rng.randint(3, 50), host=host)
    if kind == "batch":
        return _case("", kind, n=rng.randint(16, 64), lo=500, hi=rng.randint(2_000, 20_000), dim=3,
                     k=rng.randint(5, 10), clusters=5, epochs=rng.choice([100, 200]), host=host)
    if kind == "knn":
        k = rng.choice([rng.randint(5, 32), rng.randint(5, 32), rng.randint(33, 128)])
        n, dim = _log_int(rng, 300, 70_000 if k <= 32 else 20_000), _log_int(rng, 3, 100)
        return _case("", kind, n=n, dim=dim, k=k, host=host)
    n = _log_int(rng, 50_000, 1_000_000)
    return _case("", kind, n=n, dim=rng.choice([32, 64]), clusters=50, sub=max(5_000, n // 20), epochs=100,
                 rate=0.003)


# ------------------------------------------------------------------ inputs
def _points(n, dim, clusters, seed):
    """A Gaussian mixture (centres ~N(0, 5^2 I), std 1), as the benchmark's configurations use."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    centres = torch.randn((clusters, dim), generator=g, device="cuda") * 5.0
    label = torch.randint(0, clusters, (n,), generator=g, device="cuda")
    return torch.randn((n, dim), generator=g, device="cuda") + centres[label]


def _pixels(n, seed):
    """Images of 28 x 28 pixels in [0, 1], mostly zero: ten prototypes of a few Gaussian strokes,
    shifted by up to 2 pixels, scaled, with pixel noise, zeroed below 0.2."""
    g = torch.Generator(device="cuda").manual_seed(seed)

    def u(*size):
        return torch.rand(size, generator=g, device="cuda")

    at = torch.arange(28, device="cuda", dtype=torch.float32)
    cy, cx, sy, sx = 6 + 16 * u(10, 5), 6 + 16 * u(10, 5), 1 + 3 * u(10, 5), 1 + 3 * u(10, 5)
    strokes = torch.exp(-((at[:, None] - cy[..., None, None]) ** 2 / (2 * sy[..., None, None] ** 2)
                          + (at - cx[..., None, None]) ** 2 / (2 * sx[..., None, None] ** 2)))
    proto = strokes.sum(1)
    proto = proto / proto.amax((1, 2), keepdim=True)
    label = torch.randint(0, 10, (n,), generator=g, device="cuda")
    shift = torch.randint(-2, 3, (n, 2), generator=g, device="cuda")
    yy = (torch.arange(28, device="cuda") - shift[:, :1]) % 28
    xx = (torch.arange(28, device="cuda") - shift[:, 1:]) % 28
    img = proto[label[:, None, None], yy[:, :, None], xx[:, None, :]] * (0.6 + 0.4 * u(n, 1, 1))
    img += 0.1 * torch.randn((n, 28, 28), generator=g, device="cuda")
    img.clamp_(0.0, 1.0)
    return torch.where(img < 0.2, torch.zeros_like(img), img).reshape(n, 784).contiguous()


def _init(x, components):
    """The first principal components."""
    xc = x - x.mean(0, keepdim=True)
    v = torch.linalg.eigh(xc.double().T @ xc.double()).eigenvectors
    return (xc @ v[:, -components:].flip(1).float()).contiguous()


def _knn_plain(x, k):
    """Exact kNN, the point itself first: plain torch, distances recomputed in f32."""
    torch.backends.cuda.matmul.allow_tf32 = False
    n = x.shape[0]
    xc = x - x.mean(0, keepdim=True)
    sq = (xc * xc).sum(1)
    idx = torch.empty((n, k), dtype=torch.int32, device=x.device)
    dist = torch.empty((n, k), dtype=torch.float32, device=x.device)
    kc = min(n, k + 8)
    step = max(64, min(4096, (1 << 27) // n))
    for s in range(0, n, step):
        e = min(n, s + step)
        d = sq[s:e, None] + sq[None, :] - 2.0 * (xc[s:e] @ xc.T)
        d[torch.arange(e - s, device=x.device), torch.arange(s, e, device=x.device)] = -1.0
        cand = torch.topk(d, kc, dim=1, largest=False).indices
        ex = torch.sqrt(((x[s:e, None, :] - x[cand]) ** 2).sum(2))
        ex, o = torch.sort(ex, dim=1, stable=True)
        idx[s:e] = torch.gather(cand, 1, o)[:, :k]
        dist[s:e] = ex[:, :k]
    return idx, dist


def _knn(x, k):
    """The program's kNN: self first, then the k - 1 nearest others."""
    n = x.shape[0]
    if n <= 100_000:
        return _knn_plain(x, k)
    i, d = ub.knn_bruteforce(x, k - 1)
    own = torch.arange(n, dtype=torch.int32, device=x.device)[:, None]
    return torch.cat([own, i], 1), torch.cat([torch.zeros_like(own, dtype=torch.float32), d], 1)


def _config(case):
    c = ub.UmapConfig(n_components=case["components"])
    c.graph.n_neighbors = case["k"]
    c.optimization.learning_rate = case["rate"]
    if case["epochs"]:
        c.optimization.n_epochs = case["epochs"]
    return c


def _place(case, *arrays):
    """The arrays as the program holds them: CUDA tensors, or numpy on the host (kNN ids as u32)."""
    if not case["host"]:
        return arrays
    return tuple(a.cpu().numpy().view(np.uint32) if a.dtype == torch.int32 else a.cpu().numpy() for a in arrays)


def _graph_points(case, seed):
    """The points of a graph case: one set of points for the case, whose order and scale the seed
    deals, so that the graph's arrays have the same sizes for every seed."""
    x = _points(case["n"], case["dim"], case["clusters"], 11)
    g = torch.Generator(device="cuda").manual_seed(seed)
    scale = 0.5 + torch.rand((1,), generator=g, device="cuda")
    return x[torch.randperm(case["n"], generator=g, device="cuda")] * scale


def _batch_sizes(case):
    """The sizes are the case's, the points the seed's."""
    g = np.random.Generator(np.random.PCG64(4))
    return np.exp(g.uniform(math.log(case["lo"]), math.log(case["hi"]), size=case["n"])).astype(np.int64)


def prepare(case, seed):
    kind, n, k = case["kind"], case["n"], case["k"]
    s = {"kind": kind, "n": n, "k": k}
    if kind == "knn":
        x = _pixels(n, seed) if case["dim"] == 784 else _points(n, case["dim"], case["clusters"], seed)
        (s["data"],) = _place(case, x)
        return s
    s["umap"] = ub.Umap(_config(case))
    if kind == "manifold":
        s["idx"], s["dist"] = _place(case, *_knn_plain(_graph_points(case, seed), k))
    elif kind == "batch":
        sizes = _batch_sizes(case)
        sets = [_points(int(m), case["dim"], case["clusters"], seed * 1009 + i) for i, m in enumerate(sizes)]
        parts = [_knn_plain(x, k) for x in sets]
        s["offsets"] = np.concatenate([[0], np.cumsum(sizes)]).astype(np.uint64)
        s["idx"], s["dist"], s["init"] = _place(case, torch.cat([p[0] for p in parts]),
                                                torch.cat([p[1] for p in parts]),
                                                torch.cat([_init(x, case["components"]) for x in sets]))
    elif kind == "fit_roll":
        x = workloads.swiss_roll_torch(n, seed=seed)
        s["idx"], s["dist"], _ = workloads.knn_grid_torch(x, k)
        s["init"] = _init(x, case["components"])
    else:
        x = _points(n, case["dim"], case["clusters"], seed)
        s["idx"], s["dist"], s["init"] = _place(case, *_knn(x, k), _init(x, case["components"]))
        if kind == "warm":
            g = torch.Generator(device="cuda").manual_seed(seed + 5)
            rows = torch.randperm(n, generator=g, device="cuda")[:case["sub"]].sort().values
            s["data"], s["rows"] = x, rows.to(torch.int32)
            s["sub_idx"], s["sub_dist"] = _knn(x[rows], k)
            s["sub_init"] = s.pop("init")[rows]
    return s


def run(s):
    kind = s["kind"]
    if kind in ("fit", "fit_roll"):
        return s["umap"].fit(s["n"], s["idx"], s["dist"], s["init"]).embedding()
    if kind == "manifold":
        m = s["umap"].learn_manifold(s["n"], s["idx"], s["dist"])
        g = m.graph()
        return (g.indptr, g.indices, g.data) + tuple(m.sigmas_rhos())
    if kind == "batch":
        return ub.batch_fit(s["umap"].config, s["offsets"], s["idx"], s["dist"], s["init"])
    if kind == "knn":
        return ub.knn_bruteforce(s["data"], s["k"])
    return ub.warm_start_fit(s["umap"].config, s["data"], s["idx"], s["dist"], s["rows"], s["sub_idx"],
                             s["sub_dist"], sub_init=s["sub_init"], epochs=s["umap"].config.optimization.n_epochs
                             ).embedding()


# ------------------------------------------------------------------ work
def _sgd_work(points, k, d, epochs):
    """Edges kept after the union are about 1.45 per directed edge, 0.28 of them fire in an epoch,
    each with 5 negatives (measured on the mixtures; k and the data move them by some percent)."""
    edges = 1.45 * points * (k - 1)
    fired = 0.28 * edges
    return (epochs * (4 * edges + fired * (8 + 16 * d) + 4 * d * 5 * fired),
            epochs * fired * (6 * (6 * d + 10)))


def _fit_work(points, k, d, epochs):
    b, f = _sgd_work(points, k, d, epochs)
    return points * (8 * k + 8 * d) + b, f + points * (k - 1) * 60


def work(case):
    kind, n, k, d = case["kind"], case["n"], case["k"], case["components"]
    if kind == "knn":
        return {"bytes": 4 * n * case["dim"] + 8 * n * k, "flops": 2 * n * n * case["dim"]}
    if kind == "manifold":
        return {"bytes": 8 * n * k + 8 * n + 8 * 1.45 * n * (k - 1) + 8 * n, "flops": n * (k - 1) * 60}
    if kind == "warm":
        b0, f0 = _fit_work(case["sub"], k, d, 500)
        b1, f1 = _fit_work(n, k, d, case["epochs"])
        net = 2 * (case["dim"] * 256 + 256 * 256 + 256 * d)
        steps = 20 * (case["sub"] // 4096)
        return {"bytes": b0 + b1 + 4 * n * case["dim"] + 4 * steps * 4096 * case["dim"],
                "flops": f0 + f1 + net * (n + 3 * steps * 4096)}
    if kind == "batch":  # the mean of log-uniform sizes
        n = int(n * (case["hi"] - case["lo"]) / math.log(case["hi"] / case["lo"]))
    points = n
    epochs = case["epochs"] or (500 if points <= 10_000 else 200)
    b, f = _fit_work(points, k, d, epochs)
    return {"bytes": b, "flops": f}


# ------------------------------------------------------------------ 64-bit values
def _exact_manifold(case, seed):
    n, k = case["n"], case["k"]
    idx, dist = _knn_plain(_graph_points(case, seed), k)
    d = dist.double()
    first = (d > 0).to(torch.int8).argmax(1, keepdim=True)
    rho = torch.gather(d, 1, first)                       # local_connectivity = 1
    t = (d[:, 1:] - rho).clamp(min=0.0)
    target = math.log2(k)
    lo, hi = torch.zeros_like(rho), torch.full_like(rho, float("inf"))
    mid = torch.ones_like(rho)
    for _ in range(100):
        high = torch.exp(-t / mid).sum(1, keepdim=True) > target
        hi = torch.where(high, mid, hi)
        lo = torch.where(high, lo, mid)
        mid = torch.where(torch.isinf(hi), mid * 2.0, (lo + hi) / 2.0)
    sigma = torch.maximum(mid, 1e-3 * d.mean(1, keepdim=True))
    w = torch.exp(-(d - rho).clamp(min=0.0) / sigma)
    row = torch.arange(n, device=d.device)[:, None].expand(n, k)
    col = idx.long()
    keep = (col != row) & (w > 0)
    r, c, w = row[keep], col[keep], w[keep]
    key = torch.cat([r * n + c, c * n + r])
    uniq, inv = torch.unique(key, return_inverse=True)    # row major, columns ascending
    m = r.numel()
    a = torch.zeros(uniq.numel(), dtype=torch.float64, device=d.device).index_add_(0, inv[:m], w)
    b = torch.zeros_like(a).index_add_(0, inv[m:], w)
    return None, None, (a + b - a * b).cpu().numpy(), sigma[:, 0].cpu().numpy(), rho[:, 0].cpu().numpy()


def _exact_knn(case, seed):
    x = prepare(case, seed)["data"]
    x = (x if isinstance(x, torch.Tensor) else torch.from_numpy(x).cuda()).double()
    n, k = x.shape[0], case["k"]
    x = x - x.mean(0, keepdim=True)
    sq = (x * x).sum(1)
    dist = torch.zeros((n, k), dtype=torch.float64, device=x.device)
    kk = min(k, n - 1)
    step = max(64, min(2048, (1 << 27) // n))
    for s in range(0, n, step):
        e = min(n, s + step)
        d = sq[s:e, None] + sq[None, :] - 2.0 * (x[s:e] @ x.T)
        d[torch.arange(e - s, device=x.device), torch.arange(s, e, device=x.device)] = float("inf")
        cand = torch.topk(d, kk, dim=1, largest=False).indices
        for q in range(s, e, 256):
            near = x[cand[q - s:q - s + 256]]
            dq = torch.sqrt(((x[q:min(q + 256, e), None, :] - near) ** 2).sum(2))
            dist[q:min(q + 256, e), :kk] = torch.sort(dq, dim=1).values
    return None, (dist.cpu().numpy() if case["host"] else dist)


def exact(case, seed):
    if case["kind"] == "manifold":
        return _exact_manifold(case, seed)
    if case["kind"] == "knn":
        return _exact_knn(case, seed)
    return None
