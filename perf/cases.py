"""The work that users of pacmap_b200 have it do, as cases that can be timed and compared.

Eight kinds of call, each through a public entry point (the Python package or the C ABI of
include/pacmap.h), over the sizes of this repository's configurations and of the reference's own use:

``fit``        fit_transform from host arrays, the plain schedule: the interactive call on a few thousand rows
               (the reference's usual input) up to the 60,000 x 784 image-like configuration.
``learned``    fit_transform_learned_device: a large fresh draw started from a trained network, the benchmark's
               headline (1,000,000 x 128 -> 2-D, schedule (0, 50, 150)).
``knn``        knn.find_k_nearest_neighbors from host arrays: exact kNN alone, as `pacmap::knn` offers it.
``knn_device`` pacmap_knn_exact_shard_device: the same on device buffers, one shard (the multi-GPU path's
               per-rank call, here with one rank).
``pairs``      stages.generate_pairs: the three pair lists for a caller with an optimiser of its own.
``steps``      stages.optimize_steps: gradient + Adam iterations from an explicit state and pair lists.
``train``      learned.train: epochs of the initialiser's AdamW training.
``transform``  LearnedModel.transform: new points into a fitted embedding, from one batch to a million rows.

Inputs are drawn on the GPU from the seed alone; host entry points get numpy arrays, as a user holds them.
"""
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "pacmap-rs_b200"))
import pacmap_b200 as pm  # noqa: E402
from pacmap_b200 import _abi, learned, stages  # noqa: E402

DEV = "cuda"


def listed():
    return [
        # The default configuration (PCA start, 450 iterations) on the CPU-runnable configuration's 2,000 x 100:
        # a notebook user's call, where launches and host latency count.
        {"name": "fit_2k", "kind": "fit", "data": "iso", "n": 2000, "d": 100, "dim": 2, "init": "pca", "snapshots": False},
        # An ordinary embedding with a seeded Random start, odd row count, three snapshots kept.
        {"name": "fit_9k", "kind": "fit", "data": "iso", "n": 9001, "d": 50, "dim": 3, "init": "random", "snapshots": True},
        # The 60,000 x 784 image-like configuration with the defaults: PCA to 100 columns first.
        {"name": "fit_image", "kind": "fit", "data": "image", "n": 60000, "d": 784, "dim": 2, "init": "pca", "snapshots": False},
        # The benchmark's headline: a fresh 1M x 128 draw from the network's prediction, shortened schedule.
        {"name": "learned_1m", "kind": "learned", "data": "aniso", "n": 1000000, "d": 128, "dim": 2},
        # The kNN alone on a small table and on an ordinary one (a ragged row count below the larger sizes).
        {"name": "knn_3k", "kind": "knn", "data": "iso", "n": 3000, "d": 100, "k": 15, "mode": 0},
        {"name": "knn_15k", "kind": "knn", "data": "aniso", "n": 15001, "d": 64, "k": 60, "mode": 0},
        # Raw image-like rows, whose distances are small against their norms (all-black images among them).
        {"name": "knn_image", "kind": "knn", "data": "image", "n": 60000, "d": 784, "k": 72, "mode": 0},
        # A 256-column slice of the 4M x 256 configuration's subspace mixture, on the device.
        {"name": "knn_dev_400k", "kind": "knn_device", "data": "subspace", "n": 400000, "d": 256, "k": 84, "mode": 0},
        # Pair lists of a mid-sized data set with a ragged row count, Euclidean as in the reference.
        {"name": "pairs_90k", "kind": "pairs", "data": "aniso", "n": 90001, "d": 96, "angular": False},
        # A caller's own loop resumes a running optimisation for twenty iterations across the last change of phase:
        # 200,000 points in 3-D, lists and state in host arrays.
        {"name": "steps_200k", "kind": "steps", "n": 200000, "dim": 3, "begin": 190, "iters": 20},
        # One epoch of the initialiser's training at the benchmark's batch and row count.
        {"name": "train_200k", "kind": "train", "n": 200000, "d": 128, "dim": 2, "epochs": 1, "batch": 4096},
        # A service's batch of new points.
        {"name": "transform_5k", "kind": "transform", "n": 5000, "d": 128, "dim": 2},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["fit", "fit", "learned", "knn", "knn", "knn_device", "pairs", "steps", "train", "transform"])
    if kind == "fit":
        if rng.random() < 0.2:
            return {"kind": kind, "data": "image", "n": _log(rng, 3000, 50000), "d": rng.choice([256, 400, 784]), "dim": 2,
                    "init": rng.choice(["pca", "random"]), "snapshots": False}
        return {"kind": kind, "data": rng.choice(["iso", "aniso"]), "n": _log(rng, 400, 30000), "d": _log(rng, 8, 100),
                "dim": rng.choice([2, 2, 3]), "init": rng.choice(["pca", "random"]), "snapshots": rng.random() < 0.3}
    if kind == "learned":
        return {"kind": kind, "data": rng.choice(["aniso", "subspace"]), "n": _log(rng, 100000, 900000),
                "d": _log(rng, 48, 160), "dim": rng.choice([2, 2, 3])}
    if kind == "knn":
        data = rng.choice(["iso", "aniso", "aniso", "image"])
        return {"kind": kind, "data": data, "n": _log(rng, 1000, 50000), "d": 784 if data == "image" else _log(rng, 8, 256),
                "k": rng.choice([10, 15, 30, 60, 75]), "mode": 0}
    if kind == "knn_device":
        return {"kind": kind, "data": rng.choice(["aniso", "subspace"]), "n": _log(rng, 30000, 400000), "d": _log(rng, 32, 256),
                "k": rng.choice([15, 60, 80, 90]), "mode": rng.choice([0, 0, 2])}
    if kind == "pairs":
        return {"kind": kind, "data": rng.choice(["iso", "aniso"]), "n": _log(rng, 2000, 200000), "d": _log(rng, 16, 128),
                "angular": rng.random() < 0.3}
    if kind == "steps":
        return {"kind": kind, "n": _log(rng, 5000, 500000), "dim": rng.choice([2, 2, 3]), "begin": rng.choice([20, 90, 190]),
                "iters": rng.choice([10, 20])}
    if kind == "train":
        return {"kind": kind, "n": _log(rng, 5000, 200000), "d": _log(rng, 16, 256), "dim": rng.choice([2, 3]), "epochs": rng.choice([1, 2]),
                "batch": rng.choice([1024, 4096])}
    return {"kind": kind, "n": _log(rng, 200, 1000000), "d": _log(rng, 16, 256), "dim": rng.choice([2, 3])}


# ---------------------------------------------------------------------------------------------
# Inputs
# ---------------------------------------------------------------------------------------------
class _Rng:
    def __init__(self, seed):
        self.g = torch.Generator(device=DEV)
        self.g.manual_seed(int(seed) * 1000003 + 17)

    def normal(self, *s):
        return torch.randn(*s, generator=self.g, device=DEV)

    def uniform(self, *s):
        return torch.rand(*s, generator=self.g, device=DEV)

    def integers(self, hi, *s):
        return torch.randint(0, hi, s, generator=self.g, device=DEV)


def _rotations(r, k, d):
    q, u = torch.linalg.qr(r.normal(k, d, d))
    return q * torch.sign(torch.diagonal(u, dim1=-2, dim2=-1))[:, None, :]


def _data(kind, n, d, r):
    """n x d rows of one of the benchmark's generators (pacmap_b200.datasets, drawn on the GPU), and their labels."""
    if kind == "iso":  # 10 isotropic Gaussians
        lab = r.integers(10, n)
        return 5.0 * r.normal(10, d)[lab] + r.normal(n, d), lab
    if kind == "aniso":  # 50 Gaussians, each with its own rotation and axis scales in [0.3, 3]
        c, rot = 4.0 * r.normal(50, d), _rotations(r, 50, d)
        s = torch.exp(r.uniform(50, d) * math.log(10.0) + math.log(0.3))
        w = torch.rand(50, generator=r.g, device=DEV) + 0.05
        lab = torch.multinomial(w, n, replacement=True, generator=r.g)
        x = r.normal(n, d)
        for q in range(50):
            at = (lab == q).nonzero().squeeze(1)
            x[at] = c[q] + (x[at] * s[q]) @ rot[q].T
        return x, lab
    if kind == "subspace":  # 200 Gaussians on a min(32, d / 2)-dimensional subspace, noise 0.05 elsewhere
        sub = max(2, min(32, d // 2))
        basis = _rotations(r, 1, d)[0]
        c = 4.0 * r.normal(200, sub)
        lab = r.integers(200, n)
        z = torch.cat([c[lab] + r.normal(n, sub), 0.05 * r.normal(n, d - sub)], 1)
        return z @ basis.T, lab
    # image-like: 10 classes of clipped rank-20 images, multiples of 1 / 255
    lab = r.integers(10, n)
    w, mu = 0.15 * r.uniform(10, d, 20), r.normal(10, 20)
    x = torch.empty(n, d, device=DEV)
    for q in range(10):
        at = (lab == q).nonzero().squeeze(1)
        z = mu[q] + r.normal(at.numel(), 20)
        x[at] = torch.round((z @ w[q].T + 0.1 * r.normal(at.numel(), d)).clamp(0, 1) * 255) / 255
    return x, lab


def _host(t):
    return np.ascontiguousarray(t.cpu().numpy())


def _constants(x):
    """preprocess_x's constants of the rows x: min, max of the shifted data, column means."""
    mn = x.min()
    y = x - mn
    mx = y.max()
    return float(mn), float(mx), (y / mx).mean(0)


def _layout(x, lab, dim, r):
    """An embedding-like target: class centres spread over the plane, each class a blob turned by its data."""
    spots = 10.0 * r.normal(int(lab.max()) + 1, dim)
    local = x @ r.normal(x.shape[1], dim)
    return spots[lab] + 1.5 * (local - local.mean(0)) / local.std(0)


def _network(x, lab, dim, r):
    """Weights that map preprocessed rows to a standardised layout: random hidden layers, output layer by ridge
    regression on a sample. Stands for a network trained on an earlier draw. -> (params, constants, mean, std)"""
    d, h = x.shape[1], learned.HIDDEN
    mn, mx, mean = _constants(x)
    m = min(x.shape[0], 20000)
    xs = ((x[:m] - mn) / mx - mean).double()
    t = _layout(x[:m], lab[:m], dim, r).double()
    mu, sd = t.mean(0), t.std(0)
    uni = lambda rows, cols, scale: (2 * r.uniform(rows, cols) - 1) * scale  # noqa: E731
    gain = float(1.0 / xs.std())
    w1, b1 = uni(h, d, gain * 3.0 / math.sqrt(d)), uni(1, h, 0.5)[0]
    w2, b2 = uni(h, h, 3.0 / math.sqrt(h)), uni(1, h, 0.5)[0]
    f = torch.relu(torch.relu(xs @ w1.double().T + b1.double()) @ w2.double().T + b2.double())
    f = torch.cat([f, torch.ones(m, 1, device=DEV, dtype=torch.float64)], 1)
    reg = f.T @ f + 1e-2 * m * torch.eye(h + 1, device=DEV, dtype=torch.float64)
    w3 = torch.linalg.solve(reg, f.T @ ((t - mu) / sd))
    flat = torch.cat([w1.reshape(-1), b1, w2.reshape(-1), b2, w3[:h].T.reshape(-1).float(), w3[h].float()])
    return _host(flat.float()), (mn, mx, _host(mean)), _host(mu.float()), _host(sd.float())


def _counts(n):
    k = 10 if n <= 10000 else int(round(10 + 15 * (math.log10(n) - 4)))
    return k, int(round(0.5 * k)), 2 * k


def _pair_lists(n, r):
    """Pair lists like generated ones: k near neighbours along a hidden order, uniform mid-near and far partners."""
    k, n_mn, n_fp = _counts(n)
    order = torch.randperm(n, generator=r.g, device=DEV)
    place = torch.empty_like(order)
    place[order] = torch.arange(n, device=DEV)
    own = torch.arange(n, device=DEV)[:, None]
    near = order[(place[:, None] + 1 + r.integers(4 * k, n, k)) % n]
    lists = [near] + [(own + 1 + r.integers(n - 1, n, q)) % n for q in (n_mn, n_fp)]
    return [_host(torch.stack([own.expand_as(p).reshape(-1), p.reshape(-1)], 1).int()).view(np.uint32) for p in lists]


def prepare(case, seed):
    c, r = case, _Rng(seed)
    kind, n = c["kind"], c["n"]
    if kind == "steps":
        dim = c["dim"]
        y, m, v = 4.0 * r.normal(n, dim), 0.3 * r.normal(n, dim), 0.5 + r.normal(n, dim).square()
        return {"case": c, "pairs": _pair_lists(n, r), "y": _host(y), "m": _host(m), "v": _host(v)}
    if kind == "train":
        x, lab = _data("aniso", n, c["d"], r)
        mn, mx, mean = _constants(x)
        h, d, dim = learned.HIDDEN, c["d"], c["dim"]
        parts = [(h, d), (1, h), (h, h), (1, h), (dim, h), (1, dim)]
        fan = [d, d, h, h, h, h]
        params = torch.cat([((2 * r.uniform(*s) - 1) / math.sqrt(f)).reshape(-1) for s, f in zip(parts, fan)])
        return {"case": c, "xp": _host((x - mn) / mx - mean), "y": _host(_layout(x, lab, dim, r)), "params": _host(params)}
    if kind == "transform":
        x, lab = _data("aniso", max(n, 20000), c["d"], r)
        params, (mn, mx, mean), mu, sd = _network(x, lab, c["dim"], r)
        return {"case": c, "x": _host(x[:n]), "model": learned.LearnedModel(params, c["d"], c["dim"], mn, mx, mean, mu, sd)}
    x, lab = _data(c["data"], n, c["d"], r)
    if kind == "learned":
        params, _, mu, sd = _network(x, lab, c["dim"], r)
        cfg = pm.Configuration(embedding_dimensions=c["dim"], seed=7, num_iters=learned.SHORT_SCHEDULE)
        return {"case": c, "x": x.contiguous(), "out": torch.empty(n, c["dim"], device=DEV), "params": params, "stats": (mu, sd),
                "cfg": cfg}
    if kind == "knn_device":
        kp = min(c["k"], n - 1)
        return {"case": c, "x": x.contiguous(), "idx": torch.empty(n, kp, dtype=torch.int32, device=DEV),
                "dist": torch.empty(n, kp, device=DEV), "owned": torch.empty(n, dtype=torch.uint8, device=DEV)}
    if kind == "knn":
        return {"case": c, "x": _host(x)}
    if kind == "pairs":
        metric = pm.Metric.ANGULAR if c["angular"] else pm.Metric.EUCLIDEAN
        cfg = pm.Configuration(seed=7, initialization=pm.Initialization.Random(7), metric=metric)
        return {"case": c, "x": _host(x), "cfg": cfg}
    init = pm.Initialization.Pca() if c["init"] == "pca" else pm.Initialization.Random(7)
    cfg = pm.Configuration(embedding_dimensions=c["dim"], initialization=init, seed=7,
                           snapshots=[0, 100, 200] if c["snapshots"] else None)
    return {"case": c, "x": _host(x), "cfg": cfg}


# ---------------------------------------------------------------------------------------------
# One pass
# ---------------------------------------------------------------------------------------------
def run(state):
    s = state
    c = s["case"]
    kind = c["kind"]
    if kind == "fit":
        return pm.fit_transform(s["x"], s["cfg"])
    if kind == "learned":
        learned.fit_transform_learned_device(s["x"].data_ptr(), c["n"], c["d"], s["out"].data_ptr(), s["params"], s["cfg"],
                                             target_stats=s["stats"])
        return s["out"]
    if kind == "knn":
        idx, dist = pm.knn.find_k_nearest_neighbors(s["x"], c["k"], knn_mode=c["mode"])
        return idx.view(np.int32), dist
    if kind == "knn_device":
        pm._check(_abi.lib().pacmap_knn_exact_shard_device(s["x"].data_ptr(), c["n"], c["d"], c["k"], c["mode"], 0, 1, 0,
                                                           s["idx"].data_ptr(), s["dist"].data_ptr(), s["owned"].data_ptr()))
        return s["idx"], s["dist"]
    if kind == "pairs":
        return [p.view(np.int32) for p in stages.generate_pairs(s["x"], s["cfg"])]
    if kind == "steps":
        y, m, v = s["y"].copy(), s["m"].copy(), s["v"].copy()
        g = stages.optimize_steps(y, m, v, *s["pairs"], 1.0, 100, 100, c["begin"], c["begin"] + c["iters"])
        return {"y": y, "m": m, "v": v, "grad": g[:-1], "loss": float(g[-1, 0])}
    if kind == "train":
        params, losses = learned.train(s["params"], s["xp"], s["y"], epochs=c["epochs"], batch=c["batch"], seed=3)
        return params, losses
    return s["model"].transform(s["x"])


# ---------------------------------------------------------------------------------------------
# What a pass cannot do without: its inputs read once, its outputs written once, and the arithmetic that the
# outputs are made of. An exact kNN has no fixed number of distances (a search may skip rows that cannot be
# neighbours): only the reported ones are counted.
# ---------------------------------------------------------------------------------------------
def _pairs_work(n, d):
    k, n_mn, n_fp = _counts(n)
    return {"bytes": 4.0 * n * d + 8.0 * n * (k + n_mn + n_fp), "flops": 3.0 * n * d * (k + 50 + 6 * n_mn)}


def _optimise_work(n, dim, phases):
    """Each active pair read once and the state read and written once an iteration; mid-near pairs in two phases."""
    k, n_mn, n_fp = _counts(n)
    early, late = phases
    pairs = n * (early * (k + n_mn + n_fp) + late * (k + n_fp))
    return {"bytes": 8.0 * pairs + 28.0 * n * dim * (early + late), "flops": pairs * (7.0 * dim + 8)}


def work(case):
    c = case
    n, kind = c["n"], c["kind"]
    if kind in ("knn", "knn_device"):
        return {"bytes": 4.0 * n * c["d"] + 8.0 * n * c["k"], "flops": 3.0 * n * c["k"] * c["d"]}
    if kind == "pairs":
        return _pairs_work(n, c["d"])
    if kind == "steps":
        early = min(c["iters"], max(0, 200 - c["begin"]))
        w, k = _optimise_work(n, c["dim"], (early, c["iters"] - early)), _counts(n)
        return {"bytes": w["bytes"] + 8.0 * n * sum(k) + 28.0 * n * c["dim"], "flops": w["flops"]}
    mlp = 2.0 * n * (c["d"] * 512 + 512 * 512 + 512 * c["dim"])
    if kind == "transform":
        return {"bytes": 4.0 * n * (c["d"] + c["dim"]), "flops": mlp}
    if kind == "train":
        return {"bytes": 4.0 * c["epochs"] * n * (c["d"] + c["dim"]), "flops": 3.0 * c["epochs"] * mlp}
    p, o = _pairs_work(n, c["d"]), _optimise_work(n, c["dim"], (50, 150) if kind == "learned" else (200, 250))
    return {"bytes": p["bytes"] + o["bytes"] + 4.0 * n * c["dim"],
            "flops": p["flops"] + o["flops"] + (mlp if kind == "learned" else 0.0)}


# ---------------------------------------------------------------------------------------------
# The same outputs in 64 bits, where they are numbers with one
# ---------------------------------------------------------------------------------------------
def _exact_knn(x, k):
    """Distances to the k nearest other rows, ascending."""
    x = x.double()
    n = x.shape[0]
    sq = (x * x).sum(1)
    out = torch.empty(n, k, dtype=torch.float64, device=DEV)
    step = max(1, min(n, 400_000_000 // n))
    for a in range(0, n, step):
        q = x[a:a + step]
        d2 = sq[a:a + step, None] + sq[None] - 2 * (q @ x.T)
        d2[torch.arange(q.shape[0], device=DEV), torch.arange(a, a + q.shape[0], device=DEV)] = math.inf
        near = torch.topk(d2, min(k + 8, n - 1), dim=1, largest=False).indices
        part = max(1, 30_000_000 // (near.shape[1] * x.shape[1]))
        for b in range(0, q.shape[0], part):
            e = (x[near[b:b + part]] - q[b:b + part, None]).square().sum(2).sqrt()
            out[a + b:a + b + e.shape[0]] = e.sort(1).values[:, :k]
    return out


def _exact_steps(s):
    c = s["case"]
    y, m, v = (torch.from_numpy(s[q]).to(DEV).double() for q in ("y", "m", "v"))
    lists = [torch.from_numpy(p.view(np.int32)).to(DEV).long() for p in s["pairs"]]
    for t in range(c["begin"], c["begin"] + c["iters"]):
        weights = (2.0, (1 - t / 100) * 1000 + t / 100 * 3, 1.0) if t < 100 else (3.0, 3.0, 1.0) if t < 200 else (1.0, 0.0, 1.0)
        g, loss = torch.zeros_like(y), 0.0
        for p, w, (a, b, sign) in zip(lists, weights, ((10, 20, 1), (10000, 20000, 1), (1, 2, -1))):
            i, j = p[:, 0], p[:, 1]
            diff = y[i] - y[j]
            q = 1 + diff.square().sum(1)
            f = sign * (w * b / (a + q).square())[:, None] * diff
            g.index_add_(0, i, f)
            g.index_add_(0, j, f, alpha=-1)
            loss = loss + float((w * (1 / (1 + q) if sign < 0 else q / (a + q))).sum())
        m = m + 0.1 * (g - m)
        v = v + 0.001 * (g * g - v)
        lr = math.sqrt(1 - 0.999 ** (t + 1)) / (1 - 0.9 ** (t + 1))
        y = y - lr * m / (v.sqrt() + 1e-7)
    return {"y": y, "m": m, "v": v, "grad": g, "loss": loss}


def exact(case, seed):
    c = case
    kind, n = c["kind"], c["n"]
    if kind in ("knn", "knn_device") and 2.0 * n * n * c["d"] < 6e12:
        s = prepare(c, seed)
        x = s["x"] if kind == "knn_device" else torch.from_numpy(s["x"]).to(DEV)
        return None, _exact_knn(x, min(c["k"], n - 1))
    if kind == "steps":
        return _exact_steps(prepare(c, seed))
    if kind == "transform":
        s = prepare(c, seed)
        m, h, d = s["model"], learned.HIDDEN, c["d"]
        p = torch.from_numpy(m.params).to(DEV).double()
        w1, b1, w2, b2, w3, b3 = torch.split(p, [h * d, h, h * h, h, c["dim"] * h, c["dim"]])
        out = []
        for a in range(0, n, 1 << 17):
            x = (torch.from_numpy(s["x"][a:a + (1 << 17)]).to(DEV).double() - m.pre_min) / m.pre_max
            x = x - torch.from_numpy(m.pre_mean).to(DEV).double()
            f = torch.relu(torch.relu(x @ w1.view(h, d).T + b1) @ w2.view(h, h).T + b2) @ w3.view(-1, h).T + b3
            out.append(f * torch.from_numpy(m.target_std).to(DEV).double() + torch.from_numpy(m.target_mean).to(DEV).double())
        return torch.cat(out)
    return None
