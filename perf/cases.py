"""The sampler's work as a user's program has it done, case by case.

Each case is a dict of plain values.  `listed` names twelve of them, `draw`
makes more from the same ranges, `prepare` builds what a program holds before
the call, `run` is one pass through the package's public entry points, `work`
is what the pass cannot do without, and `exact` gives the results in 64 bits
where the path has such a value.

Sizes are those of the package's own workloads: the unit cube of d = 50, the
genome-shaped polytope (n = 2600 reactions, d = 700, 16 chains, thinning 116,
pair probability 0.3, slack recompute every 2048 steps), its conditioned
variants (m = 5200..5400 rows, 8 chains each), the larger polytope of
n = 7000 and d = 1500, and the rounding network of its learned rounding.
Sample counts are cut so that a pass takes milliseconds; everything a step or
a row costs is as in a full run.
"""
import math

import numpy as np
import torch

from naja_b200 import Polytope, backmap
from naja_b200.batch import Batch, Shape
from naja_b200.learned import RoundingNet
from naja_b200.pipeline import sample_backmapped
from naja_b200.validate import ess_rhat

DEV = "cuda"


def _chains(**kw):
    c = dict(kind="chains", n=2600, d=700, rounded=False, precision="fp32", chains=16, samples=200, thinning=116,
             pair=0.3, resync=2048)
    c.update(kw)
    return c


def listed():
    return [
        # the smallest call: four short chains in the unit cube, where the
        # launch and the step's fixed latency are all there is
        dict(name="cube", kind="cube", d=50, chains=4, samples=100, thinning=8),
        # a genome-scale model as it comes (8 % of A nonzero), few chains
        _chains(name="genome"),
        # the same model rounded: every entry of A nonzero, the headline workload
        _chains(name="genome-rounded", rounded=True),
        # the rounded model in the reference's own arithmetic
        _chains(name="genome-rounded-fp64", rounded=True, precision="fp64", samples=80, resync=0),
        # a bulk of conditioned variants in one launch, as they come
        dict(name="variants", kind="variants", models=64, n=2600, d=700, rounded=False, chains=8, samples=40,
             thinning=116, pair=0.3, resync=2048),
        # rounded variants in one launch (the learned rounding's training samples)
        dict(name="variants-rounded", kind="variants", models=40, n=2600, d=700, rounded=True, chains=8, samples=20,
             thinning=116, pair=0.3, resync=2048),
        # samples to reaction space, the default mode, an odd number of rows
        dict(name="backmap", kind="backmap", n=2600, d=700, rows=50001, mode="tf32x3"),
        # the larger model, the fastest mode, ragged in every dimension
        dict(name="backmap-large", kind="backmap", n=6999, d=1501, rows=30011, mode="bf16x3"),
        # the exact map of rounded samples back to the model's own coordinates
        dict(name="backmap-fp64", kind="backmap", n=700, d=700, rows=40000, mode="fp64"),
        # the convergence check of a finished run: ESS and split-R-hat of every coordinate
        dict(name="validate", kind="validate", dim=700, chains=16, samples=2500, layout=1),
        # one training step of the rounding network at its own sizes
        dict(name="network", kind="network", n_in=2600, hidden=512, n_out=23100, batch=64, train=True),
        # a whole job: rounded chains, backmap and delivery to host memory, overlapped
        dict(name="job", kind="job", n=2600, d=700, chains=16, samples=1024, thinning=116, pair=0.3, resync=2048,
             mode="tf32x3"),
    ]


def _between(rng, lo, hi):
    """A whole number of [lo, hi], spread over its logarithm."""
    return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))))


def draw(rng):
    kind = rng.choice(["cube", "chains", "chains", "chains", "variants", "variants", "backmap", "backmap", "validate",
                       "network", "job"])
    if kind == "cube":
        return dict(kind=kind, d=_between(rng, 4, 120), chains=_between(rng, 1, 64), samples=_between(rng, 20, 400),
                    thinning=rng.randint(1, 12))
    if kind == "chains":
        precision = rng.choice(["fp32", "fp32", "fp64"])
        d = _between(rng, 40, 900)
        return _chains(n=rng.randint(2 * d, 4 * d), d=d, rounded=rng.random() < 0.6, precision=precision,
                       chains=_between(rng, 1, 64), samples=_between(rng, 10, 80), thinning=rng.randint(40, 150),
                       pair=rng.choice([0.0, 0.3, 0.5]), resync=rng.choice([0, 512, 2048]))
    if kind == "variants":
        rounded = rng.random() < 0.4
        d = rng.randint(300, 720)
        return dict(kind=kind, models=_between(rng, 8, 40 if rounded else 64), n=rng.randint(3 * d, int(3.7 * d)), d=d,
                    rounded=rounded, chains=rng.randint(2, 8), samples=rng.randint(8, 20), thinning=rng.randint(40, 116),
                    pair=0.3, resync=rng.choice([0, 2048]))
    if kind == "backmap":
        mode = rng.choice(["tf32x3", "bf16x3", "fp64"])
        d = rng.randint(64, 800)
        n = d if mode == "fp64" and rng.random() < 0.5 else rng.randint(d, 3200)
        return dict(kind=kind, n=n, d=d, rows=_between(rng, 500, 8000 if mode == "fp64" else 50000), mode=mode)
    if kind == "validate":
        return dict(kind=kind, dim=_between(rng, 50, 700), chains=rng.randint(2, 16), samples=_between(rng, 1000, 2500),
                    layout=rng.choice([0, 1, 1]))
    if kind == "network":
        d = rng.randint(40, 700)
        return dict(kind=kind, n_in=rng.randint(2 * d, 4 * d) if d < 650 else 2600, hidden=rng.choice([256, 384, 512]),
                    n_out=33 * d, batch=rng.randint(16, 64), train=rng.random() < 0.7)
    d = rng.randint(100, 700)
    return dict(kind=kind, n=rng.randint(3 * d, int(3.7 * d)), d=d, chains=rng.randint(4, 16), samples=600 + rng.randint(0, 300),
                thinning=rng.randint(16, 90), pair=0.3, resync=rng.choice([512, 2048]),
                mode=rng.choice(["tf32x3", "bf16x3"]))


# ------------------------------------------------------------------ inputs
def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(int(seed))
    return g


def _rand(g, *shape):
    return torch.rand(shape, generator=g, device=DEV, dtype=torch.float64)


def _randn(g, *shape):
    return torch.randn(shape, generator=g, device=DEV, dtype=torch.float64)


def _model(g, n, d, rounded):
    """(T, u) of {-u <= T y <= u}: bounds log-uniform on [1, 1000]; T 8 %
    nonzero as in a genome-scale model, or dense as after a rounding."""
    T = _randn(g, n, d)
    if not rounded:
        mask = _rand(g, n, d) < 0.08
        mask[torch.arange(d, device=DEV) % n, torch.arange(d, device=DEV)] = True  # no empty column
        T = torch.where(mask, T, torch.zeros_like(T))
    return T, 10.0 ** (3.0 * _rand(g, n))


def _variant(g, T, u):
    """The polytope with up to 100 reactions' bounds tightened: two more rows for each."""
    n = T.shape[0]
    r = int(torch.randint(0, min(100, n) + 1, (1,), generator=g, device=DEV))
    idx = torch.randperm(n, generator=g, device=DEV)[:r]
    f = 0.05 + 0.45 * _rand(g, r)
    E = torch.stack([T[idx], -T[idx]], dim=1).reshape(2 * r, T.shape[1])
    return torch.cat([T, -T, E]), torch.cat([u, u, (u[idx] * f).repeat_interleave(2)])


class _Chains:
    def __init__(self, A, b, c, seed):
        self.P = Polytope(A, b)
        self.X0 = torch.zeros((c["chains"], A.shape[1]), dtype=torch.float64, device=DEV)
        self.out = torch.empty((c["samples"] * c["chains"], A.shape[1]), dtype=torch.float32, device=DEV)
        self.last = torch.empty_like(self.X0)
        self.shape = (c["samples"], c["thinning"], c["chains"])
        self.kw = dict(seed=seed)

    def run(self):
        self.P.run(self.X0, *self.shape, out=self.out, X_final=self.last, **self.kw)
        return {"samples": self.out, "last": self.last}


def _prepare_cube(c, seed):
    d = c["d"]
    eye = torch.eye(d, dtype=torch.float64, device=DEV)
    one = torch.ones(d, dtype=torch.float64, device=DEV)
    s = _Chains(torch.cat([eye, -eye]), torch.cat([one, 0 * one]), c, seed)
    s.X0.fill_(0.5)
    return s


def _prepare_chains(c, seed):
    T, u = _model(_gen(seed), c["n"], c["d"], c["rounded"])
    s = _Chains(torch.cat([T, -T]), torch.cat([u, u]), c, seed)
    s.kw.update(pair_prob=c["pair"], resync_interval=c["resync"], precision=c["precision"])
    return s


class _Variants:
    def __init__(self, c, seed):
        g = _gen(seed)
        T, u = _model(g, c["n"], c["d"], c["rounded"])
        self.batch = Batch([Polytope(*_variant(g, T, u)) for _ in range(c["models"])])
        self.X0 = [torch.zeros((c["chains"], c["d"]), dtype=torch.float64, device=DEV) for _ in range(c["models"])]
        self.last = [torch.empty_like(x) for x in self.X0]
        all_out = torch.empty((c["models"], c["samples"] * c["chains"], c["d"]), dtype=torch.float32, device=DEV)
        self.all_out, self.out = all_out, list(all_out.unbind(0))
        # the shapes the package's autotuner settles on for many chains (compressed
        # columns) and its learned rounding uses (dense)
        self.launch = Shape(256, 3, 1, 0, 0) if c["rounded"] else Shape(128, 4, 1, 0, 1)
        self.shape = (c["samples"], c["thinning"], c["chains"])
        self.kw = dict(seed=seed, pair_prob=c["pair"], resync_interval=c["resync"])

    def run(self):
        self.batch.run(self.X0, self.out, *self.shape, shape=self.launch, X_finals=self.last, **self.kw)
        return {"samples": self.all_out, "last": self.last[0]}


class _Backmap:
    def __init__(self, c, seed):
        g = _gen(seed)
        dense = c["mode"] == "fp64"
        self.T, _ = _model(g, c["n"], c["d"], dense)
        self.shift = _randn(g, c["n"])
        scale = 10.0 ** (2.0 * _rand(g, 1, c["d"]) - 1.0)
        self.Y = (_randn(g, c["rows"], c["d"]) * scale).to(torch.float32)
        self.V = torch.empty((c["rows"], c["n"]), dtype=torch.float32, device=DEV)
        self.mode = c["mode"]

    def run(self):
        return backmap(self.T, self.shift, self.Y, mode=self.mode, out=self.V)


def _series(c, seed):
    """Samples of chains that mix at different speeds per coordinate: AR(1)
    series, correlation 0.3 to 0.99, in the sampler's row order."""
    g = _gen(seed)
    dim, k, n = c["dim"], c["chains"], c["samples"]
    rho = 1.0 - 10.0 ** (-0.15 - 1.85 * _rand(g, dim))
    x = _randn(g, n, k, dim)
    x[1:] *= torch.sqrt(1.0 - rho * rho)
    # x[t] = rho x[t-1] + e[t] by doubling: after step s each value sums 2 s terms
    s, w = 1, rho.clone()
    while s < n:
        x[s:] = x[s:] + w * x[:-s]
        w, s = w * w, 2 * s
    return (x.reshape(n * k, dim) * 10.0 ** (2.0 * _rand(g, dim) - 1.0) + _randn(g, dim)).to(torch.float32)


class _Validate:
    def __init__(self, c, seed):
        self.S = _series(c, seed)
        self.args = (c["chains"], c["layout"])

    def run(self):
        ess, rhat = ess_rhat(self.S, *self.args)
        return {"ess": ess, "rhat": rhat}


def _network_inputs(c, seed):
    """Bound ratios (most of them 0) and standardised targets, on the host as the training loop has them."""
    r = np.random.default_rng(seed)
    X = np.zeros((c["batch"], c["n_in"]), np.float32)
    for row in X:
        k = r.integers(1, 101)
        row[r.choice(c["n_in"], min(k, c["n_in"]), replace=False)] = np.log(r.uniform(0.05, 0.5, min(k, c["n_in"]))) / 3.0
    return X, r.standard_normal((c["batch"], c["n_out"]), dtype=np.float32)


class _Network:
    def __init__(self, c, seed):
        self.net = RoundingNet((c["n_in"], c["hidden"], c["hidden"], c["n_out"]), seed=seed)
        self.X, self.T = _network_inputs(c, seed)
        self.train = c["train"]

    def run(self):
        if not self.train:
            return {"out": self.net.predict(self.X)}
        loss = self.net.train_step(self.X, self.T)
        return {"loss": loss, "W": [L.W[:, : L.n_in] for L in self.net.layers], "b": [L.b for L in self.net.layers],
                "gW": [L.gW[:, : L.n_in] for L in self.net.layers], "gb": [L.gb for L in self.net.layers]}


class _Job:
    def __init__(self, c, seed):
        g = _gen(seed)
        self.T, u = _model(g, c["n"], c["d"], True)
        self.shift = _randn(g, c["n"])
        self.P = Polytope(torch.cat([self.T, -self.T]), torch.cat([u, u]))
        self.X0 = torch.zeros(c["d"], dtype=torch.float64, device=DEV)
        self.out = torch.empty((c["samples"] * c["chains"], c["n"]), dtype=torch.float32, pin_memory=True)
        self.shape = (c["samples"], c["thinning"], c["chains"])
        self.kw = dict(mode=c["mode"], seed=seed, pair_prob=c["pair"], resync_interval=c["resync"])

    def run(self):
        last = sample_backmapped(self.P, self.T, self.shift, self.X0, *self.shape, self.out, **self.kw)
        return {"out": self.out, "last": last}


_PREPARE = {"cube": _prepare_cube, "chains": _prepare_chains, "variants": _Variants, "backmap": _Backmap,
            "validate": _Validate, "network": _Network, "job": _Job}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, int(seed))


def run(state):
    return state.run()


# -------------------------------------------------------------------- work
def work(case):
    c, k = case, case["kind"]
    if k in ("cube", "chains", "variants", "job"):
        # per step one column of A (two for a pair step): a multiply, a divide,
        # two comparisons and an update for each of its nonzero rows; per saved
        # sample one row written
        steps = c["samples"] * c["thinning"] * c["chains"] * c.get("models", 1)
        d = c["d"]
        m = 2 * (d if k == "cube" else c["n"]) + (100 if k == "variants" else 0)
        dense = k == "job" or c.get("rounded", False)
        rows = 2 if k == "cube" else (m if dense else 0.08 * m)
        elt = 8 if c.get("precision") == "fp64" else 4
        row_ops = steps * rows * (1 + c.get("pair", 0.0))
        # each step's column has to come from somewhere; A itself is small enough to stay on chip
        size = m * d * (1.0 if dense else 0.08 if k != "cube" else 1.0 / d) * elt * c.get("models", 1)
        out = c["samples"] * c["chains"] * c.get("models", 1) * (c["n"] if k == "job" else d) * 4
        more = 2.0 * c["n"] * d * c["samples"] * c["chains"] if k == "job" else 0.0
        return {"bytes": size + out, "flops": 6.0 * row_ops + more}
    if k == "backmap":
        n, d, N = c["n"], c["d"], c["rows"]
        return {"bytes": 4.0 * N * (n + d) + 8.0 * n * (d + 1), "flops": 2.0 * n * d * N}
    if k == "validate":
        N = c["dim"] * c["chains"] * c["samples"]
        # a transform's worth of operations for the autocovariances
        return {"bytes": 4.0 * N, "flops": N * (10.0 * math.log2(2 * c["samples"]) + 8.0)}
    a, h, o, B = c["n_in"], c["hidden"], c["n_out"], c["batch"]
    p = a * h + h * h + h * o
    if not c["train"]:
        return {"bytes": 2.0 * p + 4.0 * B * (a + o), "flops": 2.0 * B * p}
    # weights and both moments read and written, the gradient written, two BF16 copies written
    return {"bytes": p * (24.0 + 4.0 + 4.0) + 4.0 * B * (a + o), "flops": 2.0 * B * (3 * p - a * h)}


# ------------------------------------------------------------------- exact
def _philox(step, chain, seed):
    """The step's first four uniforms of Philox4x32-10 (arrays over steps and chains)."""
    M = np.uint64(0xFFFFFFFF)
    step, chain = np.broadcast_arrays(np.asarray(step, np.uint64), np.asarray(chain, np.uint64))
    v = [step & M, step >> np.uint64(32), chain, np.zeros_like(chain)]
    k = [int(seed) & 0xFFFFFFFF, (int(seed) >> 32) & 0xFFFFFFFF]
    for _ in range(10):
        p0, p1 = v[0] * np.uint64(0xD2511F53), v[2] * np.uint64(0xCD9E8D57)
        v = [(p1 >> np.uint64(32)) ^ v[1] ^ np.uint64(k[0]), p1 & M, (p0 >> np.uint64(32)) ^ v[3] ^ np.uint64(k[1]),
             p0 & M]
        k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
    return [(w.astype(np.float64) + 1.0) * 2.0 ** -32 for w in v]


def _exact_cube(c, seed):
    """A coordinate step in [0, 1]^d puts the coordinate at the step's uniform."""
    d, k, n = c["d"], c["chains"], c["samples"]
    steps = n * c["thinning"]
    _, uj, ua, _ = _philox(np.arange(steps)[:, None], np.arange(k)[None, :], seed)
    j = np.minimum((uj * d).astype(np.int64), d - 1)
    x, out, chain = np.full((k, d), 0.5), np.empty((n, k, d)), np.arange(k)
    for t in range(steps):
        x[chain, j[t]] = ua[t]
        if t % c["thinning"] == 0:
            out[t // c["thinning"]] = x
    return {"samples": out.reshape(n * k, d), "last": x}


def _exact_backmap(c, seed):
    s = _Backmap(c, seed)
    return s.Y.to(torch.float64) @ s.T.t() + s.shift


def _exact_validate(c, seed):
    """Geyer's initial positive sequence per series and split-R-hat per coordinate."""
    S = _series(c, seed).to(torch.float64)
    k, n, dim = c["chains"], c["samples"], c["dim"]
    x = S.reshape(n, k, dim).permute(2, 1, 0) if c["layout"] == 1 else S.reshape(k, n, dim).permute(2, 0, 1)
    ess = torch.empty((dim, k), dtype=torch.float64)
    for i in range(dim):
        y = x[i] - x[i].mean(dim=1, keepdim=True)
        f = torch.fft.rfft(y, 2 * n)
        rho = torch.fft.irfft(f * f.conj(), 2 * n)[:, : n]
        rho = rho / rho[:, :1]
        pair = (rho[:, 1::2][:, : n // 2 - 1] + rho[:, 2::2][:, : n // 2 - 1])
        keep = torch.cumprod((pair >= 0).to(torch.float64), dim=1)
        ess[i] = (n / (1.0 + 2.0 * (pair * keep).sum(dim=1)).clamp_min(1.0)).cpu()
    h = n // 2
    y = torch.stack([x[:, :, :h], x[:, :, h: 2 * h]], dim=2).reshape(dim, 2 * k, h)
    mean, W = y.mean(dim=2), y.var(dim=2).mean(dim=1)
    rhat = torch.sqrt(((h - 1.0) / h * W + mean.var(dim=1)) / W)
    return {"ess": ess, "rhat": rhat}


def _exact_network(c, seed):
    """Forward, loss gradient and Adam's first step in 64 bits."""
    net = RoundingNet((c["n_in"], c["hidden"], c["hidden"], c["n_out"]), seed=seed)
    W = [L.W[:, : L.n_in].double() for L in net.layers]
    b = [L.b.double() for L in net.layers]
    X, T = (torch.as_tensor(v, device=DEV).double() for v in _network_inputs(c, seed))
    for p in W + b:
        p.requires_grad_(True)
    a = X
    for i in range(3):
        a = a @ W[i].t() + b[i]
        if i < 2:
            a = torch.nn.functional.gelu(a)
    if not c["train"]:
        return {"out": a.detach()}
    loss = ((a - T) ** 2).sum() / c["batch"]
    loss.backward()
    lr, eps = net.lr, net.eps
    new = [(p - lr * p.grad / (p.grad.abs() + eps)).detach() for p in W + b]
    return {"loss": float(loss.detach()), "W": new[:3], "b": new[3:], "gW": [p.grad for p in W], "gb": [p.grad for p in b]}


def exact(case, seed):
    k = case["kind"]
    if k == "cube":
        return _exact_cube(case, seed)
    if k == "backmap":
        return _exact_backmap(case, seed)
    if k == "validate":
        return _exact_validate(case, seed)
    if k == "network":
        return _exact_network(case, seed)
    # A chain in any other polytope has no value to be near to: once a rounding
    # difference changes which row ends a chord, two chains part for good.
    return None
