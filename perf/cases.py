"""The workloads whose speed this framework is built for.

Every case is a call that a program using laker_b200 makes through the public
classes: operator products (one or many right-hand sides, float32 and float64,
forward and backward), single, large, batched and multi-RHS solves, predictions
and predictive variances.  `listed()` names the cases that stand for the range,
`draw()` gives others of the same ranges.

Inputs are radio maps: locations uniform in [0, 100]^2, embedded by a random
Fourier feature network (cos features, one tanh layer) as the default position
embedding does, targets from five path-loss sources with 2 dB shadowing.
"""

from __future__ import annotations

import math

import torch

import laker_b200

DEVICE = "cuda"
EXTENT = 100.0
LAMBDA = 1e-2

# Points of the largest float32 product of many columns, and kernel entries times
# right-hand sides of the largest variance solve, that draw() gives.
MAX_MULTI_POINTS = 12_000
MAX_VARIANCE = 20_000**2 * 256


def listed():
    return [
        # The smallest call: one product for a map of 1000 points (interactive
        # use, a caller's own iterative method); launches and latency count.
        {"name": "matvec_n1000", "kind": "matvec", "n": 1000, "d": 10, "k": 1, "dtype": "float32"},
        # The operator of the largest solves: 100,000 points, one vector.
        {"name": "matvec_n100000", "kind": "matvec", "n": 100000, "d": 10, "k": 1, "dtype": "float32"},
        # Many right-hand sides: the preconditioner's probes, the operator of a
        # variance solve.  Float32 products of many columns accumulate on the
        # tensor cores with a rounding of up to 1e-5 at 12,000 points that grows
        # with the points (2e-4 at 50,000), so larger ones are measured inside
        # the variance solves below, whose float64 residuals correct it.
        {"name": "matvec_n10000_k512", "kind": "matvec", "n": 10000, "d": 10, "k": 512, "dtype": "float32"},
        # A float64 operator, ragged size: the true residual of a solve.
        {"name": "matvec_f64_n30011", "kind": "matvec", "n": 30011, "d": 10, "k": 1, "dtype": "float64"},
        # A float64 operator on a block of vectors: probes or residuals of a
        # multi-RHS solve in float64.
        {"name": "matvec_f64_n8009_k200", "kind": "matvec", "n": 8009, "d": 10, "k": 200, "dtype": "float64"},
        # A training step's product: forward, then the gradients with respect
        # to the embeddings and the vector (embedding_dim at its maximum).
        {"name": "backward_n10007_d16", "kind": "backward", "n": 10007, "d": 16, "k": 1, "dtype": "float32"},
        # Predictions of a fitted model at 2000 new locations.
        {"name": "predict_n20000_m2000", "kind": "predict", "n": 20000, "d": 10, "m": 2000},
        # A small solve at the solver's default tolerance.
        {"name": "solve_n2000", "kind": "solve", "n": 2000, "d": 10, "dtype": "float64", "tol": 1e-10},
        # The large single solve, to 1e-6, float32 targets.
        {"name": "solve_n100000", "kind": "solve", "n": 100000, "d": 10, "dtype": "float32", "tol": 1e-6},
        # A serving query: predictive variance of 16 locations on a large map.
        {"name": "variance_n30011_m16", "kind": "variance", "n": 30011, "d": 10, "m": 16, "tol": 1e-10},
        # Predictive variance of 256 locations on a map of 20,000 points.
        {"name": "variance_n20000_m256", "kind": "variance", "n": 20000, "d": 10, "m": 256, "tol": 1e-10},
        # Independent regressions of uneven size solved together.
        {"name": "batch_24", "kind": "batch", "count": 24, "n_min": 500, "n_max": 20000, "d": 10,
         "sizes": 1234, "tol": 1e-10},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "multi", "multi", "matvec_f64", "multi_f64", "backward",
                       "predict", "solve", "solve", "variance", "batch"])
    # embedding_dim 10 is the default; up to 16 can be chosen
    d = 10 if rng.random() < 0.6 else rng.randint(2, 16)
    if kind == "matvec":
        return {"kind": "matvec", "n": _log_int(rng, 500, 100000), "d": d, "k": 1, "dtype": "float32"}
    if kind == "multi":
        k = _log_int(rng, 2, 512)
        return {"kind": "matvec", "n": _log_int(rng, 1000, MAX_MULTI_POINTS), "d": d, "k": k,
                "dtype": "float32"}
    if kind == "matvec_f64":
        return {"kind": "matvec", "n": _log_int(rng, 500, 100000), "d": d, "k": 1, "dtype": "float64"}
    if kind == "multi_f64":
        k = _log_int(rng, 2, 512)
        return {"kind": "matvec", "n": _log_int(rng, 1000, 20000), "d": d, "k": k, "dtype": "float64"}
    if kind == "backward":
        return {"kind": "backward", "n": _log_int(rng, 1000, MAX_MULTI_POINTS), "d": d,
                "k": rng.choice([1, 1, 2, 4]), "dtype": "float32"}
    if kind == "predict":
        return {"kind": "predict", "n": _log_int(rng, 1000, 100000), "d": d, "m": _log_int(rng, 16, 5000)}
    if kind == "solve":
        n = _log_int(rng, 500, 90000)
        if n > 25000:
            return {"kind": "solve", "n": n, "d": 10, "dtype": "float32", "tol": 1e-6}
        return {"kind": "solve", "n": n, "d": 10, "dtype": "float64", "tol": 1e-10}
    if kind == "variance":
        m = _log_int(rng, 16, 256)
        top = min(30000, int(math.sqrt(MAX_VARIANCE / m)))
        return {"kind": "variance", "n": _log_int(rng, 1000, top), "d": 10, "m": m, "tol": 1e-10}
    return {"kind": "batch", "count": rng.randint(6, 24), "n_min": 500, "n_max": _log_int(rng, 2000, 16000),
            "d": 10, "sizes": rng.randint(0, 10**6), "tol": 1e-10}


# ---- inputs ------------------------------------------------------------------
class FieldEmbedding(torch.nn.Module):
    """Random Fourier features and one tanh layer, fixed weights: the network
    that maps locations to embeddings, as a program with its own embedding
    passes it in."""

    def __init__(self, d, device):
        super().__init__()
        g = torch.Generator().manual_seed(42)
        features = 2 * d
        self.freq = (torch.randn(2, features, generator=g) / 10.0).to(device)
        self.phase = (torch.rand(features, generator=g) * (2.0 * math.pi)).to(device)
        b1, b2 = math.sqrt(1.0 / features), math.sqrt(1.0 / d)
        uniform = lambda shape, b: (torch.rand(shape, generator=g) * (2 * b) - b).to(device)  # noqa: E731
        self.w1, self.c1 = uniform((features, d), b1), uniform((d,), b1)
        self.w2, self.c2 = uniform((d, d), b2), uniform((d,), b2)

    def forward(self, x):
        features = torch.cos(2.0 * math.pi * (x @ self.freq) + self.phase)
        return torch.tanh(features @ self.w1 + self.c1) @ self.w2 + self.c2


def _generator(seed):
    return torch.Generator(device=DEVICE).manual_seed(int(seed))


def _field(n, gen):
    """Locations (n, 2) and standardised targets (n,) of one radio map, float32."""
    x = torch.rand(n, 2, generator=gen, device=DEVICE) * EXTENT
    sources = torch.rand(5, 2, generator=gen, device=DEVICE) * EXTENT
    y = -20.0 * torch.log10(torch.cdist(x, sources) + 1.0).sum(dim=1)
    y = y + 2.0 * torch.randn(n, generator=gen, device=DEVICE)
    return x, (y - y.mean()) / y.std()


def _batch_sizes(case):
    g = torch.Generator().manual_seed(case["sizes"])
    u = torch.rand(case["count"], 2, generator=g, dtype=torch.float64)
    lo, hi = math.log(case["n_min"]), math.log(case["n_max"])
    ns = torch.exp(lo + u[:, 0] * (hi - lo)).floor()
    lams = torch.exp(math.log(1e-3) + u[:, 1] * math.log(100.0))
    return [int(v) for v in ns.tolist()], lams.tolist()


def _inputs(case, seed):
    """The case's input tensors, from the seed alone."""
    gen = _generator(seed)
    kind, d = case["kind"], case["d"]
    embed = FieldEmbedding(d, DEVICE)
    if kind == "batch":
        ns, lams = _batch_sizes(case)
        fields = [_field(n, gen) for n in ns]
        return {"E": [embed(x) for x, _ in fields], "y": [y for _, y in fields], "lams": lams}
    x, y = _field(case["n"], gen)
    got = {"embed": embed, "x": x, "y": y, "E": embed(x)}
    if kind in ("matvec", "backward"):
        dtype = torch.float32 if case["dtype"] == "float32" else torch.float64
        shape = (case["n"],) if case["k"] == 1 else (case["n"], case["k"])
        got["v"] = torch.randn(shape, generator=gen, device=DEVICE).to(dtype)
        got["E"] = got["E"].to(dtype)
        if kind == "backward":
            got["g"] = torch.randn(shape, generator=gen, device=DEVICE).to(dtype)
    if kind in ("predict", "variance"):
        got["xq"] = torch.rand(case["m"], 2, generator=gen, device=DEVICE) * EXTENT
    if kind == "predict":
        # a fitted alpha is the noise-like misfit over lambda
        got["alpha"] = 90.0 * torch.randn(case["n"], generator=gen, device=DEVICE, dtype=torch.float64)
    return got


# ---- the measured calls --------------------------------------------------------
def prepare(case, seed):
    s = _inputs(case, seed)
    s["kind"] = case["kind"]
    if case["kind"] == "batch":
        s["ops"] = [laker_b200.AttentionKernelOperator(E, lambda_reg=lam)
                    for E, lam in zip(s["E"], s["lams"])]
        s["pres"] = laker_b200.build_cccp_batched(s["ops"], seeds=list(range(len(s["ops"]))))
        s["pcg"] = laker_b200.BatchedPCG(tol=case["tol"], max_iter=2000)
        return s
    if case["kind"] == "backward":
        s["E"].requires_grad_(True)
        s["v"].requires_grad_(True)
    core = laker_b200.LAKERCore(embedding_dim=case["d"], lambda_reg=LAMBDA, embedding_module=s.get("embed"),
                                pcg_tol=case.get("tol", 1e-6), pcg_max_iter=2000, device=torch.device(DEVICE),
                                dtype=s["E"].dtype, verbose=False)
    s["core"], s["op"] = core, core.build_kernel_operator(s["E"])
    if case["kind"] in ("solve", "variance"):
        n = case["n"]
        s["pre"] = core.build_preconditioner(s["op"].matvec, n, num_probes=256 if n > 20000 else 200, seed=0)
    if case["kind"] == "solve":
        s["b"] = s["y"].to(torch.float32 if case["dtype"] == "float32" else torch.float64)
        s["pcg"] = laker_b200.PreconditionedConjugateGradient(tol=case["tol"], max_iter=2000, verbose=False)
    return s


def run(s):
    kind = s["kind"]
    if kind == "matvec":
        return s["op"].matvec(s["v"])
    if kind == "backward":
        y = s["op"].matvec(s["v"])
        gE, gv = torch.autograd.grad(y, (s["E"], s["v"]), s["g"])
        return {"y": y.detach(), "gE": gE, "gv": gv}
    if kind == "predict":
        return s["core"].predict(s["xq"], s["embed"], s["E"], s["op"], s["alpha"])
    if kind == "solve":
        return s["pcg"].solve(s["op"].matvec, s["pre"].apply, s["b"])
    if kind == "variance":
        return s["core"].predict_variance(s["xq"], s["embed"], s["E"], s["op"], s["pre"], None, LAMBDA)
    return s["pcg"].solve(s["ops"], s["pres"], s["y"])


def _iterations(n, tol):
    """PCG iterations of the float64 recurrence on these fields (156 at n = 2000,
    306 at n = 100,000 for 1e-6), in proportion to the digits asked for."""
    return 156.0 * (n / 2000.0) ** 0.172 * math.log10(1.0 / tol) / 6.0


def work(case):
    """Bytes and floating-point operations of one pass.  A product takes 2 d flops
    for each logit and 2 per right-hand side for each entry; the exponential counts
    one."""
    kind, d = case["kind"], case["d"]
    size = 8 if case.get("dtype") == "float64" else 4

    def product(m, n, k):
        return float(m) * n * (2 * d + 1 + 2 * k)

    if kind == "matvec":
        n, k = case["n"], case["k"]
        return {"bytes": size * n * (d + 2.0 * k), "flops": product(n, n, k)}
    if kind == "backward":
        n, k = case["n"], case["k"]
        return {"bytes": size * n * (2.0 * d + 4.0 * k),
                "flops": 2 * product(n, n, k) + product(n, n, 2 * k * d)}
    if kind == "predict":
        n, m = case["n"], case["m"]
        return {"bytes": 4.0 * d * (n + m) + 8.0 * n + 4.0 * m, "flops": product(m, n, 1)}
    if kind == "batch":
        ns, _ = _batch_sizes(case)
        return {"bytes": sum(n * (4.0 * d + 16.0 + 4 * 200) for n in ns),
                "flops": sum(_iterations(n, case["tol"]) * (product(n, n, 1) + 4.0 * n * 200) for n in ns)}
    n, nr = case["n"], 256 if case["n"] > 20000 else 200
    k = 1 if kind == "solve" else case["m"]
    return {"bytes": n * (4.0 * d + 4.0 * nr + 16.0 * k),
            "flops": _iterations(n, case["tol"]) * (product(n, n, k) + 4.0 * n * nr * k)}


# ---- the same in plain 64-bit torch ----------------------------------------------
def _kernel_times(rows, cols, X, entries=2.0e8):
    """exp(rows cols^T) X in float64, a block of rows at a time."""
    rows, cols, X = rows.double(), cols.double(), X.double()
    step = max(1, int(entries / max(1, cols.shape[0])))
    return torch.cat([torch.exp(rows[i:i + step] @ cols.T) @ X for i in range(0, rows.shape[0], step)])


def _factor(E, lam):
    E = E.double()
    A = torch.exp(E @ E.T)
    A.diagonal().add_(lam)
    return torch.linalg.cholesky(A)


def _solve(E, lam, b):
    """A^-1 b by Cholesky, refined once."""
    L = _factor(E, lam)
    b = b.double().reshape(E.shape[0], -1)
    x = torch.cholesky_solve(b, L)
    return x + torch.cholesky_solve(b - lam * x - _kernel_times(E, E, x), L)


def exact(case, seed):
    kind = case["kind"]
    if kind == "solve" and case["n"] > 40000:
        return None  # a dense factor of that size does not fit
    with torch.no_grad():
        s = _inputs(case, seed)
        if kind == "matvec":
            return _kernel_times(s["E"], s["E"], s["v"]) + LAMBDA * s["v"].double()
        if kind == "backward":
            E, v, g = (s[name].double() for name in ("E", "v", "g"))
            v2, g2 = v.reshape(case["n"], -1), g.reshape(case["n"], -1)
            gE = torch.zeros_like(E)
            for c in range(v2.shape[1]):
                vc, gc = v2[:, c:c + 1], g2[:, c:c + 1]
                gE += gc * _kernel_times(E, E, vc * E) + vc * _kernel_times(E, E, gc * E)
            return {"y": _kernel_times(E, E, v) + LAMBDA * v, "gE": gE,
                    "gv": _kernel_times(E, E, g) + LAMBDA * g}
        if kind == "predict":
            return _kernel_times(s["embed"](s["xq"]), s["E"], s["alpha"])
        if kind == "solve":
            return _solve(s["E"], LAMBDA, s["y"])[:, 0]
        if kind == "variance":
            q, E = s["embed"](s["xq"]).double(), s["E"].double()
            kxq = torch.exp(E @ q.T)
            return torch.exp((q * q).sum(1)) - (kxq * _solve(s["E"], LAMBDA, kxq)).sum(0)
        return [_solve(E, lam, y)[:, 0] for E, lam, y in zip(s["E"], s["lams"], s["y"])]
