"""Work that a program using smolyax_gb300 has it do, as cases that can be timed.

A case is one call of a public entry point on a built interpolant: evaluation
(``ip(x, precision=...)``), one differentiation step
(``smolyax_gb300.autograd.interpolate`` and its backward), the Jacobian
(``ip.gradient(x)``) or the integral (``ip.integral()``).  The index sets are
Lambda = {nu : sum_j k_j nu_j < t} with k_j = log((2 + j) / log 2), over Leja
nodes on [-1, 1]^d or Gauss-Hermite nodes; the targets are exponentials
f_i(x) = exp(-sum_j a_ij x_j) with decaying weights, new for every seed.

``exact`` builds the same interpolant from the mathematics alone: the targets
are products of one-dimensional functions, so that the interpolant is
sum over Lambda of the products of one-dimensional interpolation differences
I_g - I_(g-1), expanded in orthogonal polynomials in 64 bits.
"""
import math

import numpy as np
import torch

from smolyax_gb300 import SmolyakBarycentricInterpolator, nodes
from smolyax_gb300.autograd import interpolate


def listed():
    return [
        # a single query, as inside an optimisation or control loop: latency of one small call
        dict(name="leja10-fp32-1pt", op="eval", rule="leja", d_in=10, d_out=1, t=8.831421, points=1, precision="fp32"),
        # the reference's everyday size: ten parameters, |Lambda| = 1000, ten thousand points in FP64
        dict(name="leja10-fp64-10k", op="eval", rule="leja", d_in=10, d_out=1, t=8.831421, points=10000,
             precision="fp64"),
        # high-dimensional scalar surrogate, |Lambda| = 9999, a large FP32 batch (uncertainty quantification)
        dict(name="leja1000-fp32-100k", op="eval", rule="leja", d_in=1000, d_out=1, t=8.224520, points=100000,
             precision="fp32"),
        # the same surrogate in FP64 with a ragged batch
        dict(name="leja1000-fp64-20k", op="eval", rule="leja", d_in=1000, d_out=1, t=8.224520, points=20011,
             precision="fp64"),
        # a handful of outputs under Gaussian inputs, |Lambda| = 20010
        dict(name="gh100-d8-fp32-50k", op="eval", rule="gh", d_in=100, d_out=8, t=9.464636, points=50001,
             precision="fp32"),
        # a discretised field as output, the largest dense evaluation
        dict(name="gh100-d2048-fp32-64k", op="eval", rule="gh", d_in=100, d_out=2048, t=9.464636, points=65536,
             precision="fp32", memory=8.0),
        # an ordinary vector-valued batch of odd size
        dict(name="leja200-d64-fp32-3k", op="eval", rule="leja", d_in=200, d_out=64, t=7.853604, points=3001,
             precision="fp32"),
        # the faster, less precise option where the caller chooses it
        dict(name="gh100-d300-bf16x3-10k", op="eval", rule="gh", d_in=100, d_out=300, t=7.723434, points=10007,
             precision="bf16x3"),
        # a training step through the interpolant: forward, dL/dx and dL/d(nodal values), FP32 inputs
        dict(name="leja200-d64-train-100k", op="train", rule="leja", d_in=200, d_out=64, t=7.853604, points=100000,
             precision="fp32"),
        # dense Jacobians, as for sensitivities and Newton steps
        dict(name="leja200-d64-jacobian-500", op="jacobian", rule="leja", d_in=200, d_out=64, t=7.853604, points=500,
             precision="fp64"),
        # the reference's own algorithm, kept by users who compare bit patterns at grid points
        dict(name="gh100-d8-barycentric-5k", op="eval", rule="gh", d_in=100, d_out=8, t=7.723434, points=5000,
             precision="fp64_barycentric"),
        # the mean of the surrogate, one call per refinement of a quadrature study
        dict(name="gh100-d8-integral", op="integral", rule="gh", d_in=100, d_out=8, t=9.464636, points=0,
             precision="fp64"),
    ]


def draw(rng):
    """One more case of the listed ranges (sizes spread over their logarithm, odd ones among them)."""
    def logint(lo, hi):
        return max(lo, min(hi, int(round(math.exp(rng.uniform(math.log(lo), math.log(hi + 1))) - 0.25))))

    kind = rng.choice(("fp32-one", "fp64", "fp32-few", "fp32-many", "bf16x3", "train", "jacobian", "barycentric",
                       "integral"))
    rule = rng.choice(("leja", "gh"))
    c = dict(op="eval", rule=rule, precision="fp32")
    if kind == "fp32-one":
        c.update(d_in=logint(10, 1000), d_out=1, points=logint(1, 100000))
        lam = logint(300, 10000)
    elif kind == "fp64":
        c.update(d_in=logint(10, 1000), d_out=rng.choice((1, 1, logint(2, 16))), points=logint(1, 20000),
                 precision="fp64")
        lam = logint(300, 10000)
    elif kind == "fp32-few":
        c.update(d_in=logint(10, 200), d_out=rng.randint(2, 15), points=logint(100, 50000))
        lam = logint(300, 10000)
    elif kind in ("fp32-many", "bf16x3"):
        c.update(d_in=logint(10, 200), d_out=logint(16, 2048), precision="bf16x3" if kind == "bf16x3" else "fp32")
        lam = logint(300, 10000)
        c["points"] = logint(100, max(1000, min(65536, int(4e11 / (lam * c["d_out"])))))
    elif kind == "train":
        c.update(op="train", d_in=logint(10, 200), d_out=logint(1, 64), points=logint(500, 50000))
        lam = logint(300, 5000)
    elif kind == "jacobian":
        c.update(op="jacobian", d_in=logint(10, 200), d_out=logint(1, 64), points=logint(1, 500), precision="fp64")
        lam = logint(300, 5000)
    elif kind == "barycentric":
        c.update(d_in=logint(10, 100), d_out=logint(1, 8), points=logint(10, 3000), precision="fp64_barycentric")
        lam = logint(300, 5000)
    else:
        c.update(op="integral", d_in=logint(10, 200), d_out=logint(1, 64), points=0, precision="fp64")
        lam = logint(300, 10000)
    c["t"] = _threshold(_weights(c["d_in"]), lam)
    return c


def prepare(case, seed):
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    d, d_out, P = case["d_in"], case["d_out"], case["points"]
    A = _target(case, seed)

    def f(X):
        return torch.exp(-(X @ A.T))

    f.on_device = True
    rule = nodes.Leja(dim=d) if case["rule"] == "leja" else nodes.GaussHermite(dim=d)
    precision = case["precision"]
    ip = SmolyakBarycentricInterpolator(node_gen=rule, k=_weights(d), t=case["t"], d_out=d_out, f=f,
                                        memory_limit=case.get("memory", 4.0),
                                        precision="fp32" if precision == "bf16x3" else precision)
    if case["op"] == "eval" and precision != "fp64_barycentric" or case["op"] == "train":
        ip.spectral_plan()
    state = dict(op=case["op"], precision=precision, ip=ip, x=_points(case, gen))
    if case["op"] == "train":
        state["g"] = torch.randn(P, d_out, dtype=torch.float32, device="cuda", generator=gen)
        # the trained FP32 correction of the nodal values, at the start of the training
        state["delta"] = torch.zeros(ip.nodal_values.shape, dtype=torch.float32, device="cuda")
    return state


def run(state):
    ip, x = state["ip"], state["x"]
    if state["op"] == "eval":
        return ip(x, precision=state["precision"])
    if state["op"] == "jacobian":
        return ip.gradient(x)
    if state["op"] == "integral":
        return ip.integral()
    x = x.detach().requires_grad_(True)
    delta = state["delta"].detach().requires_grad_(True)
    y = interpolate(ip, x, ip.nodal_values + delta)
    y.backward(state["g"])
    return {"y": y.detach(), "dx": x.grad, "ddelta": delta.grad}


def work(case):
    P, d, o = case["points"], case["d_in"], case["d_out"]
    lam = len(_index_set(_weights(d), case["t"]))
    wide = 8 if case["precision"].startswith("fp64") else 4
    coef = wide * lam * o
    if case["op"] == "eval":
        return {"bytes": 8 * P * d + wide * P * o + coef, "flops": 2 * P * lam * o}
    if case["op"] == "train":  # x, g, coefficients in; y, dx, one value per node and output out
        return {"bytes": 4 * (2 * P * d + 2 * P * o) + 2 * coef, "flops": 6 * P * lam * o}
    if case["op"] == "jacobian":
        return {"bytes": 8 * (P * d + P * o * d) + coef, "flops": 4 * P * lam * o}
    return {"bytes": coef, "flops": 2 * lam * o}


def exact(case, seed):
    d, o, P = case["d_in"], case["d_out"], case["points"]
    entries = _index_set(_weights(d), case["t"])
    C = _coefficients(case["rule"], entries, _target(case, seed))
    if case["op"] == "integral":
        return C[0].clone()
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    x = _points(case, gen).double()
    if case["op"] == "train":
        g = torch.randn(P, o, dtype=torch.float32, device="cuda", generator=gen).double()
    basis = _Basis(case["rule"], entries, d)
    step = max(1, int(1.5e8 // len(entries)))
    ys, ds = [], []
    for p0 in range(0, P, step):
        xc = x[p0 : p0 + step]
        if case["op"] == "eval":
            ys.append(basis(xc) @ C)
            continue
        xc = xc.clone().requires_grad_(True)
        y = basis(xc) @ C
        if case["op"] == "train":
            ys.append(y.detach())
            ds.append(torch.autograd.grad(y, xc, g[p0 : p0 + step])[0])
        else:
            ds.append(torch.stack([torch.autograd.grad(y[:, i].sum(), xc, retain_graph=True)[0] for i in range(o)], 1))
    if case["op"] == "eval":
        return torch.cat(ys)
    if case["op"] == "train":
        return {"y": torch.cat(ys), "dx": torch.cat(ds), "ddelta": None}
    return torch.cat(ds)


# ---- index sets, targets and inputs -------------------------------------------------------

def _weights(d):
    return np.log((2 + np.arange(d)) / np.log(2))


def _index_set(k, t):
    """All nu with sum_j k_j nu_j < t, as tuples of (dimension, degree > 0), the empty one first."""
    out = []

    def extend(entry, first, rem):
        out.append(entry)
        for j in range(first, len(k)):
            if not k[j] < rem:
                break  # k ascends
            r, g = rem, 1
            while k[j] < r:
                r -= k[j]
                extend(entry + ((j, g),), j + 1, r)
                g += 1

    extend((), 0, float(t))
    return out


def _count(k, t, cap):
    n, stack = 0, [(0, float(t))]
    while stack and n < cap:
        first, rem = stack.pop()
        n += 1
        for j in range(first, len(k)):
            if not k[j] < rem:
                break
            r = rem
            while k[j] < r:
                r -= k[j]
                stack.append((j + 1, r))
    return n


def _threshold(k, size):
    """t (to 6 decimals) with about `size` multi-indices, and no more."""
    lo, hi = float(k[0]), 2.0 * float(k[0])
    while _count(k, hi, size + 1) <= size:
        hi *= 1.5
    for _ in range(20):
        mid = 0.5 * (lo + hi)
        lo, hi = (mid, hi) if _count(k, mid, size + 1) <= size else (lo, mid)
    return round(lo, 6)


def _target(case, seed):
    """Weights a_ij of f_i(x) = exp(-sum_j a_ij x_j)."""
    d, o = case["d_in"], case["d_out"]
    rng = np.random.default_rng([int(seed), d, o])
    j = np.arange(d) + 1
    if case["rule"] == "leja":
        a = rng.uniform(0, 1, (o, d)) / j ** 2
        a *= 0.5 / a.sum(axis=1, keepdims=True)
    else:
        a = rng.normal(0.0, 0.3, (o, d)) / j ** 1.5
    return torch.as_tensor(a, device="cuda")


def _points(case, gen):
    P, d = case["points"], case["d_in"]
    dtype = torch.float32 if case["op"] == "train" else torch.float64
    if case["rule"] == "leja":
        return torch.rand(P, d, dtype=dtype, device="cuda", generator=gen) * 2 - 1
    return torch.randn(P, d, dtype=dtype, device="cuda", generator=gen)


# ---- the interpolant in 64 bits, from the mathematics ----------------------------------------

def _nodes_1d(rule, g):
    if rule == "gh":
        return np.polynomial.hermite.hermgauss(g + 1)[0]
    z = [0.0, 1.0, -1.0, math.sqrt(0.5), -math.sqrt(0.5)]
    for j in range(5, g + 1):
        z.append(math.sqrt((z[(j + 1) // 2] + 1) / 2) if j % 2 else -z[j - 1])
    return np.array(z[: g + 1])


def _phi(rule, z, n):
    """Legendre polynomials, or Hermite polynomials normalised for exp(-z^2) / sqrt(pi): degrees 0..n."""
    out = [torch.ones_like(z), z if rule == "leja" else math.sqrt(2.0) * z]
    for m in range(1, n):
        if rule == "leja":
            out.append(((2 * m + 1) * z * out[m] - m * out[m - 1]) / (m + 1))
        else:
            out.append(math.sqrt(2.0 / (m + 1)) * z * out[m] - math.sqrt(m / (m + 1)) * out[m - 1])
    return out[: n + 1]


def _coefficients(rule, entries, A):
    """[entries, d_out]: sum over Lambda of the products of the one-dimensional
    differences I_g - I_(g-1) of exp(-a z), in the orthogonal basis."""
    index = {e: i for i, e in enumerate(entries)}
    C = torch.zeros(len(entries), A.shape[0], dtype=torch.float64, device=A.device)
    top = max((g for e in entries for _, g in e), default=0)
    diff, last = [], None  # diff[g]: [g + 1, d, d_out]
    for g in range(top + 1):
        z = torch.as_tensor(_nodes_1d(rule, g), device=A.device)
        V = torch.stack(_phi(rule, z, g), 1)
        used = max((j for e in entries for j, m in e if m >= g), default=-1) + 1 if g else A.shape[1]
        vals = torch.exp(-z[:, None] * A.T[:used].reshape(1, -1))
        b = torch.linalg.solve(V, vals).reshape(g + 1, used, -1)
        diff.append(b if g == 0 else b - torch.cat([last[:, :used], torch.zeros_like(b[:1])]))
        last = b
    groups = {}
    for e in entries:
        groups.setdefault(tuple(g for _, g in e), []).append(e)
    for degs, group in groups.items():
        n = int(np.prod([g + 1 for g in degs], initial=1))
        step = max(1, int(5e7 // (n * C.shape[1])))
        subs = list(np.ndindex(*[g + 1 for g in degs]))
        for i in range(0, len(group), step):
            part = group[i : i + step]
            T = torch.ones(1, len(part), C.shape[1], dtype=torch.float64, device=A.device)
            for q, g in enumerate(degs):
                dims = torch.tensor([e[q][0] for e in part], device=A.device)
                T = (T[:, None] * diff[g][:, dims][None]).reshape(-1, len(part), C.shape[1])
            ids = [index[tuple((e[q][0], m) for q, m in enumerate(mu) if m)] for mu in subs for e in part]
            C.index_add_(0, torch.tensor(ids, device=A.device), T.reshape(-1, C.shape[1]))
    return C


class _Basis:
    """[P, entries] products of the entries' polynomials at points x, differentiable in x."""

    def __init__(self, rule, entries, d):
        self.rule, self.entries = rule, entries
        index = {e: i for i, e in enumerate(entries)}
        self.top = max((g for e in entries for _, g in e), default=0)
        self.levels = []
        for n in range(1, max(len(e) for e in entries) + 1):
            es = [(i, e) for i, e in enumerate(entries) if len(e) == n]
            cols = torch.tensor([[i, index[e[:-1]], e[-1][0], e[-1][1]] for i, e in es], device="cuda").T
            self.levels.append(cols)

    def __call__(self, x):
        phi = torch.stack(_phi(self.rule, x, max(1, self.top)))
        order, blocks = [torch.zeros(1, dtype=torch.int64, device=x.device)], [torch.ones_like(x[:, :1])]
        place = torch.zeros(len(self.entries), dtype=torch.int64, device=x.device)
        for ids, parent, dim, deg in self.levels:
            block = blocks[-1][:, place[parent]] * phi[deg, :, dim].T
            place[ids] = torch.arange(ids.numel(), device=x.device)
            order.append(ids)
            blocks.append(block)
        inverse = torch.argsort(torch.cat(order))
        return torch.cat(blocks, 1)[:, inverse]
