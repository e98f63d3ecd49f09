"""Workloads of the monotone-map path, measured through the package's public
entry points: evaluation, log-determinants, inverses, fused and dense adjoints,
the KL objective, a torch training step, batches of maps and sigmoid maps.

Sizes are those of the package's benchmark workloads (a 2 x 2 order-3 map, the
8-D order-4 component at 1M points, the 6-D order-5 KL map on 200k banana
samples, the 16-D order-3 inverse, uneven batches), of its tests, or generic
ones between them.  `exact` is a float64 torch restatement: the terms one by
one, the same adaptive rule walked level by level over all points at once."""
import math
import random

import numpy as np
import torch

import mpart_gb300 as mp

DEV = "cuda"
F64 = torch.float64


def listed():
    return [
        # One small call, as in a sampling loop that asks for a few points at
        # a time: latency and launches.
        {"name": "eval_2d_o3_n64", "kind": "evaluate", "din": 2, "dout": 2, "order": 3, "n": 64,
         "basis": "ph", "pos": "softplus", "quad": "acc", "tol": 1e-6, "std": 0.1},
        # The small workload of the benchmark set, from numpy arrays as a user
        # of the reference's binding holds them: values, log-determinants, inverse.
        {"name": "host_2d_o3_n10000", "kind": "host", "din": 2, "dout": 2, "order": 3, "n": 10000,
         "basis": "ph", "pos": "softplus", "quad": "acc", "tol": 1e-6, "std": 0.1},
        # The reference's published timing: a 5-D degree-5 map under the
        # default AdaptiveSimpson rule; values and log-determinants.
        {"name": "eval_5d_o5_simpson_n200000", "kind": "evaluate", "din": 5, "dout": 5, "order": 5, "n": 200000,
         "basis": "ph", "pos": "softplus", "quad": "simpson", "tol": 1e-6, "std": 0.05},
        # The headline: one 8-D order-4 component, forward and coefficient
        # adjoints of value and log-determinant in one call, 1M points.
        {"name": "fused_8d_o4_n1000000", "kind": "fused", "din": 8, "dout": 1, "order": 4, "n": 1000000,
         "basis": "ph", "pos": "softplus", "quad": "acc", "tol": 1e-6, "std": 0.05, "input_grad": False},
        # A conditional map (5 inputs, 3 outputs) with coefficient and input
        # adjoints at an ordinary ragged batch.
        {"name": "fused_5d_o3_n30011", "kind": "fused", "din": 5, "dout": 3, "order": 3, "n": 30011,
         "basis": "hf", "pos": "exp", "quad": "acc", "tol": 1e-6, "std": 0.05, "input_grad": True},
        # One step of KL training at the benchmark's size.
        {"name": "kl_6d_o5_n200000", "kind": "kl", "din": 6, "dout": 6, "order": 5, "n": 200000,
         "basis": "hf", "pos": "exp", "quad": "acc", "tol": 1e-7, "std": 0.05},
        # One step of KL training on a small data set.
        {"name": "kl_3d_o4_n5003", "kind": "kl", "din": 3, "dout": 3, "order": 4, "n": 5003,
         "basis": "hf", "pos": "softplus", "quad": "acc", "tol": 1e-6, "std": 0.05},
        # A normalizing-flow layer in torch: forward with log-determinant and
        # backward to coefficients and inputs.
        {"name": "torch_4d_o3_n4096", "kind": "torch", "din": 4, "dout": 4, "order": 3, "n": 4096,
         "basis": "ph", "pos": "softplus", "quad": "acc", "tol": 1e-6, "std": 0.05},
        # Per-point coefficient gradients, as the reference's objectives ask for.
        {"name": "dense_4d_o4_n100000", "kind": "dense", "din": 4, "dout": 1, "order": 4, "n": 100000,
         "basis": "ph", "pos": "softplus", "quad": "acc", "tol": 1e-6, "std": 0.05},
        # Inverse (the reference's bracketed ITP) of a 16-D order-3 map, then
        # the implicit gradient.
        {"name": "inverse_16d_o3_n40000", "kind": "inverse", "din": 16, "dout": 16, "order": 3, "n": 40000,
         "basis": "ph", "pos": "softplus", "quad": "acc", "tol": 1e-8, "std": 0.03, "method": "Bracket"},
        # Independent maps of uneven dimension, order and size in one call.
        {"name": "batch_24maps", "kind": "batch", "maps": 24, "dim_max": 10, "order_max": 5, "n_min": 1000,
         "n_max": 50000, "layout": 7, "basis": "ph", "pos": "softplus", "quad": "acc", "tol": 1e-6, "std": 0.05},
        # Sigmoid expansions (no quadrature): forward and adjoint.
        {"name": "sigmoid_8d_o3_n100000", "kind": "sigmoid", "din": 8, "dout": 8, "order": 3, "n": 100000, "nsig": 5},
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["evaluate", "host", "fused", "kl", "torch", "dense", "inverse", "batch", "sigmoid"])
    # (The exponential goes with Hermite functions: polynomials in its argument
    # overflow on ordinary tails.)
    basis, pos = rng.choice([("ph", "softplus"), ("ph", "softplus"), ("hf", "softplus"), ("hf", "exp")])
    c = {"kind": kind, "basis": basis, "pos": pos, "quad": rng.choice(["acc", "acc", "simpson"]),
         "tol": rng.choice([1e-6, 1e-7, 1e-8]), "std": 0.05}
    if kind == "evaluate":
        d = rng.randint(1, 6)
        c.update(din=d, dout=rng.randint(1, d), order=rng.randint(1, 5), n=_log_int(rng, 40, 200000))
    elif kind == "host":
        d = rng.randint(1, 4)
        c.update(din=d, dout=rng.randint(1, d), order=rng.randint(1, 4), n=_log_int(rng, 100, 20000), quad="acc")
    elif kind == "fused":
        d = rng.randint(2, 8)
        c.update(din=d, dout=rng.randint(1, min(d, 3)), order=rng.randint(2, 4), n=_log_int(rng, 1000, 300000),
                 input_grad=rng.random() < 0.3)
    elif kind == "kl":
        d = rng.randint(2, 6)
        c.update(din=d, dout=d, order=rng.randint(2, 5), n=_log_int(rng, 2000, 150000), quad="acc",
                 basis="hf")
    elif kind == "torch":
        d = rng.randint(2, 6)
        c.update(din=d, dout=d, order=rng.randint(2, 4), n=_log_int(rng, 128, 32768), quad="acc")
    elif kind == "dense":
        d = rng.randint(2, 6)
        c.update(din=d, dout=1, order=rng.randint(2, 4), n=_log_int(rng, 1000, 100000))
    elif kind == "inverse":
        d = rng.randint(2, 16)
        c.update(din=d, dout=rng.randint(1, d), order=rng.randint(2, 3), n=_log_int(rng, 300, 30000), quad="acc",
                 basis="ph", pos="softplus", std=0.03, method=rng.choice(["Bracket", "Newton"]))
    elif kind == "batch":
        c.update(maps=rng.randint(4, 24), dim_max=rng.randint(3, 9), order_max=rng.randint(2, 5), n_min=1000,
                 n_max=_log_int(rng, 5000, 40000), layout=rng.randint(0, 10 ** 6), quad="acc")
    else:
        d = rng.randint(2, 8)
        c = {"kind": kind, "din": d, "dout": rng.randint(1, d), "order": rng.randint(1, 3),
             "n": _log_int(rng, 500, 100000), "nsig": rng.randint(2, 6)}
    return c


# ---------------------------------------------------------------------------
# Maps and inputs
# ---------------------------------------------------------------------------
def _options(case):
    return mp.MapOptions(
        basisType=mp.BasisTypes.ProbabilistHermite if case["basis"] == "ph" else mp.BasisTypes.HermiteFunctions,
        posFuncType=mp.PosFuncTypes.SoftPlus if case["pos"] == "softplus" else mp.PosFuncTypes.Exp,
        quadType=mp.QuadTypes.AdaptiveSimpson if case["quad"] == "simpson" else mp.QuadTypes.AdaptiveClenshawCurtis,
        quadAbsTol=case["tol"], quadRelTol=case["tol"])


def _multis(dim, order):
    """Total-order terms: first input outermost, last fastest."""
    out, work = [], [0] * dim

    def rec(d, left):
        for p in range(left + 1):
            work[d] = p
            if d < dim - 1:
                rec(d + 1, left - p)
            else:
                out.append(tuple(work))
    rec(0, order)
    return out


def _rng(seed, tag):
    return np.random.default_rng([int(seed) & 0x7fffffff, tag])


def _coeffs(case, seed, din, dout, order, tag=0):
    """N(0, std^2) coefficients.  A KL map is near the linear map that whitens
    the banana samples, as in a training run, with smaller coefficients on the
    terms of higher degree (the samples have long tails)."""
    r = _rng(seed, 100 + tag)
    parts = []
    for i in range(dout):
        d = din - dout + i + 1
        m = _multis(d, order)
        c = r.normal(0.0, case["std"], len(m))
        if case["kind"] == "kl":
            c *= 8.0 ** -np.maximum(np.array([sum(t) for t in m]) - 1, 0)
            at = {t: j for j, t in enumerate(m)}
            scale = 1.0 if d == 1 else (0.5 if d == 2 else 0.6)
            lin = math.log(1.0 / scale) if case["pos"] == "exp" else math.log(math.expm1(1.0 / scale))
            c[at[(0,) * (d - 1) + (1,)]] += lin
            if d > 2:
                c[at[(0,) * (d - 2) + (1, 0)]] -= 0.8 / 0.6
        parts.append(c)
    return np.concatenate(parts)


def _banana(n, din, seed):
    """x1 ~ N(0,1), x2 = x1^2 + 0.5 N(0,1), x_k = 0.8 x_{k-1} + 0.6 N(0,1)."""
    z = _rng(seed, 1).standard_normal((din, n))
    x = np.empty_like(z)
    x[0] = z[0]
    for k in range(1, din):
        x[k] = x[0] ** 2 + 0.5 * z[1] if k == 1 else 0.8 * x[k - 1] + 0.6 * z[k]
    return x


def _points(case, seed):
    if case["kind"] == "kl":
        return _banana(case["n"], case["din"], seed)
    return _rng(seed, 1).standard_normal((case["din"], case["n"]))


def _batch_layout(case):
    """(dimension, order, points) of every map of a batch."""
    r = random.Random(case["layout"])
    return [(r.randint(2, case["dim_max"]), r.randint(2, case["order_max"]), _log_int(r, case["n_min"], case["n_max"]))
            for _ in range(case["maps"])]


def _sigmoid_parts(case, seed):
    """Centers (sorted, edges outside) per output and coefficients (positive on
    the terms with a last-input factor, as training keeps them)."""
    r = _rng(seed, 7)
    cen = np.stack([np.concatenate([[-3.0, 3.0], np.sort(r.uniform(-2.5, 2.5, case["nsig"])) +
                                    0.2 * np.arange(case["nsig"])]) for _ in range(case["dout"])], axis=1)
    coef = []
    for i in range(case["dout"]):
        for lead, k in _sigmoid_terms(case, i):
            coef.append(r.normal(0.0, 0.05) if k == 0 else 0.05 + 0.1 * r.random())
    return cen, np.array(coef)


def _sigmoid_terms(case, i):
    """(leading multi-index, last order) of output i: the leading set at order
    0, then leading x {1, .., nsig + 3}."""
    d, top = case["din"] - case["dout"] + i + 1, case["nsig"] + 3
    if d == 1:
        return [((), k) for k in range(top + 1)]
    lead = _multis(d - 1, case["order"])
    return [(m, 0) for m in lead] + [(m, k) for m in lead for k in range(1, top + 1)]


def _dev(a):
    return torch.as_tensor(a, dtype=F64, device=DEV)


def _empty(*shape):
    return torch.zeros(shape, dtype=F64, device=DEV)


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "batch":
        maps, pts, sens, val, ld, cg = [], [], [], [], [], []
        for j, (d, o, n) in enumerate(_batch_layout(case)):
            m = mp.CreateTriangular(d, d, o, _options(case))
            m.SetCoeffs(_coeffs(case, seed, d, d, o, j))
            r = _rng(seed, 1000 + j)
            maps.append(m)
            pts.append(_dev(r.standard_normal((d, n))))
            sens.append(_dev(r.standard_normal((d, n))))
            val.append(_empty(d, n))
            ld.append(_empty(n))
            cg.append(_empty(m.numCoeffs))
        s.update(maps=maps, batch=mp.MapBatch(maps), pts=pts, sens=sens, val=val, ld=ld, cg=cg)
        return s
    if kind == "sigmoid":
        cen, coef = _sigmoid_parts(case, seed)
        m = mp.CreateSigmoidTriangular(case["din"], case["dout"], case["order"], cen, mp.MapOptions(
            basisType=mp.BasisTypes.HermiteFunctions, sigmoidBasisSumType=mp.SigmoidSumSizeType.Constant))
    elif case["dout"] == 1 and kind in ("fused", "dense"):
        m = mp.CreateComponent(mp.FixedMultiIndexSet(case["din"], case["order"]), _options(case))
        coef = _coeffs(case, seed, case["din"], 1, case["order"])
    else:
        m = mp.CreateTriangular(case["din"], case["dout"], case["order"], _options(case))
        coef = _coeffs(case, seed, case["din"], case["dout"], case["order"])
    m.SetCoeffs(coef)
    n, din, dout = case["n"], case["din"], case["dout"]
    x = _points(case, seed)
    s["map"] = m
    if kind == "host":
        s["x"] = x
        s["x1"] = np.ascontiguousarray(x[:din - dout])
        s["kw"] = {"xtol": 1e-10, "ytol": 1e-10}
        return s
    s["x"] = _dev(x)
    if kind in ("fused", "sigmoid", "dense"):
        s["sens"] = _dev(_rng(seed, 2).standard_normal((dout, n)))
    if kind in ("fused", "sigmoid"):
        s.update(lsens=_dev(_rng(seed, 3).standard_normal(n)), val=_empty(dout, n), ld=_empty(n),
                 cg=_empty(m.numCoeffs), ig=_empty(din, n) if case.get("input_grad") else None)
    if kind == "torch":
        s["module"] = m.torch(store_coeffs=True, return_logdet=True)
        s["x"] = s["x"].T.contiguous().requires_grad_(True)
    if kind == "inverse":
        # Targets are images of points, as when reference samples of a trained
        # map are pulled back; conditioning inputs are the points' own.
        s["r"] = m.Evaluate(s["x"])
        s["x1"] = s["x"][:din - dout].contiguous()
        s["w"] = _dev(_rng(seed, 2).standard_normal((dout, n)))
        s["kw"] = {"xtol": 1e-10, "ytol": 1e-10, "method": case["method"]}
        s["x"] = None
    return s


def run(s):
    kind = s["kind"]
    if kind == "evaluate":
        return {"value": s["map"].Evaluate(s["x"]), "logdet": s["map"].LogDeterminant(s["x"])}
    if kind == "host":
        m = s["map"]
        y = m.Evaluate(s["x"])
        return {"value": y, "logdet": m.LogDeterminant(s["x"]), "inverse": m.Inverse(s["x1"], y, **s["kw"])}
    if kind in ("fused", "sigmoid"):
        s["map"].FusedForwardAdjointImpl(s["x"], sens=s["sens"], logdet_sens=s["lsens"], out_eval=s["val"],
                                         out_logdet=s["ld"], coeff_grad=s["cg"], input_grad=s["ig"])
        out = {"value": s["val"], "logdet": s["ld"], "coeff_grad": s["cg"]}
        return out if s["ig"] is None else {**out, "input_grad": s["ig"]}
    if kind == "kl":
        loss, grad = s["map"].KLObjective(s["x"])
        return {"loss": loss, "grad": grad}
    if kind == "torch":
        x, mod = s["x"], s["module"]
        x.grad = None
        mod.coeffs.grad = None
        y, ld = mod(x)
        loss = (0.5 * (y * y).sum(dim=1) - ld).mean()
        loss.backward()
        return {"loss": loss.detach(), "value": y.detach(), "logdet": ld.detach(), "grad": mod.coeffs.grad,
                "x_grad": x.grad}
    if kind == "dense":
        return {"grad": s["map"].CoeffGrad(s["x"], s["sens"]), "ld_grad": s["map"].LogDeterminantCoeffGrad(s["x"])}
    if kind == "inverse":
        x = s["map"].Inverse(s["x1"], s["r"], **s["kw"])
        gc, gx1, gr = s["map"].InverseCoeffGrad(s["x1"], x, s["w"])
        return {"x": x, "grad": gc, "grad_x1": gx1, "grad_r": gr}
    s["batch"].FusedForwardAdjoint(s["pts"], s["sens"], logdet_sens_scale=1.0, out_eval=s["val"],
                                   out_logdet=s["ld"], coeff_grad=s["cg"])
    # (one tensor per kind of output: every map's values one after another)
    return {"value": torch.cat([v.reshape(-1) for v in s["val"]]), "logdet": torch.cat(s["ld"]),
            "coeff_grad": torch.cat(s["cg"])}


# ---------------------------------------------------------------------------
# Work
# ---------------------------------------------------------------------------
def _comp_work(d, order, adjoint):
    """Floating-point operations of one point of a total-order component:
    prefix products and per-order sums, a quadrature of three bisections of a
    five-point rule, and (adjoint) the products with the per-order weights."""
    terms = math.comb(d + order, order)
    nodes = math.comb(d - 1 + order, order)
    quad = 17 * (7 * order + 10 + (3 * order if adjoint else 0))
    return nodes + 2 * terms + quad + (2 * terms if adjoint else 0)


def work(case):
    kind = case["kind"]
    if kind == "batch":
        b = f = 0
        for d, o, n in _batch_layout(case):
            terms = sum(math.comb(i + o, o) for i in range(1, d + 1))
            b += 8 * (n * (3 * d + 1) + 2 * terms)
            f += n * sum(_comp_work(i, o, True) for i in range(1, d + 1))
        return {"bytes": b, "flops": f}
    n, din, dout, order = case["n"], case["din"], case["dout"], case["order"]
    dims = [din - dout + i + 1 for i in range(dout)]
    if kind == "sigmoid":
        terms = [len(_sigmoid_terms(case, i)) for i in range(dout)]
        return {"bytes": 8 * (n * (din + 2 * dout + 2) + 2 * sum(terms)),
                "flops": n * sum(4 * t + 40 * (case["nsig"] + 3) for t in terms)}
    terms = sum(math.comb(d + order, order) for d in dims)
    fwd = n * sum(_comp_work(d, order, False) for d in dims)
    adj = n * sum(_comp_work(d, order, True) for d in dims)
    vals = {"evaluate": din + dout + 1, "host": 3 * dout + 2 * din + 1, "kl": din, "dense": din + dout + 2 * terms,
            "fused": din + 2 * dout + 2 + (din if case.get("input_grad") else 0),
            "torch": 2 * (din + dout + 1), "inverse": 3 * din + 3 * dout}[kind]
    steps = {"evaluate": 1, "host": 8, "inverse": 8}.get(kind, 0)
    return {"bytes": 8 * (n * vals + 2 * terms), "flops": steps * fwd if steps else adj}


# ---------------------------------------------------------------------------
# The same in float64 torch, term by term
# ---------------------------------------------------------------------------
def _rect(pos, x):
    """g and g'."""
    if pos == "exp":
        g = torch.exp(x)
        return g, g
    e = torch.exp(-x.abs())
    return torch.log1p(e) + x.clamp(min=0), torch.where(x < 0, e / (1 + e), 1 / (1 + e))


def _basis(basis, x, p):
    """[values], [first], [second derivatives] of orders 0..p (order 0 is 1)."""
    one, zero = torch.ones_like(x), torch.zeros_like(x)
    if basis == "ph":
        he = [one, x]
        for k in range(2, p + 1):
            he.append(x * he[-1] - (k - 1) * he[-2])
        nrm = [1 / math.sqrt(math.sqrt(2 * math.pi) * math.factorial(k)) for k in range(p + 1)]
        v = [one] + [he[k] * nrm[k] for k in range(1, p + 1)]
        d = [zero] + [k * he[k - 1] * nrm[k] for k in range(1, p + 1)]
        d2 = [zero, zero] + [k * (k - 1) * he[k - 2] * nrm[k] for k in range(2, p + 1)]
        return v, d, d2[:p + 1]
    env = torch.exp(-0.5 * x * x)
    psi = []
    for j in range(max(0, p - 1)):
        if j == 0:
            psi.append(math.pi ** -0.25 * env)
        elif j == 1:
            psi.append(math.sqrt(2.0) * x * psi[0])
        else:
            psi.append((x * psi[-1] - math.sqrt((j - 1) / 2) * psi[-2]) / math.sqrt(j / 2))
    v = [one, x] + psi
    d = [zero, one] + [-x * psi[j] + (math.sqrt(2.0 * j) * psi[j - 1] if j else 0) for j in range(len(psi))]
    d2 = [zero, zero] + [-(2 * j + 1 - x * x) * psi[j] for j in range(len(psi))]
    return v[:p + 1], d[:p + 1], d2[:p + 1]


class _Component:
    """One component at points x (d x n): leading products by prefix, the
    per-order sums a_k, and everything that follows from them."""

    def __init__(self, case, d, order, coef, x):
        self.case, self.d, self.P, self.x = case, d, order, x
        self.lead = {}
        for c, m in zip(coef.tolist(), enumerate(_multis(d, order))):
            self.lead.setdefault(m[1][:-1], []).append((m[1][-1], m[0], c))
        self.nterms = len(coef)
        self.tab = [_basis(case["basis"], x[j], order) for j in range(d - 1)]
        self.a = [torch.zeros_like(x[0]) for _ in range(order + 1)]
        for m, ks in self.lead.items():
            p = self.phi(m)
            for k, _, c in ks:
                self.a[k] += c * p

    def phi(self, m, skip=-1):
        p = torch.ones_like(self.x[0])
        for j, o in enumerate(m):
            if o and j != skip:
                p = p * self.tab[j][0][o]
        return p

    def df(self, y, idx=None):
        _, d1, d2 = _basis(self.case["basis"], y, self.P)
        a = self.a if idx is None else [t[idx] for t in self.a]
        return sum(a[k] * d1[k] for k in range(1, self.P + 1)), sum(a[k] * d2[k] for k in range(1, self.P + 1)), d1

    def integrate(self, xd, grad=False):
        """Integral over [0, 1] of x_D g(d_D f(t x_D)), and with grad the
        integrals of x_D g' phi'_k(t x_D) and of d/dx_D of the integrand."""
        tol, n = self.case["tol"], xd.shape[0]
        off = 0.5 if self.case["quad"] == "simpson" else math.sqrt(0.5)
        cw = (1 / 3, 4 / 3, 1 / 3)
        fw = (1 / 6, 2 / 3, 1 / 3, 2 / 3, 1 / 6) if self.case["quad"] == "simpson" else (1 / 15, 8 / 15, 4 / 5, 8 / 15, 1 / 15)
        out = torch.zeros(n, dtype=F64, device=xd.device)
        J = [torch.zeros_like(out) for _ in range(self.P)] if grad else []
        E = torch.zeros_like(out)
        idx = torch.arange(n, device=xd.device)
        lo, hi = torch.zeros_like(xd), torch.ones_like(xd)
        for level in range(30):
            xs, mid, half = xd[idx], 0.5 * (lo + hi), 0.5 * (hi - lo)
            ts = [lo, mid - half * off, mid, mid + half * off, hi]
            ev = []
            for t in ts:
                df, d2, d1 = self.df(t * xs, idx)
                g, gp = _rect(self.case["pos"], df)
                ev.append((xs * g, g, gp, d2, d1, t))
            ic = half * (cw[0] * ev[0][0] + cw[1] * ev[2][0] + cw[2] * ev[4][0])
            ih = half * sum(w * e[0] for w, e in zip(fw, ev))
            ok = (ih - ic).abs() < torch.clamp(tol * ic.abs(), min=tol)
            if level == 29:
                ok = torch.ones_like(ok)
            out.index_add_(0, idx[ok], ih[ok])
            if grad:
                for k in range(self.P):
                    v = half * sum(w * xs * e[2] * e[4][k + 1] for w, e in zip(fw, ev))
                    J[k].index_add_(0, idx[ok], v[ok])
                v = half * sum(w * (xs * e[5] * e[2] * e[3] + e[1]) for w, e in zip(fw, ev))
                E.index_add_(0, idx[ok], v[ok])
            no = ~ok
            if not bool(no.any()):
                break
            idx = torch.cat([idx[no], idx[no]])
            lo, hi = torch.cat([lo[no], mid[no]]), torch.cat([mid[no], hi[no]])
        return out, J, E

    def f0(self, like):
        v, _, _ = _basis(self.case["basis"], torch.zeros_like(like), self.P)
        return sum(self.a[k] * v[k] for k in range(self.P + 1))

    def full(self, grad):
        """T, log det, and with grad dT/da_k, dlogdet/da_k, dT/dx_D, dlogdet/dx_D."""
        xd = self.x[self.d - 1]
        I, J, E = self.integrate(xd, grad)
        self.T = I + self.f0(xd)
        df, d2, d1 = self.df(xd)
        g, gp = _rect(self.case["pos"], df)
        self.g, self.logdet = g, torch.log(g)
        if grad:
            v0, _, _ = _basis(self.case["basis"], torch.zeros_like(xd), self.P)
            self.wT = [v0[k] + (J[k - 1] if k else 0) for k in range(self.P + 1)]
            self.wL = [gp / g * d1[k] for k in range(self.P + 1)]
            self.dTx, self.dLx = E, gp / g * d2
        return self

    def coef_reduced(self, w):
        out = torch.zeros(self.nterms, dtype=F64, device=self.x.device)
        for m, ks in self.lead.items():
            p = self.phi(m)
            for k, t, _ in ks:
                out[t] = (p * w[k]).sum()
        return out

    def coef_dense(self, w):
        out = torch.empty(self.nterms, self.x.shape[1], dtype=F64, device=self.x.device)
        for m, ks in self.lead.items():
            p = self.phi(m)
            for k, t, _ in ks:
                out[t] = p * w[k]
        return out

    def lead_grad(self, w, out):
        """out[j] += d/dx_j of sum_k a_k w_k, leading inputs."""
        for m, ks in self.lead.items():
            if any(m):
                b = sum(c * w[k] for k, _, c in ks)
                for j, o in enumerate(m):
                    if o:
                        out[j] += b * self.phi(m, skip=j) * self.tab[j][1][o]


def _components(case, coef, x, din, dout, order):
    off = 0
    for i in range(dout):
        d = din - dout + i + 1
        nt = math.comb(d + order, order)
        yield i, d, _Component(case, d, order, coef[off:off + nt], x[:d]), slice(off, off + nt)
        off += nt


def _fused_exact(case, coef, x, din, dout, order, sens, lsens, want_x):
    n = x.shape[1]
    val, ld = torch.zeros(dout, n, dtype=F64, device=x.device), torch.zeros(n, dtype=F64, device=x.device)
    cg, ig = torch.zeros(len(coef), dtype=F64, device=x.device), torch.zeros(din, n, dtype=F64, device=x.device)
    for i, d, c, at in _components(case, coef, x, din, dout, order):
        c.full(True)
        val[i], ld = c.T, ld + c.logdet
        s = sens[i] if sens is not None else c.T / n
        w = [s * c.wT[k] + lsens * c.wL[k] for k in range(order + 1)]
        cg[at] = c.coef_reduced(w)
        if want_x:
            c.lead_grad(w, ig)
            ig[d - 1] += s * c.dTx + lsens * c.dLx
    return val, ld, cg, ig


def _root(c, r):
    """x_D with T(x_<D, x_D) = r: bracket by doubling, then safeguarded Newton."""
    f0 = c.f0(r)

    def T(y):
        df, _, _ = c.df(y)
        return c.integrate(y)[0] + f0, _rect(c.case["pos"], df)[0]
    x = torch.zeros_like(r)
    lo, hi = x - 1, x + 1
    for _ in range(40):
        bad = T(lo)[0] > r
        if not bool(bad.any()):
            break
        lo = torch.where(bad, 2 * lo, lo)
    for _ in range(40):
        bad = T(hi)[0] < r
        if not bool(bad.any()):
            break
        hi = torch.where(bad, 2 * hi, hi)
    for _ in range(25):
        y, s = T(x)
        lo, hi = torch.where(y <= r, x, lo), torch.where(y >= r, x, hi)
        nx = x - (y - r) / s
        nx = torch.where((nx >= lo) & (nx <= hi), nx, 0.5 * (lo + hi))
        if bool(((nx - x).abs() <= 1e-14 * (1 + x.abs())).all()):
            return nx
        x = nx
    return x


def _inverse_exact(case, coef, x1, r, w=None):
    din, dout, order = case["din"], case["dout"], case["order"]
    extra, n = din - dout, r.shape[1]
    x = torch.cat([x1, torch.zeros(dout, n, dtype=F64, device=r.device)])
    for i, d, c, _ in _components(case, coef, x, din, dout, order):
        x[d - 1] = _root(c, r[i])
    if w is None:
        return x[extra:]
    # (dT/dx)^T lambda = w, last component first; dL/dc = -sum lambda dT/dc.
    grad, acc = torch.zeros(len(coef), dtype=F64, device=r.device), torch.zeros_like(x)
    for i, d, c, at in reversed(list(_components(case, coef, x, din, dout, order))):
        c.full(True)
        lam = (w[i] - acc[d - 1]) / c.g
        wt = [lam * c.wT[k] for k in range(order + 1)]
        grad[at] = -c.coef_reduced(wt)
        c.lead_grad(wt, acc)
        acc[d - 1] = lam
    return x[extra:], grad, -acc[:extra], acc[extra:]


def _sigmoid_exact(case, seed, x, sens, lsens):
    cen, coef = _sigmoid_parts(case, seed)
    n, dout, top, off = x.shape[1], case["dout"], case["nsig"] + 3, 0
    val, ld = torch.zeros(dout, n, dtype=F64, device=x.device), torch.zeros(n, dtype=F64, device=x.device)
    cg = torch.zeros(len(coef), dtype=F64, device=x.device)
    for i in range(dout):
        d = case["din"] - dout + i + 1
        y, h = x[d - 1], np.concatenate([cen[:2, i], np.sort(cen[2:, i])])
        f, fp = [torch.ones_like(y), y], [torch.zeros_like(y), torch.ones_like(y)]
        for sgn, c0 in ((-1.0, h[0]), (1.0, h[1])):  # edge terms: width 1.5, weight 1/1.5
            g, gp = _rect("softplus", sgn * 1.5 * (y - c0))
            f.append(sgn * g / 1.5)
            fp.append(gp)
        for j in range(2, len(h)):
            b = 4 / (h[3] - h[2]) if j == 2 else (4 / (h[j] - h[j - 1]) if j == len(h) - 1 else 8 / (h[j + 1] - h[j - 1]))
            sg = 0.5 + 0.5 * torch.tanh(0.5 * b * (y - h[j]))
            f.append(sg)
            fp.append(b * sg * (1 - sg))
        terms = _sigmoid_terms(case, i)
        tab = [_basis("hf", x[j], max(case["order"], 1))[0] for j in range(d - 1)]
        lead = {}
        for t, (m, k) in enumerate(terms):
            lead.setdefault(m, []).append((k, off + t))
        T, dT = torch.zeros_like(y), torch.zeros_like(y)
        prods = {}
        for m, ks in lead.items():
            p = torch.ones_like(y)
            for j, o in enumerate(m):
                if o:
                    p = p * tab[j][o]
            r = _rect("softplus", p)[0] if d > 1 else p
            prods[m] = (p, r)
            for k, t in ks:
                T += coef[t] * (r if k else p) * f[k]
                dT += coef[t] * (r if k else p) * fp[k]
        val[i], ld = T, ld + torch.log(dT)
        for m, ks in lead.items():
            for k, t in ks:
                cg[t] = (prods[m][1 if k else 0] * (sens[i] * f[k] + lsens * fp[k] / dT)).sum()
        off += len(terms)
    return val, ld, cg


def exact(case, seed):
    kind = case["kind"]
    dev = DEV if torch.cuda.is_available() else "cpu"
    t = lambda a: torch.as_tensor(a, dtype=F64, device=dev)  # noqa: E731
    if kind == "batch":
        val, ld, cg = [], [], []
        for j, (d, o, n) in enumerate(_batch_layout(case)):
            r = _rng(seed, 1000 + j)
            x, sens = t(r.standard_normal((d, n))), t(r.standard_normal((d, n)))
            v, l, g, _ = _fused_exact(case, _coeffs(case, seed, d, d, o, j), x, d, d, o, sens, 1.0, False)
            val.append(v.reshape(-1))
            ld.append(l)
            cg.append(g)
        return {"value": torch.cat(val), "logdet": torch.cat(ld), "coeff_grad": torch.cat(cg)}
    n, din, dout, order = case["n"], case["din"], case["dout"], case["order"]
    x = t(_points(case, seed))
    if kind == "sigmoid":
        v, l, g = _sigmoid_exact(case, seed, x, t(_rng(seed, 2).standard_normal((dout, n))),
                                 t(_rng(seed, 3).standard_normal(n)))
        return {"value": v, "logdet": l, "coeff_grad": g}
    coef = _coeffs(case, seed, din, dout, order)
    if kind in ("evaluate", "host", "inverse"):
        val, ld = torch.zeros(dout, n, dtype=F64, device=dev), torch.zeros(n, dtype=F64, device=dev)
        for i, d, c, _ in _components(case, coef, x, din, dout, order):
            c.full(False)
            val[i], ld = c.T, ld + c.logdet
        if kind == "evaluate":
            return {"value": val, "logdet": ld}
        if kind == "host":
            return {"value": val, "logdet": ld, "inverse": _inverse_exact(case, coef, x[:din - dout], val)}
        xi, gc, gx1, gr = _inverse_exact(case, coef, x[:din - dout], val, t(_rng(seed, 2).standard_normal((dout, n))))
        return {"x": xi, "grad": gc, "grad_x1": gx1, "grad_r": gr}
    if kind == "dense":
        c = next(_components(case, coef, x, din, 1, order))[2].full(True)
        s = t(_rng(seed, 2).standard_normal((1, n)))[0]
        return {"grad": c.coef_dense([s * w for w in c.wT]), "ld_grad": c.coef_dense(c.wL)}
    if kind == "kl":
        loss, grad = torch.zeros(dout, dtype=F64, device=dev), torch.zeros(len(coef), dtype=F64, device=dev)
        for i, d, c, at in _components(case, coef, x, din, dout, order):
            c.full(True)
            loss[i] = (0.5 * c.T * c.T - c.logdet).mean()
            grad[at] = c.coef_reduced([(c.T * c.wT[k] - c.wL[k]) / n for k in range(order + 1)])
        return {"loss": loss, "grad": grad}
    if kind == "torch":
        v, l, g, gx = _fused_exact(case, coef, x, din, dout, order, None, -1.0 / n, True)
        return {"loss": (0.5 * (v * v).sum(dim=0) - l).mean(), "value": v.T, "logdet": l, "grad": g, "x_grad": gx.T}
    v, l, g, gx = _fused_exact(case, coef, x, din, dout, order, t(_rng(seed, 2).standard_normal((dout, n))),
                               t(_rng(seed, 3).standard_normal(n)), True)
    out = {"value": v, "logdet": l, "coeff_grad": g}
    return {**out, "input_grad": gx} if case.get("input_grad") else out
