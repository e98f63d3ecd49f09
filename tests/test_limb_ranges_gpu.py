"""Coefficients, inputs and adjoint weights of very different sizes: the
fixed-point phase A and reduced adjoint hold each sum to its own terms, as FP64
does.  Sums over points are compared with the per-point gradients (FP64
products) relative to the sum of their magnitudes: no floor.

Tolerances.  A sum of products whose magnitudes add up to 2^-8 of the largest
product and weight of their tile keeps 2^-53.5 of the latter, 2e-14 of its own
size; below that it is formed in FP64.  The per-point gradients and their sum
add a few 1e-16: 3e-14.  Log-determinants of a map whose constant term changes
are compared with the same map without it: a_k, k >= 1, does not meet the
constant, so they agree to the rounding of a_k, 1e-15 relative to terms of at
most 10."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _dev(a):
    import torch
    return torch.as_tensor(np.ascontiguousarray(a), dtype=torch.float64, device="cuda")


def _opts(M, pos="SoftPlus", basis="ProbabilistHermite"):
    return M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis, posFuncType=getattr(M.PosFuncTypes, pos),
                        basisType=getattr(M.BasisTypes, basis))


def _check_gradient(M, comp, x, sens, ld_scale=0.0):
    import torch
    n = x.shape[1]
    y, ld, cg = (torch.zeros(s, dtype=torch.float64, device="cuda") for s in ((1, n), (n,), (comp.numCoeffs,)))
    comp.FusedForwardAdjointImpl(_dev(x), sens=_dev(sens), logdet_sens_scale=ld_scale, out_eval=y, out_logdet=ld,
                                 coeff_grad=cg)
    dense = comp.CoeffGrad(_dev(x), _dev(sens)).cpu().numpy().astype(np.longdouble)
    if ld_scale:
        dense = dense + ld_scale * comp.LogDeterminantCoeffGrad(_dev(x)).cpu().numpy().astype(np.longdouble)
    err = np.abs(cg.cpu().numpy() - dense.sum(1))
    size = np.abs(dense).sum(1)
    assert np.all(err <= 3e-14 * size), float(np.max(err / np.maximum(size, 1e-300)))
    return y, ld


@pytest.mark.parametrize("n", [1, 100, 1000, 20_000])
@pytest.mark.parametrize("scale", [0.3, 1e-1, 1e-2, 1e-3, 1e-4, 1e-6, 1e-9])
def test_small_inputs(gpu, oracle, scale, n):
    M = gpu
    r = np.random.default_rng(n)
    comp = M.CreateComponent(M.FixedMultiIndexSet(4, 4), _opts(M))
    c = r.normal(0.0, 0.1, comp.numCoeffs)
    comp.SetCoeffs(c)
    x = r.standard_normal((4, n))
    x[:3] *= scale
    _check_gradient(M, comp, x, r.standard_normal((1, n)), 0.7)


@pytest.mark.parametrize("n", [100, 1000, 20_000])
@pytest.mark.parametrize("kind", ["mixed", "one_hot", "plus_minus_one", "masked"])
def test_inputs_and_weights_that_do_not_meet(gpu, kind, n):
    """Products that are small at every point although each input is not, and
    weights whose largest lie where the products vanish."""
    M = gpu
    r = np.random.default_rng(7)
    comp = M.CreateComponent(M.FixedMultiIndexSet(4, 4), _opts(M))
    comp.SetCoeffs(r.normal(0.0, 0.1, comp.numCoeffs))
    x, sens = r.standard_normal((4, n)), r.standard_normal((1, n))
    if kind == "mixed":  # each input large at a third of the points, tiny elsewhere
        x[:3] *= np.where(np.arange(n) % 3 == np.arange(3)[:, None], 1.0, 1e-5)
    elif kind == "one_hot":
        x[:3] = np.where(np.arange(n) % 3 == np.arange(3)[:, None], 1.0, 1e-7 * x[:3])
    elif kind == "plus_minus_one":  # He_2 vanishes up to noise
        x[:3] = np.sign(x[:3]) * (1.0 + 1e-6 * r.standard_normal((3, n)))
    else:  # the points with weights up to 1e12 have no second input
        sens *= 10.0 ** np.where(np.arange(n) % 4 == 0, r.uniform(0, 12, n), 0.0)
        x[1, ::4] = 0.0
    _check_gradient(M, comp, x, sens)


@pytest.mark.parametrize("pos", ["SoftPlus", "Exp"])
@pytest.mark.parametrize("c0", [1.0, 1e3, 1e6, 1e9, 1e12, 1e16])
def test_constant_term(gpu, oracle, c0, pos):
    import torch
    M = gpu
    r = np.random.default_rng(11)
    mset = M.FixedMultiIndexSet(3, 3)
    comp, plain = M.CreateComponent(mset, _opts(M, pos)), M.CreateComponent(mset, _opts(M, pos))
    c = r.normal(0.0, 0.1, comp.numCoeffs)
    c[0] = 0.0
    plain.SetCoeffs(c)
    c[0] = c0
    comp.SetCoeffs(c)
    x, sens = r.standard_normal((3, 5000)), r.standard_normal((1, 5000))
    d = (comp.LogDeterminant(_dev(x)) - plain.LogDeterminant(_dev(x))).abs().max()
    assert float(d) <= 1e-14
    # (T itself: the constant plus T without it, each rounded)
    t, t0 = comp.Evaluate(_dev(x)), plain.Evaluate(_dev(x))
    assert torch.all((t - c0 - t0).abs() <= 2.0 ** -51 * c0 + 1e-13)
    _check_gradient(M, comp, x, sens, 0.5)


@pytest.mark.parametrize("c", [[0.0, 1e8, 0.3, 0.0, 1.0], [1.0, 1e-9, 1e8, 0.5, 0.2], [1e-7, 1e-7, 2e-7, 1e-8, 1e-7]])
def test_coefficients_of_one_order(gpu, c):
    """Terms of one order whose largest coefficient meets a vanishing product:
    the others keep their digits (a_0 = sum c phi in float64, few roundings)."""
    import torch
    M = gpu
    comp = M.CreateComponent(M.FixedMultiIndexSet.from_multis([[0, 0, 0], [1, 0, 0], [0, 1, 0], [1, 1, 0], [0, 0, 1]]),
                             _opts(M))
    comp.SetCoeffs(np.array(c))
    r = np.random.default_rng(2)
    x = r.standard_normal((3, 999))
    x[0, ::2], x[1, ::3] = 1e-9, 0.0
    ref = M.CreateComponent(M.FixedMultiIndexSet.from_multis([[0, 0, 1]]), _opts(M))
    ref.SetCoeffs(np.array(c[4:]))
    got = comp.Evaluate(_dev(x)) - ref.Evaluate(_dev(x))
    nrm = (2.0 * np.pi) ** -0.25
    terms = np.stack([c[0] + 0 * x[0], c[1] * nrm * x[0], c[2] * nrm * x[1], c[3] * nrm ** 2 * x[0] * x[1]])
    size = _dev(np.abs(terms).sum(0) + 2.0 * np.abs(c[4]) + 2.0 * np.abs(x[2]))
    assert torch.all((got.reshape(-1) - _dev(terms.sum(0))).abs() <= 1e-14 * size)


def _mixed(r, dim, n):
    """Each input large at a part of the points where the others are tiny."""
    return r.standard_normal((dim, n)) * np.where(np.arange(n) % dim == np.arange(dim)[:, None], 1.0, 1e-5)


@pytest.mark.parametrize("tpb", [64, 128])
def test_batch_of_maps_with_mixed_inputs(gpu, tpb):
    M = gpu
    import torch
    r = np.random.default_rng(4)
    maps, x, s = [], [], []
    for d, o, n in ((2, 5, 1500), (4, 3, 700), (6, 2, 65)):
        maps.append(M.CreateTriangular(d, d, o, _opts(M)))
        maps[-1].SetCoeffs(r.normal(0.0, 0.1, maps[-1].numCoeffs))
        x.append(_dev(_mixed(r, d, n)))
        s.append(_dev(r.standard_normal((d, n))))
    b = M.MapBatch(maps)
    b.SetTuning(tpb, b.Tuning()[1])
    z = lambda *q: torch.zeros(*q, dtype=torch.float64, device="cuda")  # noqa: E731
    cg = [z(m.numCoeffs) for m in maps]
    b.FusedForwardAdjoint(x, s, logdet_sens_scale=0.0, out_eval=[torch.zeros_like(a) for a in s],
                          out_logdet=[z(a.shape[1]) for a in x], coeff_grad=cg)
    for m, a, w, g in zip(maps, x, s, cg):
        dense = m.CoeffGrad(a, w).cpu().numpy().astype(np.longdouble)
        assert np.all(np.abs(g.cpu().numpy() - dense.sum(1)) <= 3e-14 * np.abs(dense).sum(1))


@pytest.mark.parametrize("n", [100, 20_000])
def test_implicit_gradient_with_mixed_inputs(gpu, n):
    """-sum_p dT/dc lambda with lambda from the triangular solve in torch: the
    solves agree to some 1e-15 of lambda's size."""
    import torch
    M = gpu
    dim = 4
    r = np.random.default_rng(9)
    tm = M.CreateTriangular(dim, dim, 3, _opts(M))
    tm.SetCoeffs(r.normal(0.0, 0.1, tm.numCoeffs))
    x, w = _dev(_mixed(r, dim, n)), _dev(r.standard_normal((dim, n)))
    g = tm.InverseCoeffGrad(torch.zeros(0, n, dtype=torch.float64, device="cuda"), x, w)[0]
    J = torch.zeros(n, dim, dim, dtype=torch.float64, device="cuda")
    one = torch.ones(1, n, dtype=torch.float64, device="cuda")
    for i in range(dim):
        c, xi = tm.GetComponent(i), x[:i + 1].contiguous()
        J[:, i, :i + 1] = c.Gradient(xi, one).T
        J[:, i, i] = torch.exp(c.LogDeterminant(xi))
    lam = torch.linalg.solve(J.transpose(1, 2), w.T[:, :, None])[:, :, 0].T.contiguous()
    dense = tm.CoeffGrad(x, lam)
    assert torch.all((g + dense.sum(1)).abs() <= 1e-12 * dense.abs().sum(1))
