"""The fixed-point phase A and reduced adjoint against the oracle where they
change form: ragged tiles (one point, tile and warp edges), points whose
products leave the fixed-point range (few, and more than one round of them),
coefficients over many magnitudes, components of one input and of deep
prefixes, and a batch of maps beside the same maps alone.

Tolerance: the parity bar of the other GPU tests (1e-10 relative, with a floor
of 1e-6 of the largest entry, 1e-3 for sums over points)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _close(a, b, floor):
    a, b = np.asarray(a), np.asarray(b)
    err = np.abs(a - b) / np.maximum(np.abs(b), floor * np.max(np.abs(b)))
    assert np.max(err) <= 1e-10


def _run(M, oracle, dim, order, basis, pos, n, scale_far, n_far, coef_scale, seed):
    import torch
    r = np.random.default_rng(seed)
    hf = basis == "hf"
    opts = M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis,
                        basisType=M.BasisTypes.HermiteFunctions if hf else M.BasisTypes.ProbabilistHermite,
                        posFuncType=M.PosFuncTypes.Exp if pos == "exp" else M.PosFuncTypes.SoftPlus)
    tm = M.CreateTriangular(dim, dim, order, opts)
    c = r.normal(0.0, 0.05, tm.numCoeffs)
    if coef_scale:
        c *= 10.0 ** r.uniform(-6, 0, c.size)
    tm.SetCoeffs(c)
    x = r.standard_normal((dim, n))
    if n_far:
        x[0, r.choice(n, n_far, replace=False)] *= scale_far
    sens, ls = r.standard_normal((dim, n)), 0.7
    dev = lambda a: torch.as_tensor(a, dtype=torch.float64, device="cuda")  # noqa: E731
    y, ld, cg = dev(np.zeros((dim, n))), dev(np.zeros(n)), dev(np.zeros(c.size))
    tm.FusedForwardAdjointImpl(dev(x), sens=dev(sens), logdet_sens_scale=ls, out_eval=y, out_logdet=ld, coeff_grad=cg)
    om = oracle.OracleTriangularMap(dim, dim, order, basis=oracle.BASIS_HERMITE_FUNCTIONS if hf else oracle.BASIS_PROB_HERMITE,
                                    posfunc=oracle.POS_EXP if pos == "exp" else oracle.POS_SOFTPLUS)
    _close(y.cpu(), om.evaluate(c, x), 1e-6)
    _close(ld.cpu(), om.logdet(c, x), 1e-6)
    _close(cg.cpu(), om.coeff_grad(c, x, sens).sum(1) + ls * om.logdet_coeff_grad(c, x).sum(1), 1e-3)
    return tm, dev(x), dev(sens), y, ld, cg


@pytest.mark.parametrize("n", [1, 31, 33, 127, 129, 1000])
def test_ragged_tiles(gpu, oracle, n):
    _run(gpu, oracle, 4, 3, "ph", "softplus", n, 1.0, 0, False, n)


@pytest.mark.parametrize("basis,pos", [("ph", "softplus"), ("hf", "softplus"), ("hf", "exp")])
@pytest.mark.parametrize("n_far", [1, 8, 9, 70])
def test_points_out_of_range(gpu, oracle, basis, pos, n_far):
    # (the far inputs have Hermite polynomials, and linear terms of the Hermite
    # functions, beyond the fixed-point bounds)
    _run(gpu, oracle, 3, 3, basis, pos, 300, 6.0 if basis == "ph" else 40.0, n_far, True, n_far)


@pytest.mark.parametrize("dim,order", [(1, 6), (2, 1), (7, 6), (12, 2)])
def test_shapes_and_coefficient_ranges(gpu, oracle, dim, order):
    _run(gpu, oracle, dim, order, "ph", "softplus", 257, 1.0, 0, True, 10 * dim + order)


@pytest.mark.parametrize("tpb", [64, 128])
def test_batch_matches_single_maps(gpu, oracle, tpb):
    import torch
    runs = [_run(gpu, oracle, d, o, "ph", "softplus", n, 6.0, 9, True, 7 * d + o) for d, o, n in
            ((2, 5, 1500), (5, 3, 700), (9, 2, 65))]
    b = gpu.MapBatch([q[0] for q in runs])
    b.SetTuning(tpb, b.Tuning()[1])
    out = [(torch.zeros_like(q[3]), torch.zeros_like(q[4]), torch.zeros_like(q[5])) for q in runs]
    b.FusedForwardAdjoint([q[1] for q in runs], [q[2] for q in runs], logdet_sens_scale=0.7,
                          out_eval=[o[0] for o in out], out_logdet=[o[1] for o in out], coeff_grad=[o[2] for o in out])
    for q, o in zip(runs, out):
        _close(o[0].cpu(), q[3].cpu(), 1e-6)
        _close(o[1].cpu(), q[4].cpu(), 1e-6)
        _close(o[2].cpu(), q[5].cpu(), 1e-3)
