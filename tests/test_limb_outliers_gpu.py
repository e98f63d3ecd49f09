"""Outliers of the fixed-point reduction at the counts where its form changes: a
tile of 64 (128) points takes up to 2 (4) points with basis values out of range
beside its limbs and goes to FP64 with one more; points with weights that are
not finite follow in rounds of eight, whatever their number.

Tolerance: as for the sums of ordinary points, 3e-14 of the sum of the terms'
magnitudes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _run(M, x, sens):
    import torch
    n = x.shape[1]
    dev = lambda a: torch.as_tensor(np.ascontiguousarray(a), device="cuda")  # noqa: E731
    comp = M.CreateComponent(M.FixedMultiIndexSet(3, 3), M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis))
    comp.SetCoeffs(np.random.default_rng(1).normal(0.0, 0.1, comp.numCoeffs))
    y, ld, cg = (torch.zeros(s, dtype=torch.float64, device="cuda") for s in ((1, n), (n,), (comp.numCoeffs,)))
    comp.FusedForwardAdjointImpl(dev(x), sens=dev(sens), out_eval=y, out_logdet=ld, coeff_grad=cg)
    return cg.cpu().numpy(), comp.CoeffGrad(dev(x), dev(sens)).cpu().numpy()


def _tiles(n):
    """Points of a tile: consecutive in order of |x_3| (128-point tiles above 64
    points an SM, else 64), so far inputs at consecutive |x_3| share one."""
    import torch
    return 64 if n <= 64 * torch.cuda.get_device_properties(0).multi_processor_count else 128


@pytest.mark.parametrize("large", [False, True])
@pytest.mark.parametrize("far", [1, 2, 3, 4, 5, 8, 20])
def test_far_points_of_one_tile(gpu, far, large):
    n = 20_000 if large else 1000
    r = np.random.default_rng(far)
    x = r.standard_normal((3, n))
    x[2] = np.linspace(0.001, 2.9, n)  # (already in order: tile t holds points t tpb ...)
    tpb = _tiles(n)
    for tile in (0, 3, n // tpb):
        pts = tile * tpb + r.choice(min(tpb, n - tile * tpb), min(far, n - tile * tpb), replace=False)
        x[0, pts] = 40.0 + np.arange(pts.size)
    cg, dense = _run(gpu, x, r.standard_normal((1, n)))
    err, size = np.abs(cg - dense.astype(np.longdouble).sum(1)), np.abs(dense).sum(1)
    assert np.all(err <= 3e-14 * size)


@pytest.mark.parametrize("bad", [1, 7, 8, 9, 17, 64])
@pytest.mark.parametrize("kind", ["nan", "inf"])
def test_weights_that_are_not_finite(gpu, kind, bad):
    """x_1 = 0 at the points with bad weights: entries of terms that vanish there
    become NaN (0 times inf or NaN) like the others; with no bad point among the
    first tile's the rest of the sum is untouched.  Every entry's class (finite,
    NaN, infinite) is that of the dense entries' sum."""
    n = 1000
    r = np.random.default_rng(bad)
    x = r.standard_normal((3, n))
    x[2] = np.linspace(0.001, 2.9, n)
    sens = r.standard_normal((1, n))
    pts = 64 + r.choice(64, bad, replace=False)
    x[0, pts[::2]] = 0.0
    sens[0, pts] = np.nan if kind == "nan" else np.inf
    cg, dense = _run(gpu, x, sens)
    with np.errstate(invalid="ignore"):
        want = dense.sum(1)
    assert np.array_equal(np.isnan(cg), np.isnan(want))
    assert np.array_equal(np.isinf(cg), np.isinf(want))
    assert np.array_equal(np.sign(cg[np.isinf(cg)]), np.sign(want[np.isinf(want)]))
