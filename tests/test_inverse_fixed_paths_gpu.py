"""The fixed-point Inverse in its two launch shapes, and NaN coefficients of
either sign.  Four lanes a point serve up to 128 points an SM, one lane more:
targets just below, at and above that, solved together and in slices that all
take the small shape, give the same roots to the bit, among them points that
wait for the warp pass (a tight tolerance and far targets: wide quadratures)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["Bracket", "Newton"])
@pytest.mark.parametrize("pos,basis,tol", [("SoftPlus", "ProbabilistHermite", 1e-6), ("Exp", "ProbabilistHermite", 1e-8),
                                           ("SoftPlus", "HermiteFunctions", 1e-11), ("Exp", "HermiteFunctions", 1e-6)])
def test_one_and_four_lanes_agree(gpu, method, pos, basis, tol):
    import torch
    M = gpu
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    r = np.random.default_rng(5)
    tm = M.CreateTriangular(2, 2, 3, M.MapOptions(
        quadType=M.QuadTypes.AdaptiveClenshawCurtis, quadAbsTol=tol, quadRelTol=tol,
        posFuncType=getattr(M.PosFuncTypes, pos), basisType=getattr(M.BasisTypes, basis)))
    tm.SetCoeffs(r.normal(0.0, 0.05, tm.numCoeffs))
    big = 128 * sms + 131
    x = r.standard_normal((2, big))
    x[1, ::97] *= 3.0
    y = tm.Evaluate(torch.as_tensor(x, device="cuda"))
    x1 = torch.zeros(0, big, dtype=torch.float64, device="cuda")
    kw = {"xtol": 1e-10, "ytol": 1e-10, "method": method}
    small = torch.cat([tm.Inverse(x1[:, k:k + 5003], y[:, k:k + 5003].contiguous(), **kw) for k in range(0, big, 5003)],
                      dim=1)
    for n in (128 * sms - 1, 128 * sms, 128 * sms + 1, big):
        a = tm.Inverse(x1[:, :n], y[:, :n].contiguous(), **kw)
        assert torch.equal(a, small[:, :n]), n
    # and they are roots: |T(x) - r| <= ytol + slope xtol, twice that for T's rounding
    slope = torch.exp(torch.stack([tm.GetComponent(i).LogDeterminant(small[:i + 1].contiguous()) for i in range(2)]))
    assert torch.all((tm.Evaluate(small) - y).abs() <= 2.0 * (1e-10 + slope * 1e-10) + 1e-12)


@pytest.mark.parametrize("method", ["Bracket", "Newton"])
def test_nan_coefficients_of_either_sign(gpu, method):
    """A NaN coefficient of a term in x_1: points where it meets no product
    (x_1 = 0 times NaN is NaN too) all get what a NaN without sign gives."""
    import torch
    M = gpu
    out = []
    for nan in (np.nan, -np.nan):
        comp = M.CreateComponent(M.FixedMultiIndexSet(1, 2), M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis))
        c = np.array([0.1, 0.2, 0.3])
        c[0] = np.copysign(np.nan, 1.0 if nan is np.nan else -1.0)
        assert np.signbit(c[0]) == (nan is not np.nan)
        comp.SetCoeffs(c)
        y = torch.linspace(-1.0, 1.0, 300, dtype=torch.float64, device="cuda")[None, :]
        x1 = torch.zeros(0, 300, dtype=torch.float64, device="cuda")
        try:
            out.append(comp.Inverse(x1, y, xtol=1e-8, ytol=1e-8, method=method).cpu().numpy().view(np.int64) & (2 ** 63 - 1))
        except Exception as e:  # noqa: BLE001
            out.append(type(e).__name__ + str(e))
    assert np.array_equal(out[0], out[1]) if isinstance(out[0], np.ndarray) else out[0] == out[1]
