"""The fixed-point Inverse: roots found by the queue launch, by the warp pass
(quadratures of many intervals: a tight tolerance, forced subdivision) and by
the small-call path are the same to the bit, and take Evaluate back to the
target within the solver's own tolerance: |T(x) - r| <= ytol + slope xtol, twice
that for the rounding of T."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("method", ["Bracket", "Newton"])
@pytest.mark.parametrize("basis,pos,order,dim,tol,min_sub,n", [
    ("ph", "softplus", 1, 2, 1e-6, 0, 257), ("ph", "softplus", 3, 3, 1e-13, 0, 300), ("ph", "exp", 2, 2, 1e-8, 0, 511),
    ("hf", "softplus", 4, 2, 1e-8, 7, 256), ("hf", "exp", 3, 3, 1e-12, 0, 300), ("ph", "softplus", 6, 2, 1e-6, 0, 300)])
def test_paths_agree(gpu, method, basis, pos, order, dim, tol, min_sub, n):
    import torch
    M = gpu
    r = np.random.default_rng(order * 10 + dim)
    tm = M.CreateTriangular(dim, dim, order, M.MapOptions(
        quadType=M.QuadTypes.AdaptiveClenshawCurtis, quadAbsTol=tol, quadRelTol=tol, quadMinSub=min_sub,
        basisType=M.BasisTypes.HermiteFunctions if basis == "hf" else M.BasisTypes.ProbabilistHermite,
        posFuncType=M.PosFuncTypes.Exp if pos == "exp" else M.PosFuncTypes.SoftPlus))
    tm.SetCoeffs(r.normal(0.0, 0.05, tm.numCoeffs))
    x = torch.as_tensor(r.standard_normal((dim, n)), device="cuda")
    y = tm.Evaluate(x)
    x1 = torch.zeros(0, n, dtype=torch.float64, device="cuda")
    kw = {"xtol": 1e-10, "ytol": 1e-10, "method": method}
    a = tm.Inverse(x1, y, **kw)
    b = torch.cat([tm.Inverse(x1[:, k:k + 100], y[:, k:k + 100].contiguous(), **kw) for k in range(0, n, 100)], dim=1)
    assert torch.equal(a, b)
    slope = torch.exp(torch.stack([tm.GetComponent(i).LogDeterminant(a[:i + 1].contiguous()) for i in range(dim)]))
    assert torch.all((tm.Evaluate(a) - y).abs() <= 2.0 * (1e-10 + slope * 1e-10) + 1e-12)
