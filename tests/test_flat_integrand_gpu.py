"""Adjoint integrals of a SoftPlus map that is nearly flat: d_D f falls from -4
on the way to x_D.  J_k against the FP64 quadrature (quadMaxSub = 32 is outside
the fixed-point rule), relative to the integral of its integrand's magnitude:
1e-14, some thirty intervals of a few roundings each, plus one rounding of
phit_k(0), which the gradient adds (He_2(0) = -1, He_4(0) = 3, He_6(0) = -15,
psi_0(0) = pi^(-1/4))."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("basis", ["ProbabilistHermite", "HermiteFunctions"])
@pytest.mark.parametrize("slope", [1.0, 4.0, 8.0])
def test_falling_derivative(gpu, basis, slope):
    import torch
    M = gpu
    x = torch.as_tensor(np.linspace(0.5, 3.0, 200)[None, :], device="cuda")
    one = torch.ones(1, 200, dtype=torch.float64, device="cuda")
    out = []
    for max_sub in (30, 32):
        comp = M.CreateComponent(M.FixedMultiIndexSet(1, 6), M.MapOptions(
            basisType=getattr(M.BasisTypes, basis), quadType=M.QuadTypes.AdaptiveClenshawCurtis, quadAbsTol=1e-12,
            quadRelTol=1e-12, quadMaxSub=max_sub, basisNorm=False))
        c = np.zeros(comp.numCoeffs)
        # d_D f = -4 - slope y (ProbabilistHermite: He_1' = 1, He_2' = 2 y;
        # Hermite functions: phit_1' = 1 alone, and psi_0' = -pi^(-1/4) y exp(-y^2 / 2))
        c[1] = -3.99
        c[2] = -0.5 * slope if basis == "ProbabilistHermite" else slope * np.pi ** 0.25
        comp.SetCoeffs(c)
        out.append(comp.CoeffGrad(x, one).cpu().numpy())
    y = np.linspace(0.0, 3.0, 3001)
    if basis == "ProbabilistHermite":
        d = -3.99 - slope * y
        he = [np.ones_like(y), y]
        for k in range(2, 6):
            he.append(y * he[-1] - (k - 1) * he[-2])
        u, v0 = [(k + 1) * he[k] for k in range(6)], [0.0, 1.0, 0.0, 3.0, 0.0, 15.0]
    else:  # (orders 1 and 2: the others' scales are those of psi_j)
        d = -3.99 - slope * y * np.exp(-0.5 * y * y)
        u, v0 = [np.ones_like(y), np.pi ** -0.25 * y * np.exp(-0.5 * y * y)], [0.0, np.pi ** -0.25]
    for k in range(1, len(u) + 1):
        size = np.concatenate([[0.0], np.cumsum(np.abs(u[k - 1] / (1.0 + np.exp(-d)))[1:] * 1e-3)])
        size = np.interp(x.cpu().numpy()[0], y, size)
        assert np.all(np.abs(out[0][k] - out[1][k]) <= 1e-14 * size + 2.0 ** -52 * v0[k - 1]), k
