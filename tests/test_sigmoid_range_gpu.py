"""The rectifier of sigmoid expansions on both sides of the fixed-point range
(|Phi| = 31): a linear leading function of large inputs, against the oracle at
the GPU tests' parity bar (1e-10 relative, floor 1e-6 of the largest entry)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("pos", ["softplus", "exp"])
@pytest.mark.parametrize("n", [1, 129])
def test_rectifier_range(gpu, oracle, pos, n):
    import torch

    import __graft_entry__ as G
    M = gpu
    opts = M.MapOptions(basisType=M.BasisTypes.HermiteFunctions, sigmoidBasisSumType=M.SigmoidSumSizeType.Constant,
                        posFuncType=M.PosFuncTypes.Exp if pos == "exp" else M.PosFuncTypes.SoftPlus)
    comp = M.CreateSigmoidComponent(2, 2, np.array([-3.0, 3.0, -1.0, 0.5, 1.5]), opts)
    r = np.random.default_rng(n)
    lb, _ = comp.CoeffBounds()
    c = np.where(lb == 0.0, 0.2, 0.05)
    comp.SetCoeffs(c)
    x = r.standard_normal((2, n))
    x[0] = r.uniform(-60.0, 60.0, n)
    x[0, 0] = np.nextafter(31.0, 0.0)
    if n > 3:
        x[0, 1:4] = 31.0, -31.0, -0.0
    s, d, o = G._sigmoid_mset(comp)
    ref = oracle.OracleSigmoidComponent(2, s, d, o, comp.GetSigmoid(),
                                        oracle.POS_EXP if pos == "exp" else oracle.POS_SOFTPLUS).evaluate(c, x)
    y = comp.Evaluate(torch.as_tensor(x, device="cuda")).cpu().numpy()
    ref = np.asarray(ref).reshape(y.shape)
    assert np.all(np.abs(y - ref) <= 1e-10 * np.maximum(np.abs(ref), 1e-6 * np.max(np.abs(ref))))
