"""Launch plans are kept per number of points: many sizes in turn (more than
are kept), sizes seen before, two streams, and a captured call replayed after
other sizes were used give what a fresh map gives."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(M, c):
    tm = M.CreateTriangular(3, 2, 2, M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis))
    tm.SetCoeffs(c)
    return tm


def _all(tm, x, sens):
    import torch
    n = x.shape[1]
    z = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")  # noqa: E731
    y, ld, cg, ig = z(2, n), z(n), z(tm.numCoeffs), z(3, n)
    tm.FusedForwardAdjointImpl(x, sens=sens, logdet_sens_scale=0.5, out_eval=y, out_logdet=ld, coeff_grad=cg,
                               input_grad=ig)
    return y, ld, cg, ig, tm.Evaluate(x), tm.LogDeterminant(x), tm.CoeffGrad(x, sens)


@pytest.mark.parametrize("sizes", [[1, 127, 128, 129, 1], list(range(1, 70)) + [1, 2, 69]])
def test_sizes_and_streams(gpu, sizes):
    import torch
    M = gpu
    r = np.random.default_rng(5)
    probe = M.CreateTriangular(3, 2, 2, M.MapOptions())
    c = r.normal(0.0, 0.1, probe.numCoeffs)
    tm = _map(M, c)
    side = torch.cuda.Stream()
    for k, n in enumerate(sizes):
        x = torch.as_tensor(r.standard_normal((3, n)), device="cuda")
        sens = torch.as_tensor(r.standard_normal((2, n)), device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(side if k % 2 else torch.cuda.current_stream()):
            got = _all(tm, x, sens)
        torch.cuda.synchronize()
        for a, b in zip(got, _all(_map(M, c), x, sens)):
            assert torch.equal(a, b)


@pytest.mark.parametrize("warm", [True])
def test_captured_call_survives_other_sizes(gpu, warm):
    import torch
    M = gpu
    r = np.random.default_rng(6)
    probe = M.CreateTriangular(3, 2, 2, M.MapOptions())
    c = r.normal(0.0, 0.1, probe.numCoeffs)
    tm = _map(M, c)
    x = torch.as_tensor(r.standard_normal((3, 200)), device="cuda")
    y = torch.zeros(2, 200, dtype=torch.float64, device="cuda")
    tm.EvaluateImpl(x, y)
    ref = y.clone()
    s = torch.cuda.Stream()
    tm.SetAsync(True)
    g = torch.cuda.CUDAGraph()
    torch.cuda.synchronize()
    with torch.cuda.graph(g, stream=s):
        tm.EvaluateImpl(x, y)
    for n in range(1, 120):
        tm.Evaluate(x[:, :n].contiguous())
    torch.cuda.synchronize()
    y.zero_()
    g.replay()
    torch.cuda.synchronize()
    assert torch.equal(y, ref)


@pytest.mark.parametrize("dout", [1, 2, 3])
def test_input_gradient_by_component_and_whole(gpu, dout):
    """Few points are cut by component, many by tile alone: the same gradients,
    to the few roundings of adding up the components in another place."""
    import torch
    M = gpu
    r = np.random.default_rng(8 + dout)
    tm = M.CreateTriangular(3, dout, 3, M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis))
    tm.SetCoeffs(r.normal(0.0, 0.1, tm.numCoeffs))
    big, n = 100_000, 300
    x = torch.as_tensor(r.standard_normal((3, big)), device="cuda")
    s = torch.as_tensor(r.standard_normal((dout, big)), device="cuda")
    xs, ss = x[:, :n].contiguous(), s[:, :n].contiguous()
    for few, many in ((tm.Gradient(xs, ss), tm.Gradient(x, s)), (tm.LogDeterminantInputGrad(xs), tm.LogDeterminantInputGrad(x))):
        many = many[:, :n]
        assert torch.all((few - many).abs() <= 1e-13 * torch.clamp(many.abs(), min=1e-2 * float(many.abs().max())))


def test_captured_input_gradient_survives_larger_calls(gpu):
    """An asynchronous input gradient owns no buffer that a later, larger call replaces."""
    import torch
    M = gpu
    r = np.random.default_rng(13)
    tm = M.CreateTriangular(3, 2, 2, M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis))
    tm.SetCoeffs(r.normal(0.0, 0.1, tm.numCoeffs))
    x = torch.as_tensor(r.standard_normal((3, 200)), device="cuda")
    s = torch.as_tensor(r.standard_normal((2, 200)), device="cuda")
    g = torch.zeros(3, 200, dtype=torch.float64, device="cuda")
    tm.GradientImpl(x, s, g)
    ref = g.clone()
    tm.SetAsync(True)
    graph, side = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.stream(side):
        tm.GradientImpl(x, s, g)
        torch.cuda.synchronize()
        with torch.cuda.graph(graph, stream=side):
            tm.GradientImpl(x, s, g)
    torch.cuda.synchronize()
    tm.SetAsync(False)
    for n in (400, 9000):
        tm.Gradient(torch.as_tensor(r.standard_normal((3, n)), device="cuda"),
                    torch.as_tensor(r.standard_normal((2, n)), device="cuda"))
    g.zero_()
    graph.replay()
    torch.cuda.synchronize()
    assert torch.all((g - ref).abs() <= 1e-13 * torch.clamp(ref.abs(), min=1e-2 * float(ref.abs().max())))


@pytest.mark.parametrize("pos", ["SoftPlus", "Exp"])
def test_integrals_have_no_common_bias(gpu, pos):
    """T = x_2 g(0.1 x_1): the relative errors of many points average to the
    rule's own (weights that sum to 2 + 5.6e-17) and the arithmetic's few 2^-58."""
    import torch
    M = gpu
    o = M.MapOptions(basisType=M.BasisTypes.HermiteFunctions if pos == "Exp" else M.BasisTypes.ProbabilistHermite,
                     posFuncType=getattr(M.PosFuncTypes, pos), quadType=M.QuadTypes.AdaptiveClenshawCurtis,
                     basisNorm=False)
    comp = M.CreateComponent(M.FixedMultiIndexSet.from_multis([[1, 1]]), o)
    comp.SetCoeffs(np.array([0.1]))
    r = np.random.default_rng(21)
    x = r.standard_normal((2, 200_000))
    got = comp.Evaluate(torch.as_tensor(x, device="cuda")).cpu().numpy().reshape(-1).astype(np.longdouble)
    f = np.longdouble(0.1) * x[0].astype(np.longdouble)
    want = x[1].astype(np.longdouble) * (np.exp(f) if pos == "Exp" else np.log1p(np.exp(f)))
    assert abs(float((got / want - 1).mean())) <= 4e-17
