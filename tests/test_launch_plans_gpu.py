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
