"""Launch tables of sizes that vary: a call at a new size does not make the host
wait, nor other streams or a capture on another thread fail; a sequence of ever
new sizes, and components one by one, give what a fresh map gives."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _map(M, dim=2, order=2, seed=3):
    tm = M.CreateTriangular(dim, dim, order, M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis))
    tm.SetCoeffs(np.random.default_rng(seed).normal(0.0, 0.1, tm.numCoeffs))
    return tm


def _points(dim, n, seed=1):
    import torch
    return torch.as_tensor(np.random.default_rng(seed).standard_normal((dim, n)), device="cuda")


def test_new_size_does_not_wait(gpu):
    """An asynchronous call at a size not seen before returns while earlier work
    of its stream is still running."""
    import torch
    tm = _map(gpu)
    x = _points(2, 4000)
    y = torch.zeros(2, 4000, dtype=torch.float64, device="cuda")
    tm.EvaluateImpl(x, y)
    a = torch.randn(8192, 8192, device="cuda")
    b = a @ a
    tm.SetAsync(True)
    waited = []
    for n in (100, 300, 500, 700, 900):  # (several: the first may load modules)
        torch.cuda.synchronize()
        for _ in range(8):
            torch.mm(a, a, out=b)
        done = torch.cuda.Event()
        done.record()
        tm.EvaluateImpl(x[:, :n], y[:, :n])
        waited.append(done.query())
    torch.cuda.synchronize()
    assert not all(waited)


def test_many_sizes_beside_a_capture(gpu):
    """More sizes than are kept while another thread captures in the global mode."""
    import torch
    tm = _map(gpu)
    x = _points(2, 4000)
    for n in range(1, 70):
        tm.Evaluate(x[:, :n].contiguous())
    xs = [x[:, :n].contiguous() for n in range(70, 140)]
    y = torch.zeros(2, 4000, dtype=torch.float64, device="cuda")
    z = torch.zeros(4000, device="cuda")
    tm.SetAsync(True)
    go, end, err = threading.Event(), threading.Event(), []

    def capture():
        try:
            g = torch.cuda.CUDAGraph()
            s = torch.cuda.Stream()
            with torch.cuda.stream(s):
                z.add_(1.0)
                s.synchronize()
                g.capture_begin(capture_error_mode="global")
                try:
                    z.add_(1.0)
                    go.set()
                    end.wait(30)
                finally:
                    g.capture_end()
        except Exception as e:  # noqa: BLE001
            err.append(e)
        finally:
            go.set()

    torch.cuda.synchronize()
    t = threading.Thread(target=capture)
    t.start()
    go.wait(30)
    try:
        for k, n in enumerate(range(70, 140)):
            tm.EvaluateImpl(xs[k], y[:, :n])
    except Exception as e:  # noqa: BLE001
        err.append(e)
    end.set()
    t.join(60)
    assert not err
    torch.cuda.synchronize()
    assert torch.equal(y[:, :139], _map(gpu).Evaluate(xs[-1]))


def test_sizes_in_turn_on_two_streams(gpu):
    """More sizes than are kept, asynchronously on two streams that are ordered
    with one another."""
    import torch
    tm = _map(gpu, 3, 3)
    x = _points(3, 2000)
    sizes = [int(n) for n in np.random.default_rng(0).integers(1, 2000, 60)]
    out = [torch.zeros(3, n, dtype=torch.float64, device="cuda") for n in sizes]
    ref = [_map(gpu, 3, 3).Evaluate(x[:, :n].contiguous()) for n in sizes]
    xs = [x[:, :n].contiguous() for n in sizes]
    torch.cuda.synchronize()
    tm.SetAsync(True)
    st = [torch.cuda.Stream(), torch.cuda.Stream()]
    for k in range(len(sizes)):
        st[k % 2].wait_stream(st[1 - k % 2])
        with torch.cuda.stream(st[k % 2]):
            tm.EvaluateImpl(xs[k], out[k])
    torch.cuda.synchronize()
    for a, b in zip(out, ref):
        assert torch.equal(a, b)


@pytest.mark.parametrize("dim,n", [(52, 40), (3, 257), (1, 5)])
def test_implicit_gradient_of_many_components(gpu, dim, n):
    """All components' tables in one set: twice the same, and equal to the dense
    gradients' sum (w dT of each component, solved from the last to the first)."""
    import torch
    M = gpu
    tm = _map(M, dim, 1 if dim > 10 else 3)
    x = _points(dim, n)
    w = _points(dim, n, 5)
    x1 = torch.zeros(0, n, dtype=torch.float64, device="cuda")
    a = tm.InverseCoeffGrad(x1, x, w)
    b = tm.InverseCoeffGrad(x1, x, w)
    for p, q in zip(a, b):
        assert torch.equal(p, q)
    # lambda = (d T / d x)^-T w; grad = -sum_p dT/dc lambda
    J = torch.zeros(n, dim, dim, dtype=torch.float64, device="cuda")
    for i in range(dim):
        c = tm.GetComponent(i)
        J[:, i, :i + 1] = c.Gradient(x[:i + 1].contiguous(), torch.ones(1, n, dtype=torch.float64, device="cuda")).T
        # (Gradient differentiates the quadrature; the implicit gradient takes g(d_D f))
        J[:, i, i] = torch.exp(c.LogDeterminant(x[:i + 1].contiguous()))
    lam = torch.linalg.solve(J.transpose(1, 2), w.T[:, :, None])[:, :, 0].T.contiguous()
    g = -tm.CoeffGrad(x, lam).sum(1)
    assert torch.all((a[0] - g).abs() <= 1e-10 * torch.clamp(g.abs(), min=1e-3 * float(g.abs().max())))


def test_more_streams_than_are_followed(gpu):
    """One map on more streams in turn than a set keeps events for."""
    import torch
    tm = _map(gpu)
    x = _points(2, 500)
    xs = [x[:, :n].contiguous() for n in range(100, 140)]
    ref = [_map(gpu).Evaluate(a) for a in xs]
    streams = [torch.cuda.Stream() for _ in range(24)]
    out = [torch.zeros(2, a.shape[1], dtype=torch.float64, device="cuda") for a in xs]
    torch.cuda.synchronize()
    tm.SetAsync(True)
    last = torch.cuda.current_stream()
    for k in range(200):
        s = streams[k % 24]
        s.wait_stream(last)
        with torch.cuda.stream(s):
            tm.EvaluateImpl(xs[k % 40], out[k % 40])
        last = s
    torch.cuda.synchronize()
    for a, b in zip(out, ref):
        assert torch.equal(a, b)
