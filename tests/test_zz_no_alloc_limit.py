"""The no-allocation entry point near the end of its 64 MiB: a call whose tables
and partial sums fit is run, whether or not the fixed-point coefficients find
room beside them."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_call_that_leaves_no_room_for_limbs(gpu):
    import torch

    from mpart_gb300 import _capi, _mat, _ptr, _stream_of
    M = gpu
    comp = M.CreateComponent(M.FixedMultiIndexSet(15, 5), M.MapOptions(quadType=M.QuadTypes.AdaptiveClenshawCurtis))
    terms = comp.numCoeffs
    comp.SetCoeffs(np.random.default_rng(0).normal(0.0, 0.01, terms))
    # 128-point tiles, a row of partial sums each; the other tables take between
    # 48 and 64 bytes a tile and a few hundred
    limit, tiles = 64 << 20, 539
    assert 8 * terms * (tiles + 1) + 64 * tiles + 4096 <= limit < 8 * terms * (tiles + 2) + 48 * tiles
    n = 128 * tiles
    x = torch.randn(15, n, dtype=torch.float64, device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    sens = torch.ones(1, n, dtype=torch.float64, device="cuda")
    z = lambda *s: torch.zeros(*s, dtype=torch.float64, device="cuda")  # noqa: E731
    ev0, ld0, cg0, ev, ld, cg = z(1, n), z(n), z(terms), z(1, n), z(n), z(terms)
    comp.FusedForwardAdjointImpl(x, sens=sens, logdet_sens_scale=1.0, out_eval=ev0, out_logdet=ld0, coeff_grad=cg0)
    _capi.check(_capi.load().mpgb_fused_fwd_adj_noalloc(comp._h, _mat(x), _mat(sens), _mat(None), 1.0, _mat(ev), _mat(ld),
                                                        _ptr(cg), _stream_of(x)))
    torch.cuda.synchronize()
    for a, b, floor in ((ev, ev0, 1e-6), (ld, ld0, 1e-6), (cg, cg0, 1e-3)):
        assert torch.all((a - b).abs() <= 1e-10 * torch.clamp(b.abs(), min=floor * float(b.abs().max())))
