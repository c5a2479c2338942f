"""The plain line passes of 384 and 512 points keep two tile slots per CTA: grids with
more tiles than resident CTAs, so that both slots are used more than once, along y and
z, forward and inverse, with the half spectrum's edge tiles (Poisson), against the
register-tile passes (the same arithmetic: the same bits) and the FP64 transform."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

TOL = 2e-6  # of test_gpu_line_factors.py: four times a dozen roundings per point in quadrature


@pytest.mark.parametrize("n", [(64, 384, 192), (64, 192, 384), (48, 512, 128), (48, 128, 512)])
def test_two_slots_over_many_tiles(wdm, monkeypatch, n):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    L = (3.0, 2.0, 4.0)
    g = torch.Generator("cuda").manual_seed(n[1])
    x = torch.randn(n[::-1], dtype=torch.complex64, device="cuda", generator=g)
    rho = x.real.contiguous()
    torch.cuda.synchronize()
    got = {}
    for impl in ("tma", "tile"):
        monkeypatch.setenv("WDM_LINE_IMPL", impl)
        with wdm.SPEContext(n, L) as ctx:
            a, b, out = x.clone(), x.clone(), torch.empty_like(rho)
            torch.cuda.synchronize()
            got[impl] = (ctx.fft3d(a), ctx.fft3d(b, inverse=True), ctx.poisson(rho, out))
    for p, q in zip(got["tma"], got["tile"]):
        assert torch.equal(p, q)
    x128 = x.cpu().numpy().astype(np.complex128)
    for p, want in zip(got["tma"], (np.fft.fftn(x128), np.fft.ifftn(x128) * x128.size)):
        assert np.linalg.norm(p.cpu().numpy() - want) < TOL * np.linalg.norm(want)
