"""The two-factor line transforms (y and z passes) of every supported length,
through both line-pass kernels, against the FP64 transform: forward and
inverse, and the fused forward / operator / inverse pass as a drift."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SIZES = (8, 12, 16, 24, 32, 48, 64, 96, 128, 192, 256, 384, 512)
# A two-factor FP32 transform rounds about a dozen times per point along the
# way (two register transforms, one twiddle); at 6e-8 per rounding, added in
# quadrature over the three axes and doubled for a forward and inverse pair,
# that is 5e-7.  The bound is four times it.
TOL = 2e-6


@pytest.fixture(scope="module")
def wdm():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import wavedm_gb300

    return wavedm_gb300


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


@pytest.mark.parametrize("impl", ["tma", "tile"])
@pytest.mark.parametrize("n", SIZES)
def test_line_transforms_match_fp64(wdm, monkeypatch, n, impl):
    import torch

    monkeypatch.setenv("WDM_LINE_IMPL", impl)
    rng = np.random.default_rng(n)
    # the length along y, then along z; a width that leaves a part tile where 16 does not divide it
    for shape in ((24, n, 8), (24, 12, n)):
        x = (rng.standard_normal(shape[::-1]) + 1j * rng.standard_normal(shape[::-1])).astype(np.complex64)
        x128 = x.astype(np.complex128)
        with wdm.SPEContext(shape, (3.0, 2.0, 4.0)) as ctx:
            got = ctx.fft3d(torch.from_numpy(x).cuda()).cpu().numpy()
            assert _rel(got, np.fft.fftn(x128)) < TOL
            got = ctx.fft3d(torch.from_numpy(x).cuda(), inverse=True).cpu().numpy()
            assert _rel(got, np.fft.ifftn(x128) * x.size) < TOL
            ctx.set_psi(x)
            ctx.drift(0.01)
            got = ctx.get_psi()
        k = [2 * np.pi * np.fft.fftfreq(m, 1.0 / m) / L for m, L in zip(shape, (3.0, 2.0, 4.0))]
        k2 = k[0][None, None, :] ** 2 + k[1][None, :, None] ** 2 + k[2][:, None, None] ** 2
        ref = np.fft.ifftn(np.fft.fftn(x128) * np.exp(-0.005j * k2))
        assert _rel(got, ref) < TOL
