"""Diagnostics of a state whose density leaves FP32's range: |psi|^2 of finite psi
overflows.  The maximum is then infinite and reported as such, at its first cell, and
the radii, whose weights are FP64 sums, are taken about that cell."""
import numpy as np
import pytest

from oracle import spe

pytestmark = pytest.mark.gpu


# first and last lanes and tiles of the reduction's rows, first, inner and last cells of its marches
CELLS = [(0, 0, 0), (31, 5, 3), (32, 0, 4), (40, 23, 31), (63, 11, 30), (63, 23, 47), (17, 8, 28)]


@pytest.mark.parametrize("cells", [[c] for c in CELLS] + [CELLS[2:5]], ids=str)
def test_an_overflowing_density_is_the_maximum(wdm, cells):
    n = (64, 24, 48)
    g = spe.Grid(n, tuple(0.2 * m for m in n))
    rng = np.random.default_rng(5)
    psi = (1 + 0.3 * rng.standard_normal(n[::-1]) + 0.3j * rng.standard_normal(n[::-1])).astype(np.complex64)
    for x, y, z in cells:
        psi[z, y, x] = 2e19 + 1e19j  # |psi|^2 = 5e38
    first = min((z * n[1] + y) * n[0] + x for x, y, z in cells)
    with wdm.SPEContext(n, g.L, poisson_coeff=0.0) as ctx:
        ctx.set_psi(psi)
        d, r = ctx.diagnostics(), ctx.reduce()
    assert d["rho_max"] == r["rho_max"] == np.inf and d["psi_abs_max"] == np.inf
    assert d["argmax"] == r["argmax"] == first
    # FP64: the radii about the first of the cells, its weight far above all others
    rho = np.abs(psi.astype(np.complex128)) ** 2
    ref = spe.loop_diagnostics(psi.astype(np.complex128), np.zeros(n[::-1]), g, kappa=0.0)
    if len(cells) == 1:
        assert ref["argmax"] == first and rho.flat[first] > np.finfo(np.float32).max
        radii = [d[f"radius_{k}0"] for k in range(1, 10)]
        assert np.allclose(radii, ref["radii"], rtol=1e-9, atol=0)
