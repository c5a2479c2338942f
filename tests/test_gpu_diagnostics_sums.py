"""The sums of wdm_reduce and wdm_diagnostics against the FP64 oracle on the psi and
Phi that the library returns, over the edges of the reduction's tiles: rows shorter
than a warp and ragged in it, marches of every length, seams between marches, items.

Tolerances: mass, centre of mass and R are sums of exact squares or of FP32 products
of relative error 2^-23 (weights times coordinates), carried to about 2^-44, and R is
FP64: 1e-9 for mass and R, 1e-6 of the box for the centre.  W, K and Q sum FP32 terms of
about eight roundings each (8 x 2^-24 = 5e-7 of a term's parts; a difference of
neighbours of size |psi| over 2 dx adds 2^-24 |psi| / dx): 2e-6 of the sums of the
terms' magnitudes, which for Q and K are taken with the differences' parts.
"""
import numpy as np
import pytest

from oracle import spe

pytestmark = pytest.mark.gpu

SHAPES = [(8, 8, 8), (12, 16, 48), (48, 8, 12), (96, 24, 32), (64, 64, 64), (128, 48, 64), (32, 12, 192), (192, 8, 24)]


def _magnitudes(psi, phi, g):
    """Sums of |terms| of W, K and Q with every difference replaced by the size of its parts."""
    amp = np.abs(psi)
    i = slice(1, -1)

    def parts(f, axis):
        lo, hi = [i, i, i], [i, i, i]
        lo[axis], hi[axis] = slice(None, -2), slice(2, None)
        return (f[tuple(hi)] + f[tuple(lo)]) / (2 * g.spacing[2 - axis])

    return np.sum(amp[i, i, i] ** 2 * np.abs(phi[i, i, i])), np.sum(sum(parts(amp, a) ** 2 for a in range(3)))


@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("batch", [1, 3])
def test_sums_match_the_oracle(wdm, n, batch):
    g = spe.Grid(n, tuple(0.2 * m for m in n))
    X, Y, Z = g.coords()
    rng = np.random.default_rng(sum(n))
    items = []
    for b in range(batch):
        r2 = (X - 0.1 * g.L[0]) ** 2 + Y ** 2 + (Z + 0.15 * g.L[2]) ** 2
        amp = np.exp(-r2 / (0.3 * g.L[0]) ** 2) + 0.05 * rng.random(r2.shape)
        items.append((amp * np.exp(2j * np.pi * (X / g.L[0] + 2 * Z / g.L[2]))).astype(np.complex64))
    with wdm.SPEContext(n, g.L, poisson_coeff=1.0, batch=batch) as ctx:
        ctx.set_psi(np.stack(items) if batch > 1 else items[0])
        diag, red = ctx.diagnostics(), ctx.reduce()
        psi = ctx.get_psi().reshape((batch,) + n[::-1]).astype(np.complex128)
        phi = ctx.get_phi().reshape((batch,) + n[::-1]).astype(np.float64)
    diag, red = (diag, red) if batch > 1 else ([diag], [red])
    for b in range(batch):
        mag_w, mag_g = _magnitudes(psi[b], phi[b], g)
        rho = np.abs(psi[b]) ** 2
        terms = spe.virial_terms(psi[b], phi[b], g)
        ref = spe.loop_diagnostics(psi[b], phi[b], g, kappa=0.0)
        com = [np.sum(rho * c) / np.sum(rho) for c in (X, Y, Z)]
        assert diag[b]["R"] == pytest.approx(ref["R"], rel=1e-9)
        for d in (diag[b], red[b]):
            assert d["mass"] == pytest.approx(spe.mass(psi[b], g), rel=1e-9)
            for a in range(3):
                assert abs(d["com_" + "xyz"[a]] - com[a]) <= 1e-6 * g.L[a]
            for k, mag in (("VirialPotential", mag_w), ("TotalKineticE", mag_g), ("TotalQuantumE", mag_g)):
                assert abs(d[k] - terms[k]) <= 2e-6 * 0.5 * mag * g.dV, k
            assert d["Virial"] == pytest.approx(2 * d["TotalKineticE"] + 2 * d["TotalQuantumE"] - d["VirialPotential"],
                                                rel=1e-12)
