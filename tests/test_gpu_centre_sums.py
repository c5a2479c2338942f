"""The density maximum and moments for a tide centred on the halo, over batches whose
items meet inside a warp and inside a CTA, with several units per warp, and the plane
passes: every item against the FP64 oracle, which centres it by its own density.

The tide dominates the phase here, so an item that took part of another's sums or lost
part of its own is off by much more than the tolerance of a short FP32 run (2e-5)."""
import numpy as np
import pytest

from oracle import spe

pytestmark = pytest.mark.gpu

T6 = [0.8, -0.3, -0.5, 0.1, 0.05, -0.1]
# rows: pairs of an item that do not fill a warp's unit (12: 16 pairs a unit), one unit
# per item and many units per warp; planes: one item per CTA; the persistent kernel,
# whose CTAs go on
CASES = [((12, 12, 12), 5, "rows"), ((8, 8, 8), 9, "rows"), ((64, 24, 16), 3, "rows"), ((192, 12, 8), 3, "rows"),
         ((8, 384, 24), 2, "rows"), ((64, 256, 96), 1, "rows"), ((12, 12, 12), 5, "planes"), ((48, 32, 16), 2, "planes"),
         ((16, 16, 16), 5, "persistent"), ((64, 24, 16), 3, "persistent")]


def _halo(n, L, b):
    """A soliton-like blob off the centre, elsewhere for every item."""
    g = spe.Grid(n, L)
    X, Y, Z = g.coords()
    off = [0.17 * l * np.cos(1.7 * b + q) for q, l in enumerate(L)]
    r2 = sum(((x - o) / (0.2 * l)) ** 2 for x, o, l in zip((X, Y, Z), off, L))
    return ((1 + b) * np.exp(-r2 / 2) + 0.05 + 0.02j * np.sin(2 * np.pi * X / L[0])).astype(np.complex64)


@pytest.mark.parametrize("mode", ["reference", "density_max"])
@pytest.mark.parametrize("n,batch,kernels", CASES, ids=[f"{'x'.join(map(str, n))}-b{b}-{p}" for n, b, p in CASES])
def test_items_are_centred_by_their_own_density(wdm, monkeypatch, n, batch, kernels, mode):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    if kernels == "rows":
        monkeypatch.setenv("WDM_PLANES", "off")
    if kernels == "persistent":
        monkeypatch.setenv("WDM_GROUP_SCHEDULE", "persistent")
    L, dt, steps = (4.0, 3.0, 5.0), 0.02, 2
    psi0 = np.stack([_halo(n, L, b) for b in range(batch)])
    with wdm.SPEContext(n, L, batch=batch) as ctx:
        ctx.set_psi(psi0 if batch > 1 else psi0[0])
        ctx.set_tidal([T6])
        ctx.set_tidal_centering(mode)
        (ctx.step_graph if kernels == "persistent" else ctx.step)(steps, dt)
        got = ctx.get_psi().reshape(psi0.shape)
    phys = spe.Physics(tidal=lambda t: tuple(T6), tidal_centering=mode)
    for b in range(batch):
        want = spe.run(psi0[b].astype(np.complex128), spe.Grid(n, L), phys, dt, steps)
        assert spe.rel_l2(got[b], want) < 2e-5, b
