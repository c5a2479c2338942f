"""The plane passes (y transforms inside the kick and the density pass, one CTA
per z plane) against the separate passes (WDM_PLANES=off), over row and column
lengths at the edges of their range, and their bookkeeping of the potential
(kept y-spectral between calls)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# Both paths do the same transforms with the same twiddles on the same values;
# only the compiler's freedom to contract the pointwise terms could differ, a
# few roundings of 6e-8 per point over the three steps.
TOL = 1e-6


@pytest.fixture(scope="module")
def wdm():
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    import wavedm_gb300

    return wavedm_gb300


def _psi(shape, seed):
    rng = np.random.default_rng(seed)
    return (1.0 + 0.2 * rng.standard_normal(shape) + 0.2j * rng.standard_normal(shape)).astype(np.complex64)


def _rel(a, b):
    return float(np.linalg.norm(a - b) / np.linalg.norm(b))


def _run(wdm, n, batch, mode, phase, everything):
    L = (4.0, 3.0, 5.0)
    shape = ((batch,) if batch > 1 else ()) + n[::-1]
    opts = dict(kerr=0.3, absorb_alpha=0.5) if everything else {}
    with wdm.SPEContext(n, L, poisson_coeff=2.0, phase_mode=phase, batch=batch, **opts) as ctx:
        ctx.set_psi(_psi(shape, sum(n)))
        if everything:
            ctx.set_tidal([[0.3, -0.1, -0.2, 0.05, 0.0, 0.02]])
            ctx.set_tidal_centering("density_max")
            ctx.set_static_potential(np.linspace(0, 1, int(np.prod(shape)), dtype=np.float32).reshape(shape))
            if batch == 1:
                ctx.set_particles(np.array([[0.1, 0.2, 0.3], [-1.0, 0.7, -0.4]]), [0.2, 0.1])
        ctx.step(3, 0.01, mode=mode)
        phi = ctx.get_phi()
        ctx.kick(0.01)
        ctx.drift(0.01)
        ctx.step(1, 0.01, mode=mode)
        return ctx.get_psi(), phi


# shortest rows and columns, columns that do not fill a warp's row pairs, the
# longest columns that fit, planes more than SMs, several items; the last two
# are just past the rule's limits
CASES = [((8, 8, 8), 1), ((8, 256, 8), 1), ((12, 24, 8), 1), ((16, 12, 8), 2), ((24, 48, 8), 1), ((32, 32, 32), 4),
         ((48, 16, 12), 1), ((48, 256, 8), 1), ((64, 64, 8), 1), ((64, 192, 8), 1), ((96, 96, 96), 2),
         ((96, 128, 8), 1), ((128, 128, 8), 1), ((128, 8, 16), 1), ((64, 256, 8), 1), ((192, 96, 8), 1)]


@pytest.mark.parametrize("mode,phase,everything", [("strang", "precise", False), ("reference_loop", "plain", True)])
@pytest.mark.parametrize("n,batch", CASES, ids=[f"{'x'.join(map(str, n))}-b{b}" for n, b in CASES])
def test_plane_passes_equal_the_separate_passes(wdm, monkeypatch, n, batch, mode, phase, everything):
    monkeypatch.setenv("WDM_PLANES", "off")
    psi0, phi0 = _run(wdm, n, batch, mode, phase, everything)
    monkeypatch.delenv("WDM_PLANES")
    psi1, phi1 = _run(wdm, n, batch, mode, phase, everything)
    assert _rel(psi1, psi0) < TOL
    assert _rel(phi1, phi0) < TOL


def test_potential_reads_between_replays_leave_the_state(wdm):
    n = (48, 32, 24)
    x = _psi(n[::-1], 3)
    with wdm.SPEContext(n, (4.0, 3.0, 5.0)) as ctx:
        ctx.set_psi(x)
        ctx.step_graph(2, 0.01)
        ctx.get_phi()
        ctx.step_graph(2, 0.01)
        got = ctx.get_psi()
        ctx.set_psi(x)
        ctx.step_graph(2, 0.01)
        ctx.step_graph(2, 0.01)
        assert np.array_equal(got, ctx.get_psi())
        # an adjoint leaves the potential as rows; replays start from there as well
        ctx.set_psi(x)
        ctx.adjoint(2, 0.01, np.ones(n[::-1], np.float32))
        ctx.step_graph(2, 0.01)
        ctx.step_graph(2, 0.01)
        assert _rel(ctx.get_psi(), got) < TOL
