"""Passes whose launches overlap (each waits for the one in front on the device)
give the bits of passes run one by one: a run in one call, the same run as a graph,
and step by step with the device idle in between, on grids at both sides of the
size up to which a pass lets the next one in early, with line passes of both kinds
and with a memset and a kernel of the plain kind between the passes (tide frame)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# 4096 lines of 8 threads a line is the last grid that lets the next one in early:
# 64^3, and one column of tiles more; then row passes instead of planes, long lines
CASES = [(8, 8, 8), (32, 32, 32), (48, 48, 48), (64, 64, 64), (64, 96, 64), (96, 64, 48), (192, 24, 48),
         (32, 16, 512), (256, 64, 16)]


@pytest.mark.parametrize("tide", [False, True], ids=["plain", "tide-frame"])
@pytest.mark.parametrize("impl", ["tma", "tile"])
@pytest.mark.parametrize("n", CASES, ids=lambda n: "x".join(map(str, n)))
def test_overlapping_launches_match_single_passes(wdm, monkeypatch, n, impl, tide):
    monkeypatch.setenv("WDM_LINE_IMPL", impl)
    rng = np.random.default_rng(sum(n))
    psi = (1.0 + 0.2 * rng.standard_normal(n[::-1]) + 0.2j * rng.standard_normal(n[::-1])).astype(np.complex64)
    out = []
    with wdm.SPEContext(n, (4.0, 3.0, 5.0), poisson_coeff=2.0, kerr=0.2, absorb_alpha=0.3) as ctx:
        if tide:
            ctx.set_tidal([[0.3, -0.1, -0.2, 0.05, 0.0, 0.02]] * 32)
            ctx.set_tidal_centering("density_max")
        for how in ("single", "call", "graph", "graph", "call"):
            ctx.set_psi(psi)
            if how == "single":
                for _ in range(12):
                    ctx.step(1, 0.01, mode="reference_loop")
                    ctx.get_psi()
            elif how == "call":
                ctx.step(12, 0.01, mode="reference_loop")
            else:
                ctx.step_graph(12, 0.01, mode="reference_loop")
            out.append(ctx.get_psi())
    for o in out[1:]:
        assert np.array_equal(o, out[0])
