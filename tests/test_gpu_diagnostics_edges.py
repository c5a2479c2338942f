"""wdm_diagnostics at the edges of its kernels' ranges, against the FP64 oracle on
the psi and Phi that the library returns.

The reduction takes 32 neighbouring x of a row and marches along z: rows shorter
than a warp, ragged last warps, marches of every length.  The radii take eight
mirrored cells about the density maximum and sum keys in blocks of 1024: a maximum
in a corner, on a face and inside, one cell with weight, shells with empty blocks
of keys between them.

Tolerances: maxima and indices exact up to the rounding of the FP64 output; radii
and R are FP64 sums of at most 10^6 terms (1e-9 leaves a factor of ten over 10^6
eps); momenta, W, K and Q sum FP32 terms of about eight roundings each (8 x 2^-24 =
5e-7, 2e-6 with the cancellation of the differences; relative to the sum of the
terms' magnitudes).
"""
import numpy as np
import pytest

from oracle import spe

pytestmark = pytest.mark.gpu


def _check(ctx, g, n, batch):
    got = ctx.diagnostics()
    red = ctx.reduce()
    psi = ctx.get_psi().reshape((batch,) + n[::-1])
    phi = ctx.get_phi().reshape((batch,) + n[::-1])
    got, red = (got, red) if batch > 1 else ([got], [red])
    for b in range(batch):
        ref = spe.loop_diagnostics(psi[b].astype(np.complex128), phi[b].astype(np.float64), g, kappa=0.0)
        d = got[b]
        assert int(d["argmax"]) == ref["argmax"]
        for k in ("rho_max", "psi_abs_max", "phi_abs_max"):
            assert d[k] == pytest.approx(ref[k], rel=1e-12)
        scale = max(abs(ref[f"Momentum{a}"]) for a in "XYZ")
        for a in "XYZ":
            assert abs(d[f"Momentum{a}"] - ref[f"Momentum{a}"]) <= 2e-6 * (scale + abs(d["mass"]))
        assert np.allclose([d[f"radius_{k}0"] for k in range(1, 10)], ref["radii"], rtol=1e-9, atol=0, equal_nan=True)
        for k, v in red[b].items():
            assert d[k] == pytest.approx(v, rel=1e-12)


@pytest.mark.parametrize("n", [(8, 8, 8), (12, 16, 48), (48, 8, 12), (96, 24, 32), (64, 64, 64), (128, 48, 64)], ids=str)
@pytest.mark.parametrize("centre", ["corner", "face", "inside"])
@pytest.mark.parametrize("batch", [1, 2])
def test_reduction_and_radii_over_shapes(wdm, n, centre, batch):
    g = spe.Grid(n, tuple(0.2 * m for m in n))
    X, Y, Z = g.coords()
    rng = np.random.default_rng(sum(n))
    c = {"corner": (0, n[1] - 1, 0), "face": (n[0] - 1, n[1] // 2, n[2] // 3),
         "inside": (n[0] // 3, n[1] // 2, n[2] // 2 - 1)}[centre]
    items = []
    for b in range(batch):
        r2 = (X - X[0, 0, c[0]]) ** 2 + (Y - Y[0, c[1], 0]) ** 2 + (Z - Z[c[2], 0, 0]) ** 2
        amp = np.exp(-r2 / (0.5 + b)) + 0.05 * rng.random(r2.shape)
        items.append((amp * np.exp(2j * np.pi * X / g.L[0])).astype(np.complex64))
    with wdm.SPEContext(n, g.L, poisson_coeff=1.0, batch=batch) as ctx:
        ctx.set_psi(np.stack(items) if batch > 1 else items[0])
        _check(ctx, g, n, batch)


@pytest.mark.parametrize("kind", ["zero", "one cell", "far shells"])
def test_radii_with_few_weights(wdm, kind):
    n = (64, 48, 96)
    g = spe.Grid(n, tuple(0.2 * m for m in n))
    psi = np.zeros(n[::-1], np.complex64)
    if kind != "zero":
        psi[3, 5, 7] = 2 + 1j
    if kind == "far shells":
        psi[3, 5, 60] = 1
        psi[90, 5, 7] = 1 - 1j
        psi[90, 40, 60] = 0.5j
    with wdm.SPEContext(n, g.L, poisson_coeff=1.0) as ctx:
        ctx.set_psi(psi)
        d = ctx.diagnostics()
        radii = np.array([d[f"radius_{k}0"] for k in range(1, 10)])
        if kind == "zero":
            assert np.all(np.isnan(radii)) and d["mass"] == 0 and d["argmax"] == 0
        else:
            _check(ctx, g, n, 1)


@pytest.mark.parametrize("power", [-60, -51, 58, 61])
def test_radii_do_not_depend_on_the_scale(wdm, power):
    # a power of two scales every weight exactly, whether the FP32 words or FP64 sum it (components
    # outside 2^-50 .. 2^60); some components are zero
    n = (48, 32, 64)
    g = spe.Grid(n, tuple(0.2 * m for m in n))
    rng = np.random.default_rng(7)
    psi = (rng.standard_normal(n[::-1]) + 1j * rng.standard_normal(n[::-1])).astype(np.complex64)
    psi[3, 4, 5] = 0
    psi[::2, 1, ::3] = psi[::2, 1, ::3].real
    got = []
    with wdm.SPEContext(n, g.L, poisson_coeff=0.0) as ctx:
        for p in (0, power):
            ctx.set_psi(psi * np.float32(2.0 ** p))
            d = ctx.diagnostics()
            got.append([d["argmax"]] + [d[f"radius_{k}0"] for k in range(1, 10)])
    assert got[0][0] == got[1][0] == np.argmax(np.abs(psi.astype(np.complex128)) ** 2)
    assert np.allclose(got[1], got[0], rtol=1e-9, atol=0)


def test_device_outputs_of_any_alignment(wdm):
    torch = pytest.importorskip("torch")
    n = (32, 16, 24)
    g = spe.Grid(n, (4.0, 2.0, 3.0))
    rng = np.random.default_rng(1)
    cells = n[0] * n[1] * n[2]
    with wdm.SPEContext(n, g.L, poisson_coeff=1.0) as ctx:
        ctx.set_psi((rng.standard_normal(n[::-1]) + 1j * rng.standard_normal(n[::-1])).astype(np.complex64))
        for get, host in ((ctx.get_rho, ctx.get_rho()), (ctx.get_phi, ctx.get_phi())):
            for off in (0, 1):
                buf = torch.zeros(cells + 1, dtype=torch.float32, device="cuda")
                get(out=buf[off:off + cells].view(n[::-1]))
                assert np.array_equal(buf[off:off + cells].cpu().numpy().reshape(n[::-1]), host.reshape(n[::-1]))


@pytest.mark.parametrize("n,batch", [((8, 8, 8), 1), ((32, 16, 24), 3), ((96, 64, 48), 1), ((128, 128, 96), 1)], ids=str)
def test_device_inputs_match_host_inputs(wdm, n, batch):
    # a device psi is stored and summed in one kernel, a host psi copied and then summed: the same bits
    torch = pytest.importorskip("torch")
    g = spe.Grid(n, (4.0, 2.0, 3.0))
    rng = np.random.default_rng(2)
    shape = ((batch,) if batch > 1 else ()) + n[::-1]
    psi = (rng.standard_normal(shape) + 1j * rng.standard_normal(shape)).astype(np.complex64)
    with wdm.SPEContext(n, g.L, poisson_coeff=1.0, batch=batch) as ctx:
        ctx.set_psi(psi)
        phi = ctx.get_phi()
        for off in (0, 1):
            buf = torch.zeros(psi.size + 1, dtype=torch.complex64, device="cuda")
            buf[off:off + psi.size] = torch.from_numpy(psi.reshape(-1))
            torch.cuda.synchronize()
            ctx.set_psi(buf[off:off + psi.size].view(shape))
            assert np.array_equal(ctx.get_psi(), psi)
            # the block sums meet in FP64 atomics: the shift may round the other way in its last place
            assert np.allclose(ctx.get_phi(), phi, rtol=0, atol=1e-6 * np.abs(phi).max())
