"""Reading the potential while it is kept y-spectral (grids on plane passes): the same
bits as from the separate passes, as often as it is read, through every reader, and the
state goes on from there as if it had not been read."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# every row length; planes that do not fill a warp's row pairs, longest columns, several
# items, more planes than SMs
CASES = [((8, 24, 12), 1), ((12, 8, 16), 3), ((16, 256, 8), 1), ((24, 12, 8), 2), ((32, 64, 192), 1), ((48, 96, 12), 1),
         ((64, 96, 24), 1), ((96, 32, 8), 2), ((128, 16, 48), 1), ((128, 128, 128), 1)]


def _read(wdm, torch, n, batch, psi, read):
    with wdm.SPEContext(n, (4.0, 3.0, 5.0), batch=batch) as ctx:
        ctx.set_psi(psi)
        ctx.step(1, 0.01)
        got = []
        if read:
            dev = torch.empty(psi.shape, dtype=torch.float32, device="cuda")
            pos = np.array([[0.1, 0.2, 0.3], [-1.0, 0.7, -0.4]])
            for _ in range(2):
                got += [ctx.get_phi(), ctx.get_phi(dev).cpu().numpy(), ctx.reduce()]
                if batch == 1:
                    got.append(ctx.interpolate_phi(pos))
        ctx.step(1, 0.01)
        return got, ctx.get_psi()


@pytest.mark.parametrize("n,batch", CASES, ids=[f"{'x'.join(map(str, n))}-b{b}" for n, b in CASES])
def test_potential_from_planes(wdm, monkeypatch, n, batch):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator("cuda").manual_seed(2)
    psi = torch.randn(((batch,) if batch > 1 else ()) + n[::-1], dtype=torch.complex64, device="cuda", generator=g)
    torch.cuda.synchronize()
    got, after = _read(wdm, torch, n, batch, psi, True)
    _, unread = _read(wdm, torch, n, batch, psi, False)
    monkeypatch.setenv("WDM_PLANES", "off")
    want, separate = _read(wdm, torch, n, batch, psi, True)
    assert np.array_equal(after, unread) and np.array_equal(after, separate)
    for a, b in zip(got, want):
        assert np.array_equal(a, b) if isinstance(a, np.ndarray) else a == b
