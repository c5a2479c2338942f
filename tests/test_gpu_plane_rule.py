"""Which grids step on plane passes (four launches a step) and which on separate ones
(eight), at both sides of the rule's lines; either way the step equals the separate
passes bit for bit (the same transforms on the same values)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# (n, batch, plane passes): room for one CTA an SM below, at and above one wave of the
# 152 SMs, and for many waves; for two CTAs; small planes in moderate and huge
# numbers; warps per CTA between the extremes (48 x 64: six would fit, two are there)
CASES = [((128, 128, 96), 1, False), ((128, 128, 128), 1, True), ((128, 128, 192), 1, False), ((48, 256, 128), 8, True),
         ((64, 128, 48), 1, False), ((64, 128, 64), 1, True), ((8, 8, 256), 9, True), ((8, 8, 256), 10, False),
         ((48, 64, 256), 1, True), ((96, 96, 48), 2, True)]


@pytest.mark.parametrize("n,batch,planes", CASES, ids=[f"{'x'.join(map(str, n))}-b{b}" for n, b, _ in CASES])
def test_rule_and_results(wdm, monkeypatch, n, batch, planes):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    g = torch.Generator("cuda").manual_seed(1)
    psi = torch.randn(((batch,) if batch > 1 else ()) + n[::-1], dtype=torch.complex64, device="cuda", generator=g)
    out = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("WDM_PLANES", "off")
        with wdm.SPEContext(n, (4.0, 3.0, 5.0), batch=batch) as ctx:
            torch.cuda.synchronize()
            ctx.set_psi(psi)
            ctx.step(1, 0.01)
            before = ctx.launch_count
            ctx.step(2, 0.01)
            out.append(((ctx.launch_count - before), ctx.get_psi()))
    # two steps and the closing half kick
    assert out[0][0] == (4 if planes else 8) * 2 + 1 and out[1][0] == 17
    assert np.array_equal(out[0][1], out[1][1])
