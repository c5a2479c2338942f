"""wdm_get_line_schedule: its x entries are the adjoint's passes, which have two
implementations, both timed when the context is created."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

X = ("x_kick", "x_rho", "x_rho_b")


def test_both_implementations_of_the_adjoint_x_passes_are_timed(wdm, monkeypatch):
    for v in ("WDM_LINE_IMPL", "WDM_X_IMPL", "WDM_SCHEDULE"):
        monkeypatch.delenv(v, raising=False)
    times = []
    for n in ((64, 48, 32), (128, 48, 16)):
        with wdm.SPEContext(n, (4.0, 3.0, 5.0)) as ctx:
            sched = ctx.line_schedule()
            times += [sched[k]["ms"] for k in X]
            # the adjoint runs on them and does not change what is reported
            psi = np.ones(n[::-1], np.complex64)
            ctx.set_psi(psi)
            ctx.adjoint(2, 0.01, np.ones(n[::-1], np.float32))
            assert ctx.line_schedule() == sched
    assert all(0 < t < 1e3 for ms in times for t in ms.values())
    # two kernels' event times: equal in every one of six pairs only if one was measured
    assert any(ms["staged"] != ms["direct"] for ms in times)


@pytest.mark.parametrize("x_impl", ["staged", "direct"])
def test_a_schedule_from_the_environment_reaches_the_adjoint(wdm, monkeypatch, x_impl):
    monkeypatch.setenv("WDM_SCHEDULE", f"tile,tma,tile,tma,{x_impl},{x_impl},{x_impl}")
    n = (64, 48, 32)
    with wdm.SPEContext(n, (4.0, 3.0, 5.0)) as ctx:
        assert [v["impl"] for v in ctx.line_schedule().values()] == ["tile", "tma", "tile", "tma"] + [x_impl] * 3
        ctx.set_psi(np.ones(n[::-1], np.complex64))
        loss, grad, _ = ctx.adjoint(2, 0.01, np.ones(n[::-1], np.float32))
        assert np.isfinite(loss) and np.all(np.isfinite(grad.view(np.float32)))
        assert [v["impl"] for v in ctx.line_schedule().values()] == ["tile", "tma", "tile", "tma"] + [x_impl] * 3
