"""What a call returns does not depend on the reads and adjoints before it: the
adjoint runs on transforms of its own, whose potential rounds differently from the
time step's, and dL/da amplifies such a difference."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

L = (4.0, 3.0, 5.0)


def _inputs(n):
    rng = np.random.default_rng(sum(n))
    psi = (1.0 + 0.3 * rng.standard_normal(n[::-1]) + 0.3j * rng.standard_normal(n[::-1])).astype(np.complex64)
    return psi, (1.0 + 0.2 * rng.random(n[::-1])).astype(np.float32)


# on plane passes and past their range
SHAPES = [(32, 24, 16), (64, 64, 64), (192, 16, 12)]


@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("before", ["get_phi", "kick and back", "adjoint", "graph"])
def test_adjoint_does_not_depend_on_calls_before(wdm, n, before):
    psi, target = _inputs(n)
    D = (2.0, -1.0, -1.0, 0.5, 0.0, 0.0)
    out = []
    with wdm.SPEContext(n, L, poisson_coeff=2.0) as ctx:
        ctx.set_tidal([[0.02 * d for d in D]])
        for k in range(2):
            ctx.set_psi(psi)
            if k and before == "get_phi":
                ctx.get_phi()
            elif k and before == "adjoint":
                ctx.adjoint(3, 0.01, target, ckpt_every=2, tidal_dir=D)
                ctx.get_phi()
            elif k and before == "kick and back":
                ctx.kick(0.01)
                ctx.set_psi(psi)
            elif k:
                ctx.step_graph(2, 0.01)
                ctx.set_psi(psi)
                ctx.get_phi()
            out.append(ctx.adjoint(6, 0.01, target, ckpt_every=4, tidal_dir=D))
    # the loss and dL/da are FP64 sums of per-block partials added atomically: their
    # last bits depend on the order the blocks finish in
    assert out[1][0] == pytest.approx(out[0][0], rel=1e-12)
    assert np.array_equal(out[1][1], out[0][1])
    assert out[1][2] == pytest.approx(out[0][2], rel=1e-9)


@pytest.mark.parametrize("n", SHAPES, ids=lambda n: "x".join(map(str, n)))
@pytest.mark.parametrize("call", ["get_phi", "step", "step_graph", "kick"])
def test_calls_after_an_adjoint_return_what_they_do_without(wdm, n, call):
    psi, target = _inputs(n)
    out = []
    for adjoint in (False, True):
        with wdm.SPEContext(n, L, poisson_coeff=2.0) as ctx:
            ctx.set_psi(psi)
            if adjoint:
                ctx.adjoint(3, 0.01, target)
            if call == "get_phi":
                out.append(ctx.get_phi())
                continue
            if call == "kick":
                ctx.kick(0.01)
            else:
                getattr(ctx, call)(3, 0.01)
            out.append(ctx.get_psi())
    assert np.array_equal(out[0], out[1])
