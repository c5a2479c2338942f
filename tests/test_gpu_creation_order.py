"""Creating a context waits for the default stream, so that inputs queued there before
the creation are complete when a call on the context's own stream reads them."""
import pytest

pytestmark = pytest.mark.gpu

N, L = (64, 48, 32), (8.0, 6.0, 4.0)


@pytest.mark.parametrize("call", ["poisson", "set_psi"])
def test_inputs_queued_before_creation_are_complete(wdm, call):
    torch = pytest.importorskip("torch")
    if not torch.cuda.is_available():
        pytest.skip("no CUDA device")
    new = torch.randn(N[::-1], dtype=torch.complex64 if call == "set_psi" else torch.float32, device="cuda")
    data, out = torch.zeros_like(new), torch.zeros_like(new)
    a = torch.randn(4096, 4096, device="cuda") / 64
    b = a @ a
    torch.cuda.synchronize()

    def result(x):  # the calls wait for the context's stream alone
        with wdm.SPEContext(N, L) as ctx:
            if call == "poisson":
                return ctx.poisson(x, out)
            ctx.set_psi(x)
            return ctx.get_psi(out)

    want = result(new).clone()  # and this grid's passes are timed and loaded
    torch.cuda.synchronize()
    for _ in range(40):  # tens of milliseconds in front of the input
        b = b @ a
    data.copy_(new)
    got = result(data).clone()
    torch.cuda.synchronize()
    assert torch.equal(got, want)
