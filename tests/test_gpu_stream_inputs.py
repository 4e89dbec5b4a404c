"""Device inputs made by kernels that are still queued when the call is made: the autograd
functions on torch's default stream and on a stream of its own.  The result is that of the
finished inputs, to the order of the FP64 additions."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu
L, N = 9.0, 1500
WAIT = 100_000_000  # cycles that the queue is busy before the inputs change


def _pos(seed):
    g = torch.Generator(device="cuda").manual_seed(seed)
    return torch.rand((2, N, 3), generator=g, device="cuda") * L


@pytest.mark.parametrize("side", [False, True])
@pytest.mark.parametrize("what", ["gsmooth", "structure_factor"])
def test_autograd_waits_for_its_inputs(engine_mod, side, what):
    from amdat_gb300 import autograd as AG

    def value_and_grad(pos):
        out = AG.gsmooth(pos, [L] * 3, 0.05, 3.0, 60) if what == "gsmooth" else AG.structure_factor_raw(pos, [L] * 3, 4.0, 0.2)
        w = torch.cos(torch.arange(out.shape[0], device="cuda", dtype=torch.float64))
        return out.detach(), torch.autograd.grad(out, pos, w)[0]

    late = _pos(2)
    torch.cuda.synchronize()
    want, want_grad = value_and_grad(late.clone().requires_grad_(True))
    torch.cuda.synchronize()
    stream = torch.cuda.Stream() if side else torch.cuda.default_stream()
    with torch.cuda.stream(stream):
        buf = _pos(1)
        torch.cuda.synchronize()
        torch.cuda._sleep(WAIT)
        buf.copy_(late)
        got, got_grad = value_and_grad(buf.requires_grad_(True))
    torch.cuda.synchronize()
    np.testing.assert_allclose(got.cpu().numpy(), want.cpu().numpy(), rtol=1e-12)
    np.testing.assert_array_equal(got_grad.cpu().numpy(), want_grad.cpu().numpy())
