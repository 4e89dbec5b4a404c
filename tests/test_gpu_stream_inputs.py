"""Device inputs made by kernels that are still queued when the call is made: the autograd
functions on torch's default stream and on a stream of its own, and the structure factor's
adjoint on the stream set with amdat_set_stream.  The result is that of the finished
inputs, to the order of the FP64 additions."""
import ctypes as C

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


def test_adjoint_reads_its_weights_on_the_context_stream(engine_mod):
    eng = engine_mod.Engine(0)
    stream = torch.cuda.Stream()
    try:
        pos = _pos(3)
        torch.cuda.synchronize()
        eng.upload_device(pos.data_ptr(), 2, N, [L] * 3)
        eng.set_stream(stream.cuda_stream)
        h, nk, ns = eng.wave_density_lattice(0, 4.0, 0.2, L, [0, 1])
        off = eng.wave_density_vectors(h, nk, ns)[1]
        weights = torch.cos(torch.arange(ns, device="cuda", dtype=torch.float64))
        late = weights.clone()
        weights.zero_()
        grad = torch.zeros((2, N, 3), device="cuda")
        torch.cuda.synchronize()
        with torch.cuda.stream(stream):
            torch.cuda._sleep(WAIT)
            weights.copy_(late)
        engine_mod._check(engine_mod.lib().amdat_structure_factor_adjoint(
            eng.handle, h, C.c_void_p(off.ctypes.data), ns, C.c_void_p(weights.data_ptr()), engine_mod.OUT_DEVICE,
            C.c_void_p(grad.data_ptr())))
        eng.synchronize()
        want = eng.structure_factor_adjoint(h, off, late.cpu().numpy(), 2, N)
        assert np.abs(want).max() > 0
        np.testing.assert_array_equal(grad.cpu().numpy(), want)
    finally:
        eng.close()
