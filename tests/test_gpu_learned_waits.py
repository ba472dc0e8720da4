"""A network kernel whose bounded waits run out: with no polls at all every one of them gives up at its first
wait.  The call that next synchronises raises, the optimiser has changed nothing, and afterwards the
network works as before, to the last bit."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _limit(net, polls):
    from summationbyparts_b200 import _capi
    f = _capi.lib._ZN3sbp14cnn_wait_limitEP7sbp_cnni  # void sbp::cnn_wait_limit(sbp_cnn*, int)
    f.argtypes, f.restype = [ctypes.c_void_p, ctypes.c_int], None
    f(net.h, polls)


@pytest.mark.parametrize("n", [1, 40])  # fewer bands than CTAs; three for some CTAs (a stage used twice)
def test_no_polls(n):
    from summationbyparts_b200._capi import SbpError
    from summationbyparts_b200.learned import CorrectionNet
    g = torch.Generator(device="cuda").manual_seed(n)
    coarse, fine = (torch.rand((n, 4, 64, 64), dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    net, other = CorrectionNet(max_batch=n, seed=5), CorrectionNet(max_batch=n, seed=5)
    p0 = net.params()
    _limit(net, 0)
    for call in (lambda: net.output(coarse), lambda: net.apply(coarse), lambda: net.gradients(coarse, fine),
                 lambda: net.train_step(coarse, fine, 1e-3, want_loss=True)):
        with pytest.raises(SbpError, match="in time"):
            call()
    for _ in range(2):
        net.train_step(coarse, fine, 1e-3)
    with pytest.raises(SbpError, match="in time"):
        net.params()
    assert net.params().tobytes() == p0.tobytes()
    _limit(net, 1 << 22)
    net.set_params(p0)
    for m in (net, other):
        m.train_step(coarse, fine, 1e-3)
    assert net.params().tobytes() == other.params().tobytes() != p0.tobytes()
    assert torch.equal(net.apply(coarse), other.apply(coarse))
    for m in (net, other):
        m.close()
