"""A network kernel whose bounded waits run out: each gives up at its first wait, without a poll.  The call
that next synchronises raises, the optimiser has changed nothing, and afterwards the network works as
before, to the last bit."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")


def _give_up(net, on):
    from summationbyparts_b200 import _capi
    f = _capi.lib._ZN3sbp11cnn_give_upEP7sbp_cnnb  # void sbp::cnn_give_up(sbp_cnn*, bool)
    f.argtypes, f.restype = [ctypes.c_void_p, ctypes.c_bool], None
    f(net.h, on)


@pytest.mark.parametrize("n", [1, 40])  # fewer bands than CTAs; three for some CTAs (a stage used twice)
def test_no_polls(n):
    from summationbyparts_b200._capi import SbpError
    from summationbyparts_b200.learned import CorrectionNet
    g = torch.Generator(device="cuda").manual_seed(n)
    coarse, fine = (torch.rand((n, 4, 64, 64), dtype=torch.float64, device="cuda", generator=g) for _ in range(2))
    net, other = CorrectionNet(max_batch=n, seed=5), CorrectionNet(max_batch=n, seed=5)
    p0 = net.params()
    _give_up(net, True)
    for call in (lambda: net.output(coarse), lambda: net.apply(coarse), lambda: net.gradients(coarse, fine),
                 lambda: net.train_step(coarse, fine, 1e-3, want_loss=True)):
        with pytest.raises(SbpError, match="in time"):
            call()
    for _ in range(2):
        net.train_step(coarse, fine, 1e-3)
    with pytest.raises(SbpError, match="in time"):
        net.params()
    assert net.params().tobytes() == p0.tobytes()
    _give_up(net, False)
    net.set_params(p0)
    for m in (net, other):
        m.train_step(coarse, fine, 1e-3)
    assert net.params().tobytes() == other.params().tobytes() != p0.tobytes()
    assert torch.equal(net.apply(coarse), other.apply(coarse))
    for m in (net, other):
        m.close()
