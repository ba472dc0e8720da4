"""The error norm of an f64 state that has just been initialised is exactly zero: initial data and error norm
evaluate the same vortex data, to the last bit, whatever gamma, time and vortices."""
import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")


@pytest.mark.parametrize("gamma", [1.4, 1.3])
@pytest.mark.parametrize("vortices", [0, 1, 3])
@pytest.mark.parametrize("t", [0.0, 0.75])
def test_no_error_at_the_start(gamma, vortices, t):
    from summationbyparts_b200 import workloads
    from summationbyparts_b200.operators import Upwind4
    from summationbyparts_b200.system import BC_VORTEX, BlockSpec, BlockSystem, VortexParameters, Vortice
    x, y = workloads.warped(-5.0, 5.0, 71, -5.0, 5.0, 45)
    g = BlockSystem([BlockSpec(x, y, Upwind4(), [(BC_VORTEX, 0)] * 4, 0)], 1, "f64", gamma)
    g.set_vortex(VortexParameters([Vortice(-1.0 + k, 0.3 * k, 0.5 + 0.1 * k, 1.0) for k in range(vortices)], mach=0.5))
    g.set_dt(1e-3)
    g.init_vortex(t)
    g.set_time(t)
    assert g.errors()[0] == 0.0
    if vortices:
        g.advance(2)
        assert g.errors()[0] > 0.0
    g.close()
