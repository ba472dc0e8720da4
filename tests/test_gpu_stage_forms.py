"""The forms of the stage kernel against each other, where small systems take the fused form by default:
compensated states bit for bit between the fused and the separate 16-row form, autotune's schedule set again,
and the boundary kinds that read other blocks on the separate form too (against the oracle)."""
import numpy as np
import pytest
from test_gpu_interpolation import PARITY, _interpolation_example, _run_pair

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")


@pytest.mark.parametrize("op", ["upwind4", "upwind9h2", "sbp8"])
@pytest.mark.parametrize("ny,nx", [(45, 71), (150, 160)])  # 8 and 16 rows
@pytest.mark.parametrize("trad", [False, True])
def test_compensated_states(op, ny, nx, trad):
    from summationbyparts_b200 import operators, workloads
    from summationbyparts_b200.system import BC_VORTEX, BlockSpec, BlockSystem
    x, y = workloads.warped(-5.0, 5.0, nx, -5.0, 5.0, ny)
    out = []
    for separate in (False, True):
        g = BlockSystem([BlockSpec(x, y, operators.BY_NAME[op](), [(BC_VORTEX, 0)] * 4, 0)], 1, "f32c", 1.4)
        g.set_vortex(workloads.STANDARD_VORTEX)
        g.set_dt(0.1 / nx)
        g.set_force_trad(trad)
        if separate:
            g.set_tiles(16, 32)
        assert g.group_fused(0) != separate
        g.init_vortex(0.0)
        g.advance(5)
        out.append(g.state(0))
        g.close()
    assert out[0].tobytes() == out[1].tobytes()


@pytest.mark.parametrize("prec", ["f64", "f32c"])
def test_autotune_of_a_small_system(prec):
    """State and time are restored, the reported tiles are the schedule's, and they can be set."""
    from summationbyparts_b200 import workloads
    from summationbyparts_b200.system import BlockSystem
    cfg = workloads.Config0()
    g = BlockSystem(cfg.blocks(), 1, prec, 1.4)
    g.set_vortex(workloads.STANDARD_VORTEX)
    g.set_dt(cfg.dt)
    g.init_vortex(0.0)
    g.advance(2)
    q, t = g.state(0), g.time()
    tiles = g.autotune()
    assert g.state(0).tobytes() == q.tobytes() and g.time() == t
    for _ in range(2):
        ty, fused = g.group_tiles(0)[0], g.group_fused(0)
        assert tiles == (ty, 16 if ty == 8 else 32, 256 + (0 if not fused else 32 if ty == 8 else 64))
        assert g.launches_per_step() == (4 if fused else 9)
        g.set_tiles(*tiles)
    g.close()


@pytest.mark.parametrize("tiles", [(16, 32, 256), (32, 32, 256), (8, 16, 288), (16, 32, 320)])
def test_interfaces_on_every_form(orc, monkeypatch, tiles):
    from summationbyparts_b200 import system, workloads
    from summationbyparts_b200.operators import Upwind4
    from summationbyparts_b200.system import BC_GRID, BC_MULTIGRID, BC_THIS, BC_VORTEX, BlockSpec

    class Tiled(system.BlockSystem):
        def __init__(self, *a):
            super().__init__(*a)
            self.set_tiles(*tiles)

    monkeypatch.setattr(system, "BlockSystem", Tiled)
    assert max(_run_pair(orc, _interpolation_example(), 10, 0.2 / 98)) <= PARITY
    v = (BC_VORTEX, 0)
    xa, ya = workloads.cartesian(-5.0, 5.0, 41, -5.0, 0.0, 21)
    xb, yb = workloads.cartesian(-5.0, 0.0, 21, 0.0, 5.0, 21)
    xc, yc = workloads.cartesian(0.0, 5.0, 21, 0.0, 5.0, 21)
    a = BlockSpec(xa, ya, Upwind4(), [(BC_MULTIGRID, [(1, 0, 21), (2, 0, 21)]), v, (BC_THIS, 0), (BC_THIS, 0)], 0)
    b = BlockSpec(xb, yb, Upwind4(), [v, (BC_MULTIGRID, [(0, 0, 21)]), (BC_GRID, 2), v], 0)
    c = BlockSpec(xc, yc, Upwind4(), [v, (BC_MULTIGRID, [(0, 20, 41)]), v, (BC_GRID, 1)], 0)
    assert max(_run_pair(orc, [a, b, c], 10, 0.2 / 40)) <= PARITY
