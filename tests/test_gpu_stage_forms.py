"""The forms of the stage kernel, where small systems take the fused form by default: autotune's schedule is
the one that it reports, and can be set again."""
import pytest

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")


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
