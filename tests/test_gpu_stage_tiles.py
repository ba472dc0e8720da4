"""The tiled stage kernel at the edges of its tiles: lines of the least length an operator takes,
one tile, one more than a tile, and lengths whose last tile is as short or as wide as it gets.

One RK4 step of a periodic block against the f64 oracle.  Bar of the f64 form: the sums of an
output add about 21 products of size |J E| n / 10 <= 20, so one k rounds to about 21 x 20 x 1.1e-16 =
5e-14 of the state, which dt = 0.2 / 64 scales to 2e-16; 1e-13 of the largest state value leaves
room for the closure rows' larger coefficients, and is the bar of the other one-step tests.
Compensated f32: k rounds to about 2^-24 of its terms, dt |k| <= 0.1, so 1e-7 of the state; bar 1e-6.
"""
import numpy as np
import pytest
from _helpers import oracle_system, physical_state

pytestmark = pytest.mark.gpu

pytest.importorskip("torch")

SIZES = [(16, 16), (17, 24), (31, 40), (32, 33), (33, 32), (39, 48), (40, 41), (41, 63), (65, 39)]


@pytest.mark.parametrize("op", ["Upwind4", "Upwind9", "SBP8"])
@pytest.mark.parametrize("ny,nx", SIZES)
def test_one_step(orc, op, ny, nx):
    from summationbyparts_b200 import operators, workloads
    from summationbyparts_b200.system import BlockSpec, BlockSystem
    x, y = workloads.warped(-5.0, 5.0, nx, -5.0, 5.0, ny)
    blocks = [BlockSpec(x, y, getattr(operators, op)(), [(0, 0)] * 4, 0)]
    q0 = physical_state(x, y)
    dt = 0.2 / 64
    o = oracle_system(orc, blocks, workloads.STANDARD_VORTEX)
    o.set_state(0, q0)
    o.advance(1, dt)
    ref = o.state(0)
    results = {}
    for prec, ty in (("f64", 0), ("f64", 16), ("f64", 32), ("f32c", 0), ("f32c", 16)):
        g = BlockSystem(blocks, 1, prec, 1.4)
        g.set_vortex(workloads.STANDARD_VORTEX)
        if ty:
            g.set_tiles(ty, 32)
        g.set_state(0, q0)
        g.set_dt(dt)
        g.advance(1)
        results[prec, ty] = g.state(0)
        g.close()
        bar = 1e-13 if prec == "f64" else 1e-6
        assert np.abs(results[prec, ty] - ref).max() <= bar * np.abs(ref).max(), (prec, ty)
    # the f64 sums round the same way on every tile shape
    assert results["f64", 0].tobytes() == results["f64", 16].tobytes() == results["f64", 32].tobytes()
