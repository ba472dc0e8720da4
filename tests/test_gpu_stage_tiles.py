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


@pytest.mark.parametrize("case", ["block", "multiblock", "ensemble"])
def test_fused_form(case):
    """The fused stage kernel (SATs and times in the stage launches: the default of small systems)
    against the separate stage and edge kernels: the same f64 states and times bit for bit, after steps
    of every instance and after ragged ones."""
    from summationbyparts_b200 import workloads
    from summationbyparts_b200.system import BlockSystem
    if case == "block":  # 8-row tiles
        blocks, vortices, dts = workloads.Config0().blocks(), [workloads.STANDARD_VORTEX], [workloads.Config0().dt]
    elif case == "multiblock":  # 16-row tiles, coupled blocks
        blocks = workloads.multiblock()
        vortices, dts = [workloads.STANDARD_VORTEX], [workloads.multiblock_dt(blocks)]
    else:  # two operator groups on their own streams
        insts = [i for i in workloads.ensemble_instances(60, seed=1) if i.side <= 75][:6]
        assert {i.op_id for i in insts} == {workloads.UPWIND4, workloads.UPWIND9}
        blocks, vortices, dts = workloads.ensemble_blocks(insts), [i.vortex for i in insts], [i.dt for i in insts]
    out = []
    for tiles in (0, 16):
        g = BlockSystem(blocks, len(dts), "f64", 1.4)
        if tiles:
            g.set_tiles(tiles, 32)
        for k, (v, dt) in enumerate(zip(vortices, dts)):
            g.set_vortex(v, k)
            g.set_dt(dt, k)
        g.init_vortex(0.0)
        fused = g.launches_per_step() % 4 == 0
        assert fused == (tiles == 0)
        g.advance(3)
        g.advance_instances([k % 3 for k in range(len(dts))])
        out.append((np.concatenate([g.state(b).ravel() for b in range(len(blocks))]),
                    [g.time(k) for k in range(len(dts))]))
        g.close()
    assert out[0][1] == out[1][1]
    assert out[0][0].tobytes() == out[1][0].tobytes()
