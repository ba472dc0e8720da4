"""The operators at the edges of their tiles, for every tile that a size can choose: rows one more and one fewer than a
tile's, columns that just fit half a tile or do not, the whole-tile row kernel; on and off the 16-byte
boundaries.  Bit-identical to the oracle, as every operator result."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

# (fields, ny, nx): f64 takes half-width tiles up to 64 columns, f32 up to 128, as soon as the 16 x 32 tiles are too many
# for the SMs at once; the last three give f64 fewer tiles of 48 rows than there are SMs
SHAPES = [(400, 23, 17), (400, 25, 24), (260, 49, 63), (200, 48, 64), (200, 24, 65), (100, 47, 127), (100, 25, 128),
          (90, 24, 129), (150, 17, 260), (150, 16, 516), (1, 467, 1730), (1, 25, 13001), (2, 24, 6700)]


@pytest.mark.parametrize("op", ["Upwind4", "Upwind9", "SBP4", "SBP8"])
@pytest.mark.parametrize("nb,ny,nx", SHAPES)
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_tiles(orc, op, nb, ny, nx, dtype):
    from summationbyparts_b200 import operators
    o = getattr(operators, op)()
    a = np.random.default_rng(nb + nx).uniform(-1, 1, (nb, ny, nx)).astype(np.float64 if dtype == "f64" else np.float32)
    src = torch.from_numpy(a).cuda()
    for name, direction, kind in (("diffxi", orc.XI, orc.DIFF), ("diffeta", orc.ETA, orc.DIFF),
                                  ("dissxi", orc.XI, orc.DISS), ("disseta", orc.ETA, orc.DISS)):
        if not hasattr(o, name):
            continue
        out = torch.full_like(src, float("nan"))
        getattr(o, name)(src, out)
        out = out.cpu().numpy()
        for b in {0, 1, nb // 2, nb - 1} & set(range(nb)):
            assert out[b].tobytes() == orc.op_apply(o.ids[0], direction, kind, a[b]).tobytes(), (name, b)
        assert np.isfinite(out).all()
