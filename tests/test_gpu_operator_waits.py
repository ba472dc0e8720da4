"""An operator tile that stops waiting for its staged rows reads them itself: with no polls at all, so that
every tile of an application does, the result is the same to the last bit (the sums are the same code on
the same values).  The poll limit is an argument of the launcher behind the C entry points."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

OPS = {0: "upwind4", 2: "upwind9", 5: "sbp8"}


def _apply(polls, op, direction, kind, dtype, a, out, ny, nx, nb):
    from summationbyparts_b200 import _capi
    # cudaError_t sbp::op_apply(int, int, int, int, const void*, void*, int64_t x 4, cudaStream_t, int)
    f = _capi.lib._ZN3sbp8op_applyEiiiiPKvPvllllP11CUstream_sti
    f.restype = ctypes.c_int
    f.argtypes = [ctypes.c_int] * 4 + [ctypes.c_void_p] * 2 + [ctypes.c_int64] * 4 + [ctypes.c_void_p, ctypes.c_int]
    assert f(op, direction, kind, dtype, a.data_ptr(), out.data_ptr(), ny, nx, nb, ny * nx, None, polls) == 0


@pytest.mark.parametrize("op,kind", [(0, 0), (2, 1), (5, 0)])
@pytest.mark.parametrize("nb,ny,nx", [(1, 16, 16), (2, 33, 49), (3, 130, 291), (1, 20, 1030), (4, 500, 517)])
@pytest.mark.parametrize("dtype", [0, 1])
@pytest.mark.parametrize("offset", [0, 1])
def test_no_polls(op, kind, nb, ny, nx, dtype, offset):
    t = torch.float64 if dtype == 0 else torch.float32
    g = torch.Generator(device="cuda").manual_seed(ny * nx)
    n = nb * ny * nx
    a = (2 * torch.rand(n + offset, dtype=t, device="cuda", generator=g) - 1)[offset:]
    for direction in (0, 1):
        out = [torch.full((n + 8,), float("nan"), dtype=t, device="cuda") for _ in range(2)]
        for o, polls in zip(out, (1 << 22, 0)):
            _apply(polls, op, direction, kind, dtype, a, o[4:], ny, nx, nb)
        torch.cuda.synchronize()
        assert out[0].cpu().numpy().tobytes() == out[1].cpu().numpy().tobytes()
        assert not out[0][4:-4].isnan().any() and out[0][:4].isnan().all() and out[0][-4:].isnan().all()
