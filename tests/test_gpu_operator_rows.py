"""The operator kernels on rows that do not start on 16-byte boundaries: odd lengths, input and output
pointers at every element offset (equal and unequal), batches with a gap between them, the least and
tile-edge lengths of both tile shapes.  Bit-identical to the oracle, as every operator result; the
bytes around the output stay as they were."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

torch = pytest.importorskip("torch")

FNS = {"diffxi": (0, 0), "diffeta": (1, 0), "dissxi": (0, 1), "disseta": (1, 1)}
SHAPES = [(16, 16), (17, 19), (33, 31), (47, 65), (49, 129), (20, 255), (18, 257), (16, 513), (130, 1027)]


@pytest.mark.parametrize("op", [0, 2, 4, 5])
@pytest.mark.parametrize("dtype", ["f64", "f32"])
def test_alignments(orc, op, dtype):
    from summationbyparts_b200 import _capi
    np_t, t_t = (np.float64, torch.float64) if dtype == "f64" else (np.float32, torch.float32)
    rng = np.random.default_rng(10 * op + len(dtype))
    offsets = [(0, 0), (1, 1), (1, 0), (0, 1)] if dtype == "f64" else [(0, 0), (1, 1), (2, 2), (3, 3), (1, 2), (3, 0)]
    for k, (ny, nx) in enumerate(SHAPES):
        nb, gap = (1, 0) if k % 2 else (3, k)
        stride = ny * nx + gap
        a = rng.uniform(-1, 1, (nb, ny, nx)).astype(np_t)
        refs = {}
        for name, (direction, kind) in FNS.items():
            if kind == 0 or op in (0, 2):
                refs[name] = [orc.op_apply(op, orc.XI if direction == 0 else orc.ETA,
                                           orc.DIFF if kind == 0 else orc.DISS, a[b]) for b in range(nb)]
        for oi, oo in offsets:
            total = (nb - 1) * stride + ny * nx
            src = torch.full((total + 8,), float("nan"), dtype=t_t, device="cuda")
            for b in range(nb):
                src[oi + b * stride:oi + b * stride + ny * nx] = torch.from_numpy(a[b].ravel()).cuda()
            for name, ref in refs.items():
                dst = torch.full((total + 8,), 7.0, dtype=t_t, device="cuda")
                size = src.element_size()
                _capi.check(getattr(_capi.lib, "sbp_" + name)(
                    op, _capi.F64 if dtype == "f64" else _capi.F32, src.data_ptr() + oi * size,
                    dst.data_ptr() + oo * size, ny, nx, nb, stride,
                    ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
                out = dst.cpu().numpy()
                want = np.full(total + 8, 7.0, dtype=np_t)
                for b in range(nb):
                    want[oo + b * stride:oo + b * stride + ny * nx] = ref[b].ravel()
                assert out.tobytes() == want.tobytes(), (name, ny, nx, oi, oo)


@pytest.mark.parametrize("graph", [False, True])
def test_applications_in_a_row(orc, graph):
    """Each application reads what the one before it, on the same stream, wrote: after a copy, after an
    event of another stream, and recorded in a graph.  Bit-identical to the oracle's chain."""
    from summationbyparts_b200.operators import Upwind4
    op = Upwind4()
    for shape in ((64, 64), (601, 255), (2048, 2048)):
        a = np.random.default_rng(shape[1]).uniform(-1, 1, shape)
        x = [torch.zeros(shape, dtype=torch.float64, device="cuda") for _ in range(5)]
        src = torch.from_numpy(a).cuda()
        side, main = torch.cuda.Stream(), torch.cuda.Stream()

        def chain():
            x[0].copy_(src)
            op.diffxi(x[0], x[1])
            side.wait_stream(torch.cuda.current_stream())
            with torch.cuda.stream(side):
                op.diffeta(x[1], x[2])
            torch.cuda.current_stream().wait_stream(side)
            op.dissxi(x[2], x[3])
            op.disseta(x[3], x[4])

        torch.cuda.synchronize()
        with torch.cuda.stream(main):
            chain()
        torch.cuda.synchronize()
        if graph:
            for t in x:
                t.zero_()
            torch.cuda.synchronize()
            g = torch.cuda.CUDAGraph()
            with torch.cuda.graph(g, stream=main):
                chain()
            for _ in range(3):
                g.replay()
            torch.cuda.synchronize()
        ref = a
        for t, direction, kind in zip(x[1:], (orc.XI, orc.ETA, orc.XI, orc.ETA),
                                      (orc.DIFF, orc.DIFF, orc.DISS, orc.DISS)):
            ref = orc.op_apply(0, direction, kind, ref)
            assert t.cpu().numpy().tobytes() == ref.tobytes()
