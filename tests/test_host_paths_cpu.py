"""The library's host code on a runtime without a GPU (fake_cudart.cpp): which kernels a call launches,
with which grids and shared memory, on which device, and what it returns.  CPU only; no kernel runs."""
import concurrent.futures as cf
import ctypes
import os
import shutil
import subprocess

import pytest

HERE = os.path.dirname(os.path.abspath(__file__))


class Runtime:
    """The library linked with the stand-in runtime, and what that runtime recorded."""

    def __init__(self, path):
        from summationbyparts_b200 import _capi
        self.lib = ctypes.CDLL(path, mode=os.RTLD_LOCAL | os.RTLD_NOW)
        for name, (res, args) in _capi.SIGNATURES.items():
            f = getattr(self.lib, name)
            f.restype, f.argtypes = res, args
        self.lib.fake_launch_name.restype = ctypes.c_char_p
        self.lib.fake_alloc.restype = ctypes.c_void_p
        self.device(0)

    def device(self, d):
        assert self.lib.cudaSetDevice(d) == 0

    def error(self):
        return self.lib.sbp_last_error().decode()

    def launches(self):
        """(kernel, device, grid, threads, dynamic shared memory) of every launch since the last call."""
        out = []
        for i in range(self.lib.fake_launch_count()):
            v = (ctypes.c_longlong * 6)()
            self.lib.fake_launch_shape(i, v)
            out.append((self.lib.fake_launch_name(i).decode(), v[0], tuple(v[1:4]), v[4], v[5]))
        self.lib.fake_clear_launches()
        return out

    def allocations(self, host):
        return [self.lib.fake_alloc(int(host), k) for k in range(self.lib.fake_alloc_count(int(host)))]


@pytest.fixture(scope="module")
def linked(tmp_path_factory):
    from summationbyparts_b200 import build
    with cf.ThreadPoolExecutor(os.cpu_count()) as ex:
        objs = list(ex.map(lambda u: build._compile(*u, False), build.UNITS.items()))
    out = str(tmp_path_factory.mktemp("rt") / "libsbp_host.so")
    cuda = os.path.dirname(os.path.dirname(os.path.realpath(build.nvcc())))
    # symbols bind inside the library: another cudart in the process is not used
    cmd = ["g++", "-std=c++17", "-O1", "-shared", "-fPIC", "-Wl,-Bsymbolic", "-I" + os.path.join(cuda, "include"),
           os.path.join(HERE, "fake_cudart.cpp"), *objs, "-o", out]
    r = subprocess.run(cmd, capture_output=True, text=True)
    assert r.returncode == 0, r.stderr
    return out


@pytest.fixture
def rt(linked, tmp_path):
    """A copy of the library per test: its statics are as in a new process."""
    return Runtime(shutil.copy(linked, tmp_path / "lib.so"))


PTR = 1 << 20  # an address that no host code reads


@pytest.mark.parametrize("nx", [1533, 1536])  # rows off and on the 16-byte boundaries
@pytest.mark.parametrize("dtype", [0, 1])
def test_operators_on_every_device(rt, nx, dtype):
    """A large f64 column application takes more than 48 KB of shared memory, which is allowed per function and
    device: it runs on each device of a process, whatever ran before."""
    for d in (0, 3, 0, 1):
        rt.device(d)
        assert rt.lib.sbp_diffeta(2, dtype, PTR, 2 * PTR + 8, 1021, nx, 4, 1021 * nx, None) == 0, rt.error()
        (name, dev, _, _, smem), = rt.launches()
        assert "op_eta_kernel" in name and dev == d and (dtype == 1 or smem > 48 * 1024)


def test_network_on_every_device(rt):
    for d in (0, 2, 1):
        net = ctypes.c_void_p()
        assert rt.lib.sbp_cnn_create(d, 2, 0, ctypes.byref(net)) == 0, rt.error()
        n = 2 * 4 * 64 * 64
        states = (ctypes.c_double * n)()
        assert rt.lib.sbp_cnn_gradients(net, 2, states, 0, 4 * 64 * 64, states, None, None) == 0, rt.error()
        assert any(smem > 48 * 1024 for *_, smem in rt.launches())
        assert rt.lib.sbp_cnn_destroy(net) == 0


def test_network_reports_a_wait_that_gave_up(rt):
    """The status word that a kernel sets when it gives up (a network's mapped host memory) reaches the
    caller at the next synchronising call, whichever that is, and once."""
    net = ctypes.c_void_p()
    assert rt.lib.sbp_cnn_create(0, 1, 0, ctypes.byref(net)) == 0, rt.error()
    word = ctypes.c_uint.from_address(rt.allocations(host=True)[-1])
    params = (ctypes.c_float * rt.lib.sbp_cnn_param_count(net))()
    states = (ctypes.c_double * (4 * 64 * 64))()
    loss = ctypes.c_float()
    one = (net, 1, states, 0, 4 * 64 * 64)
    calls = {"synchronize": lambda: rt.lib.sbp_cnn_synchronize(net),
             "get_params": lambda: rt.lib.sbp_cnn_get_params(net, params),
             "gradients": lambda: rt.lib.sbp_cnn_gradients(*one, states, None, params),
             "loss": lambda: rt.lib.sbp_cnn_train_step(*one, states, 1e-3, ctypes.byref(loss))}
    for name, call in calls.items():
        assert call() == 0, name
        word.value = 1
        assert rt.lib.sbp_cnn_apply(*one, states) == 0, name  # asynchronous: reports nothing yet
        assert rt.lib.sbp_cnn_train_step(*one, states, 1e-3, None) == 0, name
        assert call() != 0 and "in time" in rt.error(), name
        assert call() == 0, name
    assert rt.lib.sbp_cnn_destroy(net) == 0


SYSTEMS = {"block": ("f64", 8), "block_f32c": ("f32c", 8), "multiblock": ("f64", 16), "ensemble": ("f64", 0)}


@pytest.mark.parametrize("name", SYSTEMS)
def test_autotune_reports_a_schedule_that_can_be_set(rt, monkeypatch, name):
    """What autotune returns is the schedule (every candidate takes the same time here, so the first form
    stays), and set_tiles takes it back: small systems keep the fused form both times."""
    from summationbyparts_b200 import _capi, workloads
    from summationbyparts_b200.system import BlockSystem
    monkeypatch.setattr(_capi, "lib", rt.lib)
    prec, rows = SYSTEMS[name]
    if name == "ensemble":
        insts = workloads.ensemble_instances(40, seed=1)
        blocks, dts = workloads.ensemble_blocks(insts), [i.dt for i in insts]
    else:
        blocks, dts = workloads.multiblock() if name == "multiblock" else workloads.Config0().blocks(), [1e-3]
    s = BlockSystem(blocks, len(dts), prec, 1.4)
    for k, dt in enumerate(dts):
        s.set_dt(dt, k)
    launches = s.launches_per_step()
    tiles = s.autotune()
    assert tiles == {0: (16, 32, 256), 8: (8, 16, 288), 16: (16, 32, 320)}[rows]
    for _ in range(2):
        groups = range(len(s.groups()))
        assert [s.group_fused(g) for g in groups] == [rows > 0 for _ in groups]
        assert [s.group_tiles(g)[0] for g in groups] == [rows or 16 for _ in groups]
        assert s.launches_per_step() == launches
        rt.launches()
        s.advance(1)
        s.set_tiles(*tiles)
    s.close()


def test_tiles_that_cannot_be_set(rt, monkeypatch):
    from summationbyparts_b200 import _capi, operators, workloads
    from summationbyparts_b200.system import BC_EVAL, BC_VORTEX, BlockSpec, BlockSystem
    monkeypatch.setattr(_capi, "lib", rt.lib)
    x, y = workloads.warped(-5.0, 5.0, 64, -5.0, 5.0, 64)
    v = (BC_VORTEX, 0)
    fused = [(8, 16, 288), (16, 32, 320)]
    other = [(8, 16, 0), (8, 32, 288), (8, 16, 256), (16, 16, 320), (16, 32, 288), (32, 32, 320), (24, 32, 0), (16, 32, 128)]
    plain = [(16, 32, 0), (32, 32, 0), (16, 32, 256), (32, 32, 256)]
    one = operators.Upwind9()
    for op, bc, takes_fused in ((one, [v] * 4, True), (one, [(BC_EVAL, 0)] + [v] * 3, False),
                                (operators.Pair(operators.SBP4(), operators.Upwind9()), [v] * 4, False)):
        s = BlockSystem([BlockSpec(x, y, op, bc, 0)], 1, "f64", 1.4)
        for t in plain + (fused if takes_fused else []):
            s.set_tiles(*t)
            assert s.group_fused(0) == (t in fused)
        for t in other + ([] if takes_fused else fused):
            with pytest.raises(_capi.SbpError):
                s.set_tiles(*t)
        s.close()
