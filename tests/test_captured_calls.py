"""Calls that a caller captures on the solver's stream and replays between
steps and queries.  A one-step graph leaves the control block with the host,
and the queries read it there; a replay changes the block behind it, so after
any such capture the queries must copy it again."""
import ctypes

import numpy as np
import pytest

from host_build import EMU, HERE, link

CAPTURE_HOST = """
#include "cuda_runtime.h"
extern "C" void host_capture_begin() { cudaStreamBeginCapture(nullptr, cudaStreamCaptureModeGlobal); }
extern "C" void *host_capture_end()
{
    cudaGraph_t g = nullptr;
    cudaGraphExec_t e = nullptr;
    cudaStreamEndCapture(nullptr, &g);
    cudaGraphInstantiate(&e, g);
    cudaGraphDestroy(g);
    return e;
}
extern "C" void host_replay(void *e) { cudaGraphLaunch((cudaGraphExec_t)e, nullptr); }
"""


class HostGraphs:
    """Device memory, stream and capture of the host build."""
    stream = None

    def __init__(self, lib):
        self.lib = lib
        lib.host_capture_end.restype = ctypes.c_void_p
        lib.host_replay.argtypes = [ctypes.c_void_p]

    def device_array(self, a):
        return a, a.ctypes.data

    def capture(self, work):
        self.lib.host_capture_begin()
        work()
        e = self.lib.host_capture_end()
        return lambda: self.lib.host_replay(e)


class TorchGraphs:
    """The same on the GPU, through a torch stream and CUDA graph."""

    def __init__(self):
        import torch

        self.torch = torch
        self.torch_stream = torch.cuda.Stream()
        self.stream = self.torch_stream.cuda_stream

    def device_array(self, a):
        t = self.torch.from_numpy(a).cuda()
        self.torch.cuda.synchronize()
        return t, t.data_ptr()

    def capture(self, work):
        g = self.torch.cuda.CUDAGraph()
        with self.torch.cuda.graph(g, stream=self.torch_stream):
            work()

        def replay():
            with self.torch.cuda.stream(self.torch_stream):
                g.replay()
        return replay


def _reset(lib, h, dev):
    assert lib.rmhd2d_set_state_device(h, ctypes.cast(dev, ctypes.POINTER(ctypes.c_double)), 1) == 0


def _step(lib, h, dev):
    assert lib.rmhd2d_step_rk2(h) == 0
    assert lib.rmhd2d_step_rk2(h) == 0


def _slab_step(lib, h, dev):
    for _ in range(2):
        for k in (1, 2):
            assert lib.rmhd2d_slab_stage(h, k) == 0
            assert lib.rmhd2d_slab_fill(h, k) == 0


def _queries_follow_a_replay(lib, graphs, bc, work):
    """Steps a solver, replays `work` behind the last step, and compares what
    the queries say with a fresh solver that did the same without capture."""
    from resistivemhd_gpu_b200 import Solver, setups

    s = setups.random_smooth_state(26, 22, seed=3, bc=bc)
    cfg = Solver.make_config(s.nx, s.ny, s.dx, s.dy, gamma=s.gamma, cfl=s.cfl, eps=s.eps, eta=s.eta, bc=s.bc)
    cfg.stream = graphs.stream
    keep, dev = graphs.device_array(np.ascontiguousarray(s.state))
    dev = ctypes.c_void_p(dev)

    def answers(h):
        v, c, out = ctypes.c_double(), ctypes.c_int(), np.empty_like(s.state)
        got = []
        for q in (lib.rmhd2d_calculate_dt, lib.rmhd2d_get_dt, lib.rmhd2d_get_total_time):
            assert q(h, ctypes.byref(v)) == 0
            got.append(v.value)
        assert lib.rmhd2d_check_crashed(h, ctypes.byref(c)) == 0
        assert lib.rmhd2d_get_state(h, out.ctypes.data_as(ctypes.POINTER(ctypes.c_double))) == 0
        return got + [c.value], out

    def solver(use):
        h = ctypes.c_void_p()
        if work is _slab_step:
            assert lib.rmhd2d_create_slab(ctypes.byref(cfg), 4, ctypes.byref(h)) == 0
        else:
            assert lib.rmhd2d_create(ctypes.byref(cfg), ctypes.byref(h)) == 0
        try:
            _reset(lib, h, dev)
            return use(h)
        finally:
            lib.rmhd2d_destroy(h)

    def replayed(h):
        replay = graphs.capture(lambda: work(lib, h, dev))
        _reset(lib, h, dev)
        seen = []
        for _ in range(2):
            _step(lib, h, dev)
            before = answers(h)[0]              # from here on an unchanged block could be kept
            _step(lib, h, dev)
            replay()
            seen.append((before, *answers(h)))
        return seen

    def direct(h):
        _reset(lib, h, dev)
        seen = []
        for _ in range(2):
            _step(lib, h, dev)
            before = answers(h)[0]
            _step(lib, h, dev)
            work(lib, h, dev)
            seen.append((before, *answers(h)))
        return seen

    for (b0, g, state), (b1, want, want_state) in zip(solver(replayed), solver(direct)):
        assert b0 == b1
        assert g == want
        assert np.array_equal(state, want_state)


@pytest.fixture(scope="module")
def host_abi(shared_host_abi):
    _, d = shared_host_abi
    src = d / "capture_host.cpp"
    src.write_text(CAPTURE_HOST)
    lib = link(d, sorted(str(o) for o in d.glob("*.o")), [HERE / "host_tma.cpp", src], "librmhd2d_capture.so", (EMU,))
    from resistivemhd_gpu_b200 import _lib

    for name, res, args in _lib.SIGNATURES:
        fn = getattr(lib, name)
        fn.restype = res
        fn.argtypes = args
    return lib


@pytest.mark.parametrize("bc", ["periodic", "symmetric"])
@pytest.mark.parametrize("work", [_reset, _step, _slab_step])
def test_queries_follow_a_replay_on_the_host_build(host_abi, monkeypatch, bc, work):
    from resistivemhd_gpu_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", host_abi)
    _queries_follow_a_replay(host_abi, HostGraphs(host_abi), bc, work)


@pytest.mark.gpu
@pytest.mark.parametrize("bc", ["periodic", "symmetric"])
@pytest.mark.parametrize("work", [_reset, _step, _slab_step])
def test_queries_follow_a_replay(gpu, bc, work):
    _queries_follow_a_replay(gpu, TorchGraphs(), bc, work)
