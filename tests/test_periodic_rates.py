"""A periodic domain's dt comes from its interior cells alone, however it is
stepped: by itself, in a batch beside runs with walls, or decomposed into
slabs.  The contracted variants would otherwise mix in the ghost fill's
uncontracted rates where one runs, and differ in the last bit."""
import ctypes

import numpy as np
import pytest

PRECISIONS = ["fp64_exact", "fp64_fast", "fp32_bulk"]
SEEDS = (1, 2, 3)   # states whose largest rate the two evaluations round differently


@pytest.fixture
def on_host(shared_host_abi, monkeypatch):
    from resistivemhd_gpu_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", shared_host_abi[0])


def _check_batch(precision):
    from resistivemhd_gpu_b200 import Batch, setups

    walls = setups.random_smooth_state(14, 14, seed=2, bc="symmetric")
    for seed in SEEDS:
        p = setups.random_smooth_state(24, 20, seed=seed, bc="periodic")
        got = []
        for sets in ([p], [p, walls]):
            with Batch(sets, precision=precision) as b:
                b.run(4)
                got.append((b[0].dt, b[0].total_time, b[0].get_state()))
        assert got[0][:2] == got[1][:2], seed
        assert np.array_equal(got[0][2], got[1][2]), seed


def _check_slabs(precision, torch_device):
    from resistivemhd_gpu_b200 import Solver, setups
    from resistivemhd_gpu_b200.slab import SlabGroup

    for seed in SEEDS:
        s = setups.random_smooth_state(24, 20, seed=seed, bc="periodic")
        for parts in (1, 2):
            with Solver.from_setup(s, precision=precision) as whole, \
                    SlabGroup(s, parts, torch_device=torch_device, precision=precision) as g:
                for _ in range(4):
                    whole.step()
                    g.step()
                assert np.array_equal(g.get_state(), whole.get_state()), (seed, parts)


def _check_slab_without_halos(lib, precision):
    """The whole domain as one slab with no halo columns, through the C ABI."""
    from resistivemhd_gpu_b200 import Solver, setups

    D = ctypes.POINTER(ctypes.c_double)
    for seed in SEEDS:
        s = setups.random_smooth_state(24, 20, seed=seed, bc="periodic")
        with Solver.from_setup(s, precision=precision) as whole:
            whole.run(4)
            want = whole.get_state()
        cfg = Solver.make_config(s.nx, s.ny, s.dx, s.dy, gamma=s.gamma, cfl=s.cfl, eps=s.eps, eta=s.eta, bc=s.bc,
                                 precision=precision)
        h, st = ctypes.c_void_p(), np.ascontiguousarray(s.state)
        assert lib.rmhd2d_create_slab(ctypes.byref(cfg), 4, ctypes.byref(h)) == 0
        try:
            assert lib.rmhd2d_set_state(h, st.ctypes.data_as(D), 1) == 0
            for _ in range(4):
                for k in (1, 2):
                    assert lib.rmhd2d_slab_stage(h, k) == 0
                    assert lib.rmhd2d_slab_fill(h, k) == 0
            got = np.empty_like(st)
            assert lib.rmhd2d_get_state(h, got.ctypes.data_as(D)) == 0
        finally:
            lib.rmhd2d_destroy(h)
        assert np.array_equal(got, want), seed


@pytest.mark.parametrize("precision", PRECISIONS)
def test_slab_without_halos_on_the_host_build(on_host, shared_host_abi, precision):
    _check_slab_without_halos(shared_host_abi[0], precision)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", PRECISIONS)
def test_slab_without_halos(gpu, precision):
    _check_slab_without_halos(gpu, precision)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_batch_on_the_host_build(on_host, precision):
    _check_batch(precision)


@pytest.mark.parametrize("precision", PRECISIONS)
def test_slabs_on_the_host_build(on_host, precision):
    _check_slabs(precision, "cpu")


@pytest.mark.gpu
@pytest.mark.parametrize("precision", PRECISIONS)
def test_batch(gpu, precision):
    _check_batch(precision)


@pytest.mark.gpu
@pytest.mark.parametrize("precision", PRECISIONS)
def test_slabs(gpu, precision):
    _check_slabs(precision, "cuda:0")
