"""A periodic domain's dt comes from its interior cells alone, however it is
stepped: by itself, in a batch beside runs with walls, or decomposed into
slabs.  The contracted variants would otherwise mix in the ghost fill's
uncontracted rates where one runs, and differ in the last bit."""
import numpy as np
import pytest

from host_build import build_host_abi, has_fma

PRECISIONS = ["fp64_exact", "fp64_fast", "fp32_bulk"]
SEEDS = range(6)


@pytest.fixture(scope="module")
def host_abi(tmp_path_factory):
    if not has_fma():
        pytest.skip("the host has no fused multiply-add to model the device build with")
    return build_host_abi(tmp_path_factory.mktemp("periodic"))


@pytest.fixture
def on_host(host_abi, monkeypatch):
    from resistivemhd_gpu_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", host_abi)


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
