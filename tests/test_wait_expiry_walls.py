"""A bounded wait that expires is reported by the next query whatever the
walls: with periodic walls the stage-2 kernel itself leaves the control block
with the host, so its CTAs have to count there on the way out of an expired
wait as well.  The test build (test_gpu_wait_expiry.py) issues no tile load,
so nothing is in flight when a CTA gives up."""
import ctypes

import numpy as np
import pytest

from host_build import build_host_abi, has_fma
from test_gpu_wait_expiry import ERR_KERNEL, WAIT_TEST_LIB, _load

WALLS = ("periodic", "symmetric")
PRECISIONS = ("fp64_exact", "fp64_fast", "fp32_bulk")


def _queries_after_each_step(lib, bc, precision, steps=3):
    """The status of every query after each of `steps` steps of a solver whose
    stage kernels never get their tile."""
    from resistivemhd_gpu_b200 import Solver, setups

    s = setups.random_smooth_state(40, 36, seed=9, bc=bc, with_table=True)
    cfg = Solver.make_config(s.nx, s.ny, s.dx, s.dy, gamma=s.gamma, cfl=s.cfl, eps=s.eps, eta=s.eta, bc=s.bc,
                             precision=precision)
    D = ctypes.POINTER(ctypes.c_double)
    h, st, v, c = ctypes.c_void_p(), np.ascontiguousarray(s.state), ctypes.c_double(), ctypes.c_int()
    out = np.empty_like(st)
    assert lib.rmhd2d_create(ctypes.byref(cfg), ctypes.byref(h)) == 0
    try:
        assert lib.rmhd2d_set_state(h, st.ctypes.data_as(D), 1) == 0
        got = []
        for _ in range(steps):
            assert lib.rmhd2d_step_rk2(h) == 0
            got.append([lib.rmhd2d_check_crashed(h, ctypes.byref(c)), lib.rmhd2d_get_dt(h, ctypes.byref(v)),
                        lib.rmhd2d_calculate_dt(h, ctypes.byref(v)), lib.rmhd2d_get_state(h, out.ctypes.data_as(D))])
        return got
    finally:
        lib.rmhd2d_destroy(h)


@pytest.fixture(scope="module")
def expiring_host_abi(tmp_path_factory):
    if not has_fma():
        pytest.skip("the host has no fused multiply-add to model the device build with")
    return build_host_abi(tmp_path_factory.mktemp("expiry"), extra=("-DRMHD_TEST_WAIT_EXPIRY",))


@pytest.mark.parametrize("bc", WALLS)
def test_expired_wait_is_reported_on_the_host_build(expiring_host_abi, bc):
    for status in _queries_after_each_step(expiring_host_abi, bc, "fp64_exact"):
        assert status == [ERR_KERNEL] * 4


@pytest.mark.gpu
@pytest.mark.parametrize("bc", WALLS)
@pytest.mark.parametrize("precision", PRECISIONS)
def test_expired_wait_is_reported(gpu, bc, precision):
    for status in _queries_after_each_step(_load(WAIT_TEST_LIB), bc, precision):
        assert status == [ERR_KERNEL] * 4
