"""The stage kernels' tile shape for grids too small to fill the SMs (4 x 16
cells, one interface per thread), which the library picks by itself: its host
build against the oracle on ragged grids, and on the GPU the default solver
on both sides of the rule against the oracle."""
import numpy as np
import pytest

from test_stage_host import host_stage, run_host  # noqa: F401

SMALL = 6   # rmhd2d_internal.h: SHAPE_SMALL


@pytest.mark.parametrize("dims,bc,bc_y,with_table", [
    ((6, 6), "periodic", None, False),
    ((7, 17), "symmetric", None, True),
    ((13, 33), "periodic", "symmetric", True),
    ((9, 31), "flare", "wall", False),
])
def test_host_small_shape_equals_oracle(host_stage, oracle, dims, bc, bc_y, with_table):  # noqa: F811
    from resistivemhd_gpu_b200 import setups

    s = setups.random_smooth_state(*dims, seed=17, bc=bc, bc_y=bc_y, with_table=with_table)
    want, want_dts, want_crash = oracle.run(s, s.state, 2)
    got, got_dts, got_crash = run_host(host_stage, s, 2, SMALL)
    assert got_crash == want_crash
    assert np.array_equal(got_dts, want_dts)
    assert np.array_equal(got, want, equal_nan=True)


@pytest.mark.gpu
@pytest.mark.parametrize("dims", [(6, 6), (97, 49), (148, 128), (149, 128), (512, 512)])
def test_default_shapes_equal_oracle(gpu, oracle, dims):
    """148 x 128 has the most 4 x 16 tiles that run at once (296), 149 x 128
    the fewest that do not; from 2^18 cells another rule holds."""
    from resistivemhd_gpu_b200 import Solver, setups

    s = setups.random_smooth_state(*dims, seed=5, bc="symmetric" if dims[0] % 2 else "periodic", with_table=True)
    want, want_dts, crashed = oracle.run(s, s.state, 3)
    with Solver.from_setup(s) as sol:
        dts = []
        for _ in range(3):
            sol.step()
            dts.append(sol.dt)
        got = sol.get_state()
        sol.autotune(2)
        sol.set_state(s.state)
        sol.run(3)
        again = sol.get_state()
    assert crashed == -1
    assert np.array_equal(dts, want_dts)
    assert np.array_equal(got, want) and np.array_equal(again, want)
