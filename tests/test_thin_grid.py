"""Grids with a long x side: the shapes a solver starts with give no more rows
of tiles than a launch takes (gridDim.y, 65535)."""
import numpy as np
import pytest

LIMIT = 65535


def _start_shapes(n):
    from resistivemhd_gpu_b200 import Solver

    with Solver(n + 6, 12, 1.0 / n, 1.0 / 6) as sol:
        return sol.stage_shapes


def test_start_shapes_launch_on_the_host_build(shared_host_abi, monkeypatch):
    from resistivemhd_gpu_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", shared_host_abi[0])
    assert _start_shapes(7 * LIMIT) == (4, 5)
    assert _start_shapes(7 * LIMIT + 1) == (4, 4)


@pytest.mark.gpu
@pytest.mark.parametrize("n", [7 * LIMIT, 7 * LIMIT + 1, 8 * LIMIT])
def test_thin_grid_steps_equal_oracle(gpu, oracle, n):
    from resistivemhd_gpu_b200 import Solver, setups

    s = setups.random_smooth_state(85, 6, seed=2, bc="symmetric")
    core = np.tile(s.state[3:-3], (n // 85 + 1, 1, 1))[:n]
    s.state = np.concatenate([s.state[:3], core, s.state[-3:]])
    want, want_dts, _ = oracle.run(s, s.state, 1)
    with Solver.from_setup(s) as sol:
        sol.step()
        assert sol.dt == want_dts[0]
        assert np.array_equal(sol.get_state(), want, equal_nan=True)   # (some cells start with a negative pressure)
