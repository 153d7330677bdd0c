"""Periodic walls: the stage kernels write every ghost cell themselves, and
fold the reductions the ghost fill would add -- the dt candidate of ghost cell
0, the image of the last interior cell, included."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("dims", [(6, 6), (6, 40), (33, 7), (64, 65), (200, 170)])
def test_ghosts_equal_oracle(gpu, oracle, dims):
    from resistivemhd_gpu_b200 import Solver, setups

    s = setups.random_smooth_state(*dims, seed=31, bc="periodic", with_table=True)
    want, want_dts, crashed = oracle.run(s, s.state, 5)
    assert crashed == -1
    with Solver.from_setup(s) as sol:
        dts = []
        for _ in range(2):                       # one-step graphs, whose last kernel mirrors the control block
            sol.step()
            dts.append(sol.dt)
        sol.run(3)
        assert np.array_equal(dts, want_dts[:2]) and sol.dt == want_dts[4]
        assert np.array_equal(sol.get_state(), want)


@pytest.mark.parametrize("cell", [(-4, -4), (3, 3), (-4, 3), (20, 17)])
def test_dt_after_a_crash_equals_oracle(gpu, oracle, cell):
    """A NaN candidate never wins the dt minimum unless it is cell 0's, which
    under periodic walls holds the last interior cell."""
    from resistivemhd_gpu_b200 import Solver, setups

    s = setups.random_smooth_state(40, 36, seed=5, bc="periodic", eta=2e-3)
    state = s.state.copy()
    state[cell[0], cell[1], 7] = np.nan
    with Solver.from_setup(s) as sol:
        sol.set_state(state)
        sol.step()
        assert sol.check_crashed()
        got = sol.calculate_dt()
        after = sol.get_state()
    want = oracle.calc_dt(s, after)
    assert got == want or (np.isnan(got) and np.isnan(want))
