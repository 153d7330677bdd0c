"""The shape getters report what the next step runs: the library's own choice
on a new solver, the caller's after a set, the autotuner's after a tune.
Setting the shapes that were read changes nothing."""
import numpy as np
import pytest

LARGE = {"fp64_exact": (4, 5), "fp64_fast": (4, 5), "fp32_bulk": (4, 4)}


@pytest.fixture
def on_host(shared_host_abi, monkeypatch):
    from resistivemhd_gpu_b200 import _lib

    monkeypatch.setattr(_lib, "_lib", shared_host_abi[0])


def _solver(n, m, precision="fp64_exact", ct="stage1"):
    from resistivemhd_gpu_b200 import Solver

    return Solver(n + 6, m + 6, 1.0 / n, 1.0 / m, precision=precision, ct=ct)


def _check_reports(oracle):
    from resistivemhd_gpu_b200 import Solver, _lib, setups

    for precision, large in LARGE.items():
        # 148 x 128 is the largest grid of 296 tiles of 4 x 16 cells
        for dims, want in (((6, 6), (6, 6)), ((148, 128), (6, 6)), ((149, 128), (0, 0)), ((512, 511), (0, 0)),
                           ((512, 512), large)):
            with _solver(*dims, precision) as sol:
                assert sol.stage_shapes == want and sol.tile_shape == want[0]
                sol.set_stage_shapes(*want)
                assert sol.stage_shapes == want
                with pytest.raises(_lib.RMHDError):
                    sol.set_tile_shape(7)
                assert sol.stage_shapes == want
    with _solver(512, 512, ct="contact") as sol:      # does not run the tiled kernels
        assert sol.stage_shapes == (0, 0)
    s = setups.random_smooth_state(13, 17, seed=7, bc="symmetric", with_table=True)
    want, _, _ = oracle.run(s, s.state, 2)
    with Solver.from_setup(s) as sol:
        best = sol.autotune(2)
        t = sol.tuning()
        assert sorted(t) == list(range(7))
        s1, s2 = sol.stage_shapes
        assert best == s1 == sol.tile_shape
        assert t[s1][0] == min(a for a, _ in t.values()) and t[s2][1] == min(b for _, b in t.values())
        for shapes in ((s1, s2), (6, 6), (6, 2)):
            sol.set_stage_shapes(*shapes)
            sol.set_state(s.state)
            sol.run(2)
            assert sol.stage_shapes == shapes
            assert np.array_equal(sol.get_state(), want)


def test_reported_shapes_on_the_host_build(on_host, oracle):
    _check_reports(oracle)


@pytest.mark.gpu
def test_reported_shapes(gpu, oracle):
    _check_reports(oracle)
