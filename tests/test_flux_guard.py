"""The exact HLLD flux's common path forms only the selected candidate and
tests fewer values than the candidates hold: wherever it accepts an
interface, its flux is the reference's weighted sum of six bit for bit, from
ordinary states to values next to the guard's limits, zeros, negative
pressures and densities, infinities and NaN."""
import ctypes
from pathlib import Path

import numpy as np
import pytest

from host_build import EMU, link, shim_dir

HERE = Path(__file__).resolve().parent


@pytest.fixture(scope="module")
def lib(tmp_path_factory):
    d = shim_dir(tmp_path_factory.mktemp("fluxguard"))
    return link(d, [], [HERE / "flux_guard_host.cpp"], "libfluxguard.so", (EMU,))


def _states(kind, n, rng):
    """(L, R) of n interfaces with one normal B."""
    s = rng.standard_normal((2, n, 8))
    s[..., 0] = np.exp(s[..., 0])
    s[..., 7] = np.exp(s[..., 7])
    if kind == "supersonic":
        s[..., 1] *= 30.0
    elif kind == "flat":          # zeros and equal sides, as uniform flows have
        s[..., 2:7] *= rng.integers(0, 2, (2, n, 5))
        s[1][rng.random(n) < 0.5] = s[0][rng.random(n) < 0.5][0]
    elif kind == "limits":        # one value next to 2^+-240 or 2^+-400
        k, side = rng.integers(0, 8, n), rng.integers(0, 2, n)
        e = rng.choice([-400, -240, -120, 79, 80, 119, 120, 160, 239, 240, 241, 400], n) + rng.integers(-1, 2, n)
        s[side, np.arange(n), k] = np.ldexp(1.0 + rng.random(n), e)
    elif kind == "all_large":
        s *= np.ldexp(1.0, rng.integers(-130, 131, (2, n, 8)))
    elif kind == "broken":
        k, side = rng.integers(0, 8, n), rng.integers(0, 2, n)
        s[side, np.arange(n), k] = rng.choice([0.0, -0.0, -1.0, 1e80, np.inf, -np.inf, np.nan], n)
    s[1, :, 4] = s[0, :, 4]
    return np.ascontiguousarray(s[0]), np.ascontiguousarray(s[1])


@pytest.mark.parametrize("kind,least", [("ordinary", 0.99), ("supersonic", 0.9), ("flat", 0.5), ("limits", 0.01),
                                        ("all_large", 0.0), ("broken", 0.0)])
def test_accepted_fluxes_are_the_full_sum(lib, kind, least):
    n = 200_000
    L, R = _states(kind, n, np.random.default_rng(3))
    sel, full, taken = np.zeros((n, 8)), np.zeros((n, 8)), np.zeros(n, dtype=np.int32)
    D, I = ctypes.POINTER(ctypes.c_double), ctypes.POINTER(ctypes.c_int)
    lib.host_fluxes(n, L.ctypes.data_as(D), R.ctypes.data_as(D), ctypes.c_double(5.0 / 3.0), ctypes.c_double(1e-20),
                    sel.ctypes.data_as(D), full.ctypes.data_as(D), taken.ctypes.data_as(I))
    t = taken.astype(bool)
    assert t.mean() >= least
    assert np.all(np.isfinite(full[t]))
    # f4 is identically 0 and is not formed by either path's caller
    use = [0, 1, 2, 3, 5, 6, 7]
    assert np.array_equal(sel[t][:, use].view(np.uint64), full[t][:, use].view(np.uint64))
