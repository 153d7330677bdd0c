"""The single-precision minmod's bit form against the reference's formula
sign_x * max(min(|x|, sign_x * y), EPS) (minmod.hpp:6-16) with its own min
and max, on every pairing of ordinary, huge, tiny, equal, zero, infinite and
NaN arguments."""
import ctypes
from pathlib import Path

import numpy as np
import pytest

from host_build import EMU, link, shim_dir

HERE = Path(__file__).resolve().parent


@pytest.mark.parametrize("eps", [1e-20, 1e-3, 0.0])
def test_float_minmod_is_the_reference_formula(tmp_path, eps):
    d = shim_dir(tmp_path)
    src = d / "minmod_host.cpp"
    src.write_text('#include "physics.cuh"\n'
                   'extern "C" void host_minmod(int n, const float *x, const float *y, float eps, float *r)\n'
                   '{ for (int k = 0; k < n; ++k) r[k] = rmhd2d::minmod(x[k], y[k], eps); }\n')
    lib = link(d, [], [src], "libminmod.so", (EMU,))
    rng = np.random.default_rng(1)
    v = np.concatenate([rng.standard_normal(200), 10.0 ** rng.uniform(-30, 30, 200) * rng.choice([-1, 1], 200),
                        [0.0, -0.0, 1.0, -1.0, np.inf, -np.inf, np.nan, 1e-20, -1e-20, 3e38, -3e38]]).astype(np.float32)
    x, y = (np.ascontiguousarray(a.ravel()) for a in np.meshgrid(v, v))
    r = np.zeros_like(x)
    P = ctypes.POINTER(ctypes.c_float)
    lib.host_minmod(x.size, x.ctypes.data_as(P), y.ctypes.data_as(P), ctypes.c_float(eps), r.ctypes.data_as(P))
    e = np.float32(eps)
    with np.errstate(invalid="ignore"):
        s = np.where(x > 0, np.float32(1), np.where(x < 0, np.float32(-1), np.float32(0)))
        ax, sy = np.abs(x), s * y
        sy = np.where(s == 0, np.float32(0) * y, sy)
        m = np.where(sy < ax, sy, ax)
        m = np.where(m < e, e, m)
        want = s * m
        want = np.where(np.isnan(x), np.float32(np.nan), want)
    assert np.array_equal(r, want, equal_nan=True)
