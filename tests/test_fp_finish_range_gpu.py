"""Differences and squared errors far outside the range in which the projector's closing pass works
in pairs of floats, and factors outside the range of a float: the double product of the residual and
the factor, rounded once for the difference and squared in full for the error."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w, h, n", [(100, 6, 3), (300, 5, 2), (16, 515, 40)])
@pytest.mark.parametrize("level", [1.0, 1e-18, 1e18, 1e-30, 1e25])
def test_errors_of_any_magnitude(engine, w, h, n, level):
    rng = np.random.default_rng(w)
    D = 9
    vol = (rng.random((D, h, w)) * level).astype(np.float32)
    ser = (rng.random((n, h, w)) * 9 * level).astype(np.float32)
    ser[:, 0, w // 2], ser[0, 1, 1] = np.nan, 0
    eul = np.ascontiguousarray([O.euler_tilt_y(a) for a in np.linspace(-60, 60, n)])
    geo, prm = _abi.make_geom(w, h, D, w, h, n), _abi.make_params()
    hd = C.c_void_p()
    _abi.check(engine.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))
    try:
        _abi.check(engine.tomo_load_series(hd, ser.ctypes.data, 0, _abi.ptr(eul, C.c_double), None, None))
        _abi.check(engine.tomo_set_volume(hd, vol.ctypes.data, 0, 0, h))
        for t in range(n):
            _abi.check(engine.tomo_add_projection(hd, t))
        for factor in (0.37, 1e-45, 3e-41, 1e60, 0.0, -2e39, 1e-19):
            err = np.zeros(n)
            _abi.check(engine.tomo_project_and_difference(hd, factor, 0, h, _abi.ptr(err, C.c_double)))
            for t in range(n):
                out = []
                for fn in (engine.tomo_get_projection, engine.tomo_get_norm, engine.tomo_get_difference):
                    x = np.empty((h, w), np.float32)
                    _abi.check(fn(hd, t, _abi.ptr(x)))
                    out.append(x)
                proj, norm, diff = out
                ok = np.isfinite(proj) & ~np.isnan(ser[t])
                with np.errstate(all="ignore"):
                    v = np.where(ok, ((ser[t] - proj) / norm).astype(np.float32).astype(np.float64) * factor, 0.0)
                    d = v.astype(np.float32)
                    sq = (v * v).sum()
                fin = np.isfinite(d)
                assert np.array_equal(d[~fin], diff[~fin]), (t, factor)
                # once rounded from 48 bits or more: the same float but for ties
                assert np.all(np.abs(d[fin] - diff[fin]) <= np.spacing(np.abs(d[fin]))), (t, factor)
                assert np.mean(d == diff) > 0.999, (t, factor)
                # terms to 2^-46, sums of w of them
                assert abs(err[t] - sq) <= sq * (w + 16) * 2.0 ** -46, (t, factor)
    finally:
        engine.tomo_destroy(hd)
