"""The aligned series read where it lies: weighting straight from picked images, and fills that no
pixel takes."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


def _load(lib, series, T=None, fill=_abi.FILL_NAN, D=24):
    n, h, w = series.shape
    geo, prm = _abi.make_geom(w, h, D, w, h, n), _abi.make_params(fill=fill)
    hd = C.c_void_p()
    _abi.check(lib.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))
    eul = np.ascontiguousarray([O.euler(0.0, a, 0.0) for a in np.linspace(-60, 60, n)], np.float64)
    stats = np.column_stack([series.reshape(n, -1).mean(1), np.ones(n)]).astype(np.float64)
    _abi.check(lib.tomo_load_series(hd, series.ctypes.data, 0, _abi.ptr(eul, C.c_double),
                                    None if T is None else _abi.ptr(T, C.c_double), _abi.ptr(stats, C.c_double)))
    return hd


@pytest.mark.parametrize("w, h", [(64, 9), (50, 7), (33, 1)])
@pytest.mark.parametrize("picks", [(3, 0, 3), (5, 2), (4,)])
def test_weighting_of_picked_images(engine, w, h, picks):
    # a NaN in an image that is not picked sends the batch through the copies and their scan
    series = np.random.default_rng(w).standard_normal((6, h, w)).astype(np.float32)
    out = []
    for flagged in (False, True):
        s = series.copy()
        if flagged:
            s[1, h // 2, w // 2] = np.nan
        hd = _load(engine, s)
        try:
            _abi.check(engine.tomo_set_weighting(hd, _abi.WEIGHT_RADERMACHER, 0.5, None, None))
            for k in picks:
                _abi.check(engine.tomo_add_projection(hd, k))
            vols = []
            for _ in range(2):  # the second call weights the batch's own images again
                _abi.check(engine.tomo_backproject(hd, 0, h))
                v = np.empty((24, h, w), np.float32)
                _abi.check(engine.tomo_get_volume(hd, v.ctypes.data, 0, 0, h))
                vols.append(v)
            out.append(vols)
        finally:
            engine.tomo_destroy(hd)
    assert np.array_equal(out[0][0], out[1][0]) and np.array_equal(out[0][1], out[1][1])
    assert np.any(out[0][0])


@pytest.mark.parametrize("shift", [None, 0.0, 2.0, -0.25])
def test_a_changed_fill_gives_the_images_of_a_fresh_load(engine, shift):
    series = np.random.default_rng(2).standard_normal((3, 8, 20)).astype(np.float32)
    T = None if shift is None else np.array([[1, 0, 0, 1, shift, 0]] * 3, np.float64)
    for first, then in ((_abi.FILL_NAN, _abi.FILL_AVG), (_abi.FILL_NONE, _abi.FILL_NAN), (_abi.FILL_AVG, _abi.FILL_NONE)):
        a, b = _load(engine, series, T, first), _load(engine, series, T, then)
        try:
            _abi.check(engine.tomo_set_fill(a, then))
            for k in range(3):
                x, y = np.empty((8, 20), np.float32), np.empty((8, 20), np.float32)
                _abi.check(engine.tomo_get_aligned(a, k, _abi.ptr(x)))
                _abi.check(engine.tomo_get_aligned(b, k, _abi.ptr(y)))
                assert np.array_equal(x, y, equal_nan=True)
        finally:
            engine.tomo_destroy(a)
            engine.tomo_destroy(b)
