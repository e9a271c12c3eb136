"""16-bit volumes backprojected two rows per thread (large grids) and one row per thread (a few rows
at a time): the same bits."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu

W, H, D, N = 500, 257, 70, 100  # 8 x 2 x 129 CTAs of row pairs


@pytest.fixture(scope="module")
def series():
    return np.random.default_rng(1).standard_normal((N, H, W)).astype(np.float32)


@pytest.mark.parametrize("precision", [_abi.PREC_FP16, _abi.PREC_BF16])
@pytest.mark.parametrize("T", [1, 7, 16, 17, 32, 33, 64, 65, 100])
def test_row_pairs_equal_single_rows(engine, series, precision, T):
    vol = np.random.default_rng(2).standard_normal((D, H, W)).astype(np.float32)
    eul = np.ascontiguousarray([O.euler(0.0, a, 0.0) for a in np.linspace(-65, 65, N)], np.float64)
    out = []
    for ranges in ([(0, H)], [(y, min(y + 20, H)) for y in range(0, H, 20)]):
        geo, prm = _abi.make_geom(W, H, D, W, H, N), _abi.make_params(precision=precision)
        hd = C.c_void_p()
        _abi.check(engine.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))
        try:
            _abi.check(engine.tomo_load_series(hd, series.ctypes.data, 0, _abi.ptr(eul, C.c_double), None, None))
            _abi.check(engine.tomo_set_volume(hd, vol.ctypes.data, 0, 0, H))
            for t in range(T):
                _abi.check(engine.tomo_add_projection(hd, (37 * t) % N))
            for y0, y1 in ranges:
                _abi.check(engine.tomo_backproject(hd, y0, y1))
            v = np.empty((D, H, W), np.float32)
            _abi.check(engine.tomo_get_volume(hd, v.ctypes.data, 0, 0, H))
            out.append(v)
        finally:
            engine.tomo_destroy(hd)
    assert np.array_equal(out[0], out[1])
    assert not np.array_equal(out[0], vol)
