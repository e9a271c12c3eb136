"""Row filter passes at every transform length: one projection at zero tilt (whose backprojection
is the filtered image itself) against the 64-bit transform of the same mask."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import np_oracle as N
from oracle import oracle as O
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows", [1, 3, 4])
@pytest.mark.parametrize("w", [1, 2, 3, 4, 5, 8, 9, 16, 31, 32, 33, 64, 100, 128, 200, 256, 512, 513, 750, 1024, 1500,
                               2048, 2049, 4095, 4096])
def test_filtered_rows_match_the_64_bit_transform(engine, oracle_lib, w, rows):
    angles = np.array([-40.0, -13.0, 0.0, 21.0, 55.0])
    n, at = angles.size, 2
    series = np.zeros((n, rows, w), np.float32)
    series[at] = np.random.default_rng(w).standard_normal((rows, w)) + 0.5
    eul = np.ascontiguousarray([O.euler(0.0, a, 0.0) for a in angles], np.float64)
    geo, prm = _abi.make_geom(w, rows, 1, w, rows, n), _abi.make_params(fill=_abi.FILL_NAN)
    hd = C.c_void_p()
    _abi.check(engine.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))
    try:
        _abi.check(engine.tomo_load_series(hd, series.ctypes.data, 0, _abi.ptr(eul, C.c_double), None, None))
        _abi.check(engine.tomo_set_weighting(hd, _abi.WEIGHT_RADERMACHER, 0.5, _abi.ptr(angles, C.c_double), None))
        _abi.check(engine.tomo_run_wbp(hd, 0, rows))
        got = np.empty((1, rows, w), np.float32)
        _abi.check(engine.tomo_get_volume(hd, got.ctypes.data, 0, 0, rows))
    finally:
        engine.tomo_destroy(hd)
    mask = O.weighting_mask(w, rows, angles, np.zeros(n), 0.5 * w)
    ref = N.weighting_apply(series[at], mask)
    # two transforms of at most M points, each level rounding at most twice per component, the
    # spectrum and its product; a factor 4 for the doubled row and the kernel's own spectrum
    log_m = int(np.ceil(np.log2(2 * w)))
    tol = 2.0 ** -24 * (2 * log_m + 8) * 4 * np.abs(mask).max() * np.linalg.norm(series[at])
    assert np.linalg.norm(got[0] - ref) <= tol
