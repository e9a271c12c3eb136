"""The TV step and closing pass four columns per thread at the edges of their tiles: bitwise the
oracle's updateP / updateU sequence."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


def _handle(lib, W, H, D, precision=_abi.PREC_FP32):
    geo = _abi.make_geom(W, H, D, W, H, 2)
    prm = _abi.make_params(precision=precision)
    hd = C.c_void_p()
    _abi.check(lib.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))
    return hd


# one column group, a row of one tile and of two, ragged rows and planes, one row, one plane,
# more planes than a CTA marches
@pytest.mark.parametrize("shape", [(4, 1, 3), (128, 8, 33), (132, 17, 70), (260, 9, 1), (256, 1, 32), (380, 16, 65)])
def test_tv_four_columns_per_thread(engine, oracle_lib, shape):
    W, H, D = shape
    vol = (np.random.default_rng(W).standard_normal((D, H, W)) * 3.0).astype(np.float32)
    vol[:, :, : W // 3] = 0.5  # flat parts: zero differences and zero dual variables
    hd = _handle(engine, W, H, D)
    try:
        _abi.check(engine.tomo_set_volume(hd, vol.ctypes.data, 0, 0, H))
        _abi.check(engine.tomo_set_tvm(hd, 25.0, 1.0, 0.01, 4))
        _abi.check(engine.tomo_end_iteration(hd))
        got = np.empty_like(vol)
        _abi.check(engine.tomo_get_volume(hd, got.ctypes.data, 0, 0, H))
    finally:
        engine.tomo_destroy(hd)
    O.tv_denoise(vol, 25.0, 1.0, 0.01, 4)
    assert np.array_equal(got.view(np.uint32), vol.view(np.uint32))
