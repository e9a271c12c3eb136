"""Samples that are the raw voxel at floor(x) (the volume's last plane, its last column) ignore the
next column, also where that is NaN or infinite and the handle does not know of it (voxels written
through the device pointer, or overflowed in an iteration): the values of a handle that was given
the same volume through tomo_set_volume, whose projections run on the one-row form."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("W, H, D, w, h, n, amax, scale", [
    (64, 8, 31, 64, 8, 3, 60.0, 1.0), (601, 10, 29, 601, 10, 6, 61.0, 1.0), (1024, 9, 20, 1024, 9, 7, 66.0, 1.0),
    (90, 12, 30, 180, 24, 5, 58.0, 2.0), (40, 16, 24, 33, 16, 1, 0.0, 1.0)])
def test_nonfinite_neighbours_of_raw_voxels(engine, W, H, D, w, h, n, amax, scale):
    torch = pytest.importorskip("torch")
    rng = np.random.default_rng(W)
    vol = rng.random((D, H, W), dtype=np.float32)
    bad = vol.copy()
    bad[D - 1, 2:, [W // 2, W // 3]], bad[D - 1, :, 3] = np.nan, np.inf
    bad[D // 2, 1, W - 1], bad[D // 3, 3, W - 1], bad[D // 2, 4, 0] = np.inf, np.nan, -np.inf
    eul = np.ascontiguousarray([O.euler_tilt_y(a) for a in (np.linspace(-amax, amax, n) if n > 1 else [amax])])
    ser = np.zeros((n, h, w), np.float32)
    out = []
    for known in (True, False):
        geo, prm = _abi.make_geom(W, H, D, w, h, n, scale=scale), _abi.make_params()
        hd = C.c_void_p()
        _abi.check(engine.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))
        try:
            _abi.check(engine.tomo_load_series(hd, ser.ctypes.data, 0, _abi.ptr(eul, C.c_double), None, None))
            _abi.check(engine.tomo_set_volume(hd, (bad if known else vol).ctypes.data, 0, 0, H))
            if not known:
                dev = C.c_void_p()
                _abi.check(engine.tomo_volume_device_ptr(hd, C.byref(dev)))
                view = type("V", (), {"__cuda_array_interface__": dict(shape=(D, H, W), typestr="<f4", strides=None,
                                                                       data=(dev.value, False), version=3)})()
                torch.as_tensor(view, device="cuda").copy_(torch.from_numpy(bad))
                torch.cuda.synchronize()
            for i in range(n):
                _abi.check(engine.tomo_add_projection(hd, i))
            _abi.check(engine.tomo_project(hd, 0, H))
            p = np.empty((n, h, w), np.float32)
            for i in range(n):
                _abi.check(engine.tomo_get_projection(hd, i, _abi.ptr(p[i])))
            out.append(p)
        finally:
            engine.tomo_destroy(hd)
    ref, got = out
    fin = np.isfinite(ref)
    assert np.array_equal(fin, np.isfinite(got))
    assert np.array_equal(got[np.isinf(ref)], ref[np.isinf(ref)]) and np.isinf(ref).any()
    # sums of up to D terms below 1 (ray increments up to 1 / cos), in other orders
    assert np.max(np.abs(got[fin] - ref[fin])) <= D * D * 2.0 ** -23 / np.cos(np.radians(amax))
