"""16-bit volumes packed from and unpacked into device buffers in one pass: bitwise what the copies
through host buffers give."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


def _handle(lib, W, H, D, precision=_abi.PREC_FP32):
    geo = _abi.make_geom(W, H, D, W, H, 2)
    prm = _abi.make_params(precision=precision)
    hd = C.c_void_p()
    _abi.check(lib.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))
    return hd


@pytest.mark.parametrize("precision", [_abi.PREC_FP16, _abi.PREC_BF16])
@pytest.mark.parametrize("shape, rows, shift", [((64, 9, 5), (0, 9), 0), ((72, 6, 3), (1, 5), 0), ((37, 4, 7), (0, 4), 0),
                                                ((64, 5, 4), (2, 3), 1)])
def test_device_copies_of_16_bit_volumes(engine, precision, shape, rows, shift):
    torch = pytest.importorskip("torch")
    W, H, D = shape
    y0, y1 = rows
    scale = 10.0 ** np.random.default_rng(1).integers(-3, 3, (1, H, 1))
    vol = (np.random.default_rng(W).standard_normal((D, H, W)) * scale).astype(np.float32)
    hd, other = _handle(engine, W, H, D, precision), _handle(engine, W, H, D, precision)
    try:
        _abi.check(engine.tomo_set_volume(hd, vol.ctypes.data, 0, 0, H))
        host = np.empty((D, y1 - y0, W), np.float32)
        _abi.check(engine.tomo_get_volume(hd, host.ctypes.data, 0, y0, y1))
        buf = torch.zeros(host.size + shift, dtype=torch.float32, device="cuda")
        torch.cuda.synchronize()
        _abi.check(engine.tomo_get_volume(hd, C.c_void_p(buf.data_ptr() + 4 * shift), 1, y0, y1))
        assert np.array_equal(buf.cpu().numpy()[shift:].view(np.uint32), host.ravel().view(np.uint32))
        # and in: a device buffer packs as a host one does
        src = torch.from_numpy(vol).cuda()
        torch.cuda.synchronize()
        _abi.check(engine.tomo_set_volume(other, C.c_void_p(src.data_ptr()), 1, 0, H))
        a, b = np.empty_like(vol), np.empty_like(vol)
        _abi.check(engine.tomo_get_volume(hd, a.ctypes.data, 0, 0, H))
        _abi.check(engine.tomo_get_volume(other, b.ctypes.data, 0, 0, H))
        assert np.array_equal(a.view(np.uint32), b.view(np.uint32))
    finally:
        engine.tomo_destroy(hd)
        engine.tomo_destroy(other)
