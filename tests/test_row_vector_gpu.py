"""The row-vector forward projector (eight rows per CTA) against the oracle at the sizes
where its cuts change: rows that do not fill a group of eight, columns off 16-byte
boundaries, widths that need column windows, depths that do not fill a chunk, one tilt to
more tilts than a CTA takes, steep tilts, rows and detectors larger than the volume, 16-bit
storage, fractional rows, and two passes over one CTA's rays."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import np_oracle as N
from oracle import oracle as O
from tests.cases import rel_l2
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu

# W, H, D, w, h, tilts, largest angle, scale, precision
FORMS = [
    (1, 3, 5, 4, 3, 2, 40.0, 1.0, "fp32"),
    (37, 1, 9, 37, 1, 1, 55.0, 1.0, "fp32"),
    (64, 8, 31, 64, 8, 3, 60.0, 1.0, "fp32"),
    (96, 17, 33, 130, 23, 19, 80.0, 1.0, "fp32"),
    (130, 9, 64, 101, 9, 7, 60.0, 1.0, "bf16"),
    (256, 15, 40, 256, 15, 17, 66.0, 1.0, "fp16"),
    (601, 10, 29, 601, 10, 6, 61.0, 1.0, "fp32"),
    (1304, 7, 50, 1304, 7, 18, 70.0, 1.0, "fp32"),
    (1000, 5, 21, 1000, 5, 9, 70.0, 1.0, "fp16"),
    (90, 12, 30, 180, 24, 11, 58.0, 2.0, "fp32"),
    (100, 20, 24, 80, 16, 5, 60.0, 0.8, "fp32"),
]


def _on_a_column(W, D, w, R, scale):
    """Rays that cross some plane on a whole column to within rounding.  The samples of the
    volume's last row are the raw voxel at floor(x), which jumps there: either neighbour is a
    rounding of the other, and the projection of that row says nothing."""
    i, z = np.arange(w)[:, None], np.arange(D)[None]
    x = ((i - (w - 1) / 2) / scale - R[0, 2] * (z - (D - 1) / 2)) / R[0, 0] + (W - 1) / 2
    return (np.abs(x - np.rint(x)) < 1e-8).any(1)[None, :]


def _last_row(g, H):
    """Projection rows that sample the volume's last row."""
    y = (np.arange(g.h) - g.pc[1]) / g.scale + g.vc[1]
    return (y >= H - 1) & (y < H)


@pytest.mark.parametrize("form", FORMS, ids=lambda f: f"{f[0]}x{f[1]}x{f[2]}-{f[5]}t-{f[8]}-s{f[7]}")
def test_projections_match_the_oracle(engine, oracle_lib, form):
    W, H, D, w, h, n, amax, scale, prec = form
    vol = np.random.default_rng(W + D).random((D, H, W), dtype=np.float32)
    eul = np.ascontiguousarray([O.euler_tilt_y(a) for a in (np.linspace(-amax, amax, n) if n > 1 else [amax])])
    geo = _abi.make_geom(W, H, D, w, h, n, scale=scale)
    prm = _abi.make_params(precision=_abi.precision_code(prec))
    hd = C.c_void_p()
    _abi.check(engine.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))
    try:
        ser = np.zeros((n, h, w), np.float32)
        _abi.check(engine.tomo_load_series(hd, ser.ctypes.data, 0, _abi.ptr(eul, C.c_double), None, None))
        _abi.check(engine.tomo_set_volume(hd, vol.ctypes.data, 0, 0, H))
        _abi.check(engine.tomo_get_volume(hd, vol.ctypes.data, 0, 0, H))  # as stored
        for i in range(n):
            _abi.check(engine.tomo_add_projection(hd, i))
        err = np.zeros(n)
        _abi.check(engine.tomo_project_and_difference(hd, 0.25, 0, H, _abi.ptr(err, C.c_double)))
        g = O.Geom(W, H, D, w, h, scale=scale)
        for i in range(n):
            got, norm = np.empty((h, w), np.float32), np.empty((h, w), np.float32)
            _abi.check(engine.tomo_get_projection(hd, i, _abi.ptr(got)))
            _abi.check(engine.tomo_get_norm(hd, i, _abi.ptr(norm)))
            ref, ref_norm = O.project(vol, g, eul[i])
            assert np.array_equal(np.isnan(got), np.isnan(ref)), i
            assert np.array_equal(norm, ref_norm), i
            # against the FP64 twin (the float oracle rounds positions to 24 bits, 3e-5 of a column
            # at x = 600): a float sum of up to 64 positive terms, a few ulps
            with np.errstate(divide="ignore", invalid="ignore"):
                d = np.nan_to_num((0.0 - got.astype(np.float64)) / ref_norm * 0.25)
            ref = N.project(vol, g, eul[i])[0]
            got = np.where(_on_a_column(W, D, w, eul[i], scale) & (_last_row(g, H)[:, None]), ref, got)
            assert rel_l2(got, ref) <= 1e-6, i
            assert abs(err[i] - (d * d).sum()) <= 2e-6 * (d * d).sum(), i
    finally:
        engine.tomo_destroy(hd)
