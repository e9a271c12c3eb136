"""The projector's closing pass over four rows at a time (many rows) and one row at a time (few):
the same projections, norms, differences and residuals."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import np_oracle as N
from oracle import oracle as O
from tests.test_row_vector_gpu import _on_a_column
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w, h, n", [(16, 515, 40), (130, 1023, 11), (700, 66, 150)])
def test_rows_in_groups_equal_single_rows(engine, oracle_lib, w, h, n):
    rng = np.random.default_rng(w)
    D = 12
    vol = rng.standard_normal((D, h, w)).astype(np.float32)
    series = rng.standard_normal((n, h, w)).astype(np.float32)
    series[:, 3, w // 2] = np.nan
    series[::2, 5, 0] = 1e30
    eul = np.ascontiguousarray([O.euler(0.0, a, 0.0) for a in np.linspace(-66, 66, n)], np.float64)
    geo, prm = _abi.make_geom(w, h, D, w, h, n), _abi.make_params()
    hd = C.c_void_p()
    _abi.check(engine.tomo_create(C.byref(geo), C.byref(prm), C.byref(hd)))

    def run(batch):
        _abi.check(engine.tomo_clear_projections(hd))
        for t in batch:
            _abi.check(engine.tomo_add_projection(hd, t))
        err = np.zeros(len(batch))
        _abi.check(engine.tomo_project_and_difference(hd, 0.37, 0, h, _abi.ptr(err, C.c_double)))
        out = []
        for k in range(len(batch)):
            for fn in (engine.tomo_get_projection, engine.tomo_get_norm, engine.tomo_get_difference):
                x = np.empty((h, w), np.float32)
                _abi.check(fn(hd, k, _abi.ptr(x)))
                out.append(x)
        return out, err

    try:
        _abi.check(engine.tomo_load_series(hd, series.ctypes.data, 0, _abi.ptr(eul, C.c_double), None, None))
        _abi.check(engine.tomo_set_volume(hd, vol.ctypes.data, 0, 0, h))
        whole, err = run(list(range(n)))
        for t in (0, n // 3, n - 1):
            one, e1 = run([t])
            # a projection's own plan cuts its rays into other segments: sums of D terms differ by
            # their order only; norms are exact
            assert np.array_equal(one[1], whole[3 * t + 1])
            ok = np.isfinite(one[0])
            assert np.array_equal(ok, np.isfinite(whole[3 * t]))
            assert np.max(np.abs(one[0][ok] - whole[3 * t][ok])) <= D * 2.0 ** -23 * np.abs(one[0][ok]).max()
            ref, ref_norm = O.project(vol, O.Geom(w, h, D, w, h), eul[t])
            assert np.array_equal(np.isnan(ref), ~ok)
            # the FP64 twin (the float oracle rounds positions to 24 bits), but for rays on a whole
            # column of the volume's last row
            twin = N.project(vol, O.Geom(w, h, D, w, h), eul[t])[0]
            ok &= ~(_on_a_column(w, D, w, eul[t], 1.0) & (np.arange(h) == h - 1)[:, None])
            assert np.max(np.abs(twin[ok] - whole[3 * t][ok])) <= D * 2.0 ** -23 * np.abs(twin[ok]).max()
            ok = np.isfinite(whole[3 * t])
            d = np.where(np.isnan(series[t]) | ~ok, 0, (series[t] - whole[3 * t]) / np.where(ok, ref_norm, 1) * 0.37)
            assert np.allclose(whole[3 * t + 2], d, rtol=1e-6, atol=1e-6)
            sq = np.sum(whole[3 * t + 2].astype(np.float64) ** 2)
            assert abs(err[t] - sq) <= 1e-6 * sq and abs(e1[0] - err[t]) <= 1e-5 * sq
    finally:
        engine.tomo_destroy(hd)
