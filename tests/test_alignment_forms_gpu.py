"""Alignment in fixed-point coordinates and pairs of floats: the oracle's pixels for transforms whose
coordinates are whole, dyadic, nearly whole, out of the fixed-point range or of the image."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_parity_gpu import Handle
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


def _rot(deg, s=1.0):
    c, n = s * np.cos(np.radians(deg)), s * np.sin(np.radians(deg))
    return [c, n, -n, c]


TRANSFORMS = [
    [1, 0, 0, 1, 0, 0], [1, 0, 0, 1, 3, -2], [1, 0, 0, 1, 0.5, 2], [1, 0, 0, 1, 1.3, 2], [1, 0, 0, 1, -2, 0.7],
    [1, 0, 0, 1, 1 + 1e-9, -1e-12], _rot(90) + [0, 0], _rot(180) + [0, 0], _rot(1.3) + [0.4, -0.8],
    _rot(33, 1.4) + [2.1, 1.7], [1.01, 0.2, -0.1, 0.97, 0.3, 0.2], [1, 0, 0, 1, 20000.5, 0],
    _rot(5, 1e-3) + [0, 0], [0, 1, 1, 0, 0, 0], [0.5, 0, 0, 0.25, 0.75, 0], [1, 0, 0, 1, 500.25, 1],
]


@pytest.mark.parametrize("normalize", [False, True])
@pytest.mark.parametrize("w, h, kind", [(33, 9, "plain"), (64, 16, "nonfinite"), (257, 31, "plain"), (40, 12, "extreme"),
                                        (1, 1, "plain"), (1025, 3, "plain")])
def test_aligned_pixels_are_the_oracles(engine, oracle_lib, w, h, kind, normalize):
    rng = np.random.default_rng(w)
    n = len(TRANSFORMS)
    series = (rng.standard_normal((n, h, w)) * 3 + 1).astype(np.float32)
    if kind == "nonfinite":
        series[:, 3, 5], series[:, 7, 40], series[1::3, 9, 20] = np.nan, np.inf, -np.inf
    if kind == "extreme":
        series *= (10.0 ** rng.integers(-36, 37, (n, 1, 1))).astype(np.float32)
    T = np.array(TRANSFORMS, np.float64)
    stats = np.column_stack([series.reshape(n, -1).astype(np.float64).mean(1),
                             series.reshape(n, -1).astype(np.float64).std(1)])
    stats = np.where(np.isfinite(stats) & (stats != 0), stats, 1.0)
    eul = np.tile(np.eye(3).ravel(), (n, 1))
    case = dict(W=w, H=h, D=2, w=w, h=h, n=n, series=series, T=T, eul=eul)
    for fill in (_abi.FILL_NAN, _abi.FILL_NONE):
        hd = Handle(engine, case, fill=fill, normalize=normalize)
        try:
            _abi.check(engine.tomo_load_series(hd.h, series.ctypes.data, 0, _abi.ptr(eul, _abi.C.c_double),
                                               _abi.ptr(T, _abi.C.c_double),
                                               _abi.ptr(np.ascontiguousarray(stats), _abi.C.c_double)))
            for i in range(n):
                of = O.FILL_NAN if fill == _abi.FILL_NAN else O.FILL_NONE
                ref = O.align(series[i], T[i], normalize, stats[i, 0], stats[i, 1], of)
                raw = O.align(series[i], T[i], False, stats[i, 0], stats[i, 1], of).astype(np.float64)
                got = hd.slot(engine.tomo_get_aligned, i)
                same = (got == ref) | (np.isnan(got) & np.isnan(ref))
                fin = np.isfinite(ref)
                assert np.all(same[~fin]), (i, fill)
                # one float rounding apart, plus coordinates known to 2^-39 pixel, plus the
                # rounding of the normalised value
                top = np.abs(series[i][np.isfinite(series[i])]).astype(np.float64).max()
                tol = np.abs(raw[fin]) * 2.0 ** -23 + top * 2.0 ** -36 + 2.0 ** -149
                if normalize:
                    tol = tol / stats[i, 1] + np.abs(ref[fin].astype(np.float64)) * 2.0 ** -23
                assert np.all(np.abs(got[fin].astype(np.float64) - ref[fin]) <= tol), (i, fill)
        finally:
            hd.close()
