"""Alignment at the far end of wide images: fixed-point coordinates as exact there as at the first
column, seen where neighbours cancel (columns of alternating sign, sampled half way)."""
from __future__ import annotations

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_parity_gpu import Handle
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu


def _scale(near, at):
    """A scale near `near` whose inverse lies just beside the middle between two multiples of 2^-48."""
    for k in range(1, 2000):
        s = near + k * 1e-7
        r = (1.0 / s) * 2.0 ** 48
        if abs(r - np.rint(r)) > 0.45 and (r > np.rint(r)) == at:
            return s
    raise AssertionError


@pytest.mark.parametrize("w, h", [(4096, 24), (2047, 65)])
def test_cancelling_neighbours_far_out(engine, oracle_lib, w, h):
    T = np.array([[_scale(s, at), 0, 0, 1, 0.3, 0] for s in (1.004, 1.05, 1.3) for at in (False, True)])
    n, A = len(T), 8.0
    sign = np.where(np.arange(w) % 2 == 0, A, -A)
    series = np.ascontiguousarray(np.broadcast_to(sign, (n, h, w)), np.float32)
    case = dict(W=16, H=h, D=2, w=w, h=h, n=n, series=series, T=T, eul=np.tile(np.eye(3).ravel(), (n, 1)))
    hd = Handle(engine, case, fill=_abi.FILL_NONE)
    try:
        for i in range(n):
            ref = O.align(series[i], T[i], False, 0.0, 1.0, O.FILL_NONE).astype(np.float64)
            got = hd.slot(engine.tomo_get_aligned, i).astype(np.float64)
            # the reference's coordinate: two products and three sums below 2^12, each rounded to 2^-42;
            # here 2^-47; slope 2 A, sums to 2^-44 A, one rounding of either result
            tol = np.abs(ref) * 2.0 ** -23 + 2 * A * (5 * 2.0 ** -42 + 2.0 ** -47) + A * 2.0 ** -44
            assert np.all(np.abs(got - ref) <= tol), (i, np.max(np.abs(got - ref) / tol))
    finally:
        hd.close()
