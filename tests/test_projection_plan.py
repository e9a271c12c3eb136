"""The cut of a forward projection into CTAs (host code): the same as simulating every candidate grid
would choose, wide enough for every column its rays sample, and chosen in a small part of the time of
the smallest projection, which waits for it on a handle's first call."""
from __future__ import annotations

import ctypes as C
import time

import numpy as np
import pytest

from oracle import oracle as O
from tomoj_gb300 import _abi

# W, H, D, w, h, tilts, largest angle, update, scale, precision -> planes per chunk and segment, segments,
# windows, columns of a plane buffer, tilts per CTA, as chosen by simulating all candidates (152 SMs)
PLANS = [
    ((128, 32, 128, 128, 32, 41, 60.0, 7, 1.0, 0), (6, 6, 22, 1, 136, 7)),
    ((333, 67, 150, 333, 67, 41, 60.0, 1, 1.0, 0), (6, 12, 13, 1, 344, 1)),
    ((256, 64, 256, 256, 64, 61, 60.0, 61, 1.0, 0), (8, 80, 4, 1, 264, 13)),
    ((512, 256, 512, 512, 256, 61, 60.0, 7, 1.0, 0), (4, 112, 5, 1, 520, 7)),
    ((2048, 512, 2048, 2048, 512, 121, 60.0, 121, 1.0, 0), (4, 68, 31, 8, 528, 11)),
    ((1024, 1024, 256, 1024, 1024, 61, 60.0, 61, 1.0, 2), (4, 112, 3, 6, 520, 16)),
    ((512, 512, 128, 512, 512, 41, 60.0, 5, 1.0, 0), (4, 68, 2, 1, 520, 5)),
    ((256, 64, 256, 128, 32, 41, 60.0, 41, 0.5, 0), (6, 24, 11, 1, 264, 14)),
    ((90, 12, 30, 180, 24, 11, 58.0, 11, 2.0, 0), (4, 4, 8, 1, 96, 11)),
    ((1304, 7, 50, 1304, 7, 18, 70.0, 18, 1.0, 0), (4, 8, 7, 5, 496, 9)),
    ((37, 1, 9, 37, 1, 1, 55.0, 1, 1.0, 0), (8, 16, 1, 1, 48, 1)),
    ((4000, 300, 900, 4000, 300, 50, 66.0, 10, 1.0, 0), (4, 28, 33, 14, 536, 10)),
    ((64, 5, 20000, 64, 5, 9, 50.0, 9, 1.0, 0), (8, 136, 148, 1, 72, 9)),
    ((24, 12, 1537, 24, 12, 2, 30.0, 2, 1.0, 0), (8, 32, 49, 1, 32, 2)),
    ((757, 2, 852, 757, 2, 102, 70.0, 53, 1.0, 0), (4, 24, 36, 3, 536, 11)),
]


def _call(engine, W, H, D, w, h, n, amax, update, scale, prec):
    geo = _abi.make_geom(W, H, D, w, h, n, scale=scale)
    eul = np.ascontiguousarray([O.euler_tilt_y(a) for a in (np.linspace(-amax, amax, n) if n > 1 else [amax])])
    out = np.zeros(8, np.int64)
    args = (C.byref(geo), prec, _abi.ptr(eul, C.c_double), update, _abi.ptr(out, C.c_int64))

    def call():
        _abi.check(engine.tomo_projection_plan(*args))
    call.keep = (geo, eul)
    return call, out


@pytest.fixture(autouse=True)
def no_gpu():
    torch = pytest.importorskip("torch")
    if torch.cuda.is_available():
        pytest.skip("the plans are those for 152 multiprocessors")


@pytest.mark.parametrize("case, plan", PLANS)
def test_plans(engine, case, plan):
    call, out = _call(engine, *case)
    call()
    assert tuple(out[:6]) == plan
    W, H, D, w, h, n, amax, update, scale, _ = case
    assert out[7] == 4 * out[2] * w * h * out[6] and 1 <= out[6] <= min(update, n)
    zc, seg, nseg, nwin, pitch, _ = plan
    if nwin == 1:
        assert pitch >= W + 3
        return
    # every chunk of a middle window: the tilts' fan from the segment's middle plane, a block of 32
    # rays, the neighbour column and the rounding of each bound
    step, space, xw = np.tan(np.radians(amax)), 1 / np.cos(np.radians(amax)) / scale, -(-W // nwin)
    for z_lo in range(0, D, seg):
        z_hi = min(D, z_lo + seg)
        zm = (z_lo + z_hi) // 2
        for z0 in range(z_lo, z_hi, zc):
            far = max(abs(z0 - zm), abs(min(z0 + zc, z_hi) - 1 - zm)) * step
            assert 2 * np.ceil(far) + xw + np.ceil(31 * space) + 6 <= pitch, (z0, far)


def test_a_plan_takes_microseconds(engine):
    # simulating all candidates took 118 us here; a projection of this size takes about 100
    call, _ = _call(engine, *PLANS[2][0])
    best = 1.0
    for _ in range(300):
        t = time.perf_counter()
        call()
        best = min(best, time.perf_counter() - t)
    assert best < 60e-6, best


def test_request_bytes_count_the_projectors_scratch(engine):
    from tomoj_gb300.serving import SIRT, WBP, Request, request_bytes
    angles = np.linspace(-60, 60, 41)
    series = np.lib.stride_tricks.as_strided(np.zeros(1, np.float32), (41, 256, 512), (0, 0, 0))
    wbp, sirt = [request_bytes(Request(0, 0.0, k, series, angles, 512, 256, 512)) for k in (WBP, SIRT)]
    call, out = _call(engine, 512, 256, 512, 512, 256, 41, 60.0, 0, 1.0, 0)
    call()
    assert sirt - wbp == out[7] > 0
    assert wbp >= 4 * (512 * 256 * 512 + 6 * 41 * 256 * 512)
