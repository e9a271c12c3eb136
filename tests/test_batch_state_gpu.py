"""A batch whose members change between its iterations, without tomo_batch_set: the next iteration
runs on what the members hold now, as if the membership had been set again."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_parity_gpu import Handle
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu

# 1024 columns run in column windows whose widths and margins follow from the steepest tilt: the
# cut for 40 degrees holds 264 columns of a plane, 75 degrees need 301
W, H, D, N = 1024, 16, 40, 7


def _case(amax, seed):
    rng = np.random.default_rng(seed)
    eul = np.array([O.euler_tilt_y(a) for a in np.linspace(-amax, amax, N)])
    T = np.tile(np.array([1, 0, 0, 1, 0, 0], np.float64), (N, 1))
    return dict(W=W, H=H, D=D, w=W, h=H, n=N, eul=eul, T=T, series=rng.random((N, H, W), dtype=np.float32))


def _load(lib, hd, c):
    _abi.check(lib.tomo_load_series(hd.h, c["series"].ctypes.data, 0, _abi.ptr(np.ascontiguousarray(c["eul"]), C.c_double),
                                    None, None))
    hd.c = c


def _nonfinite(lib, hd):
    v = hd.volume()
    v[D - 1, :, 100], v[7, 3, 200], v[D // 2, 5, W - 1] = np.inf, np.nan, -np.inf
    hd.set_volume(v)


CHANGES = {
    "steeper series": lambda lib, hd: _load(lib, hd, _case(75.0, 2)),
    "flatter series": lambda lib, hd: _load(lib, hd, _case(5.0, 3)),
    "non-finite volume": _nonfinite,
    "centres": lambda lib, hd: _abi.check(lib.tomo_set_centers(
        hd.h, None, _abi.ptr(np.array([np.nan, (H - 1) / 2 + 1, np.nan, (H - 1) / 2 + 1]), C.c_double))),
    "positivity": lambda lib, hd: _abi.check(lib.tomo_set_positivity(hd.h, 1)),
    "tvm": lambda lib, hd: _abi.check(lib.tomo_set_tvm(hd.h, 25.0, 1.0, 0.01, 2)),
}


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("change", list(CHANGES))
def test_iterations_follow_a_members_changes(engine, change, use_graph):
    got = {}
    for again in (False, True):  # True: the membership is set again after the change
        hds = [Handle(engine, _case(40.0, 1)), Handle(engine, _case(60.0, 4))]
        b = C.c_void_p()
        _abi.check(engine.tomo_batch_create(C.byref(b)))
        try:
            arr = (C.c_void_p * 2)(*[h.h.value for h in hds])
            rel, upd, first = np.ones(2), np.array([0, 3], np.int32), np.array([2, 5], np.int32)

            def step():
                e = np.zeros((2, 5))
                _abi.check(engine.tomo_batch_iteration(b, _abi.ptr(rel, C.c_double), _abi.ptr(upd, C.c_int32),
                                                       _abi.ptr(first, C.c_int32), use_graph, _abi.ptr(e, C.c_double)))
                return e

            _abi.check(engine.tomo_batch_set(b, arr, 2))
            step()
            CHANGES[change](engine, hds[0])
            if again:
                _abi.check(engine.tomo_batch_set(b, arr, 2))
            e = step()
            got[again] = [h.volume() for h in hds] + [e]
        finally:
            engine.tomo_batch_destroy(b)
            for h in hds:
                h.close()
    for x, y in zip(got[False], got[True]):
        assert np.array_equal(x, y, equal_nan=True)
