"""The forward projector's scratch under a memory limit: what was refused leaves the sums of the
scratch at hand, in more launches, bit for bit; a handle that cannot hold one tilt's sums runs the
one-row form; and memory that comes back is used again."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from oracle import oracle as O
from tests.test_parity_gpu import Handle
from tomoj_gb300 import _abi

pytestmark = pytest.mark.gpu

W, H, D, N = 200, 16, 96, 20
TILT = -(-D // 4) * W * H * 4  # bytes of one tilt's sums at most (chunks of four planes and more)


def _handle(lib, seed=3):
    rng = np.random.default_rng(seed)
    eul = np.array([O.euler_tilt_y(a) for a in np.linspace(-60, 60, N)])
    c = dict(W=W, H=H, D=D, w=W, h=H, n=N, eul=eul, T=np.tile(np.array([1, 0, 0, 1, 0, 0], np.float64), (N, 1)),
             series=rng.random((N, H, W), dtype=np.float32))
    return Handle(lib, c, vol=rng.random((D, H, W), dtype=np.float32))


def _project(lib, hd, tilts):
    _abi.check(lib.tomo_clear_projections(hd.h))
    for t in tilts:
        _abi.check(lib.tomo_add_projection(hd.h, t))
    err = np.zeros(len(tilts))
    _abi.check(lib.tomo_project_and_difference(hd.h, 0.3, 0, H, _abi.ptr(err, C.c_double)))
    return [hd.slot(lib.tomo_get_projection, k) for k in range(len(tilts))] + [err]


def _limit(lib, extra):
    """At most `extra` bytes more than now (None: no limit)."""
    _abi.check(lib.tomo_set_memory_limit(0 if extra is None else lib.tomo_memory_in_use() + extra))


def _same(a, b):
    return all(np.array_equal(x, y, equal_nan=True) for x, y in zip(a, b))


def test_refused_scratch_keeps_what_the_handle_holds(engine):
    hd = _handle(engine)
    try:
        free = _project(engine, hd, range(N))
    finally:
        hd.close()
    hd = _handle(engine)
    try:
        one = _project(engine, hd, [4])  # scratch of one tilt's sums
        held = engine.tomo_memory_in_use()
        _limit(engine, 0)
        for _ in range(2):
            assert _same(_project(engine, hd, range(N)), free)
            assert engine.tomo_memory_in_use() == held
        assert _same(_project(engine, hd, [4]), one)
        _limit(engine, None)
        assert _same(_project(engine, hd, range(N)), free)
        assert engine.tomo_memory_in_use() > held
    finally:
        _limit(engine, None)
        hd.close()


@pytest.mark.parametrize("tilts", [1, 3, 9])
def test_smaller_scratch_is_tried(engine, tilts):
    hd = _handle(engine)
    try:
        free = _project(engine, hd, range(N))
    finally:
        hd.close()
    hd = _handle(engine)
    try:
        _limit(engine, tilts * TILT)
        assert _same(_project(engine, hd, range(N)), free)
    finally:
        _limit(engine, None)
        hd.close()


def test_no_scratch_at_all(engine):
    hd = _handle(engine)
    try:
        free = _project(engine, hd, range(N))
    finally:
        hd.close()
    hd = _handle(engine)
    try:
        _limit(engine, 4096)
        got = _project(engine, hd, range(N))
    finally:
        _limit(engine, None)
        hd.close()
    for x, y in zip(got, free):
        ok = np.isfinite(y)
        # sums of up to D terms below 1 in other orders
        assert np.array_equal(ok, np.isfinite(x)) and np.allclose(x[ok], y[ok], rtol=D * 2.0 ** -22, atol=0)


@pytest.mark.parametrize("use_graph", [0, 1])
@pytest.mark.parametrize("update", [0, 7])
def test_iterations_under_a_limit(engine, update, use_graph):
    """OS-SART iterations of a handle, in row streams and of a batch whose scratch holds a few tilts' sums, or one
    update size's only (20 tilts in updates of 7: the last takes 6), equal those without a limit."""
    runs = {}
    for mode in ("handle", "streams", "batch"):
        for extra in (None, 4 * TILT, 4096):
            hd = _handle(engine)
            b = C.c_void_p()
            _abi.check(engine.tomo_batch_create(C.byref(b)))
            try:
                _project(engine, hd, [4])
                _limit(engine, extra)
                if mode == "batch":
                    _abi.check(engine.tomo_batch_set(b, (C.c_void_p * 1)(hd.h.value), 1))
                    for it in range(2):
                        first = np.array([engine.tomo_first_index(9, it, N)], np.int32)
                        _abi.check(engine.tomo_batch_iteration(b, _abi.ptr(np.ones(1), C.c_double),
                                                               _abi.ptr(np.array([update], np.int32), C.c_int32),
                                                               _abi.ptr(first, C.c_int32), use_graph, None))
                else:
                    _abi.check(engine.tomo_set_row_streams(hd.h, 3 if mode == "streams" else 1))
                    _abi.check(engine.tomo_run_ossart(hd.h, 2, 1.0, update, 9, 0, H, use_graph, None))
                runs[mode, extra] = hd.volume()
            finally:
                _limit(engine, None)
                engine.tomo_batch_destroy(b)
                hd.close()
    for v in runs.values():
        assert np.array_equal(v, runs["handle", None])


@pytest.mark.parametrize("kind, update, precision", [("SIRT", 0, "fp32"), ("OS-SART", 7, "fp32"), ("TVM", 0, "fp32"),
                                                     ("TVM", 0, "fp16"), ("OS-SART", 3, "bf16"), ("WBP", 0, "fp32")])
def test_request_bytes_hold_the_footprint(engine, kind, update, precision):
    """Admission counts what a request takes, the projector's scratch included, and the scratch is
    there when the request is admitted: its iterations allocate nothing more."""
    from tomoj_gb300.serving import WBP, EngineAdapter, Request, request_bytes
    rng = np.random.default_rng(1)
    req = Request(0, 0.0, kind, rng.random((41, 64, 256), dtype=np.float32), np.linspace(-60, 60, 41), 256, 64, 128,
                  n_iter=2, update=update, precision=_abi.precision_code(precision))
    eng = EngineAdapter(lanes=1)
    base = engine.tomo_memory_in_use()
    hd = eng.create(req)
    try:
        admitted = engine.tomo_memory_in_use() - base
        if kind == WBP:
            eng.run_wbp(hd, req)
        else:
            eng.set_members([hd])
            for it in range(2):
                eng.iterate([hd], [req], [it])
            eng.set_members([])
        used = engine.tomo_memory_in_use() - base
    finally:
        eng.destroy(hd)
        eng.close()
    assert used == admitted
    assert used <= request_bytes(req) <= used * 1.05 + (1 << 20), (used, request_bytes(req))
