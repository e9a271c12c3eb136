"""Workloads of the reconstruction engine for timing and accuracy comparisons.

Each case is one call, or one job of a few calls, through the package's public entry
points (the Projector mirror or the C ABI binding), as a program that reconstructs
tilt-series makes it.  `listed` are fixed sizes, `draw` gives further sizes of the same
ranges, `exact` is the same computation in plain 64-bit torch.
"""
from __future__ import annotations

import ctypes as C
import math

import numpy as np
import torch

from tomoj_gb300 import _abi
from tomoj_gb300.projector import CompressedSensingProjector, VoxelProjector3D
from tomoj_gb300.reconstruction import TomoReconstruction2
from tomoj_gb300.tiltseries import TiltSeries

DEV = "cuda"


# --- cases --------------------------------------------------------------------------------

def _case(kind, W, H, D, n, amax=60.0, w=None, h=None, iters=1, update=0, relax=1.0, precision="fp32",
          positivity=False, misalign=False, weight="none", tv=0, series=1, name=None):
    c = dict(kind=kind, W=W, H=H, D=D, w=w or W, h=h or H, n=n, amax=amax, iters=iters, update=update, relax=relax,
             precision=precision, positivity=positivity, misalign=misalign, weight=weight, tv=tv, series=series)
    if name:
        c["name"] = name
    return c


def listed():
    return [
        # the smallest call: one subset of a small preview reconstruction driven through the
        # Projector surface, as a host program that owns the iteration loop makes it
        _case("update", 128, 32, 128, 41, update=7, relax=1.0, name="update_128"),
        # a whole small job: ramp WBP, then ten SIRT iterations from its volume
        _case("job", 256, 64, 256, 61, iters=10, weight="ramp", name="sirt_256"),
        # the drop-in job at 512: misaligned series, Hamming WBP, then OS-SART iterations
        # in subsets of seven (two of the twenty iterations of a full run)
        _case("job", 512, 256, 512, 61, iters=2, update=7, misalign=True, weight="hamming", name="ossart_512"),
        # one SIRT iteration at the largest volume
        _case("iterate", 2048, 512, 2048, 121, name="sirt_2048"),
        # a served request: a 1024 x 1024 series into a thin section stored in 16 bits
        _case("iterate", 1024, 1024, 256, 61, precision="fp16", name="sirt_1024_fp16"),
        # a served OS-SART request of a thin section
        _case("iterate", 512, 512, 128, 41, update=5, name="ossart_512_thin"),
        # weighted backprojection of a series of odd sizes (the backprojection direction alone)
        _case("job", 750, 333, 201, 73, amax=66.3, iters=0, weight="radermacher", name="wbp_odd"),
        # ART (one projection per update) with positivity, odd sizes
        _case("iterate", 333, 67, 150, 41, amax=57.7, update=1, relax=0.3, positivity=True, name="art_odd"),
        # one total-variation regularised iteration
        _case("iterate", 512, 256, 512, 41, tv=5, relax=1.0, name="tvm_512"),
        # reconstruction at half the projections' sampling (projections twice as wide)
        _case("iterate", 256, 128, 256, 61, w=512, h=256, name="half_scale_256"),
        # many independent series of mixed sizes iterated together
        _case("batch", 512, 64, 160, 61, series=12, name="batch_mixed"),
        # the compressed-sensing filter that ends an iteration
        _case("wavelet", 256, 64, 256, 3, name="wavelet_256"),
    ]


def _log(rng, a, b):
    return int(round(math.exp(rng.uniform(math.log(a), math.log(b)))))


def draw(rng):
    kind = rng.choice(["update", "sirt", "sirt", "fp16", "ossart", "ossart", "wbp", "art", "tvm", "half", "batch",
                       "wavelet"])
    amax = round(rng.uniform(50.0, 70.0), 2)
    for _ in range(1000):
        W, D = _log(rng, 96, 2048), _log(rng, 64, 1024)
        H = _log(rng, 24, 1024)
        n = rng.choice([41, 61, 73, 81, 121])
        if rng.random() < 0.5:
            W, D = 16 * (W // 16), 16 * (D // 16)
        nv = W * H * D
        if kind == "update" and 4e5 <= nv <= 2e7:
            return _case("update", W, H, D, n, amax, update=rng.randint(3, 12))
        if kind == "sirt" and 4e6 <= nv and nv * n <= 8e10:
            it = 1 if nv * n > 1e10 else rng.randint(1, 5)
            return _case("job" if it > 1 else "iterate", W, H, D, n, amax, iters=it,
                         weight="ramp" if it > 1 else "none")
        if kind == "fp16" and 1e7 <= nv and nv * n <= 6e10:
            return _case("iterate", W, H, D, n, amax, precision="fp16")
        if kind == "ossart" and 4e6 <= nv and nv * n <= 3e10:
            return _case("iterate", W, H, D, n, amax, update=rng.randint(4, 13), misalign=rng.random() < 0.5)
        if kind == "wbp" and 4e6 <= nv and nv * n <= 3e10:
            return _case("job", W, H, D, n, amax, iters=0, weight=rng.choice(["radermacher", "hamming"]))
        if kind == "art" and 1e6 <= nv <= 2e7:
            return _case("iterate", W, H, D, n, amax, update=1, relax=0.3, positivity=True)
        if kind == "tvm" and 4e6 <= nv <= 2e8:
            return _case("iterate", W, H, D, n, amax, tv=rng.randint(3, 8))
        if kind == "half" and 1e6 <= nv <= 3e7 and W <= 1024:
            return _case("iterate", W, H, D, n, amax, w=2 * W, h=2 * H)
        if kind == "batch":
            return _case("batch", 512, rng.choice([32, 48, 64]), 160, 61, amax, series=rng.randint(4, 16))
        if kind == "wavelet":
            return _case("wavelet", 64 * rng.randint(2, 8), 32 * rng.randint(1, 4), 32 * rng.randint(2, 8), 3, amax)
    return _case("update", 128, 32, 128, 41, amax, update=7)


def _members(case):
    """The series of a mixed batch: widths, thicknesses and tilt counts of the batched workload."""
    g = np.random.Generator(np.random.PCG64(1000 + case["series"]))
    out = []
    for _ in range(case["series"]):
        W = int(g.choice([256, 384, 512, 768, 1024]))
        D, n = int(g.integers(64, 257)), int(g.choice([41, 61, 81, 121]))
        out.append(_case("iterate", W, case["H"], D, n, round(float(g.uniform(50, 70)), 2)))
    return out


# --- inputs --------------------------------------------------------------------------------

def _angles(case):
    return np.linspace(-case["amax"], case["amax"], case["n"])


def _eulers(angles):
    a = np.deg2rad(np.asarray(angles, np.float64))
    e = np.zeros((a.size, 3, 3))
    e[:, 0, 0], e[:, 0, 2], e[:, 1, 1], e[:, 2, 0], e[:, 2, 2] = np.cos(a), -np.sin(a), 1.0, np.sin(a), np.cos(a)
    return e


def _transforms(case, seed):
    """Per-tilt rotation up to a degree and shifts up to five pixels (flat affine matrices)."""
    g = np.random.Generator(np.random.PCG64(seed + 77))
    T = np.zeros((case["n"], 6))
    for i in range(case["n"]):
        r = math.radians(g.uniform(-1.0, 1.0)) if case["misalign"] else 0.0
        t = g.uniform(-5.0, 5.0, 2) if case["misalign"] else (0.0, 0.0)
        T[i] = (math.cos(r), math.sin(r), -math.sin(r), math.cos(r), t[0], t[1])
    return T


def _series(case, seed, device=DEV):
    """Noisy projections of a phantom of random ellipsoids (line integrals in closed form),
    float32 (n, h, w); misaligned images are taken at the transformed coordinates."""
    W, H, D, w, h, n = (case[k] for k in ("W", "H", "D", "w", "h", "n"))
    g = np.random.Generator(np.random.PCG64(seed))
    s = w / W
    ang = np.deg2rad(_angles(case))
    T = _transforms(case, seed)
    f32 = dict(dtype=torch.float32, device=device)
    I = (torch.arange(w, **f32) - w / 2.0)[None, None, :]
    J = (torch.arange(h, **f32) - h / 2.0)[None, :, None]

    def per_tilt(v):
        return torch.as_tensor(np.asarray(v, np.float64), **f32)[:, None, None]

    if case["misalign"]:
        u = per_tilt(T[:, 0]) * I + per_tilt(T[:, 2]) * J + per_tilt(T[:, 4]) + 0.5
        v = per_tilt(T[:, 1]) * I + per_tilt(T[:, 3]) * J + per_tilt(T[:, 5]) + 0.5
    else:
        u, v = (I + 0.5) / s, (J + 0.5) / s
    dims = np.array([W, H, D], np.float64)
    out = torch.zeros((n, h, w), **f32)
    for _ in range(20):
        axes = g.uniform(0.05, 0.25, 3) * dims
        cen = g.uniform(-0.5, 0.5, 3) * (dims - 2 * axes)
        q, _ = np.linalg.qr(g.normal(size=(3, 3)))
        A = q / axes[:, None]
        dens = float(g.uniform(0.0, 1.0))
        dirs = np.stack([np.sin(ang), np.zeros(n), np.cos(ang)], 1) @ A.T
        eu = np.stack([np.cos(ang), np.zeros(n), -np.sin(ang)], 1) @ A.T
        ev, c0 = A[:, 1], A @ cen
        a = (dirs ** 2).sum(1)
        bu, bv, b0 = (dirs * eu).sum(1), dirs @ ev, -(dirs @ c0)
        # discriminant of the chord, a quadratic form in (u, v)
        k = [bu * bu - a * (eu ** 2).sum(1), bv * bv - a * (ev @ ev), 2 * bu * bv - 2 * a * (eu @ ev),
             2 * bu * b0 + 2 * a * (eu @ c0), 2 * bv * b0 + 2 * a * (ev @ c0), b0 * b0 - a * (c0 @ c0 - 1.0)]
        k = [per_tilt(x) for x in k]
        d = (k[0] * u + k[2] * v + k[3]) * u + (k[1] * v + k[4]) * v + k[5]
        out += d.clamp_(min=0.0).sqrt_().mul_(per_tilt(2.0 * dens / a))
    gen = torch.Generator(device=device).manual_seed(int(seed))
    noise = 0.01 * float(out.max())
    for t in range(0, n, 16):
        part = out[t:t + 16]
        part += noise * torch.randn(part.shape, generator=gen, **f32)
    return out


def _stats(pix):
    """Mean (the fill value of aligned images' borders) and deviation of every image."""
    mean = pix.double().mean((1, 2)).cpu().numpy()
    return np.stack([mean, np.ones_like(mean)], 1)


def _start_volume(case, seed, device=DEV):
    """A smooth start volume (what earlier iterations leave): products of slow waves."""
    g = np.random.Generator(np.random.PCG64(seed + 5))

    def wave(n):
        x = torch.arange(n, dtype=torch.float32, device=device) / n
        return 0.5 + 0.3 * torch.cos(2 * math.pi * (float(g.uniform(0.5, 4)) * x + float(g.uniform(0, 1))))

    x, y, z = wave(case["W"]), wave(case["H"]), wave(case["D"])
    return z[:, None, None] * (y[:, None] * x[None, :])[None]


class _DeviceArray:
    def __init__(self, ptr, shape, owner):
        self.owner = owner  # the memory lives as long as the tensor made from this
        self.__cuda_array_interface__ = dict(shape=shape, typestr="<f4", data=(int(ptr), False), version=2)


def _volume_view(lib, h, case, owner):
    """The handle's resident FP32 volume as a torch tensor (no copy) that keeps `owner`."""
    p = C.c_void_p()
    _abi.check(lib.tomo_volume_device_ptr(h, C.byref(p)))
    return torch.as_tensor(_DeviceArray(p.value, (case["D"], case["H"], case["W"]), owner),
                           device=DEV)


class _Handle:
    """An engine handle with its series resident, as a serving program keeps one per request."""

    def __init__(self, case, seed):
        self.lib = lib = _abi.load()
        self.case = c = case
        prec = _abi.precision_code(c["precision"])
        self.geom = _abi.make_geom(c["W"], c["H"], c["D"], c["w"], c["h"], c["n"], scale=c["w"] / c["W"])
        prm = _abi.make_params(positivity=c["positivity"], precision=prec,
                               fill=_abi.FILL_NAN)
        self.h = C.c_void_p()
        _abi.check(lib.tomo_create(C.byref(self.geom), C.byref(prm), C.byref(self.h)))
        pix = _series(c, seed)
        torch.cuda.synchronize()
        eul = np.ascontiguousarray(_eulers(_angles(c)))
        T = np.ascontiguousarray(_transforms(c, seed))
        stats = np.ascontiguousarray(_stats(pix))
        _abi.check(lib.tomo_load_series(self.h, C.c_void_p(pix.data_ptr()), 1, _abi.ptr(eul, C.c_double),
                                        _abi.ptr(T, C.c_double) if c["misalign"] else None,
                                        _abi.ptr(stats, C.c_double)))
        kind = dict(none=_abi.WEIGHT_NONE, radermacher=_abi.WEIGHT_RADERMACHER, ramp=_abi.WEIGHT_RAMP,
                    hamming=_abi.WEIGHT_HAMMING_RAMP)[c["weight"]]
        if kind != _abi.WEIGHT_NONE:
            deg = np.ascontiguousarray(_angles(c))
            _abi.check(lib.tomo_set_weighting(self.h, kind, 0.5, _abi.ptr(deg, C.c_double), None))
        if c["tv"]:
            _abi.check(lib.tomo_set_tvm(self.h, 25.0, 1.0, 0.01, c["tv"]))
        if c["kind"] != "job":
            vol = _start_volume(c, seed)
            torch.cuda.synchronize()
            _abi.check(lib.tomo_set_volume(self.h, C.c_void_p(vol.data_ptr()), 1, 0, c["H"]))
            torch.cuda.synchronize()  # the copy has read `vol`
        if prec != _abi.PREC_FP32:
            self.volume = torch.empty((c["D"], c["H"], c["W"]), dtype=torch.float32, device=DEV)
        self.seed = int(seed) & 0xFFFF

    def result(self):
        if self.case["precision"] == "fp32":
            return _volume_view(self.lib, self.h, self.case, self)
        # 16-bit storage: the values have 16 bits (a row's scale is a power of two)
        _abi.check(self.lib.tomo_get_volume(self.h, C.c_void_p(self.volume.data_ptr()), 1, 0, self.case["H"]))
        return self.volume.half()

    def __del__(self):
        if getattr(self, "h", None):
            self.lib.tomo_destroy(self.h)


class _Batch:
    def __init__(self, case, seed):
        self.lib = lib = _abi.load()
        self.handles = [_Handle(m, seed + 31 * k) for k, m in enumerate(_members(case))]
        self.b = C.c_void_p()
        _abi.check(lib.tomo_batch_create(C.byref(self.b)))
        n = len(self.handles)
        _abi.check(lib.tomo_batch_set(self.b, (C.c_void_p * n)(*[h.h.value for h in self.handles]), n))
        self.relax, self.update = np.ones(n), np.zeros(n, np.int32)
        self.first = np.array([h.case["n"] // 3 for h in self.handles], np.int32)

    def __del__(self):
        if getattr(self, "b", None):
            self.lib.tomo_batch_destroy(self.b)


def prepare(case, seed):
    if case["kind"] == "batch":
        return _Batch(case, seed)
    if case["kind"] == "update":
        ts = TiltSeries(_series(case, seed).cpu().numpy(), _angles(case))
        ts.setNormalize(False)
        ts.setFillType(_abi.FILL_NAN)
        rec = TomoReconstruction2(case["W"], case["H"], case["D"], _start_volume(case, seed).cpu().numpy())
        p = VoxelProjector3D(ts, rec)
        return dict(case=case, p=p, rec=rec)
    if case["kind"] == "wavelet":
        ts = TiltSeries(np.zeros((case["n"], case["h"], case["w"]), np.float32), _angles(case))
        rec = TomoReconstruction2(case["W"], case["H"], case["D"])
        p = CompressedSensingProjector(ts, rec)
        p.setWaveletsIterations(_levels(case["W"]), _levels(case["H"]), _levels(case["D"]))
        gen = torch.Generator(device=DEV).manual_seed(int(seed))
        start = _start_volume(case, seed)
        start = start + 0.05 * torch.randn(start.shape, generator=gen, device=DEV)
        torch.cuda.synchronize()
        return dict(case=case, p=p, rec=rec, start=start)
    return _Handle(case, seed)


def _levels(n):
    k = 0
    while k < 3 and n % (2 << k) == 0 and n >> k > 32:
        k += 1
    return max(k, 1)


def _subset(case):
    """The tilts of one update: evenly spread, as a subset of an ordering."""
    return [int(round(i * (case["n"] - 1) / (case["update"] - 1))) for i in range(case["update"])]


# --- one pass ------------------------------------------------------------------------------

def run(state):
    if isinstance(state, _Batch):
        lib = state.lib
        err = np.zeros((len(state.handles), 5))
        _abi.check(lib.tomo_batch_iteration(state.b, _abi.ptr(state.relax, C.c_double),
                                            _abi.ptr(state.update, C.c_int32), _abi.ptr(state.first, C.c_int32), 1,
                                            _abi.ptr(err, C.c_double)))
        return dict(volumes=[h.result() for h in state.handles], residual=err[:, 0].astype(np.float32))
    if isinstance(state, dict):
        case, p = state["case"], state["p"]
        if case["kind"] == "wavelet":
            _abi.check(_abi.load().tomo_set_volume(p.handle, C.c_void_p(state["start"].data_ptr()), 1, 0, case["H"]))
            p.endOfIteration()
            return _volume_view(p._lib, p.handle, case, p)
        sub = _subset(case)
        p.clearAllProjections()
        for i in sub:
            p.addProjection(i)
        err = p.projectAndDifference(case["relax"] / len(sub))
        p.backproject()
        # sums of squared single-precision differences
        return dict(volume=_volume_view(p._lib, p.handle, case, p), errors=err.astype(np.float32))
    lib, h, c = state.lib, state.h, state.case
    if c["kind"] == "job":
        # mean-filled borders for the weighted backprojection, unknown ones for the iterations
        _abi.check(lib.tomo_fill_volume(h, 0.0))
        _abi.check(lib.tomo_set_fill(h, _abi.FILL_AVG))
        _abi.check(lib.tomo_run_wbp(h, 0, c["H"]))
        _abi.check(lib.tomo_set_fill(h, _abi.FILL_NAN))
    if c["iters"] == 0:
        return state.result()
    err = np.zeros((c["iters"], 5))
    _abi.check(lib.tomo_run_ossart(h, c["iters"], c["relax"], c["update"], state.seed, 0, c["H"], 1,
                                   _abi.ptr(err, C.c_double)))
    # the average residual of each iteration (of single-precision differences)
    return dict(volume=state.result(), residual=err[:, 0].astype(np.float32))


def work(case):
    """One read and one write of the volume and one read of the projections per pass; four
    operations (an interpolation's multiply-add and difference, and the sum) per voxel-update
    of each direction."""
    if case["kind"] == "batch":
        ws = [work(m) for m in _members(case)]
        return {k: sum(x[k] for x in ws) for k in ("bytes", "flops")}
    nv, npix = case["W"] * case["H"] * case["D"], case["w"] * case["h"] * case["n"]
    vb = 4 if case["precision"] == "fp32" else 2
    if case["kind"] == "wavelet":
        # three axes and levels of an analysis and a synthesis transform (n log n) in 64 bits
        return {"bytes": 8.0 * nv, "flops": 2 * 3 * 10.0 * nv * math.log2(max(case["W"], 2))}
    if case["kind"] == "update":
        npix = case["w"] * case["h"] * case["update"]
        return {"bytes": 2.0 * vb * nv + 4.0 * npix, "flops": 8.0 * nv * case["update"]}
    wbp = case["kind"] == "job"
    f = 4.0 * nv * case["n"] * (int(wbp) + 2 * case["iters"])
    if wbp:
        f += npix * 10.0 * math.log2(case["w"])
    if case["tv"]:
        f += 40.0 * nv * case["tv"]
    return {"bytes": 2.0 * vb * nv + 4.0 * npix, "flops": f}


# --- the same in 64 bits -------------------------------------------------------------------

ACC = float(np.float32(1e-10))


class _Exact:
    """Forward projection and backprojection of one geometry in float64 torch."""

    def __init__(self, case, device):
        self.c, self.dev = case, device
        self.s = case["w"] / case["W"]
        self.ang = _angles(case)
        self.eul = _eulers(self.ang)

    def _f(self, v):
        return torch.as_tensor(v, dtype=torch.float64, device=self.dev)

    def project(self, vol, t):
        c, s = self.c, self.s
        W, H, D, w, h = (c[k] for k in ("W", "H", "D", "w", "h"))
        R00, R02 = self.eul[t, 0, 0], self.eul[t, 0, 2]
        step = -R02 / R00
        ninc = math.sqrt(step * step + 1.0)
        i = torch.arange(w, dtype=torch.float64, device=self.dev)
        x0 = ((i - (w - 1) / 2.0) / s - R02 * (-1 - (D - 1) / 2.0)) / R00 + (W - 1) / 2.0
        y = (torch.arange(h, dtype=torch.float64, device=self.dev) - (h - 1) / 2.0) / s + (H - 1) / 2.0
        yin = (y + ACC >= 0) & (y < H)
        yb = torch.where(y < 0, torch.zeros_like(y), y.trunc()).long().clamp(0, H - 1)
        yf = torch.where(y < 0, torch.zeros_like(y), y - yb)
        yb1 = (yb + 1).clamp(max=H - 1)
        ray = torch.zeros((h, w), dtype=torch.float64, device=self.dev)
        cnt = torch.zeros(w, dtype=torch.float64, device=self.dev)
        last = torch.full((w,), -1, dtype=torch.long, device=self.dev)
        nz = max(1, int(3e7 // max(1, h * w)))
        for z0 in range(0, D, nz):
            z = torch.arange(z0, min(D, z0 + nz), device=self.dev)
            x = x0[None] + (z[:, None] + 1).double() * step
            ok = (x + ACC >= 0) & (x < W)
            xb = torch.where(x < 0, torch.zeros_like(x), x.trunc()).long().clamp(0, W - 1)
            xf = torch.where(x < 0, torch.zeros_like(x), x - xb)
            xf = torch.where((xb == W - 1) | (z[:, None] == D - 1), torch.zeros_like(xf), xf)
            xb1 = (xb + 1).clamp(max=W - 1)
            p = vol[z0:z0 + z.numel()]
            lo = p[:, yb, :] if s != 1 else p

            def lerp(rows):
                a = rows.gather(2, xb[:, None, :].expand(-1, rows.shape[1], -1))
                b = rows.gather(2, xb1[:, None, :].expand(-1, rows.shape[1], -1))
                return a, a + xf[:, None, :] * (b - a)

            raw, val = lerp(lo)
            if s != 1:
                val = val + yf[None, :, None] * (lerp(p[:, yb1, :])[1] - val)
            flat = (yb == H - 1)[None, :, None] | ((xb == W - 1) | (z[:, None] == D - 1))[:, None, :]
            val = torch.where(flat, raw, val)
            ray += torch.where(ok[:, None, :], val, torch.zeros_like(val)).sum(0)
            cnt += ok.sum(0)
            last = torch.maximum(last, torch.where(ok, z[:, None].expand_as(ok), -1).amax(0))
        incr = cnt + ((cnt > 0) & (last < D - 1))
        hit = (cnt > 0)[None, :] & yin[:, None]
        nan = torch.full((), float("nan"), dtype=torch.float64, device=self.dev)
        return torch.where(hit, ray * ninc, nan), torch.where(hit, (incr * ninc)[None, :], torch.zeros_like(ray))

    def backproject(self, vol, t, img):
        c, s = self.c, self.s
        W, H, D, w, h = (c[k] for k in ("W", "H", "D", "w", "h"))
        R00, R02 = self.eul[t, 0, 0], self.eul[t, 0, 2]
        X = torch.arange(W, dtype=torch.float64, device=self.dev) - (W - 1) / 2.0
        Z = torch.arange(D, dtype=torch.float64, device=self.dev) - (D - 1) / 2.0
        y = (torch.arange(H, dtype=torch.float64, device=self.dev) - (H - 1) / 2.0) * s + (h - 1) / 2.0
        yok = (y >= 0) & (y < h)
        yb = y.floor().long().clamp(0, h - 1)
        yf = (y - yb).clamp(min=0.0)
        img = img[yb] + yf[:, None] * (img[(yb + 1).clamp(max=h - 1)] - img[yb])
        img = torch.where(yok[:, None], img, torch.zeros_like(img))
        nz = max(1, int(3e7 // max(1, H * W)))
        for z0 in range(0, D, nz):
            xx = (X[None] * R00 + Z[z0:z0 + nz, None] * R02) * s + (w - 1) / 2.0
            ok = (xx >= 0) & (xx < w)
            xb = xx.floor().long().clamp(0, w - 1)
            xf = (xx - xb).clamp(min=0.0)
            k = xb.shape[0]
            a = img[:, xb.reshape(-1)].reshape(H, k, W)
            b = img[:, (xb + 1).clamp(max=w - 1).reshape(-1)].reshape(H, k, W)
            v = (a + xf * (b - a)) * ok
            part = vol[z0:z0 + k]
            part += v.transpose(0, 1)
            if c["positivity"]:
                part.clamp_(min=0.0)

    def align(self, img, T, fill):
        h, w = img.shape
        m00, m10, m01, m11, m02, m12 = (float(v) for v in T)
        det = m00 * m11 - m01 * m10
        i00, i10, i01, i11 = m11 / det, -m10 / det, -m01 / det, m00 / det
        i02, i12 = (m01 * m12 - m11 * m02) / det, (m10 * m02 - m00 * m12) / det
        J = (torch.arange(h, dtype=torch.float64, device=self.dev) - h / 2.0)[:, None]
        I = (torch.arange(w, dtype=torch.float64, device=self.dev) - w / 2.0)[None]
        xx, yy = (i00 * I + i01 * J + i02) + w / 2.0, (i10 * I + i11 * J + i12) + h / 2.0
        ix, iy = xx.trunc().long(), yy.trunc().long()
        dx, dy = xx - ix, yy - iy
        ok = (ix >= 0) & (ix < w) & (iy >= 0) & (iy < h)
        edge = (ix == w - 1) | (iy == h - 1)
        a, b = ix.clamp(0, w - 1), iy.clamp(0, h - 1)
        a1, b1 = (ix + 1).clamp(0, w - 1), (iy + 1).clamp(0, h - 1)
        f4 = dx * dy
        v = img[b, a] * (1 - dx - dy + f4) + img[b, a1] * (dx - f4) + img[b1, a] * (dy - f4) + img[b1, a1] * f4
        v = torch.where(edge, img[b, a], v)
        return torch.where(ok, v, torch.full_like(v, fill))

    def weighted(self, imgs):
        c = self.c
        w, n = c["w"], c["n"]
        k = np.arange(w, dtype=np.float64)
        k = np.where(k > w / 2.0, k - w, k)
        if c["weight"] == "radermacher":
            v = (0.5 * w) * np.pi * k[None] * np.sin(np.deg2rad(self.ang))[:, None] / w
            wt = np.where(v == 0, 1.0, np.sin(v) / np.where(v == 0, 1.0, v)).sum(0)
            m = 1.0 / (np.where(wt < 0.005, float(np.float32(0.005)), wt) * (0.5 * w))
        else:
            d = (self.ang.max() - self.ang.min()) * (math.pi / 180.0) / (n - 1)
            m = np.where(k == 0, d / (4.0 * w), d * np.abs(k) / w)
            if c["weight"] == "hamming":
                m = m * (0.54 + 0.46 * np.cos(2.0 * math.pi * k / w))
        return torch.fft.ifft(torch.fft.fft(imgs, dim=2) * self._f(m), dim=2).real

    def order(self, first):
        b = self.eul[:, 2, :]
        n, out, im = len(b), [], first
        todo = [True] * n
        while len(out) < n:
            if out:
                best, at = float("inf"), -1
                for o in range(n):
                    if todo[o]:
                        sp = abs(float(b[im][0] * b[o][0] + b[im][1] * b[o][1] + b[im][2] * b[o][2]))
                        if sp < best:
                            best, at = sp, o
                im = at
            out.append(im)
            todo[im] = False
        return out

    def subset(self, vol, meas, tilts, factor):
        diffs, errs = [], []
        for t in tilts:
            th, nm = self.project(vol, t)
            ok = ~torch.isnan(meas[t]) & ~torch.isnan(th)
            d = torch.where(ok, (meas[t] - th) / nm * factor, torch.zeros_like(th))
            diffs.append(d)
            errs.append(float((d * d).sum()))
        for t, d in zip(tilts, diffs):
            self.backproject(vol, t, d)
        return errs

    def iteration(self, vol, meas, first):
        c = self.c
        n = c["n"]
        upd = n if c["update"] == 0 else min(c["update"], n)
        factor = float(np.float32(c["relax"] / upd))
        order = self.order(first)
        som = 0.0
        for s in range(0, n, upd):
            som += sum(self.subset(vol, meas, order[s:s + upd], factor))
        return math.sqrt(som / (n * c["W"] * c["H"]))


def _first_index(seed, it, n):
    """SplitMix64 of (seed, iteration), the documented first projection of an ordering."""
    m = (1 << 64) - 1
    z = (seed + 0x9E3779B97F4A7C15 * (it + 1)) & m
    z = ((z ^ (z >> 30)) * 0xBF58476D1CE4E5B9) & m
    z = ((z ^ (z >> 27)) * 0x94D049BB133111EB) & m
    return (z ^ (z >> 31)) % n


def _tv64(f, theta, g, dt, steps):
    u = f.clone()
    p = [torch.zeros_like(f) for _ in range(3)]
    for _ in range(steps):
        du = []
        for ax in (2, 1, 0):
            d = torch.zeros_like(u)
            n = u.shape[ax]
            d.narrow(ax, 0, n - 1).copy_(u.narrow(ax, 1, n - 1) - u.narrow(ax, 0, n - 1))
            du.append(d)
        dd = 1 + dt / theta / g * (du[0] ** 2 + du[1] ** 2 + du[2] ** 2).sqrt()
        p = [(a - dt / theta * d) / dd for a, d in zip(p, du)]
        div = torch.zeros_like(u)
        for a, ax in zip(p, (2, 1, 0)):
            n = u.shape[ax]
            div += a
            div.narrow(ax, 1, n - 1).sub_(a.narrow(ax, 0, n - 1))
            # the far face takes minus its own value alone
            div.narrow(ax, n - 1, 1).sub_(2 * a.narrow(ax, n - 1, 1) - a.narrow(ax, n - 2, 1))
        u = f - theta * div
    return u


def _cost(case):
    return case["W"] * case["H"] * case["D"] * (case["n"] if case["kind"] != "update" else case["update"]) * \
        (2 * case["iters"] + 1)


def exact(case, seed):
    if case["kind"] == "wavelet":
        return None
    if case["kind"] == "batch":
        ms = _members(case)
        if sum(_cost(m) for m in ms) > 9e10:
            return None
        got = [_exact_one(m, seed + 31 * k, [m["n"] // 3]) for k, m in enumerate(ms)]
        return dict(volumes=[g["volume"] for g in got], residual=np.array([g["residual"][0] for g in got]))
    if _cost(case) > 9e10:
        return None
    return _exact_one(case, seed, [_first_index(int(seed) & 0xFFFF, it, case["n"]) for it in range(case["iters"])])


def _exact_one(case, seed, firsts):
    dev = DEV if torch.cuda.is_available() else "cpu"
    E = _Exact(case, dev)
    raw = _series(case, seed, dev)
    mean = _stats(raw)[:, 0]
    raw = raw.double()
    T = _transforms(case, seed)

    def aligned(fill):
        if not case["misalign"]:
            return raw
        return torch.stack([E.align(raw[t], T[t], fill(t)) for t in range(case["n"])])

    if case["kind"] == "job":
        vol = torch.zeros((case["D"], case["H"], case["W"]), dtype=torch.float64, device=dev)
        imgs = E.weighted(aligned(lambda t: float(mean[t])))
        for t in range(case["n"]):
            E.backproject(vol, t, imgs[t])
        if case["iters"] == 0:
            return vol
    else:
        vol = _start_volume(case, seed, dev).double()
    meas = aligned(lambda t: float("nan"))
    if case["kind"] == "update":
        errs = E.subset(vol, meas, _subset(case), case["relax"] / case["update"])
        return dict(volume=vol, errors=np.array(errs))
    res = []
    for f in firsts:
        res.append(E.iteration(vol, meas, f))
        if case["tv"]:
            vol = _tv64(vol, 25.0, 1.0, 0.01, case["tv"])
    return dict(volume=vol, residual=np.array(res))
