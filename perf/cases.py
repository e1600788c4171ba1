"""The calls a program makes of oceanlib_b200, with their sizes: listed cases,
drawn cases of the same ranges, how each is set up and run through the public
entry points, the bytes and operations a pass cannot do without, and its
results in 64-bit arithmetic.

Kinds of case:
  ocean     one Ocean, reference-style: update(t), results in the host mirror
  batch     an OceanBatch on the device, any form, with or without foam
  cascade   a CascadeStack updated on the device
  query     surface queries of a cascade, points and records on the device
  ensemble  an OceanEnsemble of uneven sizes
  field     one InteractionField: sources added, update(dt), host mirror
  serve     an OceanServer: every session sends an update and a query

Every state advances in time by one 60 Hz frame per pass, as a program does.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

import oceanlib_b200 as ob
from oceanlib_b200 import abi
from oceanlib_b200.interaction import Disturbance, InteractionDesc, InteractionField
from oceanlib_b200.serve import DISTURBANCE_DTYPE, OceanServer

DT = 1.0 / 60.0
FOAM_WARM = 3  # frames a foam batch has behind it when it is timed

FORMS = {"exact": abi.OCEAN_FFT_EXACT, "fast": abi.OCEAN_FFT_FAST, "tensor": abi.OCEAN_FFT_TENSOR,
         "precise": abi.OCEAN_FFT_PRECISE}


def listed():
    return [
        # A small patch for a game tick: the smallest call, one ocean on the CPU side.
        {"name": "ocean_64", "kind": "ocean", "n": 64, "velocity": True},
        # The default patch of the reference's README and bench: one 256^2 ocean read on the host.
        {"name": "ocean_256", "kind": "ocean", "n": 256, "velocity": False},
        # A renderer's three-level cascade, left on the device for drawing.
        {"name": "cascade_3x256", "kind": "cascade", "sizes": "256,256,256", "velocity": True, "depth": 30.0},
        # The reference bench's 512^2 update over a batch of worlds.
        {"name": "batch_64x512", "kind": "batch", "n": 512, "count": 64, "velocity": False, "foam": False,
         "form": "exact"},
        # The foam patch (orbital velocity, persistent foam) over a batch of worlds: the benchmark's workload.
        {"name": "foam_64x512", "kind": "batch", "n": 512, "count": 64, "velocity": True, "foam": True,
         "form": "exact"},
        # The tensor-core form, for results within 2e-6 of FP64.
        {"name": "tensor_16x512", "kind": "batch", "n": 512, "count": 16, "velocity": True, "foam": False,
         "form": "tensor"},
        # The FP64-block form at an odd batch count, for accuracy at any size.
        {"name": "precise_21x256", "kind": "batch", "n": 256, "count": 21, "velocity": True, "foam": False,
         "form": "precise"},
        # The largest grid the library takes, for film-quality patches.
        {"name": "large_4096", "kind": "batch", "n": 4096, "count": 1, "velocity": True, "foam": False,
         "form": "exact"},
        # Independent sea states of uneven size, as in Monte-Carlo sweeps.
        {"name": "ensemble_64", "kind": "ensemble", "count": 64, "velocity": False},
        # Buoyancy and ray queries: a million points against a three-level cascade.
        {"name": "query_1m", "kind": "query", "sizes": "256,256,256", "velocity": True, "depth": 30.0,
         "points": 1000000},
        # One interactive field around the player, with boats and swimmers.
        {"name": "field_512", "kind": "field", "n": 512, "extent": 64.0, "radius": 6, "sources": 8, "substeps": 1},
        # A server tick: sessions of three ocean sizes, each with an interaction field.
        {"name": "serve_32", "kind": "serve", "sessions": 32, "sizes": "128,256,512", "field": 512, "points": 4096,
         "sources": 8},
    ]


def draw(rng: random.Random):
    kind = rng.choice(["ocean", "batch", "batch", "batch", "cascade", "query", "ensemble", "field", "serve"])
    if kind == "ocean":
        return {"kind": kind, "n": 16 << rng.randrange(7), "velocity": rng.random() < 0.5,
                "choppiness": round(rng.uniform(0.5, 1.8), 3)}
    if kind == "batch":
        n = 32 << rng.randrange(8)
        most = max(1, (1 << 24) // (n * n))
        count = min(most, 512, max(1, round(math.exp(rng.uniform(0.0, math.log(min(most, 512) + 1))))))
        forms = ["exact", "exact", "precise", "fast"] + (["tensor"] if 64 <= n <= 512 else [])
        form = rng.choice(forms)
        if form == "tensor":
            count = min(count, max(1, (1 << 22) // (n * n)))
        velocity = rng.random() < 0.6
        return {"kind": kind, "n": n, "count": count, "velocity": velocity,
                "foam": velocity and rng.random() < 0.5, "form": form, "choppiness": round(rng.uniform(0.5, 1.8), 3)}
    if kind in ("cascade", "query"):
        sizes = ",".join(str(rng.choice([64, 128, 256, 256, 512])) for _ in range(rng.randint(1, 4)))
        c = {"kind": kind, "sizes": sizes, "velocity": rng.random() < 0.6, "depth": rng.choice([0.0, 30.0])}
        if kind == "query":
            c["points"] = round(math.exp(rng.uniform(math.log(1000), math.log(1000000))))
        return c
    if kind == "ensemble":
        return {"kind": kind, "count": rng.randint(3, 48), "velocity": rng.random() < 0.4}
    if kind == "field":
        n = rng.choice([64, 128, 256, 512, 1024])
        return {"kind": kind, "n": n, "extent": round(n * rng.uniform(0.11, 0.3), 2), "radius": rng.randint(3, 8),
                "sources": rng.randint(0, 24), "substeps": rng.randint(1, 3)}
    return {"kind": kind, "sessions": rng.randint(2, 32), "sizes": rng.choice(["64,128", "128,256,512", "256"]),
            "field": rng.choice([128, 256, 512]), "points": rng.randint(100, 4096), "sources": rng.randint(1, 16)}


# ---------------------------------------------------------------------------
# Inputs, from the seed alone
# ---------------------------------------------------------------------------
def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0x7FFFFFFF, 77])


def _descs(case, seed):
    """The case's ocean descriptors, in the order the program lists them."""
    r = _rng(case, seed)
    seeds = [int(s) for s in r.integers(1, 1 << 40, size=512)]
    kind = case["kind"]
    chop = float(case.get("choppiness", 1.2))
    if kind == "ocean":
        return [ob.OceanDesc(size=case["n"], patch_length=200.0, wind_speed=12.0, choppiness=chop,
                             compute_velocity=case["velocity"], seed=seeds[0])]
    if kind == "batch":
        wave = dict(patch_length=250.0, wind_speed=22.0) if case["velocity"] else dict(patch_length=200.0,
                                                                                      wind_speed=12.0)
        return [ob.OceanDesc(size=case["n"], choppiness=chop, compute_velocity=case["velocity"], seed=seeds[i],
                             wind_direction=0.4, **wave) for i in range(case["count"])]
    if kind in ("cascade", "query"):
        lengths = (800.0, 150.0, 25.0, 7.0)
        return [ob.OceanDesc(size=int(n), patch_length=lengths[i], wind_speed=15.0, depth=case["depth"],
                             compute_velocity=case["velocity"], seed=seeds[i])
                for i, n in enumerate(case["sizes"].split(","))]
    if kind == "ensemble":
        # Sizes from {64 .. 1024} in the same shares for every seed, the rest at random.
        sizes = [(64, 128, 256, 512, 1024, 256, 512, 128)[i % 8] for i in range(case["count"])]
        return [ob.OceanDesc(size=sizes[i], patch_length=float(np.float32(r.uniform(50.0, 1000.0))),
                             wind_speed=float(np.float32(r.uniform(5.0, 25.0))),
                             wind_direction=float(np.float32(r.uniform(0.0, 2.0 * math.pi))),
                             choppiness=float(np.float32(r.uniform(0.5, 1.8))), seed=seeds[i],
                             compute_velocity=case["velocity"]) for i in range(case["count"])]
    sizes = [int(s) for s in case["sizes"].split(",")]
    return [ob.OceanDesc(size=sizes[i % len(sizes)], seed=seeds[i]) for i in range(case["sessions"])]


def _points(count, extent, seed, salt=0):
    r = np.random.default_rng([int(seed) & 0x7FFFFFFF, 5, salt])
    return r.uniform(0.0, extent, (count, 2)).astype(np.float32)


class _Discs:
    """Continuous disc sources circling slowly inside a field of `extent` metres. A program moves its
    sources itself; here their positions are worked out beforehand, LOOP frames that come round again."""

    LOOP = 16

    def __init__(self, count, extent, seed, salt=0):
        r = np.random.default_rng([int(seed) & 0x7FFFFFFF, 9, salt])
        self.at = r.uniform(0.3 * extent, 0.7 * extent, (count, 2))
        self.ring = r.uniform(0.05 * extent, 0.2 * extent, count)
        self.phase = r.uniform(0.0, 2.0 * math.pi, count)
        self.speed = r.uniform(0.5, 6.0, count)
        self.radius = r.uniform(0.5, 3.0, count)
        self.strength = r.uniform(0.05, 0.4, count)
        self.frames = [self._frame(k) for k in range(self.LOOP)]

    def frame(self, k):
        return self.frames[k % self.LOOP]

    def _frame(self, k):
        a = self.phase + self.speed / self.ring * (k * DT)
        out = np.zeros(len(self.ring), DISTURBANCE_DTYPE)
        out["world_x"] = self.at[:, 0] + self.ring * np.cos(a)
        out["world_z"] = self.at[:, 1] + self.ring * np.sin(a)
        out["radius"] = self.radius
        out["strength"] = self.strength
        out["velocity_x"] = -self.speed * np.sin(a)
        out["velocity_z"] = self.speed * np.cos(a)
        out["kind"] = abi.OCEAN_SOURCE_CONTINUOUS
        return out


def _t0(seed):
    return 10.0 + (int(seed) % 97) * 0.25


def _frame_dt(desc, steps):
    """A frame length that gives exactly `steps` substeps of the field."""
    return float(np.nextafter(np.float32(steps * desc.fixed_dt), np.float32(1.0)))


def _field_desc(case):
    n, extent = (case["field"], 0.125 * case["field"]) if case["kind"] == "serve" else (case["n"], case["extent"])
    steps = case.get("substeps", 1)
    return InteractionDesc(size=n, extent=float(np.float32(extent)), kernel_radius=case.get("radius", 6),
                           fixed_dt=float(np.float32(DT / steps)))


class _DeviceArray:
    """Device memory of `owner`, which it keeps alive."""

    def __init__(self, owner, ptr, shape):
        self.owner = owner
        self.__cuda_array_interface__ = {"shape": shape, "typestr": "<f4", "data": (ptr, False), "version": 3}


class _HostArray:
    """Host memory of `owner`, which it keeps alive."""

    def __init__(self, owner, array):
        self.owner = owner
        self.__array_interface__ = array.__array_interface__


def _view(owner, ptr, shape):
    return torch.as_tensor(_DeviceArray(owner, ptr, shape), device="cuda")


def _views(owner, buffers, velocity):
    """One tensor per output and size over the oceans' buffers, which lie one after the other."""
    out = {}
    for n in sorted({b.size for b in buffers}):
        group = [b for b in buffers if b.size == n]
        for name in ("displacement", "normal") + (("velocity",) if velocity else ()):
            ptrs = [getattr(b, name) for b in group]
            if any(q - p != n * n * 16 for p, q in zip(ptrs, ptrs[1:])):
                raise RuntimeError("the oceans' buffers do not lie one after the other")
            out["%s_%d" % (name, n)] = _view(owner, ptrs[0], (len(group), n * n, 4))
    return out


def prepare(case, seed):
    kind = case["kind"]
    s = {"case": case, "frame": 0, "t0": _t0(seed)}
    if kind == "field":
        fd = _field_desc(case)
        s["field"] = InteractionField(fd)
        s["out"] = np.asarray(_HostArray(s["field"], s["field"].buffers()["field"]))
        s["dt"] = _frame_dt(fd, case["substeps"])
        s["sources"] = [[Disturbance(*(float(d[m]) for m in ("world_x", "world_z", "radius", "strength", "velocity_y",
                                                             "velocity_x", "velocity_z")), int(d["kind"]))
                         for d in f] for f in _Discs(case["sources"], case["extent"], seed).frames]
        return s
    descs = _descs(case, seed)
    if kind == "ocean":
        s["ocean"] = ob.Ocean(descs[0])
        b = s["ocean"].buffers()  # the host mirror, rewritten by every update
        s["out"] = {k: np.asarray(_HostArray(s["ocean"], b[k]))
                    for k in ("displacement", "normal") + (("velocity",) if case["velocity"] else ())}
    elif kind == "batch":
        b = ob.OceanBatch(descs, form=FORMS[case["form"]], foam=ob.FoamDesc() if case["foam"] else None)
        s["batch"] = b
        s["dt"] = DT if case["foam"] else 0.0
        if case["foam"]:
            for k in range(FOAM_WARM):
                b.update(s["t0"] + (k - FOAM_WARM) * DT, foam_dt=DT)
            b.synchronize()
        s["out"] = _views(b, [b.device_buffers(i) for i in range(case["count"])], case["velocity"])
        s["foam"] = {}
    elif kind in ("cascade", "query"):
        c = ob.CascadeStack(descs)
        s["cascade"] = c
        if kind == "cascade":
            s["out"] = [_views(c, [c.device_buffers(i)], case["velocity"]) for i in range(len(descs))]
        else:
            c.update(s["t0"])
            c.synchronize()
            s["xz"] = torch.from_numpy(_points(case["points"], descs[0].patch_length, seed)).cuda()
            s["rec"] = torch.zeros((case["points"], 10), dtype=torch.float32, device="cuda")
    elif kind == "ensemble":
        e = ob.OceanEnsemble(descs, autotune=False)
        e.set_schedule(ob.OceanEnsemble.ONE_LAUNCH)  # what the autotuner picks, without its timing runs
        s["ensemble"] = e
        s["out"] = _views(e, [e.device_buffers(i) for i in range(case["count"])], case["velocity"])
    else:
        srv = OceanServer(hbm_budget=8e9)
        fd = _field_desc(case)
        s["server"] = srv
        s["dt"] = _frame_dt(fd, 1)
        s["sessions"] = [srv.open_session(d, fd) for d in descs]
        s["discs"] = [_Discs(case["sources"], fd.extent, seed, i) for i in range(case["sessions"])]
        s["xz"] = [_points(case["points"], fd.extent, seed, i) for i in range(case["sessions"])]
        s["heights"] = np.zeros((case["sessions"], case["points"]), np.float32)
    return s


def run(s):
    case, k = s["case"], s["frame"]
    kind = case["kind"]
    s["frame"] = k + 1
    t = s["t0"] + k * DT
    if kind == "ocean":
        s["ocean"].update(t)
        return s["out"]
    if kind == "batch":
        b = s["batch"]
        b.update(t, foam_dt=s["dt"])
        if not case["foam"]:
            return s["out"]
        ptr = b.device_buffers(0).foam  # the foam planes swap each frame
        if ptr not in s["foam"]:
            s["foam"][ptr] = _view(b, ptr, (case["count"], case["n"] * case["n"]))
        return {**s["out"], "foam": s["foam"][ptr]}
    if kind == "cascade":
        s["cascade"].update(t)
        return s["out"]
    if kind == "query":
        s["cascade"].sample_many_device(s["xz"].data_ptr(), case["points"], s["rec"].data_ptr())
        return s["rec"]
    if kind == "ensemble":
        s["ensemble"].update(t)
        return s["out"]
    if kind == "field":
        f = s["field"]
        for d in s["sources"][k % _Discs.LOOP]:
            f.add(d)
        f.update(s["dt"])
        return s["out"]
    srv = s["server"]
    for i, sid in enumerate(s["sessions"]):
        srv.submit_update(sid, t, s["dt"], s["discs"][i].frame(k))
        srv.submit_query(sid, s["xz"][i], s["heights"][i])
    srv.drain()
    return s["heights"]


# ---------------------------------------------------------------------------
# What a pass cannot do without
# ---------------------------------------------------------------------------
def _frame_work(n, velocity, foam=False):
    """h0 read and the RGBA32F outputs (and foam, in and out) written once; the transforms and ~120 operations a cell."""
    nf = 6 if velocity else 4
    cells = n * n
    return cells * (8 + 16 * (3 if velocity else 2) + (8 if foam else 0)), cells * (nf * 10 * math.log2(n) + 120)


def _field_work(n, radius, substeps):
    return n * n * (16 + 8 + 16), n * n * substeps * (2 * (2 * radius + 1) ** 2 + 10)


def work(case):
    kind = case["kind"]
    if kind == "field":
        b, f = _field_work(case["n"], case["radius"], case["substeps"])
    elif kind == "query":
        levels = [int(n) for n in case["sizes"].split(",")]
        b = case["points"] * 48 + sum(n * n * 16 * (3 if case["velocity"] else 2) for n in levels)
        f = case["points"] * len(levels) * 400
    else:
        if kind == "batch":
            parts = [_frame_work(case["n"], case["velocity"], case["foam"])] * case["count"]
        elif kind == "ocean":
            parts = [_frame_work(case["n"], case["velocity"])]
        else:
            parts = [_frame_work(d.size, d.compute_velocity) for d in _descs(case, 0)]
        if kind == "serve":
            parts += [_field_work(case["field"], 6, 1)] * case["sessions"]
            parts += [(case["points"] * 12, case["points"] * 200)] * case["sessions"]
        b, f = sum(p[0] for p in parts), sum(p[1] for p in parts)
    return {"bytes": float(b), "flops": float(f)}


# ---------------------------------------------------------------------------
# The same results in 64 bits: the FP32 tables the model is defined by (h0,
# omega, 1/|k|, wavenumbers, stencil taps, damping), everything after in FP64
# ---------------------------------------------------------------------------
_M64 = (1 << 64) - 1
_PCG = 6364136223846793005


def _dev():
    return "cuda" if torch.cuda.is_available() else "cpu"


def _f32(v):
    return float(np.float32(v))


def _i64(values):
    return torch.from_numpy(np.array([v & _M64 for v in values], dtype=np.uint64).view(np.int64)).to(_dev())


def _shr(x, k):
    return (x >> k) & ((1 << (64 - k)) - 1)


def _mix(x):
    x = (x + 0x9E3779B97F4A7C15) & _M64
    x = ((x ^ (x >> 30)) * 0xBF58476D1CE4E5B9) & _M64
    x = ((x ^ (x >> 27)) * 0x94D049BB133111EB) & _M64
    return x ^ (x >> 31)


def _draws(seed, n):
    """(n, 2 n) uniforms: row y's PCG32 stream (stream 0, increment 1)."""
    start = []
    for y in range(n):
        s = _mix((seed ^ (0x9E3779B97F4A7C15 * (y + 1))) & _M64)
        start.append(((1 + s) * _PCG + 1) & _M64)
    a, c, at, ct = 1, 0, [], []
    for _ in range(2 * n):
        at.append(a)
        ct.append(c)
        a, c = (a * _PCG) & _M64, (c * _PCG + 1) & _M64
    st = _i64(start)[:, None] * _i64(at)[None, :] + _i64(ct)[None, :]
    xs = _shr(_shr(st, 18) ^ st, 27) & 0xFFFFFFFF
    rot = _shr(st, 59)
    u = ((xs >> rot) | (xs << ((32 - rot) & 31))) & 0xFFFFFFFF
    return (u.to(torch.float64) + 0.5) * (1.0 / 4294967296.0)


def _wavenumbers(n, length):
    si = np.arange(n)
    si = np.where(si < n // 2, si, si - n).astype(np.float32)
    k = np.float32(6.28318530717958647692) * si / np.float32(length)
    return torch.from_numpy(k.astype(np.float64)).to(_dev())


def _tables(d):
    """h0 (complex), omega, 1/|k|, kx, kz of one ocean, rounded to FP32 and widened."""
    n = d.size
    g, u, fetch, depth = _f32(d.gravity), _f32(d.wind_speed), _f32(d.fetch), _f32(d.depth)
    kv = _wavenumbers(n, d.patch_length)
    kx, kz = kv[None, :].expand(n, n), kv[:, None].expand(n, n)
    k2 = kx * kx + kz * kz
    k = torch.sqrt(k2)
    safe = torch.where(k > 0, k, torch.ones_like(k))
    om = torch.sqrt(g * safe) if depth <= 0 else torch.sqrt(g * safe * torch.tanh(safe * depth))
    if depth <= 0:
        dw = g / (2.0 * om)
    else:
        th = torch.tanh(safe * depth)
        dw = g * (th + safe * depth * (1.0 - th * th)) / (2.0 * om)
    wp = 22.0 * np.cbrt(g * g / (u * fetch))
    alpha = 0.076 * (g * fetch / (u * u)) ** -0.22
    ratio = wp / om
    pm = alpha * g * g / om ** 5 * torch.exp(-1.25 * ratio ** 4)
    sigma = torch.where(om <= wp, 0.07, 0.09).to(torch.float64)
    peak = torch.exp(-((om - wp) ** 2) / (2.0 * sigma * sigma * wp * wp))
    spec = pm * _f32(d.peak_enhancement) ** peak
    inv = om / wp
    s = torch.where(inv < 1.0, 6.97 * inv ** 4.06, 9.77 * inv ** (-2.33 - 1.45 * ((u * wp / g) - 1.17)))
    if d.swell > 0:
        s = s + 16.0 * torch.tanh(ratio) * _f32(d.swell) ** 2
    dth = torch.remainder(torch.atan2(kz, kx) - _f32(d.wind_direction) + math.pi, 2 * math.pi) - math.pi
    c = torch.cos(0.5 * dth)
    q = torch.exp(torch.lgamma(s + 1.0) - torch.lgamma(s + 0.5)) / (2.0 * math.sqrt(math.pi))
    spread = torch.where(c > 0, q * torch.where(c > 0, c, torch.ones_like(c)) ** (2.0 * s), torch.zeros_like(c))
    psi = spec * dw * spread / safe * torch.exp(-k2 * (_f32(d.small_wave_cutoff) / (2 * math.pi)) ** 2)
    psi = torch.where((k > 0) & (spec > 0), psi, torch.zeros_like(psi))
    amp = 0.5 * torch.sqrt(psi) * (2 * math.pi / _f32(d.patch_length))
    uu = _draws(d.seed, n)
    rad, ang = torch.sqrt(-2.0 * torch.log(uu[:, 0::2])), 2 * math.pi * uu[:, 1::2]
    f = lambda v: v.to(torch.float32).to(torch.float64)  # noqa: E731
    h0 = torch.complex(f(f(rad * torch.cos(ang)) * amp), f(f(rad * torch.sin(ang)) * amp))
    zero = torch.zeros_like(k)
    return h0, f(torch.where(k > 0, om, zero)), f(torch.where(k > 0, 1.0 / safe, zero)), kx, kz


def _frame64(d, tables, t):
    """(displacement, normal, velocity or None) of one ocean, (N * N, 4) float64."""
    h0, w, ki, kx, kz = tables
    n = d.size
    e = torch.polar(torch.ones_like(w), torch.remainder(w * t, 2 * math.pi))
    mirror = torch.roll(torch.flip(h0, (0, 1)), (1, 1), (0, 1)).conj()
    fwd, bwd = h0 * e, mirror * e.conj()
    h = fwd + bwd
    sx, sz = kx * ki, kz * ki

    def back(z):
        z = torch.fft.ifft2(z) * (n * n)
        return z.real, z.imag

    hh, dx = back(h + 1j * (-1j * sx * h))
    dz, hx = back(-1j * sz * h + 1j * (1j * kx * h))
    hz, jxx = back(1j * kz * h + 1j * (kx * sx * h))
    jzz, jxz = back(kz * sz * h + 1j * (kx * sz * h))
    lam, thr = _f32(d.choppiness), _f32(d.foam_threshold)
    axx, azz, axz = 1.0 + lam * jxx, 1.0 + lam * jzz, lam * jxz
    jac = axx * azz - axz * axz
    nx, nz = -(hx * azz - axz * hz), -(axx * hz - hx * axz)
    ln = torch.sqrt(nx * nx + jac * jac + nz * nz)
    inv = torch.where(ln > 0, 1.0 / ln, torch.zeros_like(ln))
    foam = ((thr - jac) * (1.0 / thr if thr > 1e-6 else 0.0)).clamp(0.0, 1.0)
    flat = lambda *c: torch.stack([v.reshape(-1) for v in c], -1)  # noqa: E731
    vel = None
    if d.compute_velocity:
        v = fwd - bwd
        ux, uy = back(-w * sx * v + 1j * (1j * w * v))
        uz, _ = back(-w * sz * v + 0j)
        vel = flat(ux, uy, uz, torch.zeros_like(ux))
    return flat(lam * dx, hh, lam * dz, foam), flat(nx * inv, jac * inv, nz * inv, jac), vel


def _foam64(d, cur, disp, vel):
    """One foam substep of 1/60 s at the default FoamDesc."""
    n = d.size
    dt = _f32(DT)
    cell = _f32(np.float32(d.patch_length) / np.float32(n))
    z, x = torch.meshgrid(torch.arange(n, device=cur.device), torch.arange(n, device=cur.device), indexing="ij")
    u = x.reshape(-1).double() - vel[:, 0] * dt / cell
    v = z.reshape(-1).double() - vel[:, 2] * dt / cell
    f = _bilinear(cur[:, None], u, v, n)[:, 0]
    return (f * math.exp(-_f32(0.35) * dt) + disp[:, 3] * 4.0 * dt).clamp(0.0, 1.0)


def _bilinear(buf, gu, gv, n):
    """Periodic bilinear taps of (N * N, C) at grid coordinates."""
    fu, fv = torch.floor(gu), torch.floor(gv)
    tu, tv = (gu - fu)[:, None], (gv - fv)[:, None]
    x0, z0 = torch.remainder(fu.long(), n), torch.remainder(fv.long(), n)
    x1, z1 = torch.remainder(x0 + 1, n), torch.remainder(z0 + 1, n)
    return (buf[z0 * n + x0] * (1 - tu) * (1 - tv) + buf[z0 * n + x1] * tu * (1 - tv) +
            buf[z1 * n + x0] * (1 - tu) * tv + buf[z1 * n + x1] * tu * tv)


def _sample64(d, frame, xz):
    """(displacement, unit normal, velocity) at world points, after four inversion steps."""
    n = d.size
    inv = _f32(np.float32(n) / np.float32(d.patch_length))
    p = xz
    for _ in range(4):
        p = xz - _bilinear(frame[0], p[:, 0] * inv, p[:, 1] * inv, n)[:, [0, 2]]
    g = (p[:, 0] * inv, p[:, 1] * inv, n)
    nm = _bilinear(frame[1], *g)[:, :3]
    nm = nm / torch.linalg.norm(nm, dim=1, keepdim=True)
    vel = _bilinear(frame[2], *g)[:, :3] if frame[2] is not None else torch.zeros_like(nm)
    return _bilinear(frame[0], *g), nm, vel


def _taps64(p, cell):
    """The deep-water iWave stencil: taps equal within each orbit {(+-a, +-b), (+-b, +-a)}, a zero
    symbol at k = 0, fitted to |k| over the first quadrant of the band by weighted least squares."""
    kmax = math.pi / cell
    ks = kmax * np.arange(97) / 96.0
    kz, kx = (v.ravel() for v in np.meshgrid(ks, ks, indexing="ij"))
    kk = np.sqrt(kx * kx + kz * kz)
    lo = 0.125 * kmax
    band = (kk >= lo) & (kk <= kmax)
    ref = np.where(band, kk, np.where(kk < lo, lo, kmax))
    w = np.where(band, 1.0, 0.02) / (ref * ref)
    orbits = [sorted({(i, j) for x, y in ((a, b), (b, a)) for i in (x, -x) for j in (y, -y)})
              for a in range(1, p + 1) for b in range(a + 1)]
    psi = np.stack([sum(np.cos((kx * i + kz * j) * cell) for i, j in o) - len(o) for o in orbits])
    ata = (psi * w) @ psi.T
    ata[np.diag_indices(len(orbits))] += 1e-12 * np.trace(ata) / len(orbits)
    g = np.linalg.solve(ata, (psi * w) @ kk)
    taps = np.zeros((2 * p + 1, 2 * p + 1), np.float32)
    for v, o in zip(g, orbits):
        for i, j in o:
            taps[j + p, i + p] = v
    taps[p, p] = -sum(v * len(o) for v, o in zip(g, orbits))
    return taps.astype(np.float64)


def _damping(d, dt):
    """The two FP32 coefficients of the damped step, with the absorbing rim."""
    i = np.arange(d.size)
    edge = np.minimum(i, d.size - 1 - i)
    dd = np.minimum(edge[:, None], edge[None, :])
    f = np.float32
    t = (d.absorb_cells - dd).astype(f) / f(d.absorb_cells)
    rim = f(4.0) / max(f(dt) * f(d.absorb_cells), f(1e-6)) * t * t
    ad = (f(d.damping) + np.where(dd < d.absorb_cells, rim, f(0.0))) * f(dt)
    return (f(1.0) / (f(1.0) + ad)).astype(np.float64), (f(1.0) - ad).astype(np.float64)


def _field64(d, discs, substeps):
    """A still field after its first frame of `substeps` steps: (N, N, 4) of height, slopes, velocity."""
    n, p = d.size, d.kernel_radius
    cell, dt, g = _f32(d.extent) / n, _f32(d.fixed_dt), _f32(d.gravity)
    dev = _dev()
    taps = torch.from_numpy(_taps64(p, cell)).to(dev)[None, None]
    c1, c2 = (torch.from_numpy(v).to(dev) for v in _damping(d, dt))
    cur = torch.zeros((n, n), dtype=torch.float64, device=dev)
    old = torch.zeros_like(cur)
    at = torch.arange(n, device=dev).double() + 0.5
    for k in range(substeps):
        for s in discs.frame(0):
            sig = max(float(s["radius"]), 0.25 * cell)
            gx = (float(s["world_x"]) + float(s["velocity_x"]) * k * dt) / cell
            gz = (float(s["world_z"]) + float(s["velocity_z"]) * k * dt) / cell
            r = math.ceil(4.0 * sig / cell)
            x0, x1 = max(0, math.floor(gx) - r), min(n - 1, math.floor(gx) + r)
            z0, z1 = max(0, math.floor(gz) - r), min(n - 1, math.floor(gz) + r)
            u = ((at[None, x0:x1 + 1] - gx) ** 2 + (at[z0:z1 + 1, None] - gz) ** 2) * cell * cell / (2 * sig * sig)
            stamp = (1.0 - u) * torch.exp(-u)
            add = -float(s["strength"]) * dt * (stamp - stamp.mean())
            cur[z0:z1 + 1, x0:x1 + 1] += add
            old[z0:z1 + 1, x0:x1 + 1] += add
        conv = torch.nn.functional.conv2d(cur[None, None], taps, padding=p)[0, 0]
        cur, old = c1 * (2.0 * cur - c2 * old - g * dt * dt * conv), cur
    pad = torch.nn.functional.pad(cur, (1, 1, 1, 1))
    dx = (pad[1:-1, 2:] - pad[1:-1, :-2]) * (0.5 / cell)
    dz = (pad[2:, 1:-1] - pad[:-2, 1:-1]) * (0.5 / cell)
    return torch.stack([cur, dx, dz, (cur - old) / dt], -1)


def _field_height64(d, field, xz):
    """The field's height at world points, bilinear between cell centres, zero outside."""
    n = d.size
    g = xz / (_f32(d.extent) / n) - 0.5
    inside = ((g >= 0) & (g < n - 1)).all(1)
    g = torch.where(inside[:, None], g, torch.zeros_like(g))
    h = _bilinear(field[..., 0].reshape(-1, 1), g[:, 0], g[:, 1], n)[:, 0]
    return torch.where(inside, h, torch.zeros_like(h))


def exact(case, seed):
    kind = case["kind"]
    if kind == "field":
        discs = _Discs(case["sources"], case["extent"], seed)
        return _field64(_field_desc(case), discs, case["substeps"]).reshape(-1, 4)
    descs = _descs(case, seed)
    t = _t0(seed)
    if kind == "serve":
        fd = _field_desc(case)
        rows = []
        for i, d in enumerate(descs):
            xz = torch.from_numpy(_points(case["points"], fd.extent, seed, i)).to(_dev()).double()
            field = _field64(fd, _Discs(case["sources"], fd.extent, seed, i), 1)
            rows.append(_sample64(d, _frame64(d, _tables(d), t), xz)[0][:, 1] + _field_height64(fd, field, xz))
        return torch.stack(rows)
    if kind == "query":
        xz = torch.from_numpy(_points(case["points"], descs[0].patch_length, seed)).to(_dev()).double()
        rec = torch.zeros((case["points"], 10), dtype=torch.float64, device=xz.device)
        clear = torch.ones_like(rec[:, 0])
        for d in descs:
            disp, nm, vel = _sample64(d, _frame64(d, _tables(d), t), xz)
            rec[:, 0] += disp[:, 1]
            rec[:, 1] += disp[:, 0]
            rec[:, 2] += disp[:, 2]
            rec[:, 3:6] += nm
            rec[:, 7:10] += vel
            clear = clear * (1.0 - disp[:, 3])
        rec[:, 3:6] /= torch.linalg.norm(rec[:, 3:6], dim=1, keepdim=True)
        rec[:, 6] = 1.0 - clear
        return rec
    frames, foams = [], []
    for d in descs:
        tables = _tables(d)
        if kind == "batch" and case["foam"]:
            foam = torch.zeros(d.size * d.size, dtype=torch.float64, device=_dev())
            for k in range(FOAM_WARM + 1):
                f = _frame64(d, tables, t + (k - FOAM_WARM) * DT)
                foam = _foam64(d, foam, f[0], f[2])
            foams.append(foam)
        else:
            f = _frame64(d, tables, t)
        frames.append(f)
    names = ("displacement", "normal") + (("velocity",) if case["velocity"] else ())
    if kind == "ocean":
        return {m: frames[0][i] for i, m in enumerate(names)}
    if kind == "cascade":
        return [{"%s_%d" % (m, d.size): f[i][None] for i, m in enumerate(names)} for d, f in zip(descs, frames)]
    out = {}
    for n in sorted({d.size for d in descs}):
        for i, m in enumerate(names):
            out["%s_%d" % (m, n)] = torch.stack([f[i] for d, f in zip(descs, frames) if d.size == n])
    if foams:
        out["foam"] = torch.stack(foams)
    return out
