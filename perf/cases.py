"""Timed cases of the Kirchhoff and Fresnel paths, through the package's public calls.

Each case is one call (or one batch of calls) as a diffraction program makes it.
The sizes and distributions are those of ``xrt_rs.synth``'s benchmark
configurations, ``bench.py``'s workloads and the reference's own pipeline
(beam -> mirror -> screen); ``draw`` spreads more cases over the same ranges.

Fields of the phase-reduced path and of the tensor-core Fresnel product are
single-precision results (requested tolerance 1e-4) in float64 buffers, and a
program keeps them as such: those cases return float32 / complex64. The FP64
paths return float64.
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

_PKG = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "xrt-rs_b200")
if _PKG not in sys.path:
    sys.path.insert(0, _PKG)

import xrt_rs  # noqa: E402

CHBAR = 1973.2697177417986  # eV * Angstrom
RAY = ("x", "y", "z", "nx", "ny", "nz", "nl", "es_re", "es_im", "ep_re", "ep_im", "energy")
PIX = ("x", "y", "z")


# ---- the cases ------------------------------------------------------------------

def _aperture(screen, n, nx, nz, half, energy, dist, sigma, path="f32pr", host=False,
              radius=30000.0):
    return {"kind": "aperture", "screen": screen, "rays": n, "nx": nx, "nz": nz, "half": half,
            "energy": energy, "dist": dist, "sigma": sigma, "radius": radius, "path": path,
            "host": host}


def listed():
    return [
        # The smallest call in use: one line scan, as a program issues it many
        # times while it looks for a focus. Launches and host steps count.
        {"name": "line_scan", **_aperture("line", 10_000, 256, 1, 0.5, 10_000.0, 1000.0, 0.05)},
        # A screen 5 m behind an aperture (a cell of the energy x distance sweep).
        {"name": "screen_far", **_aperture("grid", 1 << 18, 256, 256, 1.0, 20_000.0, 5000.0, 0.1)},
        # The same screen at 100 mm: many ray chunks, the sweep's slowest corner.
        {"name": "screen_near", **_aperture("grid", 1 << 18, 256, 256, 1.0, 20_000.0, 100.0, 0.1)},
        # The benchmark's headline solve, the largest.
        {"name": "screen_large",
         **_aperture("grid", 1 << 20, 512, 512, 0.5, 10_000.0, 1000.0, 0.1)},
        # Propagation from one mirror to the next: scattered points, one normal
        # per ray, two independent polarizations.
        {"name": "mirror_to_mirror", "kind": "mirror", "target": "mirror", "rays": 60_000,
         "nx": 50_021, "nz": 1, "half": 1.0, "energy": 9_000.0, "dist": 3000.0},
        # The reference's parity path at the size of its own benchmark and
        # fixture runs, on host arrays (the default of diffraction_integral).
        {"name": "line_f64_host",
         **_aperture("line", 10_000, 256, 1, 0.5, 10_000.0, 1000.0, 0.05, path="f64", host=True)},
        # The parity path on an ordinary screen.
        {"name": "screen_f64", **_aperture("grid", 1 << 16, 128, 128, 1.0, 10_000.0, 1000.0, 0.1,
                                           path="f64")},
        # Beam columns from a grazing mirror -> rays -> screen -> field, from
        # host arrays; odd screen, two polarizations.
        {"name": "beam_to_screen", "kind": "mirror", "target": "screen", "rays": 200_000,
         "nx": 201, "nz": 151, "half": 1.0, "energy": 10_000.0, "dist": 10_000.0},
        # kirchhoff_gpu on f32 records, the reference's GPU entry point.
        {"name": "gpu_records", "kind": "records", "rays": 50_000, "nx": 128, "nz": 96,
         "half": 0.5, "energy": 12_000.0, "dist": 2000.0, "sigma": 0.1, "radius": 30000.0},
        # bench.py's Fresnel workload: 2^20 rays, 512 x 512.
        {"name": "fresnel_large", "kind": "fresnel", "rays": 1 << 20, "nx": 512, "nz": 512,
         "half": 0.5, "energy": 10_000.0, "dist": 1000.0, "sigma": 0.1, "path": "separable"},
        # A small ragged Fresnel screen of few rays.
        {"name": "fresnel_small", "kind": "fresnel", "rays": 30_011, "nx": 133, "nz": 101,
         "half": 0.4, "energy": 8_000.0, "dist": 1500.0, "sigma": 0.08, "path": "separable"},
        # Many uneven solves at once (lines and square grids), planned and run.
        {"name": "batch_uneven", "kind": "batch", "count": 16, "mix": 17, "rays_lo": 1e3,
         "rays_hi": 2.5e5, "pix_lo": 64, "pix_hi": 65536},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["screen", "screen", "screen", "line", "f64", "mirror", "beam", "records",
                       "fresnel", "batch"])
    energy = round(rng.uniform(1_000.0, 30_000.0), 1)
    sigma = round(rng.uniform(0.02, 0.2), 4)
    radius = round(rng.uniform(10_000.0, 50_000.0), 1)
    if kind == "screen":
        n = int(_log(rng, 2e4, 1 << 19))
        nx, nz = int(_log(rng, 48, 400)), int(_log(rng, 48, 400))
        dist = round(_log(rng, 100.0, 20_000.0), 1)
        return _aperture("grid", n, nx, nz, rng.choice([0.5, 1.0]), energy, dist, sigma,
                         radius=radius)
    if kind == "line":
        n, m = int(_log(rng, 1e3, 2e5)), int(_log(rng, 64, 2e4))
        return _aperture("line", n, m, 1, rng.choice([0.5, 1.0]), energy,
                         round(_log(rng, 300.0, 20_000.0), 1), sigma, radius=radius)
    if kind == "f64":
        n, side = int(_log(rng, 1e3, 6e4)), int(_log(rng, 16, 130))
        return _aperture("grid", n, side, side + rng.randrange(9), 1.0, energy,
                         round(_log(rng, 500.0, 10_000.0), 1), sigma, path="f64",
                         host=rng.random() < 0.5, radius=radius)
    if kind == "mirror":
        return {"kind": "mirror", "target": "mirror", "rays": int(_log(rng, 2e4, 2e5)),
                "nx": int(_log(rng, 4e3, 1e5)), "nz": 1, "half": 1.0,
                "energy": round(rng.uniform(4_000.0, 20_000.0), 1),
                "dist": round(rng.uniform(2_000.0, 10_000.0), 1)}
    if kind == "beam":
        return {"kind": "mirror", "target": "screen", "rays": int(_log(rng, 2e4, 4e5)),
                "nx": int(_log(rng, 48, 300)), "nz": int(_log(rng, 48, 300)), "half": 1.0,
                "energy": round(rng.uniform(4_000.0, 20_000.0), 1),
                "dist": round(rng.uniform(3_000.0, 15_000.0), 1)}
    if kind == "records":
        return {"kind": "records", "rays": int(_log(rng, 1e3, 1e5)), "nx": int(_log(rng, 32, 200)),
                "nz": int(_log(rng, 32, 200)), "half": 0.5, "energy": energy,
                "dist": round(rng.uniform(1_000.0, 5_000.0), 1), "sigma": sigma, "radius": radius}
    if kind == "fresnel":
        return {"kind": "fresnel", "rays": int(_log(rng, 1e4, 1 << 20)),
                "nx": int(_log(rng, 40, 600)), "nz": int(_log(rng, 40, 600)),
                "half": round(rng.uniform(0.2, 1.0), 3), "energy": energy,
                "dist": round(rng.uniform(500.0, 10_000.0), 1), "sigma": sigma,
                "path": "separable"}
    return {"kind": "batch", "count": rng.randint(4, 20), "mix": rng.randrange(1 << 30),
            "rays_lo": 1e3, "rays_hi": 2.5e5, "pix_lo": 64, "pix_hi": 65536}


# ---- inputs, made on the GPU from the seed ----------------------------------------

def _k(energy):
    return energy / CHBAR * 1e7


def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _randn(n, scale, g):
    return torch.randn(n, generator=g, device="cuda", dtype=torch.float64) * scale


def _aperture_rays(n, sigma, energy, radius, g):
    """Gaussian aperture on z = 0 lit by a spherical wave, Ep = 0.1 Es."""
    x, y = _randn(n, sigma, g), _randn(n, sigma, g)
    r2 = x * x + y * y
    mag = torch.exp(-r2 / (4.0 * sigma * sigma))
    ph = _k(energy) * r2 / (2.0 * radius)
    er, ei = mag * torch.cos(ph), mag * torch.sin(ph)
    zero, one = torch.zeros_like(x), torch.ones_like(x)
    return [x, y, zero, zero.clone(), zero.clone(), one, one.clone(), er, ei, 0.1 * er, 0.1 * ei,
            torch.full_like(x, energy)]


def _axis(lo, hi, n):
    return torch.from_numpy(np.linspace(lo, hi, n)).cuda()


def _screen(kind, nx, nz, half, dist):
    """Line along x or grid (x outer, y inner) on the plane z = dist."""
    x = _axis(-half, half, nx)
    if kind == "line":
        return [x, torch.zeros_like(x), torch.full_like(x, dist)]
    y = _axis(-half, half, nz)
    gx, gy = x.repeat_interleave(nz), y.repeat(nx)
    return [gx, gy, torch.full_like(gx, dist)]


THETA = 3e-3  # grazing angle of the mirrors [rad]


def _mirror_beam(n, energy, dist, g):
    """A beam on a mirror at 3 mrad: footprint 0.2 x 15 mm (sigma), tangential
    radius 2 d / THETA, directions converging on the screen centre."""
    big_r = 2.0 * dist / THETA
    x, y = _randn(n, 0.2, g), _randn(n, 15.0, g)
    z = y * y / (2.0 * big_r)
    nrm = torch.stack([torch.zeros_like(y), -y / big_r, torch.ones_like(y)], 1)
    nrm = nrm / nrm.norm(dim=1, keepdim=True)
    d = torch.stack([-x + _randn(n, 0.05, g), dist - y, THETA * dist - z], 1)
    d = d / d.norm(dim=1, keepdim=True)
    mag = torch.exp(-x * x / 0.16 - y * y / 900.0)
    ph = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 0.6 + 20.0 * x
    rot = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 0.4
    es = mag * torch.exp(1j * ph)
    ep = 0.3 * mag * torch.exp(1j * (ph + rot))
    return {"x": x, "y": y, "z": z, "a": d[:, 0].clone(), "b": d[:, 1].clone(),
            "c": d[:, 2].clone(), "e": torch.full_like(x, energy), "es_re": es.real.clone(),
            "es_im": es.imag.clone(), "ep_re": ep.real.clone(), "ep_im": ep.imag.clone()}, nrm


def _rays_of_beam(b, nrm):
    nl = nrm[:, 0] * b["a"] + nrm[:, 1] * b["b"] + nrm[:, 2] * b["c"]
    return [b["x"], b["y"], b["z"], nrm[:, 0].clone(), nrm[:, 1].clone(), nrm[:, 2].clone(), nl,
            b["es_re"], b["es_im"], b["ep_re"], b["ep_im"], b["e"]]


def _wave_params(c):
    return xrt_rs.WaveParams((0.0, c["dist"], THETA * c["dist"]), c["half"], c["half"], c["nx"],
                             c["nz"])


def _batch_sizes(case):
    rng = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        n = int(np.exp(rng.uniform(np.log(case["rays_lo"]), np.log(case["rays_hi"]))))
        m = int(np.exp(rng.uniform(np.log(case["pix_lo"]), np.log(case["pix_hi"]))))
        e, d = float(rng.uniform(5e3, 25e3)), float(rng.uniform(500.0, 10_000.0))
        s, r = float(rng.uniform(0.02, 0.2)), float(rng.uniform(1e4, 5e4))
        side = max(1, int(round(math.sqrt(m))))
        out.append((n, ("grid", side, side) if rng.integers(0, 2) else ("line", m, 1), e, d, s, r))
    return out


def _inputs(case, seed):
    """(rays, points) as device columns, for the Kirchhoff cases."""
    g = _gen(seed)
    if case["kind"] == "aperture":
        return (_aperture_rays(case["rays"], case["sigma"], case["energy"], case["radius"], g),
                _screen(case["screen"], case["nx"], case["nz"], case["half"], case["dist"]))
    if case["kind"] == "records":
        rays = _aperture_rays(case["rays"], case["sigma"], case["energy"], case["radius"], g)
        pix = _screen("grid", case["nx"], case["nz"], case["half"], case["dist"])
        return [a.float().double() for a in rays], [a.float().double() for a in pix]
    beam, nrm = _mirror_beam(case["rays"], case["energy"], case["dist"], g)
    if case["target"] == "screen":
        w = _wave_params(case)
        # prepare_wave's grid: center + (i / (n - 1) - 0.5) * 2 d, x outer.
        fx = np.arange(w.nx) / (w.nx - 1) - 0.5
        fz = np.arange(w.nz) / (w.nz - 1) - 0.5
        x = torch.from_numpy(w.center[0] + fx * 2.0 * w.dx).cuda()
        z = torch.from_numpy(w.center[2] + fz * 2.0 * w.dz).cuda()
        gx = x.repeat_interleave(w.nz)
        return (beam, nrm), [gx, torch.full_like(gx, w.center[1]), z.repeat(w.nx)]
    # The second mirror: scattered points on a cylinder of radius 2 d / THETA.
    m, dist = case["nx"], case["dist"]
    px, py = _randn(m, 0.3, g), _randn(m, 20.0, g)
    pz = THETA * dist + THETA * py + py * py * THETA / (4.0 * dist)
    return (beam, nrm), [px, dist + py, pz]


def _pinned(t):
    out = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    out.copy_(t)
    return out.numpy()


_STREAM = None


def _stream():
    global _STREAM
    if _STREAM is None:
        _STREAM = torch.cuda.Stream()
    return _STREAM


def prepare(case, seed):
    s = {"case": case, "ctx": xrt_rs.GpuContext.shared()}
    kind = case["kind"]
    if kind == "fresnel":
        g = _gen(seed)
        n = case["rays"]
        x, z = _randn(n, case["sigma"], g), _randn(n, case["sigma"], g)
        mag = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * 0.8 + 0.2
        ph = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (2 * math.pi)
        s["rays"] = [_pinned(a) for a in (x, z, mag * torch.cos(ph), mag * torch.sin(ph))]
        h = case["half"]
        s["screen"] = xrt_rs.FresnelScreen(-h, h, case["nx"], -0.8 * h, 0.8 * h, case["nz"])
        return s
    if kind == "batch":
        s["solves"] = []
        for i, (n, scr, e, d, sg, r) in enumerate(_batch_sizes(case)):
            s["solves"].append((_aperture_rays(n, sg, e, r, _gen(seed * 1000 + i)),
                                _screen(*scr, 1.0, d)))
        total = sum(len(p[0]) for _, p in s["solves"])
        s["out"] = torch.zeros(4, total, dtype=torch.float64, device="cuda")
        s["views"], at = [], 0
        for _, p in s["solves"]:
            s["views"].append(tuple(s["out"][c, at:at + len(p[0])] for c in range(4)))
            at += len(p[0])
        torch.cuda.synchronize()
        return s
    rays, pix = _inputs(case, seed)
    if kind == "records":
        rec = np.zeros(case["rays"], dtype=xrt_rs.GPU_RAY_DTYPE)
        for name, a in zip(RAY, rays):
            rec[name] = a.cpu().numpy()
        px = np.zeros(len(pix[0]), dtype=xrt_rs.GPU_PIXEL_DTYPE)
        for name, a in zip(PIX, pix):
            px[name] = a.cpu().numpy()
        s["rec"], s["pix"] = rec, px
        return s
    if kind == "mirror" and case["target"] == "screen":
        beam, nrm = rays
        s["beam"] = {k: _pinned(a) for k, a in beam.items()}
        s["normals"] = _pinned(nrm)
        s["good"] = np.arange(case["rays"], dtype=np.uint64)
        s["params"] = _wave_params(case)
        return s
    if kind == "mirror":
        rays = _rays_of_beam(*rays)
    if case.get("host"):
        s["rays"] = [a.cpu().numpy() for a in rays]
        s["pix"] = [a.cpu().numpy() for a in pix]
        return s
    s["rays"], s["pix"] = rays, pix
    s["out"] = torch.zeros(4, len(pix[0]), dtype=torch.float64, device="cuda")
    torch.cuda.synchronize()
    return s


# ---- one pass -----------------------------------------------------------------------

def run(s):
    case = s["case"]
    kind = case["kind"]
    if kind == "fresnel":
        x, z, er, ei = s["rays"]
        res = xrt_rs.fresnel_propagate(x, z, (er, ei), case["energy"], case["dist"], s["screen"],
                                       path=case["path"], ctx=s["ctx"])
        return res.amplitude.astype(np.complex64)
    if kind == "records":
        es, ep = xrt_rs.kirchhoff_gpu(s["ctx"], s["rec"], s["pix"])
        return np.stack([es, ep]).astype(np.complex64)
    if kind == "mirror" and case["target"] == "screen":
        out = xrt_rs.diffraction_from_beam(s["beam"], s["normals"], s["good"], s["params"],
                                           path="f32pr", ctx=s["ctx"])
        return np.stack(out).astype(np.float32)
    if case.get("host"):
        return list(xrt_rs.diffraction_integral(s["rays"], s["pix"], path=case["path"],
                                                ctx=s["ctx"]))
    st = _stream()
    if kind == "batch":
        # The batch runs on its own stream: the last pass's outputs must have
        # been taken before it writes the buffers again.
        st.synchronize()
        b = xrt_rs.Batch(s["solves"], path="f32pr", ctx=s["ctx"], device_outputs=s["views"])
        b.run()
        b.close()
        with torch.cuda.stream(st):
            return s["out"].float()
    with torch.cuda.stream(st):
        xrt_rs.diffraction_integral_device(s["rays"], s["pix"], list(s["out"]),
                                           path=case.get("path", "f32pr"), ctx=s["ctx"],
                                           stream=st.cuda_stream)
        return s["out"].clone() if case.get("path") == "f64" else s["out"].float()


# ---- what a pass cannot do without ---------------------------------------------------

def work(case):
    """Inputs and outputs once. Per ray and screen point: one complex
    multiply-add (8 flops) for each amplitude column that has to be summed
    (one where all rays share a polarization); the FP64 path evaluates the
    reference's expression with its Kahan sums, 51 operations."""
    kind = case["kind"]
    if kind == "batch":
        b = f = 0.0
        for n, (_, nx, nz), *_ in _batch_sizes(case):
            b += 96.0 * n + 56.0 * nx * nz
            f += 8.0 * n * nx * nz
        return {"bytes": b, "flops": f}
    n, m = float(case["rays"]), float(case["nx"]) * case["nz"]
    if kind == "fresnel":
        return {"bytes": 32 * n + 16 * m, "flops": 8 * n * m}
    if kind == "records":
        return {"bytes": 48 * n + 48 * m, "flops": 8 * n * m}
    if kind == "mirror":
        b = 120 * n + 32 * m if case["target"] == "screen" else 96 * n + 56 * m
        return {"bytes": b, "flops": 16 * n * m}
    return {"bytes": 96 * n + 56 * m, "flops": (51 if case["path"] == "f64" else 8) * n * m}


# ---- the same in 64 bits, without the library -------------------------------------------

_EXACT_PAIRS = 1.2e11  # beyond this the sum below takes too long


def _kirchhoff64(rays, pix, formula):
    """sum_j (es, ep)_j U_j(p) in FP64. ``formula``: the phase k |p - r| as FP64
    rounds it (what the FP64 path computes); otherwise the phase is taken
    relative to one reference ray, |p - r| = |p - r0| + (r0 - r).(2p - r - r0) /
    (|p - r| + |p - r0|), with k |p - r0| reduced in extended precision, so it
    carries no rounding of the whole path."""
    rx, ry, rz, nx, ny, nz, nl, ar, ai, br, bi, e = rays
    px, py, pz = pix
    k = _k(float(e[0]))
    n, m = len(rx), len(px)
    r0 = [float(a.mean()) for a in (rx, ry, rz)]
    ld = [a.cpu().numpy().astype(np.longdouble) - np.longdouble(c) for a, c in zip(pix, r0)]
    d0 = np.sqrt(ld[0] ** 2 + ld[1] ** 2 + ld[2] ** 2)
    turns = np.longdouble(k) * d0 / (2 * np.longdouble("3.14159265358979323846264338327950288"))
    ph0 = torch.from_numpy(np.asarray((turns - np.rint(turns)) * (2 * np.pi), np.float64)).cuda()
    path0 = torch.from_numpy(np.asarray(d0, np.float64)).cuda()
    kf = k / (4.0 * math.pi)
    out = torch.zeros(4, m, dtype=torch.float64, device="cuda")
    cols = torch.stack([ar, ai, br, bi], 0)
    mb = min(m, 1 << 16)
    rows = max(1, (1 << 25) // mb)
    for m0 in range(0, m, mb):
        x, y, z = (a[None, m0:m0 + mb] for a in (px, py, pz))
        p0, f0 = path0[None, m0:m0 + mb], ph0[None, m0:m0 + mb]
        for j0 in range(0, n, rows):
            q = slice(j0, j0 + rows)
            cx, cy, cz = (a[q, None] for a in (rx, ry, rz))
            dx, dy, dz = x - cx, y - cy, z - cz
            path = dx * dx
            path += dy * dy
            path += dz * dz
            path.sqrt_()
            dot = nx[q, None] * dx
            dot += ny[q, None] * dy
            dot += nz[q, None] * dz
            dot /= path
            dot += nl[q, None]
            amp = dot.mul_(kf).div_(path)
            if formula:
                ph = path * k
            else:
                ph = (dx + (x - r0[0])) * (r0[0] - cx)
                ph += (dy + (y - r0[1])) * (r0[1] - cy)
                ph += (dz + (z - r0[2])) * (r0[2] - cz)
                ph /= path + p0
                ph *= k
                ph += f0
            del dx, dy, dz, path
            s, c = torch.sin(ph).mul_(amp), torch.cos(ph).mul_(amp)
            # i amp exp(i phase) = (-s, c)
            w = cols[:, q]
            ws, wc = w @ s, w @ c
            out[0, m0:m0 + mb] += -ws[0] - wc[1]
            out[1, m0:m0 + mb] += wc[0] - ws[1]
            out[2, m0:m0 + mb] += -ws[2] - wc[3]
            out[3, m0:m0 + mb] += wc[2] - ws[3]
    return out


def _fresnel64(case, s):
    x, z, er, ei = (torch.from_numpy(a).cuda() for a in s["rays"])
    sc = s["screen"]
    px = sc.x_min + (sc.x_max - sc.x_min) * torch.arange(sc.nx, device="cuda",
                                                         dtype=torch.float64) / max(sc.nx - 1, 1)
    pz = sc.z_min + (sc.z_max - sc.z_min) * torch.arange(sc.nz, device="cuda",
                                                         dtype=torch.float64) / max(sc.nz - 1, 1)
    a = _k(case["energy"]) / (2.0 * case["dist"])
    out = torch.zeros(sc.nz, sc.nx, dtype=torch.complex128, device="cuda")
    for j in range(0, len(x), 1 << 17):
        q = slice(j, j + (1 << 17))
        tx = (px[None, :] - x[q, None]).square_().mul_(a)
        tz = (pz[:, None] - z[None, q]).square_().mul_(a)
        w = torch.polar(torch.ones_like(tx), tx) * torch.complex(er[q], ei[q])[:, None]
        out += torch.polar(torch.ones_like(tz), tz) @ w
    return out.reshape(-1).cpu().numpy()


def exact(case, seed):
    kind = case["kind"]
    if kind == "batch":
        if work(case)["flops"] / 8 > _EXACT_PAIRS:
            return None
        s = prepare(case, seed)
        return torch.cat([_kirchhoff64(r, p, False) for r, p in s["solves"]], 1)
    if float(case["rays"]) * case["nx"] * case["nz"] > _EXACT_PAIRS and kind != "fresnel":
        return None
    if kind == "fresnel":
        return _fresnel64(case, prepare(case, seed))
    rays, pix = _inputs(case, seed)
    if kind == "mirror":
        rays = _rays_of_beam(*rays)
    out = _kirchhoff64(rays, pix, case.get("path") == "f64")
    if kind == "records":
        o = out.cpu().numpy()
        return np.stack([o[0] + 1j * o[1], o[2] + 1j * o[3]])
    if case.get("host"):
        return [a.cpu().numpy() for a in out]
    return out.cpu().numpy() if kind == "mirror" and case["target"] == "screen" else out
