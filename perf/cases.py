"""The work that users of this framework have it do, as timed cases.

Each case is one call sequence through the public entry points of the package
(``jpet_strip.capi``, ``jpet_strip.hybrid``).  Kinds of cases:

* ``iterate``: a reconstruction that a program holds (events set once) runs some
  MLEM iterations from a given image;
* ``run``: the whole drop-in call over host buffers: set-up, upload, event
  preparation, iterations, image back;
* ``batch``: many reconstructions of uneven sizes iterated together;
* ``nll``: likelihood, image gradient and width gradients of held events;
* ``hybrid``: 3D hybrid iterations and the image read back;
* ``generate``: the phantom Monte Carlo.

Sizes are those of the package's own workloads, or lie in the ranges of its
batched workload (grids of 100..500 by 100..450 pixels of 2..5 mm, widths of
6..14 and 30..60 mm, 1e4..5e6 events).  Inputs come from the seed alone; events
are drawn from ellipse phantoms, smeared by the detector widths.
"""
from __future__ import annotations

import functools
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "j-pet-mlem_gb300", "python"))

from jpet_strip import capi, hybrid, hybrid_workloads, phantom, workloads  # noqa: E402

RADIUS, LENGTH = 450.0, 1000.0  # the strip scanner of every workload, mm
PRECISIONS = {"fp32": capi.PRECISION_FP32, "compensated": capi.PRECISION_COMPENSATED,
              "fp64_den": capi.PRECISION_FP64_DEN, "fixed": capi.PRECISION_FIXED}
MODES = {"cpu": capi.MODE_CPU_REFERENCE, "gpu": capi.MODE_GPU_REFERENCE}


def _iterate(name, n, n_y, n_z, pixel, sz, sdl, iterations, phantom_name="random10",
             precision="fp32", mode="cpu"):
    return dict(name=name, kind="iterate", n=n, n_y=n_y, n_z=n_z, pixel=pixel, sigma_z=sz,
                sigma_dl=sdl, iterations=iterations, phantom=phantom_name, precision=precision,
                mode=mode)


def listed():
    return [
        # a short acquisition on a coarse odd-sized grid, as a live preview shows it:
        # launches and latency count
        _iterate("iterate-small", 20_011, 101, 117, 5.0, 10.0, 42.0, 10),
        # the CPU-runnable workload: 1e6 events at 5 mm, ten iterations
        _iterate("iterate-5mm-1M", 1_000_000, 180, 200, 5.0, 10.0, 42.0, 10, "three"),
        # the full-size workload: 2e7 events at 2 mm
        _iterate("iterate-2mm-20M", 20_000_000, 450, 500, 2.0, 10.0, 42.0, 1),
        # the stress workload's grid and widths: 1 mm pixels, narrow widths, lesions
        _iterate("iterate-1mm-6M", 6_000_003, 900, 1000, 1.0, 5.0, 20.0, 1, "lesions"),
        # reconstruction at the mis-specified widths that a recalibration starts from
        _iterate("iterate-wide-1M", 1_000_000, 450, 500, 2.0, 14.0, 55.0, 2),
        # an accuracy run: compensated sums
        _iterate("compensated-2mm-2M", 2_000_000, 450, 500, 2.0, 10.0, 42.0, 3,
                 precision="compensated"),
        # the reference GPU backend's semantics (analytic kernel, weighted denominator)
        _iterate("gpu-semantics-300k", 300_007, 180, 200, 5.0, 10.0, 42.0, 2, "three",
                 mode="gpu"),
        # the drop-in call of an ordinary scan: host events in, image after 20 iterations out
        dict(name="run-2mm-1M", kind="run", n=1_000_003, n_y=225, n_z=251, pixel=2.0,
             sigma_z=10.0, sigma_dl=42.0, iterations=20, phantom="random10"),
        # a study of uneven reconstructions, tuned once and iterated together
        dict(name="batch-12", kind="batch", instances=12, min_n=10_000, max_n=1_000_000,
             iterations=10),
        # one step of a width calibration or a gradient-based reconstruction
        dict(name="nll-2mm-500k", kind="nll", n=500_009, n_y=450, n_z=500, pixel=2.0,
             sigma_z=14.0, sigma_dl=55.0, kernel_z=12.5, kernel_dl=50.0, phantom="random10"),
        # the 3D hybrid benchmark geometry (384 detectors, 200 x 200 x 125 voxels)
        dict(name="hybrid-384-1M", kind="hybrid", geometry="hybrid-384", n=1_000_000,
             iterations=5),
        # events of a phantom for a simulation study
        dict(name="generate-2M", kind="generate", n=2_000_003, phantom="random10", sigma_z=10.0,
             sigma_dl=42.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["iterate"] * 5 + ["run", "batch", "nll", "hybrid", "generate"])
    if kind == "batch":
        return dict(kind=kind, instances=rng.randint(2, 24), min_n=_log(rng, 3e3, 2e4),
                    max_n=_log(rng, 1e5, 1e6), iterations=rng.randint(1, 6))
    if kind == "hybrid":
        return dict(kind=kind, geometry="hybrid-96", n=_log(rng, 5e3, 5e5),
                    iterations=rng.randint(1, 5))
    if kind == "generate":
        return dict(kind=kind, n=_log(rng, 1e3, 4e6), phantom=rng.choice(["three", "random10"]),
                    sigma_z=round(rng.uniform(5.0, 14.0), 2),
                    sigma_dl=round(rng.uniform(20.0, 60.0), 2))
    g = dict(n_y=rng.randint(60, 450), n_z=rng.randint(60, 500),
             pixel=round(rng.uniform(2.0, 5.0), 2), sigma_z=round(rng.uniform(6.0, 14.0), 2),
             sigma_dl=round(rng.uniform(30.0, 60.0), 2),
             phantom=rng.choice(["three", "random10"]))
    if kind == "nll":
        return dict(kind=kind, n=_log(rng, 1e4, 1e6), **g,
                    kernel_z=round(g["sigma_z"] * rng.uniform(0.8, 1.0), 2),
                    kernel_dl=round(g["sigma_dl"] * rng.uniform(0.8, 1.0), 2))
    if kind == "run":
        return dict(kind=kind, n=_log(rng, 1e4, 1e6), iterations=rng.randint(1, 20), **g)
    mode = rng.choice(["cpu"] * 7 + ["gpu"])
    precision = rng.choice(["fp32"] * 4 + ["compensated", "fixed", "fp64_den"])
    n = _log(rng, 5e3, 3e5 if mode == "gpu" else 4e6)
    return dict(kind=kind, n=n, iterations=rng.randint(1, 10 if n < 3e5 else 2), mode=mode,
                precision="fp32" if mode == "gpu" else precision, **g)


# ---- inputs --------------------------------------------------------------------------


def _ellipses(c, seed):
    if c["phantom"] == "three":
        return phantom.three_ellipse_phantom()
    if c["phantom"] == "lesions":
        return phantom.lesion_phantom(seed)
    # ten ellipses inside the part of the grid that the scanner sees
    hz = min(c.get("n_z", 500) * c.get("pixel", 2.0) / 2, LENGTH / 2)
    hy = min(c.get("n_y", 450) * c.get("pixel", 2.0) / 2, RADIUS)
    return phantom.random_ellipse_phantom(seed, half_z=hz, half_y=hy, centre_z=0.6 * hz,
                                          centre_y=0.6 * hy, axes=(10.0, 0.8 * min(hz, hy)))


def _events(ellipses, n, sz, sdl, seed):
    """float32[n, 3] detected, smeared responses of the ellipses, on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))

    def u(m):
        return torch.rand(m, generator=gen, device="cuda", dtype=torch.float64)

    par = torch.tensor([(e.z, e.y, e.a, e.b, math.radians(e.angle_deg)) for e in ellipses],
                       dtype=torch.float64, device="cuda")
    cdf = torch.tensor(np.cumsum([e.intensity * e.area for e in ellipses]), device="cuda")
    parts, have = [], 0
    while have < n:
        m = min(int((n - have) * 1.8) + 4096, 1 << 22)
        k = torch.searchsorted(cdf, u(m) * cdf[-1]).clamp_(max=len(ellipses) - 1)
        cz, cy, a, b, ang = par[k].unbind(1)
        r, th = u(m).sqrt(), 2 * math.pi * u(m)
        ex, ey = a * r * th.cos(), b * r * th.sin()
        z = ang.cos() * ex - ang.sin() * ey + cz
        y = ang.sin() * ex + ang.cos() * ey + cy
        t = torch.tan(math.atan(LENGTH / (2 * RADIUS)) * (2 * u(m) - 1))
        ev = torch.stack([z + (RADIUS - y) * t, z - (RADIUS + y) * t,
                          -2 * y * (1 + t * t).sqrt()], 1)
        noise = torch.randn(m, 3, generator=gen, device="cuda", dtype=torch.float64)
        ok = (ev[:, :2].abs() < LENGTH / 2).all(1) & (y.abs() < RADIUS)
        ev = ev + noise * torch.tensor([sz, sz, sdl], device="cuda")
        ev = ev[ok].float()
        parts.append(ev)
        have += ev.shape[0]
    return torch.cat(parts)[:n].contiguous()


def _geometry(c):
    return capi.Geometry(RADIUS, LENGTH, c["n_y"], c["n_z"], c["pixel"], c["sigma_z"],
                         c["sigma_dl"])


def _case_events(c, seed):
    # events off the grid are part of a real acquisition and stay
    return _events(_ellipses(c, seed), c["n"], c["sigma_z"], c["sigma_dl"], seed)


@functools.lru_cache(maxsize=None)
def _stream():
    """The stream that the program runs its reconstructions on, one after another."""
    return torch.cuda.Stream()


def _held(c, seed, **opts):
    ev = _case_events(c, seed)
    soa = ev.t().contiguous()
    torch.cuda.synchronize()
    rec = capi.StripReconstruction(_geometry(c), **opts)
    rec.set_stream(_stream().cuda_stream)
    rec.set_events_device(soa[0].data_ptr(), soa[1].data_ptr(), soa[2].data_ptr(), c["n"])
    return rec


class _Image:
    def __init__(self, rec):
        self.__cuda_array_interface__ = dict(
            shape=(rec.geom.n_y, rec.geom.n_z), typestr="<f4", version=2, strides=None,
            data=(rec.image_device_ptr(), False))


def _image(rec, owner):
    """A reconstruction's device image as a tensor (no copy) that keeps the owner of the
    device memory alive."""
    view = _Image(rec)
    view.owner = owner
    t = torch.as_tensor(view, device="cuda")
    t.owner = owner
    return t


def _batch_instances(c):
    # the geometries are the workload's for every seed, as a study is planned once
    return workloads.batch_instances(c["instances"], max_events=c["max_n"],
                                     min_events=c["min_n"])


def _batch_events(wl, ellipses, seed, i):
    return _events(ellipses, wl.n_events, wl.sigma_z, wl.sigma_dl, seed * 1009 + i)


@functools.lru_cache(maxsize=2)
def _hybrid_geometry(name):
    return hybrid_workloads.workload(name)[0]


def _hybrid_responses(g, n, seed):
    """int16 (lor) and float32 fields of n detected responses of an ellipsoid phantom, packed
    as the hybrid scanner's 16-byte responses on the GPU."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    f64 = dict(dtype=torch.float64, device="cuda")

    def u(m):
        return torch.rand(m, generator=gen, **f64)

    ph = hybrid_workloads.ellipsoid_phantom(g.radius, g.length, 3 + seed % 1000)
    wt = torch.tensor([p[2] * float(np.prod(p[1])) for p in ph], **f64)
    cen, axes = (torch.tensor([p[i] for p in ph], **f64) for i in (0, 1))
    seg = {k: torch.from_numpy(np.ascontiguousarray(g.segments[k])).cuda().double()
           for k in ("mid_x", "mid_y", "dir_x", "dir_y", "length")}
    parts, have = [], 0
    while have < n:
        m = int((n - have) * 1.6) + 4096
        k = torch.searchsorted(wt.cumsum(0), u(m) * wt.sum()).clamp_(max=len(ph) - 1)
        d3 = torch.randn(m, 3, generator=gen, **f64)
        p = cen[k] + d3 / d3.norm(dim=1, keepdim=True) * u(m).pow(1 / 3)[:, None] * axes[k]
        phi, tn = math.pi * u(m), 2 * u(m) - 1
        d = torch.stack([phi.cos(), phi.sin()], 1)
        pd = (p[:, :2] * d).sum(1)
        disc = pd * pd - (p[:, :2] ** 2).sum(1) + g.radius ** 2
        sq = disc.clamp(min=0).sqrt()
        step = 2 * math.pi / g.n_detectors

        def det(q):
            return torch.remainder(torch.round(torch.atan2(q[:, 1], q[:, 0]) / step),
                                   g.n_detectors).long()

        i1 = det(p[:, :2] + d * (sq - pd)[:, None])
        i2 = det(p[:, :2] - d * (sq + pd)[:, None])
        f, s = torch.maximum(i1, i2), torch.minimum(i1, i2)
        lor = f * (f + 1) // 2 + s
        up = ((p[:, 0] - seg["mid_x"][lor]) * seg["dir_x"][lor] +
              (p[:, 1] - seg["mid_y"][lor]) * seg["dir_y"][lor])
        R = seg["length"][lor] / 2
        zu, zd = p[:, 2] + (R - up) * tn, p[:, 2] - (R + up) * tn
        ok = (disc > 0) & (i1 != i2) & (zu.abs() <= g.length / 2) & (zd.abs() <= g.length / 2)
        ok &= up.abs() < R
        noise = torch.randn(m, 3, generator=gen, **f64)
        val = torch.stack([zu + noise[:, 0] * g.sigma_z, zd + noise[:, 1] * g.sigma_z,
                           -2 * up * (1 + tn * tn).sqrt() + noise[:, 2] * g.sigma_dl], 1).float()
        words = torch.empty(m, 4, dtype=torch.int32, device="cuda")
        words[:, 0] = (f + s * 65536).int()
        words[:, 1:] = val.view(torch.int32)
        parts.append(words[ok])
        have += parts[-1].shape[0]
    return torch.cat(parts)[:n].contiguous()


def prepare(case, seed):
    c, kind = dict(case), case["kind"]
    state = {"case": c, "seed": seed}
    if kind == "iterate":
        state["rec"] = _held(c, seed, precision=PRECISIONS[c["precision"]], mode=MODES[c["mode"]])
        state["start"] = torch.ones(c["n_y"], c["n_z"], device="cuda")
    elif kind == "run":
        state["events"] = _case_events(c, seed).cpu().numpy()
        state["geom"] = _geometry(c)
    elif kind == "batch":
        inst = _batch_instances(c)
        b = capi.StripBatch([capi.Geometry(*wl.geometry_args()) for wl, _ in inst])
        for i, (wl, ell) in enumerate(inst):
            ev = _batch_events(wl, ell, seed, i)
            torch.cuda.synchronize()
            b.set_events(i, ev)
        b.tune()
        state["batch"] = b
        state["start"] = [torch.ones(wl.n_y, wl.n_z, device="cuda") for wl, _ in inst]
    elif kind == "nll":
        state["rec"] = _held(c, seed)
        state["rho"] = _nll_image(c, seed)
        state["grad"] = torch.empty_like(state["rho"])
    elif kind == "hybrid":
        g = _hybrid_geometry(c["geometry"])
        resp = _hybrid_responses(g, c["n"], seed)
        torch.cuda.synchronize()
        rec = hybrid.HybridReconstruction(g)
        rec.set_responses_device(resp.data_ptr(), c["n"])
        rec.set_stream(_stream().cuda_stream)
        state["rec"] = rec
        state["start"] = np.ones(g.n_voxels, np.float32)
    elif kind == "generate":
        state["regions"] = _ellipses(c, seed)
    return state


def _nll_image(c, seed):
    """A positive, uneven image with the events' total: what an optimiser holds midway."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed) + 77)
    x = torch.rand(1, 1, c["n_y"] // 8 + 2, c["n_z"] // 8 + 2, generator=gen, device="cuda")
    x = torch.nn.functional.interpolate(x, size=(c["n_y"], c["n_z"]), mode="bilinear")[0, 0]
    x = x + 0.2
    return (x * (c["n"] / x.sum())).contiguous()


def run(state):
    c, kind = state["case"], state["case"]["kind"]
    if kind == "iterate":
        rec = state["rec"]
        rec.set_image_device(state["start"].data_ptr())
        rec.iterate(c["iterations"])
        return _image(rec, rec)
    if kind == "run":
        rho = np.ones((c["n_y"], c["n_z"]), np.float32)
        capi.run(state["geom"], state["events"], rho, 1, c["iterations"])
        return rho
    if kind == "batch":
        b = state["batch"]
        for i, start in enumerate(state["start"]):
            b.instance(i).set_image_device(start.data_ptr())
        b.iterate(c["iterations"])
        return [_image(b.instance(i), b) for i in range(len(b))]
    if kind == "nll":
        loss, gs, skipped = state["rec"].nll_grad(c["kernel_z"], c["kernel_dl"],
                                                  state["rho"].data_ptr(), None,
                                                  state["grad"].data_ptr())
        return {"loss": loss, "grad_sigma": list(gs), "skipped": skipped,
                "grad_rho": state["grad"]}
    if kind == "hybrid":
        rec = state["rec"]
        rec.rho = state["start"]
        rec.iterate(c["iterations"])
        return rec.rho
    if kind == "generate":
        return capi.generate_device(state["regions"], c["n"], RADIUS, LENGTH, c["sigma_z"],
                                    c["sigma_dl"], seed=state["seed"])
    raise ValueError(kind)


# ---- what a pass cannot do without ---------------------------------------------------------


def _pixels_per_event(pixel, sz, sdl, sec=1.1):
    # area of the 3-sigma ellipse over the pixel's
    return 9 * math.pi * sz * sdl / (math.sqrt(8) * sec) / pixel ** 2


def work(case):
    c, kind = case, case["kind"]
    if kind in ("iterate", "run"):
        ev = c["n"] * _pixels_per_event(c["pixel"], c["sigma_z"], c["sigma_dl"])
        px = c["n_y"] * c["n_z"]
        # per kernel value: its exponent (2 FMA) and exp, K rho and its sum, K rho / den added
        return {"bytes": 12.0 * c["n"] + 8.0 * px, "flops": 9.0 * ev * c["iterations"]}
    if kind == "batch":
        inst = _batch_instances(c)
        return {"bytes": sum(12.0 * w.n_events + 8.0 * w.n_y * w.n_z for w, _ in inst),
                "flops": sum(9.0 * c["iterations"] * w.n_events *
                             _pixels_per_event(w.pixel, w.sigma_z, w.sigma_dl) for w, _ in inst)}
    if kind == "nll":
        ev = c["n"] * _pixels_per_event(c["pixel"], c["sigma_z"], c["sigma_dl"])
        return {"bytes": 12.0 * c["n"] + 12.0 * c["n_y"] * c["n_z"], "flops": 15.0 * ev}
    if kind == "hybrid":
        w = hybrid_workloads.HYBRID_WORKLOADS[c["geometry"]]
        vox = w["n_pixels"] ** 2 * w["n_planes"]
        # voxels of an event: the 3-sigma ellipse along the LOR and z, times the LOR's width
        per = _pixels_per_event(w["pixel_size"], w["sigma_z"], w["sigma_dl"]) * (
            2 * w["width"] / w["pixel_size"])
        return {"bytes": 16.0 * c["n"] + 8.0 * vox, "flops": 9.0 * c["n"] * per * c["iterations"]}
    # generate: the region, the point, the angle and the three normals of a candidate
    return {"bytes": 12.0 * c["n"], "flops": 200.0 * c["n"]}


# ---- the same in 64 bits, without the package's code -----------------------------------------


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind in ("iterate", "run"):
        ev = _case_events(c, seed)
        return _mlem64(ev, c["n_y"], c["n_z"], c["pixel"], c["sigma_z"], c["sigma_dl"],
                       c["iterations"], c.get("mode") == "gpu")
    if kind == "batch":
        return [_mlem64(_batch_events(w, ell, seed, i), w.n_y, w.n_z, w.pixel, w.sigma_z,
                        w.sigma_dl, c["iterations"])
                for i, (w, ell) in enumerate(_batch_instances(c))]
    if kind == "nll":
        return _nll64(c, seed)
    if kind == "hybrid":
        return _hybrid64(c, seed)
    return _generate64(c, seed)


def _sens64(z, y, half):
    def pos(v):
        return torch.where(v <= 0, torch.ones_like(v), v)

    rp, rm = pos(RADIUS + y), pos(RADIUS - y)
    return (torch.atan(torch.minimum((half - z) / rm, (half + z) / rp)) -
            torch.atan(torch.maximum(-(half + z) / rm, -(half - z) / rp))) / math.pi


class _Grid64:
    def __init__(self, n_y, n_z, p):
        self.n_y, self.n_z, self.p = n_y, n_z, p
        self.top, self.left = n_y * p / 2, -n_z * p / 2

    def centres(self):
        z = self.left + self.p / 2 + self.p * torch.arange(self.n_z, device="cuda").double()
        y = self.top - self.p / 2 - self.p * torch.arange(self.n_y, device="cuda").double()
        return z[None, :], y[:, None]


def _supports64(ev, grid, sz, sdl):
    """Per chunk of events: (y, tan, sec, dy, dz, flat pixel index, inside) of a stripe of
    pixels around each event's 3-sigma ellipse; inside says which belong to it."""
    ipz, ipd, p = 1 / sz ** 2, 1 / sdl ** 2, grid.p
    half_cols = 3 / math.sqrt(2 * ipz) / p
    cols = torch.arange(2 * int(half_cols) + 5, device="cuda")
    max_rows = 2 * int(3 / math.sqrt(4 * ipd) / p + 1.5) + 2
    step = max(1, int(2.5e7 // (max_rows * len(cols))))
    for s in range(0, len(ev), step):
        e = ev[s:s + step].double()
        t = (e[:, 0] - e[:, 1]) / (2 * RADIUS)
        sec = (1 + t * t).sqrt()
        y = -0.5 * e[:, 2] / sec
        z = 0.5 * (e[:, 0] + e[:, 1] + 2 * y * t)
        A, B, C = 4 * sec * sec * ipd + 2 * t * t * ipz, -4 * t * ipz, 2 * ipz
        hy = 3 / (A - B * B / (4 * C)).sqrt()
        hz = 3 / (C - B * B / (4 * A)).sqrt()
        cx, cy = ((z - grid.left) / p).trunc(), ((grid.top - y) / p).trunc()
        hw, hh = (hz / p + 0.5).trunc(), (hy / p + 0.5).trunc()
        x0, x1 = (cx - hw).clamp(0, grid.n_z - 1), (cx + hw).clamp(0, grid.n_z - 1)
        y0, y1 = (cy - hh).clamp(0, grid.n_y - 1), (cy + hh).clamp(0, grid.n_y - 1)
        rows = y0[:, None] + torch.arange(max_rows, device="cuda")
        dy = grid.top - p / 2 - rows * p - y[:, None]
        left = ((z[:, None] + t[:, None] * dy - grid.left) / p - 0.5 - half_cols).floor() - 1
        col = left[:, :, None] + cols
        dz = grid.left + p / 2 + col * p - z[:, None, None]
        dy = dy[:, :, None]
        q = (A[:, None, None] * dy + B[:, None, None] * dz) * dy + C * dz * dz
        ok = (q <= 9) & (col >= x0[:, None, None]) & (col < x1[:, None, None])
        ok &= (rows < y1[:, None])[:, :, None]
        del q
        # pixels outside the support get a zero: they need an index, not its value
        idx = (rows.clamp(max=grid.n_y - 1) * grid.n_z)[:, :, None] + col.clamp(0, grid.n_z - 1)
        idx = idx.long()
        yield (v[:, None, None] if v.dim() == 1 else v for v in (y, t, sec, dy, dz, idx, ok))


def _mlem64(ev, n_y, n_z, p, sz, sdl, iterations, gpu_semantics=False):
    grid = _Grid64(n_y, n_z, p)
    ipz, ipd = 1 / sz ** 2, 1 / sdl ** 2
    rho = torch.ones(n_y * n_z, dtype=torch.float64, device="cuda")
    sens = None
    if gpu_semantics:
        cz, cy = grid.centres()
        h, half = p / 2, LENGTH / 2
        sens = (_sens64(cz, cy, half) / 3 + _sens64(cz + h, cy + h, half) / 6 +
                _sens64(cz - h, cy - h, half) / 6 + _sens64(cz - h, cy + h, half) / 6 +
                _sens64(cz + h, cy - h, half) / 6).reshape(-1)
    for _ in range(iterations):
        out = torch.zeros_like(rho)
        for y, t, sec, dy, dz, idx, ok in _supports64(ev, grid, sz, sdl):
            py = dy + y
            if gpu_semantics:
                ap, aq = -(py - RADIUS) * sec ** 2, -(py + RADIUS) * sec ** 2
                ar, br = -2 * py * sec * t, -2 * dy * sec
                orr = -py * sec * (1 + 2 * t * t)
                b = dz - dy * t
                a_a = (ap * ap + aq * aq) * ipz + ar * ar * ipd
                b_a = b * (ap + aq) * ipz + br * ar * ipd
                b_b = 2 * b * b * ipz + br * br * ipd
                o_b = b * (ap + aq) * t * ipz + orr * br * ipd
                norm = a_a + 2 * o_b
                k = norm.rsqrt() * torch.exp(-0.5 * (b_b - b_a * b_a / norm))
            else:
                a_a = 2 * sec ** 4 * (py * py + RADIUS ** 2) * ipz + (2 * py * sec * t) ** 2 * ipd
                b = dz - dy * t
                k = a_a.rsqrt() * torch.exp(-(b * b) * ipz - 2 * (dy * sec) ** 2 * ipd)
            k = torch.where(ok, k, 0.0) * rho[idx]
            den = ((k * sens[idx]) if gpu_semantics else k).sum((1, 2), keepdim=True)
            k = torch.where(den > 0, k / torch.where(den > 0, den, 1.0), 0.0)
            out.index_add_(0, idx.reshape(-1), k.reshape(-1))
        rho = out
    return rho.reshape(n_y, n_z)


def _nll64(c, seed):
    ev = _case_events(c, seed)
    grid = _Grid64(c["n_y"], c["n_z"], c["pixel"])
    rho = _nll_image(c, seed).double().reshape(-1)
    kz, kdl = c["kernel_z"], c["kernel_dl"]
    ipz, ipd = 1 / kz ** 2, 1 / kdl ** 2
    log_c0 = math.log(1 / (2 * math.pi ** 2) * ipz * math.sqrt(ipd))
    cz, cy = grid.centres()
    s = _sens64(cz, cy, LENGTH / 2).reshape(-1)
    loss, gz, gdl, skipped = (s * rho).sum(), 0.0, 0.0, 0
    grad = s.clone()
    for y, t, sec, dy, dz, idx, ok in _supports64(ev, grid, c["sigma_z"], c["sigma_dl"]):
        py = dy + y
        pa = 2 * sec ** 4 * (py * py + RADIUS ** 2)
        qa = 4 * sec ** 2 * t ** 2 * py * py
        a_a = pa * ipz + qa * ipd
        u2 = (dz - dy * t) ** 2
        v2 = 2 * sec ** 2 * dy * dy
        k = torch.where(ok, a_a.rsqrt() * torch.exp(-u2 * ipz - v2 * ipd), 0.0)
        kr = k * rho[idx]
        den = kr.sum((1, 2), keepdim=True)
        d_z = (kr * (1 / ipz - 0.5 * pa / a_a - u2)).sum((1, 2), keepdim=True)
        d_l = (kr * (0.5 / ipd - 0.5 * qa / a_a - v2)).sum((1, 2), keepdim=True)
        good = den > 0
        safe = torch.where(good, den, 1.0)
        loss = loss - torch.where(good, safe.log() + log_c0, 0.0).sum()
        gz = gz - torch.where(good, d_z / safe, 0.0).sum() * (-2 / kz ** 3)
        gdl = gdl - torch.where(good, d_l / safe, 0.0).sum() * (-2 / kdl ** 3)
        skipped += int((~good).sum())
        grad.index_add_(0, idx.reshape(-1), torch.where(good, -k / safe, 0.0).reshape(-1))
    return {"loss": loss.reshape(1), "grad_sigma": [gz.reshape(1), gdl.reshape(1)],
            "skipped": None, "grad_rho": grad.reshape(c["n_y"], c["n_z"])}


def _hybrid64(c, seed):
    g = _hybrid_geometry(c["geometry"])
    dev = "cuda"

    def field(a):
        return torch.from_numpy(np.ascontiguousarray(a)).to(dev)

    px, py = field(g.pixels["x"]).long(), field(g.pixels["y"]).long()
    pix = px + g.n_columns * py
    pos = field(g.positions).double()
    seg = {k: field(g.segments[k]).double() for k in
           ("mid_x", "mid_y", "dir_x", "dir_y", "normal_x", "normal_y", "length",
            "distance_from_origin")}
    begin, end = field(g.info_begin.astype(np.int64)), field(g.info_end.astype(np.int64))
    lor = torch.repeat_interleave(torch.arange(g.n_lors, device=dev), end - begin)
    ps = g.pixel_size
    cx, cy = g.lower_left_x + ps / 2 + px * ps, g.lower_left_y + ps / 2 + py * ps
    d = cx * seg["normal_x"][lor] + cy * seg["normal_y"][lor] - seg["distance_from_origin"][lor]
    sw = 0.3 * field(g.widths).double()[lor]
    w = torch.exp(-d * d / (2 * sw * sw)) / (sw * math.sqrt(2 * math.pi))
    n_px = g.n_columns * g.n_rows
    sens = torch.zeros(n_px, dtype=torch.float64, device=dev).index_add_(0, pix, w)
    wn = w / sens[pix]
    # events in their LOR's frame
    words = _hybrid_responses(g, c["n"], seed)
    f, s = words[:, 0] & 0xffff, words[:, 0] >> 16
    zu, zd, dl = words[:, 1:].contiguous().view(torch.float32).double().unbind(1)
    el = (f.long() * (f.long() + 1)) // 2 + s.long()
    R = seg["length"][el] / 2
    t = (zu - zd) / (2 * R)
    sec = (1 + t * t).sqrt()
    up = -0.5 * dl / sec
    right = 0.5 * (zu + zd + 2 * up * t)
    ipz, ipd = 1 / g.sigma_z ** 2, 1 / g.sigma_dl ** 2
    A, B, C = 4 * sec * sec * ipd + 2 * t * t * ipz, -4 * t * ipz, 2 * ipz
    h_up, h_rt = 3 / (A - B * B / (4 * C)).sqrt(), 3 / (C - B * B / (4 * A)).sqrt()
    p0 = ((right - h_rt - g.z_left) / ps).trunc().clamp(min=0).long()
    p1 = (((right + h_rt - g.z_left) / ps).trunc() + 1).clamp(max=g.n_planes).long()
    key = lor * 4.0 + pos  # ascending: positions lie in [0, 1] and ascend within a LOR

    def at(v, side):
        b = torch.searchsorted(key, el * 4.0 + v.clamp(-1, 2), side=side)
        return torch.minimum(torch.maximum(b, begin[el]), end[el])

    i1 = (at((up + h_up + R) / (2 * R), "right") + 1).clamp(max=len(pos))
    i0 = at((up - h_up + R) / (2 * R), "left")
    keep = (p1 > 0) & (p0 < g.n_planes) & (p1 > p0) & (i1 > i0)
    order = torch.nonzero(keep)[:, 0]
    order = order[torch.argsort((i1 - i0)[order])]
    n_pl = int((p1 - p0)[order].max())
    rho = torch.ones(n_px * g.n_planes, dtype=torch.float64, device=dev)
    half = g.length / 2
    chunks, at_ = [], 0
    while at_ < len(order):  # events of like info counts together
        take = max(1, int(1.5e7 // (n_pl * int((i1 - i0)[order[min(len(order) - 1,
                                                                   at_ + 20000)]]) + 1)))
        chunks.append(order[at_:at_ + min(take, 20000)])
        at_ += len(chunks[-1])
    for _ in range(c["iterations"]):
        out = torch.zeros_like(rho)
        for ch in chunks:
            n_in = (i1 - i0)[ch]
            j = torch.arange(int(n_in.max()), device=dev)
            oki = j < n_in[:, None]
            info = torch.where(oki, i0[ch][:, None] + j, 0)
            last = pix[i1[ch] - 1][:, None]
            same = oki & (pix[info] == last) & (j < n_in[:, None] - 1)
            # a voxel that the range holds twice is added twice with its last value
            mult = torch.where(same, 0.0, 1.0)
            mult = mult + ((j == n_in[:, None] - 1) & same.any(1, keepdim=True))

            def ev(v):
                return v[ch][:, None]

            u = ((cx[info] - ev(seg["mid_x"][el])) * ev(seg["dir_x"][el]) +
                 (cy[info] - ev(seg["mid_y"][el])) * ev(seg["dir_y"][el]))
            eR, es, et = ev(R), ev(sec), ev(t)
            dy = u - ev(up)
            a_a = 2 * es ** 4 * (u * u + eR * eR) * ipz + (2 * u * es * et) ** 2 * ipd
            base = a_a.rsqrt() * torch.exp(-2 * (dy * es) ** 2 * ipd) * wn[info] * oki
            planes = p0[ch][:, None] + torch.arange(n_pl, device=dev)
            okp = planes < p1[ch][:, None]
            z = (g.z_left + (planes + 0.5) * ps)[:, None, :]
            b = z - ev(right)[:, :, None] - (dy * et)[:, :, None]
            rm, rp = (eR - u)[:, :, None], (eR + u)[:, :, None]
            ang = torch.atan(torch.minimum((half - z) / rm, (half + z) / rp))
            ang = ang - torch.atan(torch.maximum(-(half + z) / rm, -(half - z) / rp))
            k = base[:, :, None] * torch.exp(-b * b * ipz) * (math.pi / ang)
            k = torch.where((ang >= 0) & okp[:, None, :] & oki[:, :, None], k, 0.0)
            idx = pix[info][:, :, None] + n_px * planes.clamp(max=g.n_planes - 1)[:, None, :]
            k = k * rho[idx]
            den = (k * sens[pix[info]][:, :, None]).sum((1, 2), keepdim=True)
            k = torch.where(den > 0, k * mult[:, :, None] / torch.where(den > 0, den, 1.0), 0.0)
            out.index_add_(0, idx.reshape(-1), k.reshape(-1))
        rho = out
    return rho


def _philox(counter, seed):
    """Philox4x32-10 words (int64 tensors below 2^32) at counter (index, draw)."""
    mask = 0xFFFFFFFF
    x = list(counter)
    k0, k1 = seed & mask, (seed >> 32) & mask
    for _ in range(10):
        p0, p1 = x[0] * 0xD2511F53, x[2] * 0xCD9E8D57  # low 64 bits, wrapped
        h0, h1 = (p0 >> 32) & mask, (p1 >> 32) & mask
        x = [h1 ^ x[1] ^ k0, p1 & mask, h0 ^ x[3] ^ k1, p0 & mask]
        k0, k1 = (k0 + 0x9E3779B9) & mask, (k1 + 0xBB67AE85) & mask
    return x


def _generate64(c, seed):
    ell = _ellipses(c, seed)
    w = np.cumsum([e.intensity * e.area for e in ell])
    cdf = torch.tensor(w / w[-1], device="cuda")
    par = torch.tensor([(e.z, e.y, e.a, e.b, math.radians(e.angle_deg)) for e in ell],
                       dtype=torch.float64, device="cuda")
    got, have, first = [], 0, 0

    def u53(a, b):
        return ((a >> 5).double() * 67108864.0 + (b >> 6).double()) / 9007199254740992.0

    while have < c["n"]:
        m = 1 << 20
        i = torch.arange(first, first + m, device="cuda")
        first += m
        zero = torch.zeros_like(i)
        r = [_philox((i & 0xFFFFFFFF, i >> 32, zero + d, zero), seed) for d in range(4)]
        k = torch.searchsorted(cdf, u53(r[0][0], r[0][1])).clamp_(max=len(ell) - 1)
        cz, cy, a, b, ang = par[k].unbind(1)
        rr, th = u53(r[0][2], r[0][3]).sqrt(), 2 * math.pi * u53(r[1][0], r[1][1])
        ex, ey = a * rr * th.cos(), b * rr * th.sin()
        x = ang.cos() * ex - ang.sin() * ey + cz
        y = ang.sin() * ex + ang.cos() * ey + cy
        ok = torch.ones_like(k, dtype=torch.bool)
        for q, e in enumerate(ell):
            sn, cs = math.sin(math.radians(e.angle_deg)), math.cos(math.radians(e.angle_deg))
            dx, dy = x - e.z, y - e.y
            inside = ((dx * cs + dy * sn) / e.a) ** 2 + ((dy * cs - dx * sn) / e.b) ** 2 <= 1
            ok &= ~(inside & (q < k))
        t = torch.tan(math.atan(LENGTH / (2 * RADIUS)) * (2 * u53(r[1][2], r[1][3]) - 1))
        zu, zd = x + (RADIUS - y) * t, x - (RADIUS + y) * t
        ok &= (zu.abs() < LENGTH / 2) & (zd.abs() < LENGTH / 2)
        m0 = (-2 * torch.log(1 - u53(r[2][0], r[2][1]))).sqrt()
        m1 = (-2 * torch.log(1 - u53(r[3][0], r[3][1]))).sqrt()
        a0, a1 = 2 * math.pi * u53(r[2][2], r[2][3]), 2 * math.pi * u53(r[3][2], r[3][3])
        ev = torch.stack([zu + c["sigma_z"] * m0 * a0.cos(), zd + c["sigma_z"] * m0 * a0.sin(),
                          -2 * y * (1 + t * t).sqrt() + c["sigma_dl"] * m1 * a1.cos()], 1)[ok]
        got.append(ev)
        have += len(ev)
    return torch.cat(got)[:c["n"]]
