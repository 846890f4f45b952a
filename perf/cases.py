"""The focus engine's measured workloads: whole start() calls on host arrays, device-resident
focuses, the focus with caller-owned memory, an autofocus step and the request loop, each over
the sizes, inputs and options that users of the engine run.

A case names its `kind` (how the work is called), the radar and aperture (chirps, samples), the
focus grid (columns x rows at a spacing in metres, planes for a volume), and options. Scenes are
seeded point targets with complex Gaussian noise under a Hann window in the processor's sign
convention, at 77 GHz with 4 GHz of bandwidth.
"""
from __future__ import annotations

import ctypes
import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.getcwd(), "sarlab-tdc_gb300"))

C0 = 299792458.0
F0 = 77e9
BANDWIDTH = 4e9
CHIRP_S = 40e-6
INF = float("inf")


def _case(name, kind, nx, ny, spacing, n_pri, n_samples, **more):
    c = dict(name=name, kind=kind, nx=nx, ny=ny, planes=1, spacing=spacing, n_pri=n_pri, n_samples=n_samples,
             pitch=0.5e-3, fp64=False, band=0.0, speed=0.0, taper=True, range_win=False, motion="still", targets=3,
             jobs=1)
    c.update(more)
    return c


def listed():
    return [
        # The smallest whole call, a quick look: host arrays in (per-sample trajectory, as the
        # processor's Python interface takes them), image out.
        _case("quicklook_start", "start", 24, 20, 2e-3, 256, 128, range_win=True),
        # The ordinary whole call: a 256 x 256 ground grid from a 0.5 m rail.
        _case("stripmap_start", "start", 256, 256, 2e-3, 1024, 512),
        # The large 2-D image: jittered FP64 positions and FP64 grid, acquisition resident on the GPU.
        _case("precision_focus", "focus", 1024, 1024, 1e-3, 4096, 1024, fp64=True, targets=50),
        # Near-field volume from a planar aperture: short rows, very many chirps.
        _case("volume_focus", "focus", 256, 256, 1e-3, 16384, 256, planes=16, targets=200),
        # A moving antenna under a finite Doppler band: most chirps are out of band for a pixel.
        _case("windowed_focus", "focus", 1024, 1024, 1e-3, 4096, 1024, fp64=True, band=10.0, speed=0.05, targets=50),
        # The antenna keeps moving during each chirp: a position for every sample, smooth in the chirp.
        _case("moving_focus", "focus", 512, 64, 1e-3, 512, 1024, motion="drift", targets=20),
        # A vibrating antenna: a position for every sample with no smooth model (odd sizes).
        _case("vibrating_focus", "focus", 151, 97, 2e-3, 333, 500, motion="vibration"),
        # Position and velocity for every sample under a band: the window changes within a chirp.
        _case("sampled_window_focus", "focus", 128, 128, 2e-3, 512, 512, motion="sampled", band=30.0, speed=0.08,
              pitch=1e-3),
        # Long chirps of an odd length.
        _case("long_rows_focus", "focus", 256, 256, 2e-3, 64, 12345, pitch=4e-3),
        # One step of trajectory autofocus: image, entropy, gradient for every chirp's position.
        _case("autofocus_step", "autofocus", 512, 512, 1e-3, 4096, 1024, fp64=True, targets=30),
        # Requests of mixed sizes submitted together to the request loop; host arrays in and out.
        _case("request_loop", "serve", 512, 512, 2e-3, 1024, 512, pitch=0.25e-3, targets=30, jobs=8),
        # A real-time chain that owns all device memory.
        _case("noalloc_focus", "noalloc", 200, 150, 2e-3, 300, 256),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    """One more case: any kind, every size spread over its range."""
    kind = rng.choice(["start", "start", "focus", "focus", "focus", "banded", "motion", "autofocus", "serve", "noalloc"])
    while True:
        c = _case("", "focus", _log(rng, 16, 1024), _log(rng, 16, 1024), rng.choice([0.7e-3, 1e-3, 2e-3, 3.9e-3]),
                  _log(rng, 64, 4096), _log(rng, 100, 2000), targets=rng.randint(1, 30), fp64=rng.random() < 0.5)
        del c["name"]
        c["pitch"] = min(0.5e-3, 1.5 / c["n_pri"])
        if kind in ("start", "autofocus", "serve", "noalloc"):
            c["kind"] = kind
        if kind in ("start", "noalloc"):
            c["fp64"] = False
            c["range_win"] = kind == "start" and rng.random() < 0.5
        if kind == "autofocus":
            c["fp64"] = True
        if kind == "serve":
            c["jobs"] = rng.randint(2, 8)
        if kind == "banded":
            c.update(band=rng.choice([8.0, 12.0, 20.0]), speed=0.05, taper=rng.random() < 0.7)
        if kind == "motion":
            c.update(motion=rng.choice(["drift", "vibration", "sampled"]), fp64=False, spacing=2e-3)
            if c["motion"] == "sampled":
                c.update(band=30.0, speed=0.08)
        corr = c["nx"] * c["ny"] * c["n_pri"] * c["n_samples"]
        most = 1.5e10 if kind == "motion" else 2e11 if kind == "serve" else 8e11
        if kind == "noalloc" and c["nx"] * c["ny"] > 400000:
            continue
        if 1e6 <= corr <= most and c["n_pri"] * c["n_samples"] <= 4194304:
            return c


# ---- the scene of a case ----------------------------------------------------

def _trajectory(c, rng):
    """Per-chirp antenna positions [n_pri, 3]: a rail 0.3 m above the grid (jittered when the
    positions are FP64), or for a volume a square planar aperture at 1 mm pitch."""
    n = c["n_pri"]
    pos = np.zeros((n, 3))
    if c["planes"] > 1:
        side = int(round(math.sqrt(n)))
        ax = (np.arange(side) - (side - 1) / 2.0) * 1e-3
        pos[:, 0], pos[:, 2] = np.repeat(ax, side), np.tile(ax, side)
        return pos
    pos[:, 0] = (np.arange(n) - (n - 1) / 2.0) * c["pitch"]
    pos[:, 2] = 0.3
    if c["fp64"]:
        pos += rng.normal(0.0, 0.5e-3, pos.shape)
    return pos


def _grid(c):
    """[rows, cols, 3] focus points: a ground plane in front of the rail, or a volume's planes."""
    xs = (np.arange(c["nx"]) - (c["nx"] - 1) / 2.0) * c["spacing"]
    if c["planes"] > 1:
        zs = (np.arange(c["ny"]) - (c["ny"] - 1) / 2.0) * c["spacing"]
        ys = 0.2 + np.arange(c["planes"]) * 2e-3
        g = np.zeros((c["planes"], c["ny"], c["nx"], 3))
        g[..., 0], g[..., 1], g[..., 2] = xs, ys[:, None, None], zs[None, :, None]
        return g.reshape(-1, c["nx"], 3)
    g = np.zeros((c["ny"], c["nx"], 3))
    g[..., 0] = xs
    g[..., 1] = (0.2 + np.arange(c["ny"]) * c["spacing"])[:, None]
    return g


def _sample_times(n):
    return (np.arange(n) * (CHIRP_S / n)).astype(np.float32)


def _scene(c, seed):
    """Everything the engine is given for one acquisition, as host arrays."""
    rng = np.random.default_rng(seed)
    n, s = c["n_pri"], c["n_samples"]
    grid = _grid(c)
    nominal = _trajectory(c, rng)
    flat = grid.reshape(-1, 3)
    lo, hi = flat.min(0), flat.max(0)
    tg = rng.uniform(lo, hi, (c["targets"], 3))
    amp = rng.rayleigh(1.0, c["targets"]) * np.exp(2j * np.pi * rng.uniform(0, 1, c["targets"]))
    true = nominal
    if c["kind"] == "autofocus":
        walk = np.cumsum(rng.normal(0.0, 0.2e-3 / math.sqrt(max(1.0, n / 256)), (n, 3)), axis=0)
        true = nominal + walk - walk.mean(0)
    gen = torch.Generator(device="cuda").manual_seed(int(rng.integers(1 << 40)))
    t = torch.from_numpy(_sample_times(s)).cuda().double()
    raw = torch.zeros((n, s), dtype=torch.complex128, device="cuda")
    tau = 2.0 * torch.cdist(torch.from_numpy(true).cuda(), torch.from_numpy(tg).cuda()) / C0
    k = BANDWIDTH / CHIRP_S
    for i in range(c["targets"]):
        base = F0 * tau[:, i] - 0.5 * k * tau[:, i] ** 2
        cyc = base[:, None] + (k * tau[:, i])[:, None] * t
        raw += complex(amp[i]) * torch.polar(torch.ones_like(cyc), -2.0 * math.pi * (cyc - cyc.round()))
    noise = torch.randn((n, s, 2), dtype=torch.float64, device="cuda", generator=gen)
    raw += 0.1 / math.sqrt(2.0) * torch.view_as_complex(noise)
    raw *= 0.5 - 0.5 * torch.cos(2.0 * math.pi * torch.arange(s, device="cuda", dtype=torch.float64) / s)
    d = dict(raw=raw.to(torch.complex64).cpu().numpy(), times=_sample_times(s), nominal=nominal, grid=grid,
             position=nominal.astype(np.float32), velocity=np.zeros((n, 3), np.float32), per_sample=False)
    d["velocity"][:, 0] = c["speed"]
    u = np.arange(s) / s
    if c["motion"] != "still":
        d["per_sample"] = True
        pos = nominal[:, None, :] + u[None, :, None] * rng.normal(0.0, 0.3e-3, (n, 1, 3))
        if c["motion"] == "vibration":
            pos[..., 2] += 20e-6 * np.sin(2 * np.pi * 3 * u + rng.uniform(0, 2 * np.pi, (n, 1)))
        d["position"] = pos.astype(np.float32)
        vel = np.zeros((n, s, 3), np.float32)
        vel[..., 0] = c["speed"]
        if c["motion"] == "sampled":
            vel[..., 0] *= 1.0 + 0.02 * np.sin(2 * np.pi * u)[None, :]
        d["velocity"] = vel
    return d


def _api(d):
    """setRawData's arguments: per-sample trajectory arrays."""
    n, s = d["raw"].shape
    pos, vel = d["position"], d["velocity"]
    if not d["per_sample"]:
        pos = np.ascontiguousarray(np.broadcast_to(pos[:, None, :], (n, s, 3)))
        vel = np.ascontiguousarray(np.broadcast_to(vel[:, None, :], (n, s, 3)))
    att = np.zeros((n, s, 4), np.float32)
    att[..., 0] = 1.0
    return (d["raw"], np.arange(n, dtype=np.float32) * np.float32(1e-3), d["times"], pos, vel, att,
            np.float32(BANDWIDTH / CHIRP_S), np.float32(F0), np.array([0, 1, 0], np.float32))


def _start_args(c):
    return (0.0, c["band"] or INF, False, c["range_win"], c["taper"])


def _jobs(c):
    """The requests of one request-loop case: sizes spread below and up to the case's own."""
    if c["kind"] != "serve":
        return [c]
    scale = [1.0, 0.25, 0.5, 0.125, 0.7, 0.35, 0.9, 0.18]
    out = []
    for i in range(c["jobs"]):
        f = scale[i % len(scale)]
        q = dict(c, nx=max(16, int(c["nx"] * f)), ny=max(16, int(c["ny"] * f)), n_pri=max(64, int(c["n_pri"] * f)))
        q["spacing"] = c["spacing"] * c["nx"] / q["nx"] if i % 2 else c["spacing"]
        q["n_samples"] = [c["n_samples"], max(64, c["n_samples"] // 2)][i % 2]
        q["fp64"] = bool(c["fp64"])
        out.append(q)
    return out


# ---- calls ------------------------------------------------------------------

def prepare(case, seed):
    import _sarlabtdc

    c = case
    if c["kind"] == "serve":
        from sarlabtdc.serving import FocusServer

        scenes = [_scene(q, seed * 64 + i) for i, q in enumerate(_jobs(c))]
        for d in scenes:
            d["send_position"] = d["nominal"] if c["fp64"] else d["position"]
            d["send_grid"] = d["grid"] if c["fp64"] else d["grid"].astype(np.float32)
        return dict(case=c, scenes=scenes, server=FocusServer(max_jobs=8, memory_budget=8 << 30))
    d = _scene(c, seed)
    if c["kind"] == "noalloc":
        return _prepare_noalloc(c, d)
    api = _api(d)
    grid = d["grid"] if c["fp64"] else np.ascontiguousarray(d["grid"].astype(np.float32))
    p = _sarlabtdc.TdcProcessor(0)
    state = dict(case=c, proc=p, api=api, grid=grid)
    if c["kind"] == "start":
        return state
    p.setRawData(*api)
    if c["fp64"]:
        p.setChirpPositionsF64(d["nominal"])
        p.setFocusGridF64(grid)
    else:
        p.setFocusGrid(grid)
    if c["kind"] == "autofocus":
        from sarlabtdc import autofocus

        state["op"] = autofocus.FocusOperator(p, _start_args(c))
        # the optimiser's parameters are FP32 corrections in metres, widened for the call
        state["offsets"] = torch.zeros((c["n_pri"], 3), dtype=torch.float32, device="cuda", requires_grad=True)
        return state
    p.prepare(*_start_args(c))
    p.uploadGrid()
    state["image"] = torch.empty(p.numPixels(), dtype=torch.complex64, device="cuda")
    return state


def _prepare_noalloc(c, d):
    import _tdc_capi

    n, s = d["raw"].shape
    samples = torch.zeros((n, (s + 15) // 16 * 16), dtype=torch.complex64, device="cuda")
    samples[:, :s] = torch.from_numpy(d["raw"]).cuda()
    rec = np.zeros((n, 12), np.float32)
    rec[:, 0:3], rec[:, 8:11] = d["position"], d["velocity"]
    g = np.zeros((d["grid"].size // 3, 4), np.float32)
    g[:, :3] = d["grid"].reshape(-1, 3)
    chirps, grid = torch.from_numpy(rec).cuda(), torch.from_numpy(g).cuda()
    image = torch.empty(g.shape[0], dtype=torch.complex64, device="cuda")
    f = _frequencies(d)
    i = np.arange(s)
    f1 = ((i - i.mean()) * (f - f.mean())).sum() / ((i - i.mean()) ** 2).sum()
    a = _tdc_capi.NoallocFocusArgs()
    a.samples, a.chirps, a.grid_hi = samples.data_ptr(), chirps.data_ptr(), grid.data_ptr()
    a.skip_points = a.grid_lo = None
    a.n_pix, a.n_pri, a.n_samples = g.shape[0], n, s
    a.g0, a.g1 = 2 * (f.mean() - f1 * i.mean()) / C0, 2 * f1 / C0
    a.lambda_ = C0 / f.mean()
    a.doppler_bandwidth = INF
    a.doppler_win_taper = 1
    return dict(case=c, lib=_tdc_capi.lib(), args=a, image=image, hold=(samples, chirps, grid))


def run(state):
    c = state["case"]
    if c["kind"] == "start":
        p = state["proc"]
        p.setRawData(*state["api"])
        p.setFocusGrid(state["grid"])
        p.start(*_start_args(c))
        return p.getFocusedImage()
    if c["kind"] == "focus":
        state["proc"].focusDevice(state["image"])
        return state["image"]
    if c["kind"] == "autofocus":
        from sarlabtdc import autofocus

        x = state["offsets"]
        x.grad = None
        image = autofocus.focus(state["op"], x.double())
        autofocus.entropy(image).backward()
        return {"image": image.detach(), "grad": x.grad}
    if c["kind"] == "serve":
        srv = state["server"]
        ids = [srv.submit(d["raw"], d["times"], d["send_position"], d["send_grid"], np.float32(BANDWIDTH / CHIRP_S),
                          np.float32(F0), start=_start_args(c)) for d in state["scenes"]]
        return [srv.wait(i)[0] for i in ids]
    rc = state["lib"].tdc_focus_noalloc(ctypes.byref(state["args"]), ctypes.c_void_p(state["image"].data_ptr()),
                                        ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
    if rc != 0:
        raise RuntimeError(f"tdc_focus_noalloc returned {rc}")
    return state["image"]


# ---- the work a pass cannot do without --------------------------------------

def work(case):
    """Bytes: raw rows, trajectory and grid once, image once. Operations: where one range per
    chirp describes a chirp, a pixel needs of each chirp its range, its phase and one value of
    the chirp's (oversampled) spectrum at that range -- about 50 flops -- and each chirp one
    transform; where a chirp's samples have ranges of their own, every (pixel, chirp, sample)
    needs its range change, its phasor and a complex multiply-add, about 25 flops."""
    total = {"bytes": 0.0, "flops": 0.0}
    for c in _jobs(case):
        pix, n, s = c["nx"] * c["ny"] * c["planes"], c["n_pri"], c["n_samples"]
        traj = 6 * 4 * n * s if c["motion"] != "still" or c["kind"] == "start" else 6 * 4 * n
        total["bytes"] += 8.0 * n * s + traj + pix * (12.0 * (2 if c["fp64"] else 1) + 8.0)
        if c["motion"] in ("vibration", "sampled"):
            total["flops"] += 25.0 * pix * n * s
        else:
            times = 2.0 if c["kind"] == "autofocus" else 1.0
            share = 0.2 if c["band"] else 1.0
            total["flops"] += times * share * 50.0 * pix * n + 10.0 * n * s * math.log2(max(2, 2 * s))
    return total


# ---- the same results in 64 bits --------------------------------------------

def _frequencies(d):
    return float(np.float32(F0)) + float(np.float32(BANDWIDTH / CHIRP_S)) * d["times"].astype(np.float64)


def _wavelength(d):
    t = d["times"]
    f0 = float(np.float32(F0))
    end = f0 + float(np.float32(BANDWIDTH / CHIRP_S)) * float(np.float32(t[-1] - t[0]))
    return float(np.float32(C0 / ((f0 + end) / 2.0)))


def _azimuth(c, fd):
    """Doppler window at frequency offset fd from its centre (0 Hz)."""
    w = (fd.abs() <= c["band"] / 2.0).double()
    if c["taper"]:
        w = w * (25.0 / 46.0 - 21.0 / 46.0 * torch.cos(2.0 * math.pi * fd / c["band"] - math.pi))
    return w


def _chunk_seen(c, d, lam, k, grid):
    """The chunk skip test of 128 chirps: 1 where any of its 3 x 3 points is in band."""
    n, s = d["raw"].shape
    valid = min(128, n - 128 * k)
    best = None
    for row in (0, 63, 127):
        pri = 128 * k + row if row < valid else 128 * (k - 1) + row
        for q in (0, max(s // 2 - 1, 0), max(2 * (s // 2) - 1, 0)):
            if pri < 0:
                p, v = np.zeros(3), np.zeros(3)
            elif d["per_sample"]:
                p, v = d["position"][pri, q].astype(np.float64), d["velocity"][pri, q].astype(np.float64)
            else:
                p, v = d["position"][pri].astype(np.float64), d["velocity"][pri].astype(np.float64)
            e = grid - torch.from_numpy(p).cuda()
            fd = (2.0 / lam * (e * torch.from_numpy(v).cuda()).sum(1) / e.norm(dim=1)).abs()
            best = fd if best is None else torch.minimum(best, fd)
    return (best <= c["band"] / 2.0).double()


def _exact_parts(c, d):
    """What both exact forms start from: rows, frequencies, grid and chirp positions in 64 bits."""
    s = d["raw"].shape[1]
    rows = torch.from_numpy(d["raw"]).cuda().to(torch.complex128)
    if c["range_win"]:
        rows = rows * (25.0 / 46.0 - 21.0 / 46.0 * torch.cos(2.0 * math.pi * torch.arange(s, device="cuda").double() / s))
    g = 2.0 * torch.from_numpy(_frequencies(d)).cuda() / C0
    grid = torch.from_numpy((d["grid"] if c["fp64"] else d["grid"].astype(np.float32)).reshape(-1, 3).astype(np.float64)).cuda()
    pos = torch.from_numpy(d["nominal"] if c["fp64"] else np.asarray(d["position"], np.float64)).cuda()
    return rows, g, grid, pos


def _chirps_exact(c, d, image=None, grad_of=None):
    """I(T) = sum_c w(T, c) sum_s x[c, s] exp(2 pi j g_s R), R one range per chirp, as values of
    each row's 8-fold zero-padded spectrum carried to the exact range by its Taylor series (to
    order 9, |angle| <= 0.2: below 1e-13), plus the first-order term of what g_s deviates from a
    straight line. With `grad_of` (dL/dI of a loss): its gradient for every chirp's position."""
    rows, g, grid, pos = _exact_parts(c, d)
    n, s = rows.shape
    lam = _wavelength(d)
    mid = s // 2
    i = torch.arange(s, device="cuda").double()
    g1 = (((i - i.mean()) * (g - g.mean())).sum() / ((i - i.mean()) ** 2).sum()).item()
    gm = (g.mean() + g1 * (mid - i.mean())).item()
    rest = g - (gm + g1 * (i - mid))
    size = 8 * 2 ** math.ceil(math.log2(max(2, s)))
    order = 9
    vel = None if not c["band"] else torch.from_numpy(d["velocity"].astype(np.float64)).cuda()
    out = torch.zeros(grid.shape[0], dtype=torch.complex128, device="cuda")
    grad = torch.zeros((n, 3), dtype=torch.float64, device="cuda")
    seen = None
    batch = max(1, min(n, (1 << 25) // size // (order + 1)))
    shift = torch.polar(torch.ones(size, dtype=torch.float64, device="cuda"),
                        -2.0 * math.pi * ((torch.arange(size, device="cuda") * mid) % size).double() / size)
    for c0 in range(0, n, batch):
        x = rows[c0:c0 + batch]
        tab = []
        y = x
        for m in range(order):
            tab.append(torch.fft.ifft(y, n=size, dim=1) * size * shift)
            y = y * (2j * math.pi * (i - mid) / size) / (m + 1)
        extra = torch.fft.ifft(x * (2j * math.pi * rest), n=size, dim=1) * size * shift
        extra1 = torch.fft.ifft(x * (2j * math.pi * rest) * (2j * math.pi * (i - mid) / size), n=size, dim=1) * size * shift
        for b in range(x.shape[0]):
            k = c0 + b
            e = pos[k] - grid
            r = e.norm(dim=1)
            if c["band"] and k % 128 == 0:
                seen = _chunk_seen(c, d, lam, k // 128, grid)
            beta = g1 * r * size
            at = beta.round()
            delta = beta - at
            at = at.long() % size
            value = tab[order - 1][b][at]
            slope = torch.zeros_like(value)
            for m in range(order - 2, -1, -1):
                if grad_of is not None:
                    slope = slope * delta + value
                value = value * delta + tab[m][b][at]
            more = extra[b][at] + extra1[b][at] * delta
            cyc = gm * r
            phase = torch.polar(torch.ones_like(r), 2.0 * math.pi * (cyc - cyc.round()))
            w = 1.0
            if c["band"]:
                w = seen * _azimuth(c, -2.0 / lam * (e * vel[k]).sum(1) / r)
            if grad_of is None:
                out += w * phase * (value + r * more)
            else:
                total = value + r * more
                by_r = phase * (2j * math.pi * gm * total + (slope + r * extra1[b][at]) * (g1 * size) + more)
                grad[k] = ((grad_of.conj() * by_r).real / r) @ e
    return grad if grad_of is not None else out


def _samples_exact(c, d):
    """The same sum with a range and window of its own for every sample, added up directly."""
    rows, g, grid, pos = _exact_parts(c, d)
    n, s = rows.shape
    lam = _wavelength(d)
    out = torch.zeros(grid.shape[0], dtype=torch.complex128, device="cuda")
    vel = torch.from_numpy(d["velocity"].astype(np.float64)).cuda()
    block = max(1, (1 << 24) // s)
    for k in range(n):
        if c["band"] and k % 128 == 0:
            seen = _chunk_seen(c, d, lam, k // 128, grid)
        for p0 in range(0, grid.shape[0], block):
            t = grid[p0:p0 + block]
            ex, ey, ez = (pos[k, :, q] - t[:, q, None] for q in range(3))
            r = torch.sqrt(ex * ex + ey * ey + ez * ez)
            cyc = r * g
            z = torch.polar(torch.ones_like(r), 2.0 * math.pi * (cyc - cyc.round()))
            if c["band"]:
                dot = ex * vel[k, :, 0] + ey * vel[k, :, 1] + ez * vel[k, :, 2]
                z = z * (_azimuth(c, -2.0 / lam * dot / r) * seen[p0:p0 + block, None])
            out[p0:p0 + block] += z @ rows[k]
    return out


def exact(case, seed):
    c = case
    if c["kind"] == "serve":
        return [_chirps_exact(q, _scene(q, seed * 64 + i)) for i, q in enumerate(_jobs(c))]
    d = _scene(c, seed)
    if c["motion"] != "still":
        return _samples_exact(c, d)
    image = _chirps_exact(c, d)
    if c["kind"] == "autofocus":
        x = image.clone().requires_grad_(True)
        inten = x.real ** 2 + x.imag ** 2
        share = inten / inten.sum()
        (-(share * torch.log(share + 1e-300)).sum()).backward()
        return {"image": image, "grad": _chirps_exact(c, d, grad_of=x.grad)}
    if c["kind"] == "start":
        return image.reshape(c["planes"] * c["ny"], c["nx"])
    return image
