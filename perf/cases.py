"""The correlation work that users of ampcor_b200 give it, as cases to be timed and compared.

A case is one job through a public entry point of the framework:

* ``raster`` - device-resident rasters, corners and results (``Worker.correlate`` on CUDA tensors);
* ``host``   - page-locked host rasters in, offsets out (``Worker.correlate`` on numpy arrays);
* ``arena``  - the pair-by-pair interface ampcor binds to (``ext.ampcor_cuda``);
* ``batch``  - uneven raster pairs in one CUDA graph (``batch.UnevenBatch``);
* ``server`` - queued jobs through the continuous-batching loop (``serve.Server``).

The inputs are single-look speckle: circular complex Gaussian pixels, the secondary moved by a
constant plus a smooth quadratic field and covered by noise at 10 dB, optionally with bright point
scatterers, or band-limited and off baseband as a Doppler centroid leaves it.

What comes back is what a program goes on with: the target point of every chip centre (the
codomain of the refined offset map: the centre plus the pair's offset) and, where the program asks
for them, the three correlation peaks of every pair and both correlation surfaces.  ``exact``
computes the same from the definition of the pipeline, in 64 bits.
"""
from __future__ import annotations

import math
import random

import numpy as np
import torch

from ampcor_b200 import batch, serve
from ampcor_b200.ext import ampcor_cuda
from ampcor_b200.worker import Worker

DEVICE = "cuda:0"
FACTOR = 2  # the refinement factor of every configuration

RASTER = {"kind": "raster", "lines": 4096, "samples": 4096, "chip": 64, "margin": 32, "refine_margin": 8,
          "zoom": 8, "spacing": 33, "chunk": "default", "wait": False, "deramp": False, "heavy": False,
          "surfaces": False}


def listed():
    def job(name, **kw):
        return dict(RASTER, name=name, **kw)

    return [
        # the smallest call: 64 pairs of a 512^2 pair of rasters, the caller waiting for the answer
        # (interactive use, the first look at a scene); launches and host work count
        job("small_512", lines=512, samples=512, chip=32, margin=8, refine_margin=4, zoom=4, spacing=64,
            wait=True),
        # a job on rasters of odd size, as cropped scenes are (lines that are no multiple of 16
        # bytes), with an odd search margin
        job("ragged_odd", lines=1531, samples=1999, margin=19, spacing=37, wait=True),
        # band-limited data off baseband with the deramp, a small quick-look grid
        job("deramp_1024", lines=1024, samples=1024, margin=16, spacing=48, deramp=True),
        # quality control: both correlation surfaces kept, bright scatterers in the scene
        job("surfaces_heavy", lines=1024, samples=1024, spacing=64, heavy=True, surfaces=True),
        # a dense field of small chips (grid spacing down to 16 px)
        job("dense_32", lines=2048, samples=3072, chip=32, margin=16, spacing=16),
        # a wide search with a fine zoom, the far end of the serving range
        job("wide_search", lines=2048, samples=2048, margin=64, zoom=16, spacing=64),
        # the headline geometry at production size, the worker configured as its autotuner does
        # (all pairs in one chunk)
        job("production_4096", chunk="whole"),
        # ampcor's default geometry (128^2 chips, 32 px padding) on the same rasters
        job("default_128", chip=128, spacing=64),
        # the production job end to end, from page-locked host memory
        job("host_4096", kind="host", chunk="whole"),
        # ampcor's own calling sequence: tiles added pair by pair, then adjust
        job("arena_128", kind="arena", lines=1024, samples=1024, chip=128, spacing=128),
        # uneven raster pairs replayed as one CUDA graph
        {"name": "uneven_graph", "kind": "batch", "jobs": 6, "layout": 11, "most": 2500},
        # a queue of jobs of mixed geometry through the server, uploads included
        {"name": "server_queue", "kind": "server", "jobs": 8, "layout": 7, "most": 1200},
    ]


def draw(rng):
    """A raster, host or arena job anywhere in the ranges of the listed ones."""

    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(("raster", "raster", "raster", "raster", "host", "arena"))
    chip = rng.choice((24, 32, 48, 64, 64, 128))
    refine_margin = rng.choice((4, 8)) if chip in (24, 32) else 8
    margin = log_int(refine_margin, 64)
    least = chip + 2 * margin + 64
    most = 1024 if kind == "arena" else 4096
    case = dict(RASTER, kind=kind, chip=chip, margin=margin, refine_margin=refine_margin,
                zoom=rng.choice((4, 8, 16)), lines=log_int(max(384, least), most),
                samples=log_int(max(384, least), most), spacing=log_int(16, 128),
                chunk=rng.choice(("default", "whole")), wait=rng.random() < 0.5)
    if kind == "raster":
        case["deramp"] = rng.random() < 0.15
        case["heavy"] = rng.random() < 0.25
    while _pairs(case) > (200 if kind == "arena" else 15000) or work(case)["flops"] > _LARGEST:
        case["spacing"] = case["spacing"] * 5 // 4 + 1
    return case


# ---- geometry ----------------------------------------------------------------------------------


def _pairs(case):
    return len(serve.grid_corners(case["lines"], case["samples"], case["chip"], case["margin"], case["spacing"]))


def _members(case):
    """The raster jobs of a batch or server case: fixed by its layout, not by the seed of the data."""
    rng = random.Random(case["layout"])
    jobs = []
    for _ in range(case["jobs"]):
        if case["kind"] == "batch":
            lines, samples = rng.choice(((1024, 1024), (2048, 2048), (2048, 1024), (1024, 1536)))
            chip, margin, zoom = rng.choice((32, 64, 128)), rng.choice((8, 16, 32, 64)), 8
        else:
            lines = samples = rng.choice((1024, 2048))
            chip, margin, zoom = rng.choice(((32, 16, 16), (64, 32, 8), (128, 32, 8)))
        one = dict(RASTER, lines=lines, samples=samples, chip=chip, margin=margin, zoom=zoom,
                   spacing=rng.randint(24, 128))
        while _pairs(one) > case["most"]:
            one["spacing"] += 8
        jobs.append(one)
    return jobs


def _corners(case):
    return serve.grid_corners(case["lines"], case["samples"], case["chip"], case["margin"], case["spacing"])


def _centres(case, ulhc):
    return (ulhc[:, :2] + case["chip"] // 2).astype(np.float32)


def work(case):
    """Each raster sample and corner read once, each result written once; the arithmetic of the
    correlation by FFT (both real tiles in one complex transform, half of the inverse), of the
    band-limited upsampling and of the zoom as a matrix product."""
    if case["kind"] in ("batch", "server"):
        parts = [work(c) for c in _members(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    R, m, z, P = case["chip"], case["refine_margin"], case["zoom"], _pairs(case)
    W, E = R + 2 * case["margin"], R + 2 * m
    C, Cf = W - R + 1, 2 * FACTOR * m + 1
    Z = z * Cf

    def fft(n, rows, cols):  # `rows` + `cols` complex transforms of n points
        return 5.0 * n * math.log2(n) * (rows + cols)

    flops = 1.5 * fft(W, W, W) + 1.5 * fft(FACTOR * E, FACTOR * E, FACTOR * E)
    for n in (R, E):
        flops += fft(n, n, n) + fft(FACTOR * n, n, FACTOR * n)
    flops += 2.0 * Z * Cf * (Cf + Z)
    out = 8.0 + (12.0 if case["kind"] == "raster" else 0.0)
    if case["surfaces"]:
        out += 4.0 * (C * C + Cf * Cf)
    tiles = 8.0 * P * (R * R + W * W) if case["kind"] == "arena" else 16.0 * case["lines"] * case["samples"]
    return {"bytes": tiles + P * (16.0 + out), "flops": flops * P}


# a drawn job costs no more than the production job
_LARGEST = work(dict(RASTER))["flops"]


# ---- inputs ------------------------------------------------------------------------------------


def _noise(shape, power, gen):
    re = torch.randn(shape, generator=gen, device=DEVICE)
    im = torch.randn(shape, generator=gen, device=DEVICE)
    return torch.complex(re, im) * math.sqrt(power / 2.0)


def _rasters(case, seed):
    """The pair of complex64 rasters of a job, on the device."""
    gen = torch.Generator(device=DEVICE)
    gen.manual_seed(int(seed) * 1000003 + 17)
    rng = random.Random(int(seed))
    L, S = case["lines"], case["samples"]
    reach = min(0.5 * case["margin"], 10.0)
    dy, dx = rng.uniform(-0.6, 0.6) * reach, rng.uniform(-0.6, 0.6) * reach
    quad = rng.uniform(-0.4, 0.4) * reach
    ref = _noise((L, S), 1.0, gen)
    if case["heavy"]:  # one pixel in a hundred a point scatterer, 30 dB up
        bright = torch.rand((L, S), generator=gen, device=DEVICE) < 0.01
        ref = torch.where(bright, ref * 10.0 ** 1.5, ref)
    ky = torch.fft.fftfreq(L, device=DEVICE, dtype=torch.float64)[:, None]
    kx = torch.fft.fftfreq(S, device=DEVICE, dtype=torch.float64)[None, :]
    spectrum = torch.fft.fft2(ref.to(torch.complex128))
    if case["deramp"]:
        spectrum[(ky.abs() > 0.3).expand(L, S) | (kx.abs() > 0.3).expand(L, S)] = 0.0
        ref = torch.fft.ifft2(spectrum)
        ref = (ref / ref.abs().square().mean().sqrt()).to(torch.complex64)
        spectrum = torch.fft.fft2(ref.to(torch.complex128))
    tgt = torch.fft.ifft2(spectrum * torch.exp(-2j * math.pi * (ky * dy + kx * dx))).to(torch.complex64)
    del spectrum
    # the smooth part: out(y, x) = in(y - qy, x - qx)
    Y, X = torch.meshgrid(torch.linspace(-1.0, 1.0, L, device=DEVICE), torch.linspace(-1.0, 1.0, S, device=DEVICE),
                          indexing="ij")
    qy, qx = quad * (Y * Y - 0.5 * X * Y), quad * (X * X + 0.5 * X * Y)
    grid = torch.stack([X - qx * 2.0 / (S - 1), Y - qy * 2.0 / (L - 1)], dim=-1)[None]
    planes = torch.stack([tgt.real, tgt.imag])[None]
    planes = torch.nn.functional.grid_sample(planes, grid, mode="bicubic", padding_mode="zeros", align_corners=True)[0]
    tgt = torch.complex(planes[0], planes[1])
    tgt = tgt + _noise((L, S), 0.1 * float(ref.abs().square().mean()), gen)
    if case["deramp"]:
        y = torch.arange(L, device=DEVICE, dtype=torch.float64)[:, None]
        x = torch.arange(S, device=DEVICE, dtype=torch.float64)[None, :]
        ramp = torch.exp(2j * math.pi * (0.1 * y + 0.45 * x))
        ref, tgt = (ref * ramp).to(torch.complex64), (tgt * ramp).to(torch.complex64)
    return ref.contiguous(), tgt.contiguous()


def _pinned(t):
    host = torch.empty(t.shape, dtype=t.dtype, pin_memory=True)
    host.copy_(t)
    return host


def prepare(case, seed):
    if case["kind"] == "batch":
        jobs = []
        for k, c in enumerate(_members(case)):
            ref, tgt = _rasters(c, seed * 64 + k)
            jobs.append(batch.RasterJob(ref, tgt, _corners(c), c["chip"], c["margin"], FACTOR, c["refine_margin"],
                                        c["zoom"]))
        ub = batch.UnevenBatch(jobs, tune=False)
        ub.capture()
        centres = [torch.from_numpy(_centres(c, j.ulhc)).to(DEVICE) for c, j in zip(_members(case), jobs)]
        return {"case": case, "batch": ub, "centres": centres}
    if case["kind"] == "server":
        jobs = []
        for k, c in enumerate(_members(case)):
            ref, tgt = (_pinned(t) for t in _rasters(c, seed * 64 + k))
            jobs.append(serve.Job(k, 0.0, ref, tgt, _corners(c), c["chip"], c["margin"], FACTOR, c["refine_margin"],
                                  c["zoom"]))
        server = serve.Server(slots=3)
        server.warm(jobs)
        return {"case": case, "server": server, "jobs": jobs,
                "centres": [_centres(c, j.ulhc) for c, j in zip(_members(case), jobs)]}

    ulhc = _corners(case)
    P, R, W = len(ulhc), case["chip"], case["chip"] + 2 * case["margin"]
    ref, tgt = _rasters(case, seed)
    state = {"case": case, "ulhc": ulhc, "centres": _centres(case, ulhc)}
    if case["kind"] == "arena":
        state["ref"], state["tgt"] = ref.cpu().numpy(), tgt.cpu().numpy()
        state["worker"] = ampcor_cuda.sequential(P, (R, R), (W, W), case["refine_margin"], FACTOR, case["zoom"])
        return state
    worker = Worker(P, (R, R), (W, W), refine_factor=FACTOR, refine_margin=case["refine_margin"],
                    zoom_factor=case["zoom"], deramp=case["deramp"])
    if case["chunk"] == "whole":
        worker.configure(chunk=P)
    state["worker"] = worker
    if case["kind"] == "host":
        state["pinned"] = _pinned(ref), _pinned(tgt)
        state["ref"], state["tgt"] = (t.numpy() for t in state["pinned"])
        return state
    state["ref"], state["tgt"] = ref, tgt
    state["ulhc"] = torch.from_numpy(ulhc).to(DEVICE)
    state["centres"] = torch.from_numpy(state["centres"]).to(DEVICE)
    state["diag"] = torch.zeros((P, 12), dtype=torch.float32, device=DEVICE)
    for name, n in (("coarse_surfaces", worker.coarse_dim), ("refined_surfaces", worker.refined_dim)):
        state[name] = torch.zeros((P, n, n), device=DEVICE) if case["surfaces"] else None
    return state


# ---- the passes --------------------------------------------------------------------------------


def run(state):
    case = state["case"]
    if case["kind"] == "batch":
        ub = state["batch"]
        ub.replay()
        with torch.cuda.stream(ub.stream):
            return [{"points": c + o} for c, o in zip(state["centres"], ub.offsets)]
    if case["kind"] == "server":
        jobs = state["server"].run(state["jobs"], realtime=False)
        return [{"points": c + j.offsets} for c, j in zip(state["centres"], jobs)]
    if case["kind"] == "arena":
        worker, ref, tgt = state["worker"], state["ref"], state["tgt"]
        R, W = case["chip"], case["chip"] + 2 * case["margin"]
        for k, (rl, rs, tl, ts) in enumerate(state["ulhc"]):
            ampcor_cuda.addReference(worker, ref, k, (rl, rs), (rl + R, rs + R))
            ampcor_cuda.addTarget(worker, tgt, k, (tl, ts), (tl + W, ts + W))
        return {"points": state["centres"] + np.array(ampcor_cuda.adjust(worker), np.float32).reshape(-1, 2)}
    if case["kind"] == "host":
        return {"points": state["centres"] + state["worker"].correlate(state["ref"], state["tgt"], state["ulhc"])}
    offsets = state["worker"].correlate(
        state["ref"], state["tgt"], state["ulhc"], diag=state["diag"], coarse_surfaces=state["coarse_surfaces"],
        refined_surfaces=state["refined_surfaces"], synchronize=case["wait"])
    # the peaks of a pair's record: coarse, refined and zoomed surface
    return {"points": state["centres"] + offsets, "peaks": state["diag"][:, 8:11],
            "coarse": state["coarse_surfaces"], "refined": state["refined_surfaces"]}


# ---- the same in 64 bits -----------------------------------------------------------------------


def _tiles(raster, rows, cols, n):
    k = torch.arange(n, device=DEVICE)
    return raster[(rows[:, None] + k)[:, :, None], (cols[:, None] + k)[:, None, :]]


def _ncc(chip, win):
    """The normalised cross-correlation of each real chip with its window at every placement."""
    R, W = chip.shape[-1], win.shape[-1]
    C = W - R + 1
    r = chip - chip.mean(dim=(1, 2), keepdim=True)
    t = win - win.mean(dim=(1, 2), keepdim=True)
    num = torch.fft.irfft2(torch.fft.rfft2(r, s=(W, W)).conj() * torch.fft.rfft2(t), s=(W, W))[:, :C, :C]

    def boxes(v):
        v = torch.nn.functional.pad(v.cumsum(1).cumsum(2), (1, 0, 1, 0))
        return v[:, R:, R:] - v[:, :-R, R:] - v[:, R:, :-R] + v[:, :-R, :-R]

    s1, s2 = boxes(t), boxes(t * t)
    var = s2 - s1 * s1 / (R * R)
    return num / torch.sqrt(var * (r * r).sum(dim=(1, 2))[:, None, None])


def _upsampled(z):
    """Band-limited interpolation of complex tiles by FACTOR: zero-padded spectra, Nyquist split."""
    N = z.shape[-1]
    F, h = FACTOR * N, N // 2
    for axis in (1, 2):
        s = torch.fft.fft(z, dim=axis).movedim(axis, -1)
        p = torch.zeros(s.shape[:-1] + (F,), dtype=s.dtype, device=s.device)
        p[..., :h], p[..., F - h + 1:] = s[..., :h], s[..., h + 1:]
        p[..., h] = p[..., F - h] = 0.5 * s[..., h]
        z = torch.fft.ifft(p, dim=-1).movedim(-1, axis) * FACTOR
    return z


def _deramped(z):
    n = z.shape[-1]
    s = (z[:, :, 1:] * z[:, :, :-1].conj()).sum(dim=(1, 2)).angle()[:, None, None]
    l = (z[:, 1:] * z[:, :-1].conj()).sum(dim=(1, 2)).angle()[:, None, None]
    k = torch.arange(n, device=DEVICE, dtype=torch.float64)
    return z * torch.exp(-1j * (s * k[None, None, :] + l * k[None, :, None]))


def _first_maximum(surface):
    n = surface.shape[-1]
    best = surface.reshape(len(surface), -1).max(dim=1)
    return best.values, best.indices // n, best.indices % n


def _exact_job(case, ref, tgt, ulhc):
    R, M, m, z = case["chip"], case["margin"], case["refine_margin"], case["zoom"]
    W, E, Cf = R + 2 * M, R + 2 * m, 2 * FACTOR * m + 1
    d = torch.arange(z * Cf, device=DEVICE, dtype=torch.float64)[:, None] / z - torch.arange(Cf, device=DEVICE)
    U = torch.ones_like(d)
    for n in range(1, (Cf - 1) // 2 + 1):
        U = U + 2.0 * torch.cos(2.0 * math.pi * n * d / Cf)
    U = U / Cf
    out = {"points": [], "peaks": [], "coarse": [], "refined": []}
    ulhc = torch.from_numpy(ulhc).to(DEVICE).long()
    for u in ulhc.split(192):
        chip = _tiles(ref, u[:, 0], u[:, 1], R).to(torch.complex128)
        win = _tiles(tgt, u[:, 2], u[:, 3], W).to(torch.complex128)
        coarse = _ncc(chip.abs(), win.abs())
        peak, cy, cx = _first_maximum(coarse)
        top, left = (cy - m).clamp(0, W - E), (cx - m).clamp(0, W - E)
        near = _tiles(tgt, u[:, 2] + top, u[:, 3] + left, E).to(torch.complex128)
        if case["deramp"]:
            chip, near = _deramped(chip), _deramped(near)
        refined = _ncc(_upsampled(chip).abs(), _upsampled(near).abs())
        zoomed, p, q = _first_maximum(U @ refined @ U.T)
        fine = torch.stack([p, q], 1).double() / (FACTOR * z)
        out["points"].append(u[:, :2] + R // 2 + torch.stack([top, left], 1) - M + fine)
        out["peaks"].append(torch.stack([peak, refined.amax(dim=(1, 2)), zoomed], 1))
        if case["surfaces"]:
            out["coarse"].append(coarse)
            out["refined"].append(refined)
    return {k: torch.cat(v) if v else None for k, v in out.items()}


def exact(case, seed):
    if case["kind"] in ("batch", "server"):
        return [{"points": _exact_job(c, *_rasters(c, seed * 64 + k), _corners(c))["points"]}
                for k, c in enumerate(_members(case))]
    got = _exact_job(case, *_rasters(case, seed), _corners(case))
    return got if case["kind"] == "raster" else {"points": got["points"]}
