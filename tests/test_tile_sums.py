"""The statistics of chips keep their digits (needs a B200): coarse and refined surfaces against FP64
where the sums are hard - a strong steady return, bright scatterers, chips of nearly one value - for
every way a stage is correlated: one tile, several CTAs per multiprocessor, four parts, chip blocks
with summed spectra and block by block.

Coarse surfaces are compared with the FP64 correlation of the FP32 amplitudes that are correlated.  A
steady return of L times the speckle's level: a zero-mean chip value is rounded to 2^-24 of its size
(about 0.46 speckle levels), and the window's level L multiplies the sum of n such roundings where a
block's sub-window is centred on its own mean; against |r'||t'| of about n / 4.6 that is
L 2^-24 sqrt(n) 0.46 / (n / 4.6), 3e-7 at L = 300 and n = 128^2 for independent roundings, 4e-5 if they
all went one way.  1e-5 lies between: sums in FP32 miss it by ten times.  One tile's window is centred
on its own mean, to 2^-24 of L, so that nothing of the sort remains: 5e-7, eight roundings of 1."""
import numpy as np
import pytest

from ampcor_b200 import serve, synth
from ampcor_b200.worker import Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

DEV = "cuda:0"


def cut(raster, at, n):
    k = torch.arange(n, device=DEV)
    return raster[(at[:, :1] + k)[:, :, None], (at[:, 1:] + k)[:, None, :]]


def ncc(chip, win):
    R, W = chip.shape[-1], win.shape[-1]
    C = W - R + 1
    r = chip - chip.mean(dim=(1, 2), keepdim=True)
    t = win - win.mean(dim=(1, 2), keepdim=True)
    num = torch.fft.irfft2(torch.fft.rfft2(r, s=(W, W)).conj() * torch.fft.rfft2(t), s=(W, W))[:, :C, :C]

    def boxes(v):
        v = torch.nn.functional.pad(v.cumsum(1).cumsum(2), (1, 0, 1, 0))
        return v[:, R:, R:] - v[:, :-R, R:] - v[:, R:, :-R] + v[:, :-R, :-R]

    s1 = boxes(t)
    var = boxes(t * t) - s1 * s1 / (R * R)
    return num / torch.sqrt(var * (r * r).sum(dim=(1, 2))[:, None, None])


def coarse(R, M, ref, tgt, ulhc):
    worker = Worker(len(ulhc), (R, R), (R + 2 * M, R + 2 * M), refine_factor=2, refine_margin=8, zoom_factor=8)
    dev = [torch.from_numpy(a).to(DEV) for a in (ref, tgt, ulhc)]
    got = torch.zeros((len(ulhc), worker.coarse_dim, worker.coarse_dim), device=DEV)
    worker.correlate(*dev, coarse_surfaces=got)
    worker.close()
    at = dev[2].long()
    chip = cut(dev[0].to(torch.complex128).abs().float().double(), at[:, :2], R)
    win = cut(dev[1].to(torch.complex128).abs().float().double(), at[:, 2:], R + 2 * M)
    return got.double(), chip, win


FORMS = [(32, 16), (64, 32), (64, 64), (128, 32), (128, 64)]


def scene(n):
    ref = synth.speckle((n, n), 61)
    return ref, synth.fourier_shift(ref, 2.3, -1.7)


@pytest.mark.parametrize("R,M", FORMS)
def test_steady_return(R, M):
    ref, tgt = (a + np.float32(300.0) for a in scene(R + 2 * M + 64))
    ulhc = serve.grid_corners(*ref.shape, R, M, 31)
    got, chip, win = coarse(R, M, ref, tgt, ulhc)
    assert (got - ncc(chip, win)).abs().max() < (1e-5 if R == 128 else 5e-7)


@pytest.mark.parametrize("R,M", FORMS)
def test_chip_of_nearly_one_value(R, M):
    """A reference whose amplitudes differ in their last digit only (1 or 1 + 2^-23, at random) against a
    secondary of the same pattern, 2^-23 or 2^-22 (both tiles share one transform, whose error goes with
    the larger one's deviations: the two are of one size): the chip's deviations are a 1e-15th of its sum
    of squares, and exact, so that each chip's own place correlates to 1 (less the transform's 1.4e-7 and
    the roundings of the last products)."""
    n = R + 2 * M + 64
    k = np.random.default_rng(3).integers(0, 2, (n, n)).astype(np.float32)
    ref, tgt = (1 + np.float32(2.0 ** -23) * k).astype(np.complex64), (np.float32(2.0 ** -23) * (1 + k)).astype(np.complex64)
    ulhc = serve.grid_corners(n, n, R, M, 31)
    got, chip, win = coarse(R, M, ref, tgt, ulhc)
    dev = chip - chip.mean(dim=(1, 2), keepdim=True)
    share = (dev * dev).sum(dim=(1, 2)) / (chip * chip).sum(dim=(1, 2))
    assert (share > 0).all() and (share < 1e-14).all()
    C = got.shape[-1]
    assert (got.flatten(1).argmax(1) == M * C + M).all()
    assert (got[:, M, M] - 1.0).abs().max() < 1e-6


@pytest.mark.parametrize("R", [32, 64, 128])
def test_bright_scatterers_in_the_refined_chip(R):
    """Scatterers of 100 times the level: the refined surface's peak (the refined amplitudes carry 2^-24
    each, and |r'|^2 is a sum of squares: 1e-6 allows eight roundings of every term in one direction)."""
    M, n = 16, R + 32 + 64
    ref = synth.speckle((n, n), 62)
    bright = np.random.default_rng(7).random(ref.shape) < 1.0 / 2048
    ref[bright] *= np.float32(100.0)
    ulhc = serve.grid_corners(n, n, R, M, 9)
    worker = Worker(len(ulhc), (R, R), (R + 2 * M, R + 2 * M), refine_factor=2, refine_margin=8, zoom_factor=8)
    surf = torch.zeros((len(ulhc), worker.refined_dim, worker.refined_dim), device=DEV)
    dev = [torch.from_numpy(a).to(DEV) for a in (ref, ref, ulhc)]
    diag = torch.zeros((len(ulhc), 12), dtype=torch.float32, device=DEV)
    worker.correlate(*dev, diag=diag, refined_surfaces=surf)
    worker.close()
    at = dev[2].long()
    corner = diag.view(torch.int32)[:, 2:4].long()

    def upsampled(z):
        N = z.shape[-1]
        F, h = 2 * N, N // 2
        for axis in (1, 2):
            s = torch.fft.fft(z, dim=axis).movedim(axis, -1)
            p = torch.zeros(s.shape[:-1] + (F,), dtype=s.dtype, device=s.device)
            p[..., :h], p[..., F - h + 1:] = s[..., :h], s[..., h + 1:]
            p[..., h] = p[..., F - h] = 0.5 * s[..., h]
            z = torch.fft.ifft(p, dim=-1).movedim(-1, axis) * 2
        return z.abs()

    chip = upsampled(cut(dev[0].to(torch.complex128), at[:, :2], R))
    win = upsampled(cut(dev[1].to(torch.complex128), at[:, 2:] + corner, R + 16))
    want = ncc(chip, win)
    best = want.flatten(1).argmax(1)[:, None]
    error = (surf.double().flatten(1).gather(1, best) - want.flatten(1).gather(1, best)).abs()
    assert error.max() < 1e-6


@pytest.mark.parametrize("M", [24, 32, 64])
def test_blocks_under_a_steady_return(M):
    """The blocks of a 128 px chip (spectra summed, or block by block) keep a level of 300 out of the
    numerators: what remains is the rounding of the amplitudes' centred values and the transform, 5e-7 as
    of one tile."""
    R = 128
    ref, tgt = (a + np.float32(300.0) for a in scene(R + 2 * M + 64))
    got, chip, win = coarse(R, M, ref, tgt, serve.grid_corners(*ref.shape, R, M, 31))
    assert (got - ncc(chip, win)).abs().max() < 5e-7


@pytest.mark.parametrize("R,m,f", [(32, 4, 1), (32, 4, 3), (24, 4, 4), (56, 4, 2), (16, 4, 5)])
def test_statistics_from_the_interpolating_refinement(R, m, f):
    """Tiles and factors that have no transform of their own are refined by interpolation, which hands on the
    same statistics: the refined surfaces of a scene under a return of 30 within the 2e-5 that every form is
    held to."""
    M = 16
    ref, tgt = (a + np.float32(30.0) for a in scene(R + 2 * M + 64))
    ulhc = serve.grid_corners(*ref.shape, R, M, 17)
    worker = Worker(len(ulhc), (R, R), (R + 2 * M, R + 2 * M), refine_factor=f, refine_margin=m, zoom_factor=4)
    assert worker.form == "spectral"
    surf = torch.zeros((len(ulhc), worker.refined_dim, worker.refined_dim), device=DEV)
    diag = torch.zeros((len(ulhc), 12), dtype=torch.float32, device=DEV)
    dev = [torch.from_numpy(a).to(DEV) for a in (ref, tgt, ulhc)]
    worker.correlate(*dev, diag=diag, refined_surfaces=surf)
    worker.close()

    def upsampled(z):
        N = z.shape[-1]
        d = torch.arange(f * N, device=DEV, dtype=torch.float64)[:, None] / f - torch.arange(N, device=DEV)
        U = torch.ones_like(d)
        for n in range(1, N // 2):
            U = U + 2.0 * torch.cos(2.0 * np.pi * n * d / N)
        U = ((U + torch.cos(np.pi * d)) / N).to(z.dtype)
        return (U @ z @ U.T).abs()

    at = dev[2].long()
    corner = diag.view(torch.int32)[:, 2:4].long()
    chip = upsampled(cut(dev[0].to(torch.complex128), at[:, :2], R))
    win = upsampled(cut(dev[1].to(torch.complex128), at[:, 2:] + corner, R + 2 * m))
    assert (surf.double() - ncc(chip, win)).abs().max() < 2e-5
