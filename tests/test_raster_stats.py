"""Box statistics of whole rasters (needs a B200) through the coarse surfaces: chips at the edges of the
kernel's columns and of its row blocks, rasters of odd sizes, the host path's bands."""
import numpy as np
import pytest

from ampcor_b200 import synth
from ampcor_b200.worker import Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def coarse(chip, win):
    """The normalised cross-correlation of a real chip with its window, from the definition in FP64."""
    R = chip.shape[0]
    r = chip - chip.mean()
    boxes = np.lib.stride_tricks.sliding_window_view(win, (R, R))
    num = np.einsum("uvij,ij->uv", boxes, r, optimize=True)
    dev = boxes - boxes.mean(axis=(2, 3), keepdims=True)
    return num / np.sqrt((dev * dev).sum(axis=(2, 3)) * (r * r).sum())


# chips of 16 to 128 samples (256 and 512 threads to a CTA, 161 to 417 boxes of a row each), rasters
# narrower than a CTA's columns, one column more, and several CTAs wide
@pytest.mark.parametrize("chip,lines,samples", [(16, 97, 120), (32, 200, 256), (32, 211, 257), (64, 300, 450),
                                                (80, 330, 515), (128, 257, 641)])
def test_coarse_surfaces(chip, lines, samples):
    ref, tgt = synth.speckle((lines, samples), 41), synth.speckle((lines, samples), 42)
    W = chip + 16
    ys = sorted({0, lines - W, (lines - W) // 2, max(0, 64 - 8)} & set(range(lines - W + 1)))
    xs = sorted({0, samples - W, (samples - W) // 2, max(0, 257 - chip - 8)} & set(range(samples - W + 1)))
    ulhc = np.array([[y + 8, x + 8, y, x] for y in ys for x in xs], np.int32)
    P, dev = len(ulhc), torch.device("cuda:0")
    worker = Worker(P, (chip, chip), (W, W), refine_factor=2, refine_margin=8, zoom_factor=4)
    surf = torch.zeros((P, worker.coarse_dim, worker.coarse_dim), device=dev)
    worker.correlate(torch.from_numpy(ref).to(dev), torch.from_numpy(tgt).to(dev), torch.from_numpy(ulhc).to(dev),
                     coarse_surfaces=surf)
    got = surf.cpu().numpy()
    a, b = np.abs(ref).astype(np.float64), np.abs(tgt).astype(np.float64)
    for k, (rl, rs, tl, ts) in enumerate(ulhc):
        want = coarse(a[rl:rl + chip, rs:rs + chip], b[tl:tl + W, ts:ts + W])
        # the surface bound of the parity rule
        assert np.abs(got[k] - want).max() <= 2e-5
    worker.close()


# lines of the two rasters that are no whole 16-byte units (one, the other, both), one raster for both
@pytest.mark.parametrize("chip,margin,ref_samples,tgt_samples", [(64, 32, 515, 514), (64, 32, 512, 513),
                                                                 (128, 32, 517, 519), (32, 16, 513, 513)])
def test_lines_of_any_length(chip, margin, ref_samples, tgt_samples):
    base = synth.speckle((480, 520), 51)
    both = ref_samples == tgt_samples
    ref = np.ascontiguousarray(base[:, :ref_samples])
    tgt = ref if both else np.ascontiguousarray(synth.fourier_shift(base, 1.3, -2.2)[:, :tgt_samples])
    W, least = chip + 2 * margin, min(ref_samples, tgt_samples)
    ulhc = np.array([[y + margin, x + margin, y, x] for y in range(0, 480 - W + 1, 29)
                     for x in [*range(0, least - W, 31), least - W]], np.int32)
    ulhc[1] = (0, ref_samples - chip + 1, 0, 0)  # off the raster
    P, dev = len(ulhc), torch.device("cuda:0")

    def job(a, b):
        worker = Worker(P, (chip, chip), (W, W), refine_factor=2, refine_margin=8, zoom_factor=8)
        surf = torch.full((P, worker.coarse_dim, worker.coarse_dim), np.nan, device=dev)
        da = torch.from_numpy(a).to(dev)
        off = worker.correlate(da, da if b is a else torch.from_numpy(b).to(dev), torch.from_numpy(ulhc).to(dev),
                               coarse_surfaces=surf, synchronize=False).cpu().numpy()
        torch.cuda.synchronize()
        return worker, off, surf.cpu().numpy()

    def wide(a):  # the same samples in lines of 520
        out = np.zeros((480, 520), np.complex64)
        out[:, :a.shape[1]] = a
        return out

    worker, off, surf = job(ref, tgt)
    aligned = wide(ref)
    other, want, surf_want = job(aligned, aligned if both else wide(tgt))
    keep = np.arange(P) != 1
    assert np.isnan(off[1]).all()
    np.testing.assert_array_equal(off[keep], want[keep])
    assert np.abs(surf[keep] - surf_want[keep]).max() <= 1e-6
    worker.close()
    other.close()
    # the host path, in bands, gives the device path's offsets
    host = Worker(P - 1, (chip, chip), (W, W), refine_factor=2, refine_margin=8, zoom_factor=8)
    np.testing.assert_array_equal(host.correlate(ref, ref.copy() if both else tgt, np.ascontiguousarray(ulhc[keep])), off[keep])
    host.close()
