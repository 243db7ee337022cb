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
