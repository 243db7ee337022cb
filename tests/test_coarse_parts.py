"""Coarse searches correlated in four parts of their placements (needs a B200), against the chip blocks
that AMPCOR_STAGED=0 keeps: the same cells, peaks and surfaces on rasters whose best placements fall into
every part and onto the rows and columns that two parts share, a pair off the raster, several chunks."""
import numpy as np
import pytest

from ampcor_b200 import synth
from ampcor_b200.worker import DIAG_DTYPE, Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def run(ref, tgt, ulhc, chip, W, chunk=0):
    dev, P = torch.device("cuda:0"), len(ulhc)
    w = Worker(P, (chip, chip), (W, W), refine_factor=2, refine_margin=8, zoom_factor=4)
    if chunk:
        w.configure(chunk=chunk)
    diag = torch.zeros((P, DIAG_DTYPE.itemsize), dtype=torch.uint8, device=dev)
    surf = torch.zeros((P, w.coarse_dim, w.coarse_dim), device=dev)
    args = [torch.from_numpy(a).to(dev) for a in (ref, tgt, ulhc)]
    w.correlate(*args, diag=diag, coarse_surfaces=surf, synchronize=False)
    torch.cuda.synchronize()
    bare = torch.zeros_like(diag)
    w.correlate(*args, diag=bare, synchronize=False)  # without surfaces
    torch.cuda.synchronize()
    assert torch.equal(diag, bare)
    w.close()
    return diag.cpu().numpy().view(DIAG_DTYPE).reshape(P), surf.cpu().numpy()


@pytest.mark.parametrize("chip,margin,samples", [(64, 64, 400), (64, 64, 403), (48, 64, 400), (64, 60, 401)])
def test_parts_equal_blocks(chip, margin, samples, monkeypatch):
    W, C = chip + 2 * margin, 2 * margin + 1
    s = C // 2 // 4 * 4
    ref = synth.speckle((420, samples), 61)
    other = synth.speckle((420, samples), 62)
    rng = np.random.default_rng(3)
    cells = [(0, 0), (s, s), (C - s - 1, C - s - 1), (C - 1, C - 1), (0, C - 1), (C - 1, 0), (s, 3), (5, C - s - 1)]
    ulhc = []
    for k, (u, v) in enumerate(cells):  # the chip's own samples at placement (u, v) of the window
        tl, ts = int(rng.integers(0, 420 - W)), int(rng.integers(0, samples - W))
        ulhc.append((tl + u, ts + v, tl, ts))
    ulhc = np.array(ulhc + [(419 - chip + 2, 0, 0, 0)], np.int32)
    # chips cut from the secondary itself, whose best placement is known, and others
    for r, known in ((ref, True), (other, False)):
        got, surf = run(r.copy(), ref, ulhc, chip, W)
        again, _ = run(r.copy(), ref, ulhc, chip, W, chunk=4)
        monkeypatch.setenv("AMPCOR_STAGED", "0")
        want, wsurf = run(r.copy(), ref, ulhc, chip, W)
        monkeypatch.delenv("AMPCOR_STAGED")
        np.testing.assert_array_equal(got[:-1], again[:-1])
        for f in ("coarse_u", "coarse_v", "top", "left"):
            np.testing.assert_array_equal(got[f], want[f], err_msg=f)
        assert np.abs(surf[:-1] - wsurf[:-1]).max() <= 2e-6  # each within 1e-6 of the definition
        if known:
            np.testing.assert_array_equal(np.stack([got["coarse_u"], got["coarse_v"]], 1)[:-1], cells)
