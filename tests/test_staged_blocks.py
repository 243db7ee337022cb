"""Blocked stages through the copy engine (needs a B200) against the general path (AMPCOR_STAGED=0,
one CTA per pair and block): the same coarse cells and offsets, both surfaces within the parity
tolerance, for blocks whose spectra are summed (tiles of 104 and 128 samples), blocks taken one by
one (160 samples), windows at every sample of a 16-byte unit, a pair off the raster, rasters whose
lines the copy engine cannot take, and more pairs than a chunk holds."""
import numpy as np
import pytest

from oracle import parity
from ampcor_b200 import synth
from ampcor_b200.worker import DIAG_DTYPE, Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def run(ref, tgt, ulhc, chip, W, chunk=0):
    P = len(ulhc)
    w = Worker(P, (chip, chip), (W, W), refine_factor=2, refine_margin=8, zoom_factor=4)
    if chunk:
        w.configure(chunk=chunk)
    dev = torch.device("cuda:0")
    diag = torch.zeros((P, DIAG_DTYPE.itemsize), dtype=torch.uint8, device=dev)
    cs = torch.full((P, w.coarse_dim, w.coarse_dim), -2.0, device=dev)
    rs = torch.full((P, w.refined_dim, w.refined_dim), -2.0, device=dev)
    off = w.correlate(*(torch.from_numpy(a).to(dev) for a in (ref, tgt, ulhc)), diag=diag, coarse_surfaces=cs,
                      refined_surfaces=rs, synchronize=False)
    torch.cuda.synchronize()
    out = off.cpu().numpy(), diag.cpu().numpy().view(DIAG_DTYPE).reshape(P), cs.cpu().numpy(), rs.cpu().numpy()
    w.close()
    return out


# chip 128: +-20 sums tiles of 104 samples, +-32 of 128, +-34 takes 132-sample tiles block by block;
# the refined stage always takes four 160-sample tiles block by block
@pytest.mark.parametrize("chip,margin", [(128, 20), (128, 32), (128, 34)])
@pytest.mark.parametrize("samples", [512, 517])
def test_against_the_general_path(chip, margin, samples, monkeypatch):
    W = chip + 2 * margin
    ref = synth.speckle((400, samples), 41)
    tgt = (synth.fourier_shift(ref, -2.6, 3.2) + synth.noise(ref.shape, 10.0, 42)).astype(np.complex64)
    ulhc = np.array([[y + margin, x + margin, y, x] for y in (0, 57, 113, 401 - W) for x in range(0, samples - W + 1, 37)],
                    np.int32)
    ulhc[5, 3] = samples  # leaves the raster
    got = run(ref, tgt, ulhc, chip, W, chunk=len(ulhc) // 2)
    monkeypatch.setenv("AMPCOR_STAGED", "0")
    want = run(ref, tgt, ulhc, chip, W)
    bad = np.isnan(want[0]).any(axis=1)
    assert bad[5] and np.array_equal(np.isnan(got[0]), np.isnan(want[0]))
    ok = ~bad
    for f in ("coarse_u", "coarse_v", "top", "left"):
        assert np.array_equal(got[1][f][ok], want[1][f][ok])
    np.testing.assert_array_equal(got[0][ok], want[0][ok])
    np.testing.assert_allclose(got[2][ok], want[2][ok], atol=parity.SURF_ATOL, rtol=0)
    np.testing.assert_allclose(got[3][ok], want[3][ok], atol=parity.SURF_ATOL, rtol=0)
