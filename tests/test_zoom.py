"""The zoom's maximum (needs a B200) against the FP64 interpolation of the refined surfaces the
worker returns: sizes at the edges of the kernel's row tiles and column batches, surfaces whose
maximum stands out (few columns kept), surfaces of noise (every column kept) and flat ones."""
import numpy as np
import pytest

from ampcor_b200 import synth
from ampcor_b200.worker import DIAG_DTYPE, Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def interpolation(Cf, z):
    d = np.arange(Cf * z)[:, None] / z - np.arange(Cf)
    return (1.0 + 2.0 * sum(np.cos(2.0 * np.pi * n * d / Cf) for n in range(1, (Cf - 1) // 2 + 1))) / Cf


def rasters(kind):
    ref = synth.speckle((300, 300), 21)
    if kind == "peak":
        return ref, synth.fourier_shift(ref, 1.3, -2.2)
    if kind == "noise":
        return ref, synth.speckle((300, 300), 22)
    return np.ones((300, 300), np.complex64), np.ones((300, 300), np.complex64)


@pytest.mark.parametrize("kind", ["peak", "noise", "flat"])
# Z = 17 and 68 (one tile), 132 and 264 (a last tile of 4 and 8 rows), 272, 528 (one CTA per SM)
@pytest.mark.parametrize("m,z", [(4, 1), (4, 4), (8, 4), (8, 8), (4, 16), (8, 16)])
def test_zoom_maximum(m, z, kind):
    ref, tgt = rasters(kind)
    ulhc = np.array([[y + 16, x + 16, y, x] for y in range(0, 236, 59) for x in range(0, 236, 47)], np.int32)
    P = len(ulhc)
    worker = Worker(P, (32, 32), (64, 64), refine_factor=2, refine_margin=m, zoom_factor=z)
    dev = torch.device("cuda:0")
    diag = torch.zeros((P, DIAG_DTYPE.itemsize), dtype=torch.uint8, device=dev)
    surf = torch.zeros((P, worker.refined_dim, worker.refined_dim), device=dev)
    off = worker.correlate(torch.from_numpy(ref).to(dev), torch.from_numpy(tgt).to(dev),
                           torch.from_numpy(ulhc).to(dev), diag=diag, refined_surfaces=surf).cpu().numpy()
    d = diag.cpu().numpy().view(DIAG_DTYPE).reshape(P)
    G = surf.cpu().numpy().astype(np.float64)
    U = interpolation(worker.refined_dim, z)
    Zm = U @ G @ U.T
    # three of the four tf32 products of a split pair: 2^-21 of |U| |G| |U| each product
    lip = np.abs(U).sum(1).max()
    tol = 2.0 ** -20 * lip * lip * max(np.abs(G).max(), 1e-30)
    cells = Zm[np.arange(P), d["fine_p"], d["fine_q"]]
    best = Zm.reshape(P, -1).max(1)
    assert np.all(best - cells <= 2 * tol), (best - cells).max()
    assert np.all(np.abs(d["zoom_peak"] - best) <= tol)
    if kind == "flat":
        assert not d["fine_p"].any() and not d["fine_q"].any()
    np.testing.assert_array_equal(off[:, 0], d["top"] - 16 + d["fine_p"] / np.float32(2 * z))
    np.testing.assert_array_equal(off[:, 1], d["left"] - 16 + d["fine_q"] / np.float32(2 * z))
    worker.close()


@pytest.mark.parametrize("kind", ["peak", "noise"])
# one, two, three and four pairs to a multiprocessor: teams of nine warps, then of three
@pytest.mark.parametrize("m,z", [(4, 4), (8, 8), (8, 16)])
def test_zoom_teams_agree(m, z, kind):
    ref, tgt = rasters(kind)
    ulhc = np.array([[y + 16, x + 16, y, x] for y in range(0, 236, 59) for x in range(0, 236, 47)], np.int32)
    P, dev = len(ulhc), torch.device("cuda:0")
    sms = torch.cuda.get_device_properties(dev).multi_processor_count
    got = []
    for n in (P, 2 * sms, 2 * sms + 1, 3 * sms, 3 * sms + 1):
        many = np.ascontiguousarray(np.resize(ulhc, (n, 4)))
        worker = Worker(n, (32, 32), (64, 64), refine_factor=2, refine_margin=m, zoom_factor=z)
        diag = torch.zeros((n, DIAG_DTYPE.itemsize), dtype=torch.uint8, device=dev)
        worker.correlate(torch.from_numpy(ref).to(dev), torch.from_numpy(tgt).to(dev), torch.from_numpy(many).to(dev),
                         diag=diag)
        d = diag.cpu().numpy()
        np.testing.assert_array_equal(d, d[np.arange(n) % P])
        got.append(d[:P])
        worker.close()
    for d in got[1:]:
        np.testing.assert_array_equal(d, got[0])
