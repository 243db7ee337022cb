"""The zoom's bounds (needs a B200) where they are cut finest: odd zooms (their sampled rows miss the
surface's own, and the last interval may be short) and z = 2, on noise (every column is kept, and most rows
go) and on peaks, for each of the kernels that a call's number of pairs selects; and surfaces of NaN.

The zoomed maximum is compared with the FP64 interpolation of the refined surface the worker returns.
Each cell is two FP32 sums of Cf terms; a sum's partial sums are cells of its own kind, no larger than
about the largest cell, so that sqrt(Cf) independent roundings of 2^-24 of it, twice, bound the error."""
import numpy as np
import pytest

from ampcor_b200 import synth
from ampcor_b200.worker import DIAG_DTYPE, Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def interpolation(Cf, z):
    d = np.arange(Cf * z)[:, None] / z - np.arange(Cf)
    return (1.0 + 2.0 * sum(np.cos(2.0 * np.pi * n * d / Cf) for n in range(1, (Cf - 1) // 2 + 1))) / Cf


def pair_counts():
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    return {"one": sms, "two": sms + 52, "five": 4 * sms + 1}  # to a multiprocessor


def corners(n):
    rng = np.random.default_rng(n)
    y, x = rng.integers(0, 237, n), rng.integers(0, 237, n)
    return np.stack([y + 16, x + 16, y, x], 1).astype(np.int32)


@pytest.mark.parametrize("each", ["one", "two", "five"])
@pytest.mark.parametrize("kind", ["peak", "noise"])
# (surfaces of 17, 33 and 49 samples, and of 41 at the refinement factor 5)
@pytest.mark.parametrize("m,z,f", [(4, 2, 2), (4, 5, 2), (4, 7, 2), (8, 2, 2), (8, 3, 2), (8, 5, 2), (8, 7, 2), (8, 8, 2),
                                   (12, 4, 2), (4, 3, 5), (4, 4, 5)])
def test_maximum(m, z, f, kind, each):
    n = pair_counts()[each]
    ref = synth.speckle((300, 300), 21)
    tgt = synth.fourier_shift(ref, 1.3, -2.2) if kind == "peak" else synth.speckle((300, 300), 22)
    R = 16 if f == 5 else 32 if m < 12 else 40  # (at factor 2 chip and R + 2 m are compiled tiles of the refinement)
    ulhc = corners(n)
    worker = Worker(n, (R, R), (64, 64), refine_factor=f, refine_margin=m, zoom_factor=z)
    if worker.form != "spectral":
        pytest.skip("no spectral form of this geometry")
    dev = torch.device("cuda:0")
    diag = torch.zeros((n, DIAG_DTYPE.itemsize), dtype=torch.uint8, device=dev)
    surf = torch.zeros((n, worker.refined_dim, worker.refined_dim), device=dev)
    worker.correlate(*(torch.from_numpy(a).to(dev) for a in (ref, tgt, ulhc)), diag=diag, refined_surfaces=surf)
    d = diag.cpu().numpy().view(DIAG_DTYPE).reshape(n)
    U = torch.from_numpy(interpolation(worker.refined_dim, z)).to(dev)
    Zm = U @ surf.double() @ U.T
    best = Zm.flatten(1).amax(1)
    tol = 2.0 * np.sqrt(worker.refined_dim) * 2.0 ** -24 * Zm.abs().flatten(1).amax(1)
    pick = torch.from_numpy((d["fine_p"].astype(np.int64) * Zm.shape[-1] + d["fine_q"])).to(dev)
    cells = Zm.flatten(1).gather(1, pick[:, None])[:, 0]
    assert (best - cells <= 2 * tol).all()
    assert ((torch.from_numpy(d["zoom_peak"].copy()).to(dev).double() - best).abs() <= tol).all()
    worker.close()


@pytest.mark.parametrize("each", ["one", "two", "five"])
def test_a_surface_of_nan_has_no_maximum(each):
    n, R, W = pair_counts()[each], 32, 64
    ref = synth.speckle((300, 300), 21)
    tgt = synth.fourier_shift(ref, 1.3, -2.2)
    worker = Worker(n, (R, R), (W, W), refine_factor=2, refine_margin=8, zoom_factor=8)

    def run(bad):
        for k, (rl, rs, tl, ts) in enumerate(corners(n)):
            chip = ref[rl:rl + R, rs:rs + R].copy()
            if bad and k % 7 == 3:
                chip[5, 6] = np.nan
            worker.add_reference(k, chip)
            worker.add_target(k, tgt[tl:tl + W, ts:ts + W])
        return worker.adjust(), worker.diagnostics()

    want, _ = run(False)
    got, diag = run(True)
    nan = np.arange(n) % 7 == 3
    np.testing.assert_array_equal(got[~nan], want[~nan])
    assert np.isneginf(diag["zoom_peak"][nan]).all()
    worker.close()
