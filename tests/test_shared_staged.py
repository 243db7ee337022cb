"""Short transforms run several resident CTAs per multiprocessor (needs a B200): the compiled tile
lengths of that form against the FP64 oracle pair by pair, with more pairs than resident CTAs and
with fewer, the same offsets bit for bit."""
import numpy as np
import pytest

from oracle import parity
from ampcor_b200 import synth
from ampcor_b200.worker import DIAG_DTYPE, Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


# (chip, margin, refine margin): coarse and fine tile lengths 24/48, 32/48, 40/80, 48/80, 64/80, 80/96
@pytest.mark.parametrize("chip,margin,m", [(16, 4, 4), (16, 8, 4), (24, 8, 8), (24, 12, 8), (32, 16, 4), (32, 21, 8)])
def test_short_transforms(chip, margin, m):
    W = chip + 2 * margin
    side = 18 * 20 + W
    ref = synth.speckle((side, side), 31)
    tgt = (synth.fourier_shift(ref, 1.4, -0.7) + synth.noise(ref.shape, 10.0, 32)).astype(np.complex64)
    ulhc = np.array([[y + margin, x + margin, y, x] for y in range(0, 18 * 20, 20) for x in range(0, 18 * 20, 20)],
                    np.int32)
    P = len(ulhc)  # 324, more than two per multiprocessor
    worker = Worker(P, (chip, chip), (W, W), refine_factor=2, refine_margin=m, zoom_factor=4)
    assert worker.form == "spectral"
    dev = torch.device("cuda:0")
    r, t, u = (torch.from_numpy(a).to(dev) for a in (ref, tgt, ulhc))
    diag = torch.zeros((P, DIAG_DTYPE.itemsize), dtype=torch.uint8, device=dev)
    cs = torch.zeros((P, worker.coarse_dim, worker.coarse_dim), device=dev)
    rs = torch.zeros((P, worker.refined_dim, worker.refined_dim), device=dev)
    off = worker.correlate(r, t, u, diag=diag, coarse_surfaces=cs, refined_surfaces=rs).cpu().numpy()
    orc = parity.oracle_run(ref, tgt, ulhc, chip, W, 2, m, 4)
    rep = parity.compare(orc, off, diag.cpu().numpy().view(DIAG_DTYPE).reshape(P), cs.cpu().numpy(), rs.cpu().numpy())
    assert not rep["failures"], parity.summary(rep)
    assert rep["max_abs_err_non_excused_px"] == 0.0
    few = worker.correlate(r, t, u[:100].contiguous()).cpu().numpy()
    assert np.array_equal(few, off[:100])
    worker.close()
