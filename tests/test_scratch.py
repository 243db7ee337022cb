"""The default chunk where the device has no room for its scratch (needs a B200): one wave of pairs
at a time, with the results of the whole chunk; and a smaller job between two larger ones."""
import numpy as np
import pytest

from ampcor_b200 import serve, synth
from ampcor_b200.worker import Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_default_chunk_gives_way_to_one_wave():
    ref = synth.speckle((768, 768), 31)
    tgt = synth.fourier_shift(ref, 1.3, -2.2)
    ulhc = serve.grid_corners(768, 768, 32, 16, 8)  # 7,921 pairs of 58 KB: 460 MB, a wave 34 MB
    dev = torch.device("cuda:0")
    args = [torch.from_numpy(a).to(dev) for a in (ref, tgt, ulhc)]

    def job(worker, n=None):
        return worker.correlate(args[0], args[1], args[2][:n].contiguous()).cpu().numpy()

    worker = Worker(len(ulhc), (32, 32), (64, 64), refine_factor=2, refine_margin=8, zoom_factor=8)
    assert worker.chunk >= len(ulhc)
    want = job(worker)
    np.testing.assert_array_equal(job(worker, 100), want[:100])
    np.testing.assert_array_equal(job(worker), want)
    worker.close()

    worker = Worker(len(ulhc), (32, 32), (64, 64), refine_factor=2, refine_margin=8, zoom_factor=8)
    torch.cuda.empty_cache()
    filler = torch.empty(torch.cuda.mem_get_info()[0] - (256 << 20), dtype=torch.uint8, device=dev)
    try:
        for _ in range(2):
            np.testing.assert_array_equal(job(worker), want)
            assert worker.chunk == 592
    finally:
        del filler
        torch.cuda.empty_cache()
        worker.close()
