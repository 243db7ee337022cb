"""A chunk that a caller configures is the one that runs (needs a B200), also where it is the default
of the form before."""
import numpy as np
import pytest

from ampcor_b200 import synth
from ampcor_b200.worker import Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_chunk_equal_to_the_other_forms_default():
    w = synth.plain_512()
    worker = Worker(w.pairs, (32, 32), (48, 48), refine_factor=2, refine_margin=4, zoom_factor=4)
    args = [torch.from_numpy(a).cuda() for a in (w.ref, w.tgt, w.ulhc)]
    worker.configure("spectral")
    want = worker.correlate(*args).cpu().numpy()
    chunk = worker.chunk
    worker.configure("tensor", chunk)
    assert worker.chunk == chunk
    worker.correlate(*args)
    assert worker.chunk == chunk
    worker.configure("spectral")
    assert worker.chunk == chunk
    np.testing.assert_array_equal(worker.correlate(*args).cpu().numpy(), want)
    worker.close()
