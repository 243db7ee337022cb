"""A tuned batch also times the chunk that an untuned one takes (needs a B200)."""
import pytest

from ampcor_b200 import batch
from ampcor_b200.worker import Worker

pytest.importorskip("torch")
pytestmark = pytest.mark.gpu


def test_the_default_chunk_is_a_candidate():
    jobs = [j for j in batch.uneven_jobs(n=2, seed=3)][:1]
    c, m, f, rm, z = jobs[0].geometry
    worker = Worker(jobs[0].pairs, (c, c), (c + 2 * m, c + 2 * m), refine_factor=f, refine_margin=rm, zoom_factor=z)
    default = worker.chunk
    worker.close()
    ub = batch.UnevenBatch(jobs)
    timed = [r["chunk"] for r in ub.tuning[jobs[0].geometry]["candidates"] if r["form"] == "spectral"]
    # (of the chunks that hold the whole batch only the smallest is timed)
    assert default in timed or any(jobs[0].pairs <= t <= default for t in timed)
    ub.close()
