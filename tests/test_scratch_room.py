"""The default chunk's scratch leaves room (needs a B200): a job whose rasters fit beside one wave of
pairs but not beside the whole chunk runs, on a new worker and on one that already holds the chunk;
and a worker takes no more than a share of the memory that is free."""
import numpy as np
import pytest

from ampcor_b200 import serve, synth
from ampcor_b200.worker import Error, Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

MB = 1 << 20


def new_worker(pairs):
    return Worker(pairs, (32, 32), (64, 64), refine_factor=2, refine_margin=8, zoom_factor=8)


class Filled:
    """All but `left` bytes of the device memory taken."""

    def __init__(self, left):
        torch.cuda.synchronize()
        torch.cuda.empty_cache()
        self.block = torch.empty(torch.cuda.mem_get_info()[0] - left, dtype=torch.uint8, device="cuda:0")

    def __enter__(self):
        return self

    def __exit__(self, *exc):
        self.block = None
        torch.cuda.empty_cache()


@pytest.fixture(scope="module")
def jobs():
    """7,921 pairs, 435 MiB of scratch (a wave 33), on a corner of rasters whose amplitudes and box
    statistics take 192 MiB, and the same pairs on rasters of the corner alone (7 MiB)."""
    ref = synth.speckle((768, 768), 31)
    small = ref, synth.fourier_shift(ref, 1.3, -2.2)
    ulhc = serve.grid_corners(768, 768, 32, 16, 8)
    dev = torch.device("cuda:0")
    corner = [torch.from_numpy(a).to(dev) for a in small]
    whole = [torch.zeros((4096, 4096), dtype=torch.complex64, device=dev) for _ in small]
    for w, c in zip(whole, corner):
        w[:768, :768] = c
    u = torch.from_numpy(ulhc).to(dev)
    worker = new_worker(len(ulhc))
    assert worker.chunk >= len(ulhc)
    want = worker.correlate(*corner, u).cpu().numpy()
    # (blocks of box rows differ between the rasters: compared with their own results)
    want_whole = worker.correlate(*whole, u).cpu().numpy()
    worker.close()
    return corner, whole, u, want, want_whole


def test_rasters_come_before_the_chunk(jobs):
    corner, whole, u, want, want_whole = jobs
    worker = new_worker(len(u))
    with Filled(535 * MB):
        for _ in range(2):
            np.testing.assert_array_equal(worker.correlate(*whole, u).cpu().numpy(), want_whole)
    worker.close()


def test_chunk_held_gives_way_to_rasters(jobs):
    corner, whole, u, want, want_whole = jobs
    worker = new_worker(len(u))
    np.testing.assert_array_equal(worker.correlate(*corner, u).cpu().numpy(), want)
    with Filled(64 * MB):
        np.testing.assert_array_equal(worker.correlate(*whole, u).cpu().numpy(), want_whole)
        assert worker.chunk == 592
        np.testing.assert_array_equal(worker.correlate(*corner, u).cpu().numpy(), want)
    worker.close()


def test_chunk_held_gives_way_to_host_rasters(jobs):
    corner, _, u, want, _ = jobs
    worker = new_worker(len(u))
    np.testing.assert_array_equal(worker.correlate(*corner, u).cpu().numpy(), want)
    host = [np.zeros((2048, 2048), np.complex64) for _ in corner]
    for h, c in zip(host, corner):
        h[:768, :768] = c.cpu().numpy()
    with Filled(8 * MB):
        got = worker.correlate(*host, u.cpu().numpy())
    np.testing.assert_array_equal(got, worker.correlate(*(torch.from_numpy(h).to(u.device) for h in host), u).cpu().numpy())
    worker.close()


def test_chunk_of_a_captured_job_stays(jobs):
    corner, whole, u, want, want_whole = jobs
    worker = new_worker(len(u))
    out = torch.empty((len(u), 2), device=u.device)
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        worker.correlate(*corner, u, offsets=out, stream=stream)
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        worker.correlate(*corner, u, offsets=out, stream=stream, synchronize=False)
    graph.replay()
    torch.cuda.synchronize()
    # (the host path's own staging is what finds no room: it replaces no buffer of the captured job)
    host = [np.zeros((2048, 2048), np.complex64) for _ in corner]
    with Filled(8 * MB):
        with pytest.raises(Error):
            worker.correlate(*host, u.cpu().numpy())
        out.zero_()
        graph.replay()
        torch.cuda.synchronize()
        np.testing.assert_array_equal(out.cpu().numpy(), want)
    del graph
    worker.close()


def test_chunk_takes_a_share_of_what_is_free(jobs):
    corner, _, u, want, _ = jobs
    worker = new_worker(len(u))
    with Filled(2048 * MB):  # an eighth is 256 MiB
        np.testing.assert_array_equal(worker.correlate(*corner, u).cpu().numpy(), want)
        assert worker.chunk == 592
        assert torch.cuda.mem_get_info()[0] > (2048 - 128) * MB
    worker.close()
