"""Expired waits of the staged blocked kernels and of the calls that wait by themselves (needs a
B200): a 128 px chip's stages time out on a barrier that nothing completes, before any copy is
issued, in a raster job, the pair-by-pair interface and a banded host job; the call reports it, and
the same worker's next call gives the offsets of the one before."""
import numpy as np
import pytest

from ampcor_b200 import synth
from ampcor_b200.worker import Error, Worker

torch = pytest.importorskip("torch")
pytestmark = pytest.mark.gpu

R, M = 128, 32
W = R + 2 * M


def rasters():
    ref = synth.speckle((320, 384), 41)
    return ref, synth.fourier_shift(ref, 2.3, -1.7)


def corners(pairs):
    rng = np.random.default_rng(5)
    top, left = rng.integers(0, 320 - W + 1, pairs), rng.integers(0, 384 - W + 1, pairs)
    return np.stack([top + M, left + M, top, left], 1).astype(np.int32)


def calls():
    ref, tgt = rasters()

    def raster(worker, ulhc):
        return worker.correlate(*(torch.from_numpy(a).cuda() for a in (ref, tgt, ulhc))).cpu().numpy()

    def host(worker, ulhc):
        return worker.correlate(ref, tgt, ulhc)

    def arena(worker, ulhc):
        for k, (rl, rs, tl, ts) in enumerate(ulhc):
            worker.add_reference(k, ref[rl:rl + R, rs:rs + R])
            worker.add_target(k, tgt[tl:tl + W, ts:ts + W])
        return worker.adjust()

    return {"raster": raster, "host": host, "arena": arena}


@pytest.mark.parametrize("name", ["raster", "host", "arena"])
@pytest.mark.parametrize("pairs", [5, 40])  # (40: a banded host job, and arena blocks of one pair in several waves)
def test_expired_wait_is_reported(name, pairs):
    ulhc = corners(pairs)
    worker = Worker(pairs, (R, R), (W, W), refine_factor=2, refine_margin=8, zoom_factor=8)
    run = calls()[name]
    want = run(worker, ulhc)
    for _ in range(2):
        worker.inject_timeout(1)
        with pytest.raises(Error) as e:
            run(worker, ulhc)
        assert "AMPCOR_E_CUDA" in str(e.value) and "timed out" in str(e.value)
        np.testing.assert_array_equal(run(worker, ulhc), want)
    worker.close()


def test_the_blocked_kernels_time_out_themselves():
    """More waits run out than the zoom and the other staged kernels of a batch have CTAs."""
    ulhc = corners(40)
    worker = Worker(40, (R, R), (W, W), refine_factor=2, refine_margin=8, zoom_factor=8)
    worker.inject_timeout(1)
    with pytest.raises(Error) as e:
        calls()["raster"](worker, ulhc)
    expired = int(str(e.value).split(": ", 1)[1].split()[0])
    # coarse: a CTA per pair (summed blocks); fine: a CTA per block and multiprocessor; the zoom: a CTA
    # per pair at most
    sms = torch.cuda.get_device_properties(0).multi_processor_count
    assert 40 + min(4 * 40, sms) < expired <= 40 + min(4 * 40, sms) + 40
    worker.close()
