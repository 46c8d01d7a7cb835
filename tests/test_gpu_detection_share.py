"""Detection where the caller has a share of the GPU's SMs (a green context): the
distance rule's launch takes no more blocks than the share holds, with the share's
context current and on one of its streams, and the results are the oracle's."""
import numpy as np
import pytest

from test_detection_oracle import bits

pytestmark = pytest.mark.gpu

N, DISTANCE = 400_000, 700  # 200,000 peaks and more: a block on each SM of the device


@pytest.fixture
def share(cuda):
    import torch
    from torch.cuda import green_contexts
    if not green_contexts.SUPPORTED:
        pytest.skip("green contexts are not supported")
    torch.ones(1, device="cuda")
    return green_contexts.GreenContext.create(16, 0)


def _problem():
    from oracle import detection as odet
    rng = np.random.default_rng(4)
    x = rng.standard_normal(N).astype(np.float32)
    x[::2] += np.float32(3.0)  # every other sample is a peak
    thr = np.full(N, 5.0, np.float32)
    source = rng.integers(0, 1000, size=N).astype(np.int32)
    return x, thr, source, np.asarray(odet.find_peaks(x, DISTANCE), np.int64)


def _check(x, thr, source, want):
    from beampower_b200 import detection as det
    got, _ = det.find_peaks(x, distance=DISTANCE)
    assert np.array_equal(got, want)
    d = det.detect(x, source, threshold=thr, distance=DISTANCE)
    want = want[x[want] > thr[want]]
    assert 0 < len(want) and np.array_equal(d.peaks, want)
    assert np.array_equal(bits(d.heights), bits(x[want]))
    assert np.array_equal(d.sources, source[want])


def test_share_as_the_current_context(share):
    problem = _problem()
    share.set_context()
    try:
        _check(*problem)
    finally:
        share.pop_context()
    _check(*problem)


def test_stream_of_a_share(share):
    import torch
    problem = _problem()
    with torch.cuda.stream(share.Stream()):
        _check(*problem)
    torch.cuda.synchronize()
