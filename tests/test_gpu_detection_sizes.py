"""Detection at the sizes where its kernels can go wrong: the 4,096 samples of a
mask block, pairwise-sum leaves of 8 and 128 values and their blocks, peaks whose
distance rule takes one round or one round per kept peak, plateaus across blocks.
Everything is exact, against the oracle."""
import numpy as np
import pytest

from test_detection_oracle import bits

pytestmark = pytest.mark.gpu


def _series(kind, n, rng):
    x = rng.standard_normal(n).astype(np.float32)
    t = np.arange(n)
    if kind == "up":        # peaks that grow: one round per kept peak
        x = (t * 1e-3 + (t % 4 == 1)).astype(np.float32)
    elif kind == "down":
        x = (-t * 1e-3 + (t % 4 == 1)).astype(np.float32)
    elif kind == "equal":   # heights that are all the same
        x = (t % 2).astype(np.float32)
    elif kind == "steps":   # plateaus of many lengths, up to the end
        x = np.repeat(x, rng.integers(1, 40, size=n))[:n]
    elif kind == "flat":    # one plateau over the blocks between two steps
        x = np.ones(n, np.float32)
        x[:1] = x[n - 1:] = 0.0
    elif kind == "holes":
        x[rng.random(n) < 0.2] = np.nan
    return x


@pytest.mark.parametrize("kind", ["noise", "up", "down", "equal", "steps", "flat", "holes"])
@pytest.mark.parametrize("n", [0, 1, 2, 3, 4, 31, 33, 511, 513, 4095, 4096, 4097, 8193, 40001])
def test_peaks(cuda, n, kind):
    from oracle import detection as odet
    from beampower_b200 import detection as det
    rng = np.random.default_rng(n)
    x = _series(kind, n, rng)
    thr = np.full(n, np.nanmedian(x) if n else 0.0, np.float32)
    source = rng.integers(0, 1000, size=n).astype(np.int32)
    for distance in (None, 1, 2, 3.5, 10, 40, 700, n + 5):
        want = np.asarray(odet.find_peaks(x, distance), np.int64)
        got, _ = det.find_peaks(x, distance=distance)
        assert np.array_equal(got, want), distance
        if distance is None:
            continue
        d = det.detect(x, source, threshold=thr, distance=distance)
        want = want[x[want] > thr[want]]
        assert np.array_equal(d.peaks, want), distance
        assert np.array_equal(bits(d.heights), bits(x[want]))
        assert np.array_equal(d.sources, source[want])


@pytest.mark.parametrize("n,window", [(9, 1), (20, 7), (20, 8), (300, 127), (300, 128), (300, 129),
                                      (1100, 256), (1100, 263), (5000, 1031), (70000, 16385),
                                      (300000, 100003)])
@pytest.mark.parametrize("zeros", ["none", "some", "all but one", "all"])
def test_threshold(cuda, n, window, zeros):
    from oracle import detection as odet
    from beampower_b200 import detection as det
    rng = np.random.default_rng(n + window)
    x = (1.0 + rng.standard_normal(n)).astype(np.float32)
    if zeros == "some":
        x[rng.random(n) < 0.1] = 0.0
    elif zeros != "none":
        x[:] = 0.0
        if zeros != "all":
            x[n // 2] = 3.0
    noise = rng.standard_normal(int((x == 0).sum())).astype(np.float32)
    overlap = 0.66 if window >= 7 else 0.0
    for kind in ("rms", "mad"):
        got = det.time_dependent_threshold(x, window, overlap, kind, 8.0, white_noise=noise)
        want = odet.time_dependent_threshold(x, window, overlap, kind, 8.0, white_noise=noise)
        assert np.array_equal(bits(got), bits(want)), kind
