"""Thresholds of many short windows, whose pairwise sums share blocks: windows of every
depth of the sums' tree up to the one from which a window has blocks of its own (8,193
samples), numbers of windows that fill the last block or leave it with one.  Exact,
against the oracle."""
import numpy as np
import pytest

from test_detection_oracle import bits

pytestmark = pytest.mark.gpu


# depths 0 0 0 0 0 1 1 2 2 2 3 4 5 6 6 7
@pytest.mark.parametrize("window", [1, 2, 7, 8, 128, 129, 256, 257, 263, 512, 520, 1031, 2047,
                                    4103, 8192, 8193])
@pytest.mark.parametrize("windows", [2, 64, 65, 200])
def test_threshold(cuda, window, windows):
    from oracle import detection as odet
    from beampower_b200 import detection as det
    rng = np.random.default_rng(window + windows)
    overlap = 0.66 if window >= 7 else 0.0
    shift = int((1.0 - overlap) * window)
    n = window + shift * (windows - 1) + (1 if shift > 1 else 0)
    x = (1.0 + rng.standard_normal(n)).astype(np.float32)
    x[rng.random(n) < 0.01] = 0.0
    noise = rng.standard_normal(int((x == 0).sum())).astype(np.float32)
    got = det.time_dependent_threshold(x, window, overlap, "rms", 8.0, white_noise=noise)
    want = odet.time_dependent_threshold(x, window, overlap, "rms", 8.0, white_noise=noise)
    assert np.array_equal(bits(got), bits(want))
