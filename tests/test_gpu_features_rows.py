"""Envelope rows at the lengths where the transform and the medians change their
way -- odd and even, one complex number, up to 4,096 samples (selected by one
block), above (a sampled bracket), long single rows (radix select) -- and with the
rows that a sampled bracket does not fit: many equal values, a row whose sampled
places are unlike the rest, values that are not finite.

Two checks.  Against the oracle, with the bound of test_gpu_features.py.  And of
the statistics themselves, exactly: a feature (e - median) / MAD is a monotone
function of the envelope e in float32, so the middle values of the features lie
on both sides of 0 and (a MAD above 0) those of their moduli on both sides of 1."""
import numpy as np
import pytest

from test_gpu_features import _bound

pytestmark = pytest.mark.gpu


def _sampled_places(n, count=4096):
    j = np.arange(count, dtype=np.uint64)
    h = (j * np.uint64(2654435761)) & np.uint64(0xFFFFFFFF)
    return ((j * np.uint64(n)) // np.uint64(count) + ((h * np.uint64(n // count)) >> np.uint64(32))
            ).astype(np.int64)


def _row(kind, n, rng):
    x = rng.standard_normal(n).astype(np.float32)
    if kind == "few":        # a handful of envelope values
        return np.resize(np.array([1, 0, -1, 0, 2, 0, -2, 0], np.float32), n)
    if kind == "zero":
        return np.zeros(n, np.float32)
    if kind == "quiet":      # mostly silence
        x[: 3 * n // 4] = 0.0
    if kind == "unlike" and n > 4096:
        places = _sampled_places(n)
        x = np.zeros(n, np.float32)
        x[places] = 10.0 * rng.choice([-1.0, 1.0], size=len(places))
    return x


LENGTHS = [2, 3, 4, 5, 6, 127, 1000, 4095, 4096, 4097, 4098, 8193, 20480, 49999, 262144, 262146,
           300001]


@pytest.mark.parametrize("kind", ["noise", "few", "zero", "quiet", "unlike"])
@pytest.mark.parametrize("n", LENGTHS)
def test_row_lengths(cuda, n, kind):
    import torch
    from scipy import signal
    from oracle import features as ofeat
    from beampower_b200.features import envelope
    rng = np.random.default_rng(n)
    rows = np.stack([_row(kind, n, rng), _row("noise", n, rng), 5 * _row(kind, n, rng)])
    got = envelope(torch.from_numpy(rows).to(cuda)).cpu().numpy()
    # rows whose start is off the transforms' alignment, and a result in place
    off = torch.zeros(1 + rows.size, device=cuda)
    off[1:] = torch.from_numpy(rows.ravel()).to(cuda)
    assert np.array_equal(envelope(off[1:].view(rows.shape)).cpu().numpy(), got)
    for x, f in zip(rows, got):
        raw = np.abs(signal.hilbert(x.astype(np.float64)))
        med = np.median(raw)
        mad = np.median(np.abs(raw - med))
        if mad > 1e-4 * raw.max(initial=1e-30):
            ref = ofeat.envelope(x)
            err = np.abs(f.astype(np.float64) - ref)
            assert np.all(err <= _bound(raw, ref)), float(err.max())
        s, a = np.sort(f), np.sort(np.abs(f))
        assert s[(n - 1) // 2] <= 0 <= s[n // 2]
        if np.any(f != 0) and mad > 1e-4 * raw.max(initial=1e-30) and s[-1] < 1e5:
            assert a[(n - 1) // 2] <= 1 <= a[n // 2]


@pytest.mark.parametrize("n", [2, 3, 8, 9, 4096, 4097, 20480, 30001])
@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_values_that_are_not_finite(cuda, n, bad):
    from beampower_b200.features import envelope
    rng = np.random.default_rng(n)
    x = rng.standard_normal((3, n)).astype(np.float32)
    clean = envelope(x)
    x[1, n // 2] = bad
    got = envelope(x)
    assert np.all(np.isnan(got[1]))
    if n % 2 == 0:  # (cuFFT computes two real rows of an odd length as one complex row)
        assert np.array_equal(got[0], clean[0]) and np.array_equal(got[2], clean[2])
