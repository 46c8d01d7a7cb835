"""The order of the sources in a table's tiles decides no result: beams against
the oracle, bit for bit, at the sizes where the splits can go wrong -- around one
tile, around the 4,096 sources that one block orders by itself, above it -- and
with delays that are all equal, few, far apart or of both signs."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    a = np.ascontiguousarray(a, dtype=np.float32).copy()
    a[np.isnan(a)] = np.float32(np.nan)
    return a.view(np.uint32)


def _delays(kind, N, S, P, rng):
    if kind == "equal":
        return np.full((N, S, P), 7, np.int32)
    if kind == "two":
        return (5 + 3 * rng.integers(0, 2, size=(N, S, P))).astype(np.int32)
    if kind == "signs":
        return rng.integers(-30, 31, size=(N, S, P)).astype(np.int32)
    far = rng.integers(0, 40, size=(N, S, P))  # "far": some beyond every sample
    far[rng.random((N, S, P)) < 0.01] = 2_000_000_000
    return far.astype(np.int32)


@pytest.mark.parametrize("kind", ["equal", "two", "signs", "far"])
@pytest.mark.parametrize("N,S,P", [(64, 3, 1), (65, 3, 2), (129, 17, 2), (191, 65, 2),
                                   (4095, 4, 1), (4096, 2, 2), (4097, 3, 1), (8193, 2, 1),
                                   (12289, 1, 1)])
def test_source_order(cuda, bplib, oracle_lib, N, S, P, kind):
    import torch
    from beampower_b200.tables import TravelTimeTable
    rng = np.random.default_rng(N + S)
    T = 70
    F = rng.standard_normal((S, 1, T)).astype(np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
    D = _delays(kind, N, S, P, rng)
    W = np.ones((N, S), np.float32)
    W[rng.random((N, S)) < 0.2] = 0.0
    U = oracle_lib.prestack(F, A)
    table = TravelTimeTable(D, W)
    traces = table.traces_from_features(F, A)
    for oob in (0, 1):
        bm, am = table.beamform_max(traces, oob)
        beam = table.beamform(traces, oob)
        torch.cuda.synchronize()
        want_bm, want_am = oracle_lib.beamform_max(U, D, W, oob)
        assert np.array_equal(_bits(bm.cpu().numpy()), _bits(want_bm)), oob
        assert np.array_equal(am.cpu().numpy(), want_am), oob
        want = oracle_lib.beamform(U, D, W, oob)
        assert np.array_equal(_bits(beam.cpu().numpy()), _bits(want)), oob
    table.close()
