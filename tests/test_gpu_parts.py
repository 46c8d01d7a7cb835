"""A table whose tiles run as several launches -- the narrow ones with the
tensor-memory kernel, wider ones with a faster staged shape than the widest of
them allows -- gives the oracle's beams, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    a = np.ascontiguousarray(a, dtype=np.float32).copy()
    a[np.isnan(a)] = np.float32(np.nan)
    return a.view(np.uint32)


def _table(widths, S, P, weights, seed):
    """4,096 sources per width, in as many clusters of near delays."""
    rng = np.random.default_rng(seed)
    D, W = [], []
    for w in widths:
        D.append(rng.integers(0, w + 1, size=(4096, S, P)))
        W.append(np.ones((4096, S)))
    D, W = np.concatenate(D).astype(np.int32), np.concatenate(W).astype(np.float32)
    order = rng.permutation(len(D))
    D, W = D[order], W[order]
    if weights != "ones":
        W[rng.random(W.shape) < 0.2] = 0.0
    if weights == "real":
        W *= rng.uniform(0.5, 1.5, size=W.shape).astype(np.float32)
    return D, W


# parts: launches of the beams; planes: one that prepares the tensor-memory part
@pytest.mark.parametrize("widths,P,weights,parts,planes", [
    ((20, 3000), 2, "zero_one", 2, 1),        # tensor memory, a staged shape
    ((1500, 5000), 2, "real", 2, 0),          # two staged shapes
    ((20, 9000, 40000), 1, "zero_one", 3, 1), # all three
    ((20, 100), 2, "zero_one", 1, 1),         # narrow throughout
])
def test_parts(cuda, bplib, oracle_lib, widths, P, weights, parts, planes):
    import torch
    from beampower_b200.core import launch_count
    from beampower_b200.tables import TravelTimeTable
    S, T = 2, 62_000  # 122 time tiles: 4,880 pairs with 40 tiles
    D, W = _table(widths, S, P, weights, len(widths) + P)
    rng = np.random.default_rng(T)
    F = rng.standard_normal((S, 1, T)).astype(np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
    U = oracle_lib.prestack(F, A)
    table = TravelTimeTable(D, W)
    traces = table.traces_from_features(F, A)
    for oob in (0, 1):
        before = launch_count()
        bm, am = table.beamform_max(traces, oob)
        assert launch_count() - before == parts + planes + 1  # and the decode
        torch.cuda.synchronize()
        want_bm, want_am = oracle_lib.beamform_max(U, D, W, oob)
        assert np.array_equal(_bits(bm.cpu().numpy()), _bits(want_bm)), oob
        assert np.array_equal(am.cpu().numpy(), want_am), oob
    table.close()
    # whole response of the same table, fewer samples: one launch
    T = 700
    table = TravelTimeTable(D, W)
    traces = table.traces_from_features(F[:, :, :T], A)
    beam = table.beamform(traces, 1)
    torch.cuda.synchronize()
    want = oracle_lib.beamform(oracle_lib.prestack(np.ascontiguousarray(F[:, :, :T]), A), D, W, 1)
    assert np.array_equal(_bits(beam.cpu().numpy()), _bits(want))
    table.close()
