"""Which FP32 calls run the tensor-memory kernel, by their number of (table tile, time
tile) pairs and the tiles' work; both kernels give the oracle's beams, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    return np.ascontiguousarray(a, dtype=np.float32).view(np.uint32)


# launches of reduce='max': the staged kernel and the decode; the tensor-memory kernel
# has its traces prepared by one more
STAGED, TMEM = 2, 3


@pytest.mark.parametrize("N,S,T,masked,want", [
    (64, 20, 512, False, STAGED),            # one pair
    (64 * 37, 20, 512 * 4 - 5, False, STAGED),   # one pair per SM of 148
    (64 * 37, 20, 512 * 14 - 5, False, TMEM),    # 3.5: shares of equal tiles
    (64 * 37, 12, 512 * 40 - 5, False, TMEM),    # 10
    (64 * 37, 4, 512 * 160 - 5, False, TMEM),    # 40: shares, little work in each pair
    (64 * 37, 24, 512 * 20 - 5, True, STAGED),   # 5: tiles of few and of many stations
    (64 * 37, 24, 512 * 160 - 5, True, TMEM),    # 40
])
def test_choice(cuda, bplib, oracle_lib, N, S, T, masked, want):
    import torch
    from beampower_b200.core import launch_count
    from beampower_b200.tables import TravelTimeTable
    if torch.cuda.get_device_properties(0).multi_processor_count != 148:
        pytest.skip("sizes are for 148 SMs")
    rng = np.random.default_rng(S + T)
    P = 2
    F = rng.standard_normal((S, 1, T)).astype(np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
    D = (rng.integers(0, 20, size=(1, S, P)) + rng.integers(0, 60, size=(N, S, P)))
    W = np.ones((N, S), np.float32)
    if masked:  # 18 of the 37 tiles, far from the others, use a third of the stations
        W[:64 * 18, S // 3:] = 0.0
        D[64 * 18:] += 300
    D = D.astype(np.int32)
    table = TravelTimeTable(D, W)
    traces = table.traces_from_features(F, A)
    before = launch_count()
    bm, am = table.beamform_max(traces, 0)
    assert launch_count() - before == want
    torch.cuda.synchronize()
    # the oracle on stretches of the record: its ends and a tile's edge
    U = oracle_lib.prestack(F, A)
    reach = int(D.max()) + 1
    for a in sorted({0, max(0, min(512 * 3 - 40, T - 600)), max(0, T - 600)}):
        b = min(T, a + 600)
        end = min(T, b + reach)
        want_bm, want_am = oracle_lib.beamform_max(np.ascontiguousarray(U[:, a:end]), D, W, 0)
        n = b - a if end < T or b < T else T - a
        assert np.array_equal(_bits(bm[a:a + n].cpu().numpy()), _bits(want_bm[:n]))
        assert np.array_equal(am[a:a + n].cpu().numpy(), want_am[:n])
    table.close()
