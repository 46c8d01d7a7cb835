"""Tables whose tiles may run as several launches, in the order of their widths:
creating one takes the launches of any other table, it can be used at once on any
stream, and a launch over some of its tiles takes those."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _bits(a):
    a = np.ascontiguousarray(a, dtype=np.float32).copy()
    a[np.isnan(a)] = np.float32(np.nan)
    return a.view(np.uint32)


def _delays(widths, S, P, seed, per=1024):
    rng = np.random.default_rng(seed)
    D = np.concatenate([rng.integers(0, w + 1, size=(per, S, P)) for w in widths])
    return D[rng.permutation(len(D))].astype(np.int32)


@pytest.mark.parametrize("P", [1, 2, 3])
def test_creation_takes_no_second_build(cuda, bplib, P):
    from beampower_b200.core import launch_count
    from beampower_b200.tables import TravelTimeTable
    counts = []
    for widths in ((20, 20), (20, 3000)):  # all in tensor memory, half beyond it
        D = _delays(widths, 4, P, 1)
        before = launch_count()
        table = TravelTimeTable(D, np.ones(D.shape[:2], np.float32))
        counts.append(launch_count() - before)
        table.close()
    assert counts[0] == counts[1]


@pytest.mark.parametrize("widths", [(20, 3000), (3000, 20, 700)])
def test_used_at_once_on_another_stream(cuda, bplib, oracle_lib, widths):
    import torch
    from beampower_b200.core import launch_count
    from beampower_b200.tables import TravelTimeTable
    S, P, T = 3, 2, 300_000  # 586 time tiles of 9 or more narrow tiles: two launches
    rng = np.random.default_rng(len(widths))
    F = rng.standard_normal((S, 1, T)).astype(np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
    U = oracle_lib.prestack(F, A)
    made, used = torch.cuda.Stream(), torch.cuda.Stream()
    D = _delays(widths, S, P, 5)
    W = np.ones(D.shape[:2], np.float32)
    want = oracle_lib.beamform_max(U, D, W, 0)
    d, w = torch.from_numpy(D).cuda(), torch.from_numpy(W).cuda()
    probe = TravelTimeTable(d, w)
    traces = probe.traces_from_features(F, A)  # the layout of every table of these delays
    torch.cuda.synchronize()
    for _ in range(5):
        table = TravelTimeTable(d, w, stream=made)
        before = launch_count()
        with torch.cuda.stream(used):
            bm, am = table.beamform_max(traces, 0, stream=used)
        assert launch_count() - before >= 4  # planes, two beam launches, decode
        used.synchronize()
        assert np.array_equal(_bits(bm.cpu().numpy()), _bits(want[0]))
        assert np.array_equal(am.cpu().numpy(), want[1])
        table.close()
    probe.close()


def test_direct_table_used_at_once_on_another_stream(cuda, bplib, oracle_lib):
    """Five phases: the direct kernel, over the table's copies of the delays."""
    import torch
    from beampower_b200.tables import TravelTimeTable
    S, P, N, T = 20, 5, 40_000, 600
    rng = np.random.default_rng(7)
    D = rng.integers(0, 200, size=(N, S, P)).astype(np.int32)
    W = np.ones((N, S), np.float32)
    F = rng.standard_normal((S, 1, T)).astype(np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
    want = oracle_lib.beamform_max(oracle_lib.prestack(F, A), D, W, 1)
    d, w = torch.from_numpy(D).cuda(), torch.from_numpy(W).cuda()
    probe = TravelTimeTable(d, w)
    assert probe.info["uses_window_kernel"] == 0
    traces = probe.traces_from_features(F, A)
    made, used = torch.cuda.Stream(), torch.cuda.Stream()
    torch.cuda.synchronize()
    for _ in range(5):
        table = TravelTimeTable(d, w, stream=made)
        with torch.cuda.stream(used):
            bm, am = table.beamform_max(traces, 1, stream=used)
        used.synchronize()
        assert np.array_equal(_bits(bm.cpu().numpy()), _bits(want[0]))
        assert np.array_equal(am.cpu().numpy(), want[1])
        table.close()
    probe.close()
