"""The tensor-memory kernel (kernel config 9) against the oracle, bit for bit,
at the sizes where it can go wrong: time tiles of 512 samples, 64-source tiles
cut into groups of 4, delay windows around the widths at which TMEM holds 4, 2
or 1 fills and around its 512 columns (beyond them another shape runs), window
starts at every offset from a 16-sample boundary, weights of each kind."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CONFIG = 9


def _bits(a):
    a = np.ascontiguousarray(a, dtype=np.float32).copy()
    a[np.isnan(a)] = np.float32(np.nan)
    return a.view(np.uint32)


def _problem(N, S, P, T, span, weights, seed, shift=0):
    rng = np.random.default_rng(seed)
    F = rng.standard_normal((S, 2, T)).astype(np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 2, P)).astype(np.float32)
    base = rng.integers(0, 90, size=(1, S, P)) + shift
    D = (base + rng.integers(0, span + 1, size=(N, S, P))).astype(np.int32)
    W = np.ones((N, S), np.float32)
    if weights != "ones":
        # whole groups without a station, and single sources without it
        W[np.repeat(rng.random(((N + 3) // 4, S)) < 0.3, 4, axis=0)[:N]] = 0.0
        W[rng.random((N, S)) < 0.1] = 0.0
    if weights == "real":
        W *= rng.uniform(0.5, 1.5, size=(N, S)).astype(np.float32)
    return F, A, D, W


def _check(lib, oracle_lib, F, A, D, W, must_run=True):
    import torch
    from beampower_b200.tables import TravelTimeTable
    U = oracle_lib.prestack(F, A)
    table = TravelTimeTable(D, W)
    traces = table.traces_from_features(F, A)
    for red in (0, 1):
        lib.bp_set_kernel_config(0, red, CONFIG)
    try:
        for red in (0, 1):
            assert (lib.bp_table_kernel_config(table.handle, 0, red) == CONFIG) == must_run
        for oob in (0, 1):
            bm, am = table.beamform_max(traces, oob)
            beam = table.beamform(traces, oob)
            torch.cuda.synchronize()
            want_bm, want_am = oracle_lib.beamform_max(U, D, W, oob)
            assert np.array_equal(_bits(bm.cpu().numpy()), _bits(want_bm)), oob
            assert np.array_equal(am.cpu().numpy(), want_am), oob
            want = oracle_lib.beamform(U, D, W, oob)
            assert np.array_equal(_bits(beam.cpu().numpy()), _bits(want)), oob
    finally:
        for red in (0, 1):
            lib.bp_set_kernel_config(0, red, -1)
        table.close()


@pytest.mark.parametrize("weights", ["ones", "zero_one", "real"])
@pytest.mark.parametrize("N,T", [(1, 1), (3, 511), (64, 512), (65, 513), (130, 1537), (257, 2048)])
def test_tile_edges(cuda, bplib, oracle_lib, N, T, weights):
    _check(bplib, oracle_lib, *_problem(N, 7, 2, T, 40, weights, N + T))


@pytest.mark.parametrize("P", [1, 2, 3, 4])
@pytest.mark.parametrize("span", [0, 104, 105, 120, 232, 240, 300, 470])
def test_window_widths(cuda, bplib, oracle_lib, P, span):
    """Spans on both sides of 4, 2 and 1 fills per TMEM."""
    _check(bplib, oracle_lib, *_problem(70, 5, P, 1100, span, "zero_one", span + P))


def test_window_beyond_tensor_memory(cuda, bplib, oracle_lib):
    _check(bplib, oracle_lib, *_problem(70, 5, 2, 1100, 600, "ones", 5), must_run=False)


@pytest.mark.parametrize("shift", list(range(-33, -16)) + [-400, 5000])
def test_window_starts(cuda, bplib, oracle_lib, shift):
    """Negative delays move the traces' left padding; delays beyond the record
    leave no valid sample under the strict rule."""
    _check(bplib, oracle_lib, *_problem(66, 4, 2, 700, 50, "real", 11, shift))


def test_nan_infinite_and_lowest_values(cuda, bplib, oracle_lib):
    """NaN and infinite traces, beams at the lowest float: never candidates."""
    F, A, D, W = _problem(80, 6, 2, 900, 60, "zero_one", 3)
    F[0, 0, 100:110] = np.nan
    F[1, 0, 300] = np.inf
    F[2, 0, 305] = -np.inf
    F[3, :, 500:560] = np.float32(-3.4e38)
    _check(bplib, oracle_lib, F, A, D, W)


def test_ties_keep_the_lowest_source(cuda, bplib, oracle_lib):
    F, A, D, W = _problem(200, 5, 2, 1024, 30, "ones", 9)
    D[:] = D[:1]
    _check(bplib, oracle_lib, F, A, D, W)


def test_no_station_used(cuda, bplib, oracle_lib):
    F, A, D, W = _problem(70, 5, 2, 600, 30, "ones", 1)
    W[:] = 0.0
    _check(bplib, oracle_lib, F, A, D, W)


@pytest.mark.parametrize("weights", ["zero_one", "real"])
def test_batch_and_records(cuda, bplib, oracle_lib, weights):
    """Two tables of unlike widths, station subsets and lengths in one
    persistent launch; a record with its own time origin and output range is
    what a stream runs."""
    import torch
    from beampower_b200.batch import Window, WindowBatch
    from beampower_b200.stream import NetworkStream
    from beampower_b200.tables import TravelTimeTable
    F, A, D, W = _problem(150, 9, 2, 2100, 70, weights, 21)
    D2 = (D[:90] // 3).astype(np.int32)
    t1, t2 = TravelTimeTable(D, W), TravelTimeTable(D2, W[:90])
    bplib.bp_set_kernel_config(0, 1, CONFIG)
    try:
        windows = [Window(0, 2100), Window(1, 700, stations=[0, 2, 5, 8]),
                   Window(0, 513, stations=range(1, 9, 2), out_of_bounds="flexible")]
        batch = WindowBatch([t1, t2], windows, A, storage="fp32")
        for i, w in enumerate(windows):
            batch.set_features(i, F[:, :, :w.n_samples])
        out = batch.run()
        torch.cuda.synchronize()
        assert batch.status() == 0
        for w, (bm, am) in zip(windows, out):
            Dw, Ww = (D, W) if w.table == 0 else (D2, W[:90])
            Ww = Ww.copy()
            if w.stations is not None:
                Ww[:, [s for s in range(9) if s not in set(w.stations)]] = 0.0
            U = oracle_lib.prestack(np.ascontiguousarray(F[:, :, :w.n_samples]), A)
            want_bm, want_am = oracle_lib.beamform_max(
                U, Dw, Ww, 0 if w.out_of_bounds == "strict" else 1)
            assert np.array_equal(_bits(bm.cpu().numpy()), _bits(want_bm))
            assert np.array_equal(am.cpu().numpy(), want_am)
        batch.close()
        net = NetworkStream(t1, A, storage="fp32")
        for a in range(0, 2100, 617):
            net.push(F[:, :, a:a + 617])
        net.flush()
        bm, am = net.collect()
        want_bm, want_am = oracle_lib.beamform_max(oracle_lib.prestack(F, A), D, W, 0)
        assert np.array_equal(_bits(bm), _bits(want_bm))
        assert np.array_equal(am, want_am)
    finally:
        bplib.bp_set_kernel_config(0, 1, -1)
    t1.close()
    t2.close()
