"""Batches on the tensor-memory kernel: the traces of all records are prepared in one
launch, however many there are, at the sizes where its blocks end; the oracle's
beams, bit for bit, with each new set of data."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

CONFIG = 9


@pytest.fixture
def forced(bplib):
    for storage in range(3):
        bplib.bp_set_kernel_config(storage, 1, CONFIG)
    yield
    for storage in range(3):
        bplib.bp_set_kernel_config(storage, 1, -1)


# a block prepares 1,024 FP32 samples of a row: lengths around one and two of them
LENGTHS = (1, 2, 15, 16, 17, 900, 960, 970, 1024, 1900, 1985, 2047, 3000)


@pytest.mark.parametrize("storage", ["fp32", "bf16"])
def test_records_of_unlike_lengths(cuda, bplib, oracle_lib, forced, storage):
    import torch
    from beampower_b200.batch import Window, WindowBatch
    from beampower_b200.core import launch_count
    from beampower_b200.tables import TravelTimeTable
    rng = np.random.default_rng(6)
    S, P = 4, 2
    D = rng.integers(-20, 40, size=(130, S, P)).astype(np.int32)
    W = np.ones((130, S), np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
    table = TravelTimeTable(D, W)
    batch = WindowBatch([table], [Window(0, T) for T in LENGTHS], A, storage=storage)
    counts = []
    for turn in range(2):
        F = [rng.standard_normal((S, 1, T)).astype(np.float32) for T in LENGTHS]
        for i, f in enumerate(F):
            batch.set_features(i, f)
        before = launch_count()
        out = batch.run()
        launches = launch_count() - before
        torch.cuda.synchronize()
        assert batch.status() == 0
        for f, (bm, am) in zip(F, out):
            if storage == "fp32":
                want = oracle_lib.beamform_max(oracle_lib.prestack(f, A), D, W, 0)
            else:  # the call for this window alone
                tr = table.traces_from_features(f, A, storage=storage)
                want = [x.cpu().numpy() for x in table.beamform_max(tr, 0)]
            assert np.array_equal(bm.cpu().numpy().view(np.uint32), want[0].view(np.uint32))
            assert np.array_equal(am.cpu().numpy(), want[1])
        counts.append(launches)
    batch.close()
    # each window's prestack, then planes, beams and decode of all
    few = WindowBatch([table], [Window(0, 900)], A, storage=storage)
    few.set_features(0, np.ones((S, 1, 900), np.float32))
    before = launch_count()
    few.run()
    one = launch_count() - before
    assert counts == [one + (one - 3) * (len(LENGTHS) - 1)] * 2
    few.close()
    table.close()


@pytest.mark.parametrize("P,width,tmem", [(2, 30, True), (2, 139, False), (3, 30, False)])
def test_choice(cuda, bplib, oracle_lib, P, width, tmem):
    """Tables of narrow and of wide mean windows, and of three phases."""
    import torch
    from beampower_b200.batch import Window, WindowBatch
    from beampower_b200.core import launch_count
    from beampower_b200.tables import TravelTimeTable
    rng = np.random.default_rng(P + width)
    S, T = 20, 512 * 20
    D = rng.integers(0, width, size=(64 * 40, S, P)).astype(np.int32)
    W = np.ones(D.shape[:2], np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
    F = rng.standard_normal((S, 1, T)).astype(np.float32)
    table = TravelTimeTable(D, W)
    batch = WindowBatch([table], [Window(0, T)], A, storage="fp32")
    batch.set_features(0, F)
    before = launch_count()
    (bm, am), = batch.run()
    assert launch_count() - before == (4 if tmem else 3)  # prestack, planes, beams, decode
    torch.cuda.synchronize()
    n = 600
    want = oracle_lib.beamform_max(oracle_lib.prestack(
        np.ascontiguousarray(F[:, :, :n + width]), A), D, W, 0)
    assert np.array_equal(bm[:n].cpu().numpy().view(np.uint32), want[0][:n].view(np.uint32))
    assert np.array_equal(am[:n].cpu().numpy(), want[1][:n])
    batch.close()
    table.close()
