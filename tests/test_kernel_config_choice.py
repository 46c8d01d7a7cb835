"""What bp_get_kernel_config answers when nothing has been chosen: setting the
answer again leaves the built-in choice as it is.  A caller that saves the answer,
tries configs and restores it (the autotuner) leaves no choice behind."""
import pytest


@pytest.fixture
def lib():
    from beampower_b200.core import load_library
    lib = load_library("gpu")
    yield lib
    for storage in range(3):
        for reduce in (0, 1):
            lib.bp_set_kernel_config(storage, reduce, -1)


@pytest.mark.parametrize("reduce", [0, 1])
@pytest.mark.parametrize("storage,default", [(0, -1), (1, 2), (2, 2)])
def test_answer_without_a_choice(lib, monkeypatch, storage, reduce, default):
    monkeypatch.delenv("BEAMPOWER_B200_KERNEL_CONFIG", raising=False)
    assert lib.bp_get_kernel_config(storage, reduce) == default
    assert lib.bp_set_kernel_config(storage, reduce, default) == 0
    assert lib.bp_get_kernel_config(storage, reduce) == default
    assert lib.bp_set_kernel_config(storage, reduce, 5) == 0
    assert lib.bp_get_kernel_config(storage, reduce) == 5
    assert lib.bp_set_kernel_config(storage, reduce, -1) == 0
    assert lib.bp_get_kernel_config(storage, reduce) == default


@pytest.mark.gpu
@pytest.mark.parametrize("storage", ["fp16", "bf16"])
def test_autotune_of_a_table_without_a_shape_leaves_no_choice(cuda, lib, tmp_path, monkeypatch,
                                                              storage):
    """Delay windows that no 16-bit shape holds: the autotuner finds nothing, and
    the next tables run with what they ran before."""
    import numpy as np
    from beampower_b200 import autotune
    from beampower_b200.core import STORAGE
    from beampower_b200.tables import TravelTimeTable
    monkeypatch.setenv(autotune.CACHE_ENV, str(tmp_path / "cache.json"))
    rng = np.random.default_rng(8)
    S, P = 6, 2
    ones = np.ones((300, S), np.float32)
    tables = [TravelTimeTable(rng.integers(0, w, size=(300, S, P)).astype(np.int32), ones)
              for w in (40, 700, 4500)]
    before = [lib.bp_table_kernel_config(t.handle, STORAGE[storage], 1) for t in tables]
    assert before[0] >= 0 and before[1] >= 0 and before[2] == -1
    traces = tables[2].traces_from_features(np.ones((S, 1, 3000), np.float32),
                                            np.ones((S, 1, P), np.float32), storage=storage)
    assert autotune.autotune(tables[2], traces, repeats=1)["best"] is None
    assert [lib.bp_table_kernel_config(t.handle, STORAGE[storage], 1)
            for t in tables] == before
    for t in tables:
        t.close()


@pytest.mark.gpu
def test_restoring_the_answer_keeps_each_table_s_default(cuda, lib):
    """FP32: the default depends on the table, narrow and wide ones."""
    import numpy as np
    from beampower_b200.tables import TravelTimeTable
    rng = np.random.default_rng(9)
    ones = np.ones((300, 6), np.float32)
    tables = [TravelTimeTable(rng.integers(0, w, size=(300, 6, 2)).astype(np.int32), ones)
              for w in (40, 240, 3000)]
    for reduce in (0, 1):
        before = [lib.bp_table_kernel_config(t.handle, 0, reduce) for t in tables]
        assert len(set(before)) > 1
        prev = lib.bp_get_kernel_config(0, reduce)
        lib.bp_set_kernel_config(0, reduce, 3)
        lib.bp_set_kernel_config(0, reduce, prev)
        assert [lib.bp_table_kernel_config(t.handle, 0, reduce) for t in tables] == before
    for t in tables:
        t.close()
