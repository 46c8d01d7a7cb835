"""The autotuner beside the built-in rule: a table that the rule runs as several
launches is timed that way too and keeps the rule when it is the fastest; cached
choices of earlier versions, and of tables for which the rule has another answer,
are not applied.  On the CPU with a fake library and fake times; one real table."""
import json

import numpy as np
import pytest

from beampower_b200 import autotune
from beampower_b200.core import REDUCE_MAX, STORAGE

FP32, FP16 = STORAGE["fp32"], STORAGE["fp16"]


class FakeLib:
    """Three shapes; the built-in rule reports `default` and runs as `parts`
    launches.  Times of the call: by choice, -1 the built-in rule's."""

    def __init__(self, default=2, parts=1, ms=None):
        self.choice, self.default, self.parts = -1, default, parts
        self.ms = ms or {-1: 1.0, 0: 3.0, 1: 2.0, 2: 4.0}
        self.count = 0

    def bp_get_kernel_config(self, storage, reduce):
        return self.choice

    def bp_set_kernel_config(self, storage, reduce, config):
        self.choice = config
        return 0

    def bp_table_kernel_config(self, handle, storage, reduce):
        return self.default if self.choice < 0 else self.choice

    def call(self):
        self.count += self.parts if self.choice < 0 else 1


class FakeTable:
    handle, n_stations, n_phases, info = None, 60, 2, {"max_spread": 300}

    def __init__(self, lib):
        self.lib = lib

    def beamform_max(self, traces, out_of_bounds):
        self.lib.call()


class FakeTraces:
    storage = FP32


@pytest.fixture
def setup(tmp_path, monkeypatch):
    path = tmp_path / "autotune.json"
    monkeypatch.setenv(autotune.CACHE_ENV, str(path))
    monkeypatch.setattr(autotune, "_gpu_key", lambda: "NVIDIA B200|148")
    monkeypatch.setattr(autotune, "configs", lambda: [(c, {}) for c in range(3)])

    def use(lib):
        monkeypatch.setattr(autotune, "load_library", lambda device: lib)
        monkeypatch.setattr(autotune, "launch_count", lambda: lib.count)
        monkeypatch.setattr(autotune, "_time_ms", lambda run, repeats: lib.ms[lib.choice])
        return FakeTable(lib)
    return path, use


@pytest.mark.parametrize("default_ms,best", [(1.0, -1), (2.5, 1)])
def test_several_launches_are_timed_too(setup, default_ms, best):
    path, use = setup
    lib = FakeLib(parts=2, ms={-1: default_ms, 0: 3.0, 1: 2.0, 2: 4.0})
    table = use(lib)
    res = autotune.autotune(table, FakeTraces())
    assert res["best"] == best and res["default_ms"] == default_ms and lib.choice == best
    assert set(res["times_ms"]) == {0, 1, 2}
    lib.choice = -1
    assert autotune.apply_cached(table, "fp32") == best and lib.choice == best


def test_one_launch_is_one_of_the_shapes(setup):
    path, use = setup
    lib = FakeLib(parts=1)  # its time (1.0) would win if it were taken
    res = autotune.autotune(use(lib), FakeTraces())
    assert res["best"] == 1 and res["default_ms"] is None and lib.choice == 1


def test_cache_of_an_earlier_version_is_not_applied(setup):
    path, use = setup
    lib = FakeLib(default=9)
    table = use(lib)
    key = autotune._problem_key(table, FP32, "max")
    path.write_text(json.dumps({key: {"config": 8, "ms": {str(c): 1.0 + c for c in range(9)}}}))
    assert autotune.apply_cached(table, "fp32") is None
    assert autotune.apply_cached(None, "fp32") is None
    assert lib.choice == -1


def test_choice_of_a_table_with_another_default_is_not_applied(setup):
    path, use = setup
    narrow = use(FakeLib(default=2))
    assert autotune.autotune(narrow, FakeTraces())["best"] == 1
    wide = use(FakeLib(default=0))  # same stations, phases and widest window
    assert autotune.apply_cached(wide, "fp32") is None and wide.lib.choice == -1
    narrow = use(FakeLib(default=2))
    narrow.lib.choice = 0
    assert autotune.apply_cached(narrow, "fp32") == 1 and narrow.lib.choice == 1


@pytest.mark.gpu
def test_table_of_several_launches(cuda, bplib, tmp_path, monkeypatch):
    from beampower_b200.tables import TravelTimeTable
    monkeypatch.setenv(autotune.CACHE_ENV, str(tmp_path / "cache.json"))
    rng = np.random.default_rng(3)
    S, P, T = 2, 2, 62_000
    D = np.concatenate([rng.integers(0, w, size=(4096, S, P)) for w in (20, 3000)])
    table = TravelTimeTable(D.astype(np.int32), np.ones((len(D), S), np.float32))
    traces = table.traces_from_features(
        rng.standard_normal((S, 1, T)).astype(np.float32), np.ones((S, 1, P), np.float32))
    try:
        res = autotune.autotune(table, traces, repeats=1)
        ran = {c: t for c, t in res["times_ms"].items() if t is not None}
        ran[-1] = res["default_ms"]
        assert res["best"] == min(ran, key=ran.get)
        bplib.bp_set_kernel_config(FP32, REDUCE_MAX, -1)
        assert autotune.apply_cached(table, "fp32") == res["best"]
    finally:
        bplib.bp_set_kernel_config(FP32, REDUCE_MAX, -1)
        table.close()
