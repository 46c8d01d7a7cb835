"""Run by tests/test_gpu_tmem_lost_fill.py in a child process whose
BEAMPOWER_B200_LIBRARY names the index-checked library, in which block 0 of the
tensor-memory kernel can be told to leave out one fill.  Prints LOST FILL OK."""
import ctypes as ct
import os
import sys
import time

import numpy as np

sys.path.insert(0, os.path.dirname(os.path.dirname(os.path.abspath(__file__))))

TILE = 512      # samples of a time tile
CONFIG = 9
LIMIT_S = 2.0   # of a wait
MORE_S = 1.5    # and for the kernel to end after it


def main():
    import torch
    import beampower_b200 as bp
    from beampower_b200.batch import Window, WindowBatch
    from beampower_b200.core import BeampowerError
    from beampower_b200.tables import TravelTimeTable, _stream_ptr
    lib = bp.load_library("gpu")
    assert lib._name.endswith("libbeampower_b200_checked.so"), lib._name
    lose = lib.bp_debug_lose_fill
    lose.argtypes, lose.restype = [ct.c_int], None
    S, P = 3, 2
    fills = S * P  # of a time tile

    def problem(N, T, seed):
        rng = np.random.default_rng(seed)
        F = rng.standard_normal((S, 1, T)).astype(np.float32)
        A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
        D = rng.integers(0, 30, size=(N, S, P)).astype(np.int32)
        return F, A, D, np.ones((N, S), np.float32)

    def lost(fill, call):
        """The call's outputs with that fill left out."""
        lose(fill)
        t0 = time.perf_counter()
        try:
            out = call()
            torch.cuda.synchronize()
        finally:
            lose(0)
        s = time.perf_counter() - t0
        assert LIMIT_S <= s <= LIMIT_S + MORE_S, s
        return out

    # (sources, samples, lost fill): a block per SM with one time tile each and
    # with two, then blocks of several time tiles; one table tile each, so that
    # block 0 alone has the first samples
    for storage in ("fp32", "fp16"):
        code = {"fp32": 0, "fp16": 2}[storage]
        for N, T, fill in ((64, 700, 4), (50, 500 * TILE, fills + 3),
                           (64, 4800 * TILE, fills + 1)):
            F, A, D, W = problem(N, T, T)
            table = TravelTimeTable(D, W)
            traces = table.traces_from_features(F, A, storage=storage)
            keys = torch.empty(T, dtype=torch.int64, device="cuda")
            scales = traces.scales.data_ptr() if storage != "fp32" else None

            def beam_max():
                bm = torch.full((T,), -7.0, device="cuda")
                am = torch.full((T,), -7, dtype=torch.int32, device="cuda")
                assert lib.bp_beamform_max_dev(
                    table.handle, traces.buf.data_ptr(), code, scales, T, traces.lpad,
                    traces.pitch, 1, keys.data_ptr(), bm.data_ptr(), am.data_ptr(),
                    _stream_ptr()) == 0, lib.bp_last_error()
                torch.cuda.synchronize()
                return bm.cpu().numpy(), am.cpu().numpy()

            for red in (0, 1):
                lib.bp_set_kernel_config(code, red, CONFIG)
                assert lib.bp_table_kernel_config(table.handle, code, red) == CONFIG
            want_bm, want_am = beam_max()
            bm, am = lost(fill, beam_max)
            first = (fill - 1) // fills * TILE  # the lost fill's time tile, block 0's last one
            end = first + int(np.argmin(np.append(bm[first:] == -7.0, False)))
            assert end > first and (end - first) % TILE == 0 or end == T, (first, end)
            keep = np.ones(T, bool)
            keep[first:end] = False
            assert np.array_equal(bm[keep], want_bm[keep])
            assert np.array_equal(am[keep], want_am[keep])
            assert (am[~keep] == 0).all()
            again = beam_max()
            assert np.array_equal(again[0], want_bm) and np.array_equal(again[1], want_am)
            if T < 1000 * TILE:  # the whole response
                want = table.beamform(traces, 1).cpu().numpy()
                out = torch.full((N, T), -7.0, device="cuda")
                part = lost(fill, lambda: table.beamform(traces, 1, out=out)).cpu().numpy()
                same = (part == want) | (part == -7.0)
                assert same.all() and (part[:, first:first + TILE] == -7.0).all()
                assert np.array_equal(part[:, :first], want[:, :first])
            table.close()
            for red in (0, 1):
                lib.bp_set_kernel_config(code, red, -1)

    lib.bp_set_kernel_config(0, 1, CONFIG)
    # a call that reads the kernel's status says so
    F, A, D, W = problem(64, 700, 1)
    try:
        lost(2, lambda: bp.beamform(F, D, A, W, reduce="max"))
        raise AssertionError("no error")
    except BeampowerError as e:
        assert "status 0x1" in str(e), e

    # the persistent batch
    F, A, D, W = problem(200, 3000, 2)
    table = TravelTimeTable(D, W)
    batch = WindowBatch([table], [Window(0, 3000), Window(0, 900)], A, storage="fp32")
    batch.set_features(0, F)
    batch.set_features(1, F[:, :, :900])
    want = [(b.cpu().numpy(), a.cpu().numpy()) for b, a in batch.run()]
    torch.cuda.synchronize()
    assert batch.status() == 0
    lost(3, batch.run)
    assert batch.status() == 1
    batch.close()
    batch = WindowBatch([table], [Window(0, 3000), Window(0, 900)], A, storage="fp32")
    batch.set_features(0, F)
    batch.set_features(1, F[:, :, :900])
    got = [(b.cpu().numpy(), a.cpu().numpy()) for b, a in batch.run()]
    assert batch.status() == 0
    for (b0, a0), (b1, a1) in zip(want, got):
        assert np.array_equal(b0, b1) and np.array_equal(a0, a1)
    batch.close()
    table.close()
    print("LOST FILL OK")


if __name__ == "__main__":
    main()
