"""A batch whose traces fit the GPU a second time (as planes for the tensor-memory
kernel) but not that and its keys: it runs without planes, as it does where there
is no memory for them at all."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("left_mb", [400, 280])  # planes 240 and keys 240; keys alone
def test_batch_without_memory_for_planes(cuda, bplib, monkeypatch, left_mb):
    import torch
    from beampower_b200 import batch as batch_module
    from beampower_b200.batch import Window, WindowBatch
    from beampower_b200.tables import TravelTimeTable
    rng = np.random.default_rng(2)
    S, P, N, T = 2, 1, 64, 30_000_000
    D = rng.integers(0, 20, size=(N, S, P)).astype(np.int32)
    table = TravelTimeTable(D, np.ones((N, S), np.float32))
    A = np.ones((S, 1, P), np.float32)
    held = []

    class Library:
        """Fills the device before the batch is made."""

        def __getattr__(self, name):
            return getattr(bplib, name)

        def bp_batch_create(self, *args):
            torch.cuda.synchronize()
            torch.cuda.empty_cache()
            free, _ = torch.cuda.mem_get_info()
            held.append(torch.empty(free - (left_mb << 20), dtype=torch.uint8, device="cuda"))
            return bplib.bp_batch_create(*args)

    monkeypatch.setattr(batch_module, "load_library", lambda device: Library())
    b = WindowBatch([table], [Window(0, T)], A, storage="fp32")
    assert held
    held.clear()
    torch.cuda.empty_cache()
    x = torch.randn((S, 1, T), device="cuda", generator=torch.Generator("cuda").manual_seed(1))
    b.set_features(0, x)
    (bm, am), = b.run()
    assert b.status() == 0
    tr = table.traces_from_features(x, A)
    want_bm, want_am = table.beamform_max(tr, 0)
    torch.cuda.synchronize()
    assert torch.equal(bm.view(torch.int32), want_bm.view(torch.int32))
    assert torch.equal(am, want_am)
    b.close()
    table.close()
