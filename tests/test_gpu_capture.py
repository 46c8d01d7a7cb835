"""Plain calls in a CUDA graph: one on the tensor-memory kernel, whose planes are
allocated and given back inside the graph, and one of several launches; replayed on new
traces in the same buffers they give the oracle's beams."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("widths,T", [((30,), 8192), ((20, 3000), 62_000)])
def test_capture_and_replay(cuda, bplib, oracle_lib, widths, T):
    import torch
    from beampower_b200.tables import TravelTimeTable
    rng = np.random.default_rng(T)
    S, P = 4, 2
    D = np.concatenate([rng.integers(0, w, size=(4096, S, P)) for w in widths]).astype(np.int32)
    W = np.ones(D.shape[:2], np.float32)
    A = rng.uniform(0.2, 1.2, size=(S, 1, P)).astype(np.float32)
    table = TravelTimeTable(D, W)
    traces = table.traces_from_features(np.zeros((S, 1, T), np.float32), A)
    out = (torch.zeros(T, device="cuda"), torch.zeros(T, dtype=torch.int32, device="cuda"),
           torch.empty(T, dtype=torch.int64, device="cuda"))
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        table.beamform_max(traces, 1, stream=stream, out=out)  # warm-up outside the capture
    stream.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        table.beamform_max(traces, 1, stream=stream, out=out)
    n = 700
    for turn in range(3):
        F = rng.standard_normal((S, 1, T)).astype(np.float32)
        traces.buf.copy_(table.traces_from_features(F, A).buf)
        graph.replay()
        torch.cuda.synchronize()
        U = oracle_lib.prestack(F, A)[:, -n:]  # the end: no sample before it is read
        want_bm, want_am = oracle_lib.beamform_max(np.ascontiguousarray(U), D, W, 1)
        got = out[0][-n:].cpu().numpy()
        assert np.array_equal(got.view(np.uint32), want_bm.view(np.uint32)), turn
        assert np.array_equal(out[1][-n:].cpu().numpy(), want_am), turn
    graph.reset()
    table.close()
