"""Performance cases: the work that users of beampower_b200 have it do, each
through a public entry point, over the range of sizes and options in use.

A case is a dict of plain values with a "kind":

  resident   the repeated call of a monitoring program: a resident
             ``TravelTimeTable`` and traces, ``table.beamform_max`` or
             ``table.beamform`` (the whole response)
  call       the one-off call on device tensors: ``beampower_b200.beamform``
             builds the table, prestacks and beamforms
  host       the same call from NumPy arrays, as reference users make it
  batch      ``WindowBatch.run``: many detection windows in one launch
  features   ``features.waveform_features``: the envelope of every trace
  threshold  ``detection.time_dependent_threshold`` of a beam series
  detect     ``detection.detect``: the events of a beam series
  pipeline   ``pipeline.detect_events``: raw waveforms to events

Networks follow ``beampower_b200.synthetic``: stations at random places in a
square, a regular grid of sources below it, delays from straight rays.
"""
import math

import numpy as np
import torch

import beampower_b200 as bp
from beampower_b200 import detection, features, pipeline
from beampower_b200.batch import Window, WindowBatch
from beampower_b200.tables import TravelTimeTable

V_P, V_S = 6.0, 3.46
DEV = "cuda"


def listed():
    return [
        # A small local network, called for every new minute of data: the
        # smallest resident call, where latency counts.
        dict(name="resident small fp32", kind="resident", nx=20, ny=20, nz=10, stations=20,
             square_km=50.0, depth_km=20.0, fs=25.0, samples=6000, phases=2, reduce="max",
             oob="strict", storage="fp32", max_km=0.0, weights="unit"),
        # The headline: a dense grid under a regional network, one hour at 50 Hz.
        dict(name="resident large fp32", kind="resident", nx=100, ny=100, nz=40, stations=60,
             square_km=150.0, depth_km=40.0, fs=50.0, samples=180000, phases=2, reduce="max",
             oob="strict", storage="fp32", max_km=100.0, weights="unit"),
        # The batch workload's smaller grid with half-size traces.
        dict(name="resident mid fp16", kind="resident", nx=50, ny=50, nz=20, stations=100,
             square_km=150.0, depth_km=20.0, fs=50.0, samples=45000, phases=2, reduce="max",
             oob="strict", storage="fp16", max_km=0.0, weights="unit"),
        # Wide delay windows (20 km between sources, 100 Hz), stations weighted
        # by their quality, partial sums at the record's ends.
        dict(name="resident regional weighted", kind="resident", nx=40, ny=40, nz=10, stations=60,
             square_km=800.0, depth_km=40.0, fs=100.0, samples=60007, phases=2, reduce="max",
             oob="flexible", storage="fp32", max_km=0.0, weights="real"),
        # The whole network response of a sub-grid, kept for plots and statistics.
        dict(name="resident whole response", kind="resident", nx=40, ny=25, nz=10, stations=60,
             square_km=75.0, depth_km=40.0, fs=50.0, samples=18000, phases=2, reduce="none",
             oob="strict", storage="fp32", max_km=100.0, weights="unit"),
        # A new network geometry on every call (a moving sub-grid): device
        # tensors in, odd sizes; the table build is part of the call.
        dict(name="call mid", kind="call", nx=53, ny=47, nz=21, stations=37, square_km=120.0,
             depth_km=30.0, fs=50.0, samples=15001, phases=2, oob="strict", storage="fp32",
             max_km=80.0, weights="unit"),
        # The reference's own usage: NumPy arrays in and out, tutorial scale.
        dict(name="host small", kind="host", nx=20, ny=20, nz=10, stations=20, square_km=50.0,
             depth_km=20.0, fs=25.0, samples=6000, phases=2, oob="strict", storage="fp32",
             max_km=0.0, weights="unit"),
        # Re-locating a list of triggered windows of 1 to 15 minutes, each
        # with its own stations; the class's default storage.
        dict(name="batch", kind="batch", nx=50, ny=50, nz=20, stations=100, square_km=150.0,
             depth_km=20.0, fs=50.0, windows=12, shortest=3000, longest=45000, storage="fp16"),
        # One hour of a regional network's traces made into features.
        dict(name="features", kind="features", stations=60, samples=180000),
        # The detection threshold of a day of beam values at 25 Hz.
        dict(name="threshold", kind="threshold", samples=2160000, window=180000,
             threshold_type="rms", zeros=2864),
        # The events of the same day, one minute apart.
        dict(name="detect", kind="detect", samples=2160000, distance=1500, zeros=2864),
        # The tutorial from raw traces to events on its network's grid
        # (32 x 16 x 25 sources, 8 stations, 25 Hz), four hours of it.
        dict(name="pipeline", kind="pipeline", nx=25, ny=16, nz=32, stations=8, square_km=60.0,
             depth_km=30.0, fs=25.0, samples=360000, phases=2, storage="fp32",
             window_s=1800.0, apart_s=60.0),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["resident", "resident", "resident", "call", "host", "batch", "features",
                       "threshold", "detect", "pipeline"])
    if kind == "features":
        return dict(kind=kind, stations=_log(rng, 3, 60), samples=_log(rng, 6000, 180000))
    if kind == "threshold":
        n = _log(rng, 20000, 2160000)
        return dict(kind=kind, samples=n, window=_log(rng, 500, n // 8),
                    threshold_type=rng.choice(["rms", "rms", "mad"]),
                    zeros=rng.randrange(0, 3000))
    if kind == "detect":
        return dict(kind=kind, samples=_log(rng, 20000, 2160000), distance=_log(rng, 50, 3000),
                    zeros=rng.randrange(0, 3000))
    if kind == "batch":
        return dict(kind=kind, nx=rng.randint(20, 50), ny=rng.randint(20, 50),
                    nz=rng.randint(8, 20), stations=rng.randint(30, 100), square_km=150.0,
                    depth_km=20.0, fs=50.0,
                    windows=rng.randint(2, 12), shortest=_log(rng, 1000, 3000),
                    longest=_log(rng, 6000, 45000), storage=rng.choice(["fp16", "fp16", "fp32"]))
    if kind == "pipeline":
        return dict(kind=kind, nx=rng.randint(12, 25), ny=rng.randint(12, 20),
                    nz=rng.randint(8, 32), stations=rng.randint(6, 20),
                    square_km=rng.choice([50.0, 60.0, 80.0]),
                    depth_km=30.0, fs=25.0, samples=_log(rng, 30000, 360000), phases=2,
                    storage="fp32", window_s=rng.choice([120.0, 300.0, 600.0]),
                    apart_s=rng.choice([10.0, 30.0, 60.0]))
    case = dict(kind=kind, stations=rng.randint(8, 60),
                square_km=rng.choice([50.0, 100.0, 150.0]), depth_km=rng.choice([20.0, 40.0]),
                fs=rng.choice([25.0, 50.0, 100.0]), phases=rng.choice([2, 2, 2, 1, 3]),
                oob=rng.choice(["strict", "strict", "flexible"]),
                max_km=rng.choice([0.0, 100.0]),
                weights=rng.choice(["unit", "unit", "real"]))
    if kind == "resident":
        case["reduce"] = rng.choice(["max", "max", "max", "none"])
        case["storage"] = rng.choice(["fp32", "fp32", "fp32", "fp16", "bf16"])
        whole = case["reduce"] == "none"
        n = _log(rng, 1000, 10000 if whole else 100000)
        case["samples"] = _log(rng, 1500, 20000 if whole else 90000)
        if case["fs"] == 100.0 and rng.random() < 0.3:
            case["square_km"] = 800.0
    else:
        case["storage"] = rng.choice(["fp32", "fp32", "fp32", "fp16"])
        n = _log(rng, 1000, 50000 if kind == "call" else 10000)
        case["samples"] = _log(rng, 3000, 20000 if kind == "call" else 12000)
    nz = rng.randint(6, 20)
    nx = max(5, int(math.sqrt(n / nz) * rng.uniform(0.8, 1.25)))
    case.update(nx=nx, ny=max(5, round(n / nz / nx)), nz=nz)
    return case


# ---- inputs --------------------------------------------------------------------
def _generator(seed):
    return torch.Generator(device=DEV).manual_seed(int(seed) + 7919)


def _network(case, g):
    """Travel times in seconds (N, S, P) and station weights (N, S)."""
    nx, ny, nz = case["nx"], case["ny"], case["nz"]
    S, side, P = case["stations"], case["square_km"], case.get("phases", 2)
    sta = torch.rand((S, 2), generator=g, device=DEV, dtype=torch.float64) * side
    ax = [torch.linspace(0.0, m, n, device=DEV, dtype=torch.float64)
          for m, n in ((case["depth_km"], nz), (side, ny), (side, nx))]
    z, y, x = (v.reshape(-1) for v in torch.meshgrid(*ax, indexing="ij"))
    speeds = [V_P, V_S, 3.0][:P]
    times = torch.empty((x.numel(), S, P), device=DEV)
    weights = torch.ones((x.numel(), S), device=DEV)
    for s in range(S):
        epi2 = (x - sta[s, 0]) ** 2 + (y - sta[s, 1]) ** 2
        dist = torch.sqrt(epi2 + z * z)
        for p, v in enumerate(speeds):
            times[:, s, p] = (dist / v).float()
        if case.get("max_km"):
            weights[:, s] = (epi2 <= case["max_km"] ** 2).float()
    if case.get("weights") == "real":
        quality = torch.rand(S, generator=g, device=DEV) * 0.8 + 0.4
        weights *= quality
    return times, weights


def _delays(times, fs):
    d = torch.round(times.double() * fs).to(torch.int32)
    return d - d[:, :, 0].amin(dim=1)[:, None, None]


def _phase_weights(S, P):
    """Vertical channel to the first phase, the horizontal ones to the others."""
    a = torch.zeros((S, 3, P), device=DEV)
    a[:, 0, 0] = 1.0
    if P == 1:
        a[:, :, 0] = 1.0
    else:
        a[:, 1:, 1:] = 1.0
    return a


def _noise_features(S, T, g):
    """|noise| smoothed over 25 samples, as the synthetic workloads'."""
    x = torch.randn((S * 3, 1, T + 24), generator=g, device=DEV).abs_()
    return torch.nn.functional.avg_pool1d(x, 25, 1).reshape(S, 3, T)


def _add_events(f, delays, alpha, g, n_events):
    """Gaussian pulses at the arrivals of a few random sources."""
    S, C, T = f.shape
    taps = torch.arange(-30, 31, device=DEV)
    pulse = 5.0 * torch.exp(-0.5 * (taps / 5.0) ** 2)
    for _ in range(n_events):
        src = int(torch.randint(0, delays.shape[0], (1,), generator=g, device=DEV))
        t0 = int(torch.randint(0, max(1, T), (1,), generator=g, device=DEV))
        for p in range(delays.shape[2]):
            t = t0 + delays[src, :, p].long()[:, None] + taps[None, :]
            ok = (t >= 0) & (t < T)
            add = torch.zeros((S, T), device=DEV)
            add.scatter_add_(1, t.clamp(0, T - 1), torch.where(ok, pulse[None, :], 0.0))
            f += alpha[:, :, p, None] * add[:, None, :]
    return f


def _series(case, g):
    """A beam series: the level of a stack's maximum, slow changes, events
    well apart, zeros where no source had a valid beam."""
    n = case["samples"]
    x = torch.randn((1, 1, n + 24), generator=g, device=DEV).abs_()
    x = torch.nn.functional.avg_pool1d(x, 25, 1).reshape(n)
    t = torch.arange(n, device=DEV, dtype=torch.float32)
    x = x * (1.0 + 0.2 * torch.sin(t * (6.2831853 / (n / 3.0))))
    live = n - case["zeros"]
    slot = min(live // 2, max(10000, 4 * case.get("distance", 0)))
    at = torch.arange(live // slot, device=DEV)[:, None] * slot + slot // 4
    at = at + torch.randint(0, slot // 2, at.shape, generator=g, device=DEV)
    taps = torch.arange(-30, 31, device=DEV)
    tall = 3.0 + 4.0 * torch.rand(at.shape, generator=g, device=DEV)
    bump = tall * torch.exp(-0.5 * (taps / 5.0) ** 2)
    x.scatter_reduce_(0, (at + taps).reshape(-1), bump.reshape(-1), "amax")
    if case["zeros"]:
        x[live:] = 0.0
    return x.contiguous()


def _inputs(case, seed):
    """(features, delays, phase weights, source weights) of the beam kinds."""
    g = _generator(seed)
    times, weights = _network(case, g)
    delays = _delays(times, case["fs"])
    del times
    alpha = _phase_weights(case["stations"], case.get("phases", 2))
    f = _noise_features(case["stations"], case["samples"], g)
    return _add_events(f, delays, alpha, g, 3), delays, alpha, weights


def _batch_inputs(case, seed):
    """(delays, source weights, stations of each window, features of each window)."""
    g = _generator(seed)
    times, weights = _network(case, g)
    pick = np.random.default_rng(seed)
    S = case["stations"]
    stations, records = [], []
    for n in _window_samples(case):
        some = np.sort(pick.permutation(S)[:int(pick.integers(S // 5, S * 4 // 5 + 1))])
        stations.append([int(s) for s in some])
        records.append(_noise_features(S, int(n), g))
    return _delays(times, case["fs"]), weights, stations, records


def prepare(case, seed):
    kind = case["kind"]
    g = _generator(seed)
    if kind == "resident":
        f, delays, alpha, weights = _inputs(case, seed)
        table = TravelTimeTable(delays, weights)
        traces = table.traces_from_features(f, alpha, storage=case["storage"])
        return dict(case=case, table=table, traces=traces)
    if kind == "call":
        return dict(case=case, args=_inputs(case, seed))
    if kind == "host":
        return dict(case=case, args=[v.cpu().numpy() for v in _inputs(case, seed)])
    if kind == "batch":
        delays, weights, stations, records = _batch_inputs(case, seed)
        table = TravelTimeTable(delays, weights)
        windows = [Window(0, f.shape[2], some) for some, f in zip(stations, records)]
        batch = WindowBatch([table], windows, _phase_weights(case["stations"], 2),
                            storage=case["storage"])
        for k, f in enumerate(records):
            batch.set_features(k, f)
        batch.capture()
        return dict(case=case, batch=batch)
    if kind == "features":
        x = torch.randn((case["stations"], 3, case["samples"]), generator=g, device=DEV)
        loud = torch.rand((case["stations"], 3, case["samples"] // 600 + 1), generator=g,
                          device=DEV) ** 4
        x *= 0.2 + loud.repeat_interleave(600, dim=2)[:, :, :case["samples"]]
        return dict(case=case, x=x)
    if kind in ("threshold", "detect"):
        x = _series(case, g)
        if kind == "threshold":
            noise = torch.randn(max(case["zeros"], 1), generator=g, device=DEV)
            return dict(case=case, x=x, noise=noise)
        source = torch.randint(0, 100000, x.shape, generator=g, device=DEV, dtype=torch.int32)
        thr = 2.2 + 0.1 * torch.sin(torch.arange(x.numel(), device=DEV) * 1.0e-5)
        return dict(case=case, x=x, source=source, thr=thr)
    times, weights = _network(case, g)
    delays = _delays(times, case["fs"])
    alpha = _phase_weights(case["stations"], case["phases"])
    f = torch.zeros((case["stations"], 3, case["samples"]), device=DEV)
    f = _add_events(f, delays, alpha, g, 12)
    raw = torch.randn(f.shape, generator=g, device=DEV) * (1.0 + f)
    table = TravelTimeTable.from_travel_times(times, case["fs"], weights)
    return dict(case=case, raw=raw, times=times, alpha=alpha, weights=weights, table=table)


# ---- one pass --------------------------------------------------------------------
def run(state):
    case = state["case"]
    kind = case["kind"]
    if kind == "resident":
        oob = 1 if case["oob"] == "flexible" else 0
        if case["reduce"] == "max":
            return state["table"].beamform_max(state["traces"], oob)
        return state["table"].beamform(state["traces"], oob)
    if kind in ("call", "host"):
        f, delays, alpha, weights = state["args"]
        return bp.beamform(f, delays, alpha, weights, device="gpu", reduce="max",
                           out_of_bounds=case["oob"], storage=case["storage"])
    if kind == "batch":
        return state["batch"].run()
    if kind == "features":
        return features.waveform_features(state["x"])
    if kind == "threshold":
        return detection.time_dependent_threshold(
            state["x"], case["window"], threshold_type=case["threshold_type"], num_dev=8.0,
            white_noise=state["noise"])
    if kind == "detect":
        d = detection.detect(state["x"], state["source"], threshold=state["thr"],
                             distance=case["distance"])
        return d.peaks, d.heights, d.sources
    e = pipeline.detect_events(state["raw"], state["times"], case["fs"], state["alpha"],
                               state["weights"], window_duration_sec=case["window_s"],
                               num_dev=4.0, min_detection_interval_sec=case["apart_s"],
                               storage=case["storage"], table=state["table"])
    # the catalogue as series, as a plot over the beam takes it
    heights, sources = torch.zeros_like(e.beam_max), torch.full_like(e.beam_argmax, -1)
    heights[e.peaks], sources[e.peaks] = e.heights, e.sources.to(torch.int32)
    return heights, sources, e.beam_max, e.beam_argmax, e.threshold


def _sources(case):
    return case["nx"] * case["ny"] * case["nz"]


def _window_samples(case):
    return np.geomspace(case["shortest"], case["longest"], case["windows"]).astype(int)


def work(case):
    """Bytes: each input once, each output once.  Operations: one multiply and
    one add per beam term of the weighted stations, five per sample and
    transform level of an FFT, two per sample of a series."""
    kind = case["kind"]
    if kind == "features":
        rows, n = 3 * case["stations"], case["samples"]
        return {"bytes": 8 * rows * n, "flops": rows * n * (10 * math.log2(n) + 8)}
    if kind == "threshold":
        return {"bytes": 8 * case["samples"], "flops": 4 * 3 * case["samples"]}
    if kind == "detect":
        return {"bytes": 4 * case["samples"], "flops": 2 * case["samples"]}
    N, S, P = _sources(case), case["stations"], case.get("phases", 2)
    size = 4 if case.get("storage", "fp32") == "fp32" else 2
    table = N * S * (4 * P + 4)
    if kind == "batch":
        T = int(_window_samples(case).sum())
        return {"bytes": table + T * (12 * S + 8), "flops": 2 * N * T * P * S // 2}
    T = case["samples"]
    near = 1.0
    if case.get("max_km"):
        # share of (source, station) pairs within max_km in a square of this side
        r = min(case["max_km"] / case["square_km"], 1.0)
        near = min(1.0, math.pi * r * r - 8.0 / 3.0 * r ** 3 + 0.5 * r ** 4)
    flops = int(2 * N * T * P * S * near)
    if kind == "resident":
        out = 4 * N * T if case["reduce"] == "none" else 8 * T
        return {"bytes": table + size * S * P * T + out, "flops": flops}
    return {"bytes": table + 12 * S * T + 8 * T, "flops": flops}


# ---- the same in 64 bits ---------------------------------------------------------
def _exact_beams(f, delays, alpha, weights, strict, whole):
    """The beams of every source, or their maximum, in float64."""
    u = torch.einsum("sct,scp->spt", f.double(), alpha.double())
    S, P, T = u.shape
    N = delays.shape[0]
    used = (weights != 0)[:, :, None].expand_as(delays)
    low = torch.where(used, delays, 1 << 30).amin(dim=(1, 2)).long()
    high = torch.where(used, delays, -(1 << 30)).amax(dim=(1, 2)).long()
    best = torch.full((T,), -math.inf, device=DEV, dtype=torch.float64)
    beams = torch.zeros((N, T), dtype=torch.float64) if whole else None
    t = torch.arange(T, device=DEV)
    step = max(1, (1 << 27) // T)
    pad = torch.zeros((1,), device=DEV, dtype=torch.float64)
    for a in range(0, N, step):
        d, w = delays[a:a + step].long(), weights[a:a + step].double()
        acc = torch.zeros((d.shape[0], T), device=DEV, dtype=torch.float64)
        for s in range(S):
            for p in range(P):
                at = t[None, :] + d[:, s, p, None]
                at = torch.where((at >= 0) & (at < T), at, T)
                acc += w[:, s, None] * torch.cat([u[s, p], pad])[at]
        if strict:
            lo, hi = low[a:a + step, None], high[a:a + step, None]
            valid = (lo <= hi) & (t + lo >= 0) & (t + hi < T)
        else:
            valid = torch.ones((1, 1), device=DEV, dtype=torch.bool)
        if whole:
            beams[a:a + step] = torch.where(valid, acc, 0.0).cpu()
        else:
            best = torch.maximum(best, torch.where(valid, acc, -math.inf).amax(dim=0))
    if whole:
        return beams
    return torch.where(torch.isinf(best), 0.0, best)


def _median(x):
    """NumPy's median of the last axis."""
    n = x.shape[-1]
    s = x.sort(dim=-1).values
    return s[..., n // 2] if n % 2 else 0.5 * (s[..., n // 2 - 1] + s[..., n // 2])


def _exact_envelope(x):
    n = x.shape[-1]
    out = torch.empty(x.shape, device=DEV, dtype=torch.float64)
    for s in range(x.shape[0]):
        z = torch.fft.fft(x[s].double())
        h = torch.zeros(n, device=DEV, dtype=torch.float64)
        h[0] = 1.0
        h[1:(n + 1) // 2] = 2.0
        if n % 2 == 0:
            h[n // 2] = 1.0
        env = torch.fft.ifft(z * h).abs()
        env = env - _median(env)[..., None]
        mad = _median(env.abs())
        out[s] = torch.clamp(env / torch.where(mad == 0, 1.0, mad)[..., None], max=1.0e5)
    return out


def _exact_threshold(case, x, noise):
    x = x.double()
    n, W = x.numel(), case["window"]
    rms = case["threshold_type"] == "rms"
    kept = x[x != 0]
    centre = kept.mean() if rms else _median(kept)
    dev = torch.sqrt(((kept - centre) ** 2).mean()) if rms else _median((kept - centre).abs())
    zero = x == 0
    x[zero] = noise.double()[:int(zero.sum())] * dev + centre
    shift = int((1.0 - 0.66) * W)
    thr = []
    for i in range((n - W) // shift + 1):
        w = x[i * shift:i * shift + W]
        c = w.mean() if rms else _median(w)
        d = torch.sqrt(((w - c) ** 2).mean()) if rms else _median((w - c).abs())
        thr.append(c + 8.0 * d)
    thr = torch.stack(thr)
    thr[1:] = torch.maximum(thr[:-1], thr[1:]).clone()
    thr[:-1] = torch.maximum(thr[:-1], thr[1:]).clone()
    j = (torch.arange(n, device=DEV) - W // 2).clamp(0, n - W - 1)
    return thr[((W // 2 + j) // shift).clamp(max=thr.numel() - 1)]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("resident", "call", "host"):
        N, P = _sources(case), case.get("phases", 2)
        terms = N * case["samples"] * case["stations"] * P
        if terms > 4.6e11:
            return None
        whole = case.get("reduce", "max") == "none"
        if whole and terms > 1e10:
            return None
        beams = _exact_beams(*_inputs(case, seed), case["oob"] == "strict", whole)
        return beams if whole else (beams, None)
    if kind == "batch":
        if _sources(case) * int(_window_samples(case).sum()) * case["stations"] > 4.6e11:
            return None
        delays, weights, stations, records = _batch_inputs(case, seed)
        alpha, out = _phase_weights(case["stations"], 2), []
        for some, f in zip(stations, records):
            out.append((_exact_beams(f[some], delays[:, some], alpha[some], weights[:, some],
                                     True, False), None))
        return out
    if kind == "features":
        return _exact_envelope(prepare(case, seed)["x"])
    if kind == "threshold":
        state = prepare(case, seed)
        return _exact_threshold(case, state["x"], state["noise"])
    return None
