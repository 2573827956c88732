"""Performance cases: what a program that sorts spikes with this package asks of the GPU.

Every case goes through a public entry point.  The kinds:

* ``host``        ``binary_pursuit`` on a recording in host memory (the drop-in call of a
                  sorting pipeline): upload, pursuit, spikes and (optionally) clips back.
* ``device``      ``fbp_pursue_chunk`` of the C ABI on a voltage, templates and workspace
                  that a host program keeps on the device.
* ``segments``    ``pursue_segments``: many short independent segments, several at once.
* ``refine``      ``residual_energy`` forward and backward (template refinement).
* ``inputs``      ``templates_and_covariances``: robust templates and noise covariances of
                  the sorted spikes, before the pursuit.
* ``noise``       ``compute_separability_metrics`` and ``pairwise_separability`` of a
                  template set.
* ``duplicates``  ``remove_segment_duplicates`` on the pursuit's clips left on the device.

Recordings are synthetic: band-passed unit-variance noise, biphasic templates, Poisson spike
trains with a refractory period and a share of overlapping spikes, thresholds from the noise
model -- the distributions of ``spikesorting_fullpursuit_b200.synth`` drawn on the GPU.
"""
import ctypes
import math

import numpy as np
import torch

from spikesorting_fullpursuit_b200 import _native, binary_pursuit, synth
from spikesorting_fullpursuit_b200.adjoint import residual_energy
from spikesorting_fullpursuit_b200.overlap import full_binary_pursuit, neuron_separability
from spikesorting_fullpursuit_b200.postprocessing import remove_segment_duplicates
from spikesorting_fullpursuit_b200.segments import pursue_segments

CLIP_WIDTH = (-1.0e-3, 1.5e-3)
DEV = "cuda"

# Probe models: how a unit's template spreads over the channels ("index": a Gaussian over the
# channel index, non-zero on every channel, as templates estimated from clips are; "linear" and
# "two_column": exactly zero outside a neighbourhood), spike rates and the overlapping share.
PROBES = {
    "index": dict(layout="index", pitch_um=50.0, nbhd=None, sigma_um=60.0, rate=(10.0, 80.0), overlap=0.1),
    "linear": dict(layout="linear", pitch_um=50.0, nbhd=(4, 6), sigma_um=60.0, rate=(10.0, 80.0), overlap=0.2),
    "two_column": dict(layout="two_column", pitch_um=25.0, nbhd=8, sigma_um=40.0, rate=(8.0, 100.0), overlap=0.25),
}

# The largest drawn pursuit, in channel x unit x sample: that of the largest listed one.
MOST = 64 * 200 * 600_000


def _pursuit(name, kind, probe, chans, units, fs, seconds, recheck=True, clips=False, half_shift=False):
    return {"name": name, "kind": kind, "probe": probe, "chans": chans, "units": units, "fs": fs,
            "seconds": seconds, "recheck": recheck, "clips": clips, "half_shift": half_shift}


def listed():
    return [
        # one short tetrode segment, the smallest call a sorter makes: launches and latency count
        _pursuit("tetrode_segment_5s", "host", "index", 4, 5, 40000, 5.0),
        # the package's tetrode configuration, with the adjusted clips a sorter goes on with
        _pursuit("tetrode_30s_clips", "host", "index", 4, 6, 40000, 30.0, clips=True),
        # a 16-channel probe from host memory and back: upload, pursuit, download
        _pursuit("linear16_host_120s", "host", "linear", 16, 40, 40000, 120.0),
        # the benchmark's 16-channel probe (40 units x 101 samples), resident on the device
        _pursuit("linear16_300s", "device", "linear", 16, 40, 40000, 300.0),
        # the dense 64-channel probe with 200 units: the heaviest likelihood and recheck
        _pursuit("dense64_20s", "device", "two_column", 64, 200, 30000, 20.0),
        # templates without a zero channel, odd sizes, the default half-window shift range
        _pursuit("index11_43s_half_shift", "device", "index", 11, 27, 30000, 43.0, half_shift=True),
        # the option without the overlap recheck, odd sizes: likelihood, argmax and residual only
        _pursuit("linear23_no_recheck", "device", "linear", 23, 77, 30000, 41.0, recheck=False),
        # uneven short segments, four at once on streams of their own
        {"name": "segments_12", "kind": "segments", "segments": 12, "chans": 4, "most_chans": 12, "units": 5,
         "most_units": 30, "fs": 40000, "seconds": 3.0, "most_seconds": 12.0, "streams": 4},
        # one gradient step of template refinement on the 16-channel probe
        {"name": "refine_linear16_60s", "kind": "refine", "probe": "linear", "chans": 16, "units": 40, "fs": 40000,
         "seconds": 60.0},
        # templates and covariances of one minute of sorted spikes on the 16-channel probe
        {"name": "inputs_linear16_60s", "kind": "inputs", "probe": "linear", "chans": 16, "units": 40, "fs": 40000,
         "seconds": 60.0, "cov_samples": 10000},
        # the noise model of the dense probe's 200 templates: thresholds and all pairs
        {"name": "noise_dense64", "kind": "noise", "probe": "two_column", "chans": 64, "units": 200, "fs": 30000},
        # duplicate removal over all units of a 16-channel segment
        {"name": "duplicates_linear16", "kind": "duplicates", "probe": "linear", "chans": 16, "units": 40,
         "fs": 40000, "spikes": 12000},
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["host", "host", "device", "device", "device", "segments", "refine", "inputs", "noise",
                       "duplicates"])
    fs = rng.choice([30000, 40000])
    probe = rng.choice(sorted(PROBES))
    chans = int(round(_log(rng, 4, 12 if probe == "index" else 64)))
    units = int(round(_log(rng, 5, 60 if probe == "index" else 200)))
    if kind == "segments":
        return {"kind": kind, "segments": rng.randint(4, 12), "chans": 4, "most_chans": rng.randint(5, 12),
                "units": 5, "most_units": rng.randint(6, 30), "fs": fs, "seconds": 3.0,
                "most_seconds": round(rng.uniform(4.0, 12.0), 3), "streams": rng.choice([1, 2, 4, 8])}
    if kind in ("host", "device"):
        # templates without zero channels make more of the recheck: a third of the largest
        most = min(300.0, MOST / (chans * units * fs * (3 if probe == "index" else 1)),
                   (120.0 if kind == "host" else 300.0) * 16 / chans)
        recheck, clips = rng.random() < 0.8, kind == "host" and rng.random() < 0.5
        if clips:   # at most about 40 MB of clips
            most = min(most, 1e7 / (12 * units * chans * _window(fs)))
        seconds = round(max(0.5, min(_log(rng, 2.0, 300.0), most)), 4)
        c = _pursuit("", kind, probe, chans, units, fs, seconds, recheck, clips, rng.random() < 0.3)
        del c["name"]
        return c
    c = {"kind": kind, "probe": probe, "chans": min(chans, 32), "units": min(units, 60), "fs": fs}
    if kind == "noise":
        c.update(chans=chans, units=units)
    elif kind == "duplicates":
        c["spikes"] = int(round(_log(rng, 500, 12000)))
    else:
        c["seconds"] = round(min(_log(rng, 3.0, 60.0), 60.0 * 16 * 40 / (c["chans"] * c["units"])), 4)
        if kind == "inputs":
            c["cov_samples"] = rng.choice([2000, 10000, 50000])
    return c


# --------------------------------------------------------------------------- recordings


def _window(fs):
    return int(round(CLIP_WIDTH[1] * fs)) + 1 + int(round(-CLIP_WIDTH[0] * fs))


def _noise(gen, chans, n, fs):
    """Unit-variance noise, band-passed 300-8000 Hz (squared 4th-order Butterworth magnitude)."""
    size = 1 << (n - 1).bit_length()
    f = torch.fft.rfftfreq(size, 1.0 / fs, device=DEV).clamp_(min=1.0)
    gain = 1.0 / ((1.0 + (300.0 / f) ** 8) * (1.0 + (f / min(8000.0, 0.45 * fs)) ** 8))
    V = torch.empty((chans, n), dtype=torch.float32, device=DEV)
    for c in range(chans):
        x = torch.randn(size, generator=gen, device=DEV)
        y = torch.fft.irfft(torch.fft.rfft(x) * gain, n=size)[:n]
        V[c] = y / y.std()
    return V


def _covariances(gen, V, W, clips=2000):
    """Per-channel noise covariance from random clips (float64 [C][W][W])."""
    n = V.shape[1]
    at = torch.randint(0, n - W, (clips,), generator=gen, device=DEV)
    X = V[:, at[:, None] + torch.arange(W, device=DEV)].double()
    return torch.einsum("cni,cnj->cij", X, X) / clips


def _trains(rng, units, seconds, fs, rate, overlap):
    """Spike samples (sorted) and units: Poisson with a 1.5 ms refractory period, a share moved
    to within a millisecond of another spike."""
    times, labels = [], []
    for m in range(units):
        hz = min(math.exp(rng.normal(math.log(rate[0]), 0.6)), rate[1])
        gaps = 1.5e-3 + rng.exponential(max(1.0 / hz - 1.5e-3, 1e-4), size=int(seconds * hz * 1.2) + 40)
        t = np.cumsum(gaps)
        t = t[t < seconds]
        times.append(t)
        labels.append(np.full(t.size, m))
    t, lab = np.concatenate(times), np.concatenate(labels)
    if overlap and t.size > 1 and units > 1:
        move = rng.choice(t.size, int(overlap * t.size), replace=False)
        t[move] = t[rng.integers(0, t.size, move.size)] + rng.uniform(-1e-3, 1e-3, move.size)
    s = np.round(t * fs).astype(np.int64)
    order = np.lexsort((lab, s))
    return s[order], lab[order]


def _recording(case, seed, spikes=True):
    """Voltage on the device, sort_info, metrics, spike onsets and labels."""
    p = PROBES[case["probe"]]
    C, M, fs = case["chans"], case["units"], case["fs"]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    T, W, pre = synth.make_templates(rng, M, C, fs, list(CLIP_WIDTH), p["layout"], p["pitch_um"], p["nbhd"],
                                     p["sigma_um"])
    n = int(round(case.get("seconds", 4.0) * fs))
    V = _noise(gen, C, n, fs)
    covs = _covariances(gen, V, W)
    info = {"sampling_rate": fs, "clip_width": list(CLIP_WIDTH), "n_samples_per_chan": W, "n_channels": C,
            "n_samples": n, "do_overlap_recheck": case.get("recheck", True),
            "get_adjusted_clips": case.get("clips", False), "sigma_bp_noise": 3.719, "sigma_bp_CI": 12.0,
            "n_threshold_crossings": [n // 400] * C}
    metrics = synth.separability_metrics(T, list(covs.cpu().numpy()), C, W)
    if not spikes:
        return V, info, metrics, covs, None, None
    s, lab = _trains(rng, M, n / fs, fs, p["rate"], p["overlap"])
    on = s - pre
    keep = (on >= 0) & (on + W <= n)
    on, lab = on[keep], lab[keep]
    at = torch.from_numpy(on).to(DEV)
    lb = torch.from_numpy(lab).to(DEV)
    scale = torch.from_numpy(rng.normal(1.0, 0.1, on.size).astype(np.float32)).to(DEV)
    T3 = torch.from_numpy(T.reshape(M, C, W)).to(DEV)
    cols = (at[:, None] + torch.arange(W, device=DEV)).reshape(-1)
    for c in range(C):   # summed as whole numbers, so that overlapping spikes add up to the same value every time
        vals = torch.round(scale[:, None].double() * T3[lb, c] * 2.0 ** 24).long().reshape(-1)
        V[c] += torch.zeros(n, dtype=torch.int64, device=DEV).index_add_(0, cols, vals).double() / 2.0 ** 24
    return V, info, metrics, covs, on, lab


def _most_spikes(units, probe, seconds):
    return int(units * PROBES[probe]["rate"][1] * seconds) + 2000


def _shift(case, W):
    return W // 2 if case["half_shift"] else W - 1


def _device_pursuit(case, seed):
    V, info, metrics, _, _, _ = _recording(case, seed)
    C, N = V.shape
    W, M = info["n_samples_per_chan"], case["units"]
    flags = _native.FBP_OVERLAP_RECHECK if case["recheck"] else 0
    d = _native.dims(C, N, M, W, _shift(case, W))
    cap = 16 * (N // W + 1) + 1024
    as_f32 = lambda a: torch.from_numpy(np.ascontiguousarray(a, dtype=np.float32)).to(DEV)  # noqa: E731
    return {"dims": d, "flags": flags, "voltage": V, "work": torch.empty_like(V),
            "templates": as_f32(metrics["templates"]), "bias": as_f32(-0.5 * metrics["template_SS"]),
            "theta": as_f32(metrics["neuron_lower_thresholds"]), "cap": cap,
            "scratch": torch.empty(_native.workspace_bytes(d, flags), dtype=torch.uint8, device=DEV),
            "idx": torch.zeros(cap, dtype=torch.int32, device=DEV),
            "lab": torch.zeros(cap, dtype=torch.int32, device=DEV)}


def _segments(case, seed):
    rng = np.random.default_rng(seed)
    out = []
    for k in range(case["segments"]):
        one = {"probe": "index", "chans": int(rng.integers(case["chans"], case["most_chans"] + 1)),
               "units": int(rng.integers(case["units"], case["most_units"] + 1)), "fs": case["fs"],
               "seconds": float(rng.uniform(case["seconds"], case["most_seconds"]))}
        V, info, metrics, _, _, _ = _recording(one, seed * 1000 + k)
        out.append((V.cpu().numpy(), np.float32, info, metrics))
    most = _most_spikes(case["most_units"], "index", case["most_seconds"])
    return out, np.zeros((2, case["segments"], most), dtype=np.int64)


def _duplicates(case, seed):
    """Clips around each unit's template, ordered spike times, one in ten a near-duplicate."""
    p = PROBES[case["probe"]]
    rng = np.random.default_rng(seed)
    gen = torch.Generator(device=DEV)
    gen.manual_seed(int(seed))
    n, M, fs = case["spikes"], case["units"], case["fs"]
    T, W, _ = synth.make_templates(rng, M, case["chans"], fs, list(CLIP_WIDTH), p["layout"], p["pitch_um"], p["nbhd"],
                                   p["sigma_um"])
    lab = rng.integers(0, M, n)
    ev = np.sort(rng.integers(0, n * fs // 400, n))
    twin = np.flatnonzero(rng.random(n - 1) < 0.1)
    ev[twin + 1] = ev[twin] + rng.integers(0, 8, twin.size)
    lab[twin + 1] = lab[twin]
    order = np.argsort(ev, kind="stable")
    ev, lab = ev[order], lab[order]
    clips = torch.from_numpy(T).to(DEV)[torch.from_numpy(lab).to(DEV)]
    clips += torch.randn(clips.shape, generator=gen, device=DEV)
    return {"events": ev, "labels": lab, "clips": clips, "found": rng.random(n) < 0.9, "tol": W // 10}


def prepare(case, seed):
    kind = case["kind"]
    if kind == "device":
        return {"kind": kind, **_device_pursuit(case, seed)}
    if kind == "segments":
        segments, spikes = _segments(case, seed)
        return {"kind": kind, "segments": segments, "streams": case["streams"], "spikes": spikes}
    if kind == "duplicates":
        return {"kind": kind, **_duplicates(case, seed)}
    V, info, metrics, covs, on, lab = _recording(case, seed, spikes=kind != "noise")
    C, W, M = case["chans"], info["n_samples_per_chan"], case["units"]
    if kind == "host":
        most = _most_spikes(M, case["probe"], case["seconds"])
        return {"kind": kind, "voltage": V.cpu().numpy(), "info": info, "metrics": metrics,
                "shift": _shift(case, W), "spikes": np.zeros((2, most), dtype=np.int64),
                "clips": np.zeros((most if case["clips"] else 0, C * W), dtype=np.float32)}
    if kind == "noise":
        return {"kind": kind, "templates": list(metrics["templates"]), "covs": list(covs.cpu().numpy()),
                "info": info}
    if kind == "refine":
        rng = np.random.default_rng(seed + 1)
        f32 = lambda a: torch.from_numpy(a.astype(np.float32)).to(DEV)  # noqa: E731
        # a fixed number of the recording's spikes (topped up anywhere if it has fewer)
        want = int(8 * M * case["seconds"])
        extra = max(0, want - on.size)
        pick = np.sort(rng.permutation(on.size)[:want])
        on = np.concatenate([on[pick], rng.integers(0, info["n_samples"] - W, extra)])
        lab = np.concatenate([lab[pick], rng.integers(0, M, extra)])
        return {"kind": kind, "voltage": V, "templates": f32(metrics["templates"].reshape(M, C, W)),
                "onsets": torch.from_numpy(on).to(DEV), "labels": torch.from_numpy(lab).to(DEV),
                "amplitude": f32(rng.normal(1.0, 0.1, on.size)), "shift": f32(rng.uniform(-0.5, 0.5, on.size))}
    pre = int(round(-CLIP_WIDTH[0] * case["fs"]))
    units = [on[lab == m] + pre for m in range(M)]   # event indices: the alignment sample
    units = [u if u.size else np.array([info["n_samples"] // 2]) for u in units]
    probe = {"sampling_rate": case["fs"], "n_samples": info["n_samples"], "v_dtype": np.float32}
    return {"kind": kind, "voltage": V, "probe": probe, "units": units, "chans": C, "window": W,
            "cov_samples": case["cov_samples"], "seed": int(seed) % (1 << 32)}


# --------------------------------------------------------------------------- one pass


def _ptr(t):
    return ctypes.c_void_p(t.data_ptr())


def run(s):
    kind = s["kind"]
    if kind == "host":
        ev, lab, _, clips = binary_pursuit(s["voltage"], np.float32, s["info"], dict(s["metrics"]),
                                           n_max_shift_inds=s["shift"], verbose=False)
        s["spikes"][0, :len(ev)] = ev   # into the program's own arrays
        s["spikes"][1, :len(ev)] = lab
        if s["info"]["get_adjusted_clips"]:
            s["clips"][:len(ev)] = clips
        return [len(ev), s["spikes"], s["clips"]]
    if kind == "device":
        s["work"].copy_(s["voltage"])   # the pursuit leaves its residual in place
        n = ctypes.c_uint32(0)
        _native.check(_native.lib().fbp_pursue_chunk(
            ctypes.byref(s["dims"]), s["flags"], _ptr(s["work"]), _ptr(s["templates"]), _ptr(s["bias"]),
            _ptr(s["theta"]), _ptr(s["scratch"]), s["scratch"].numel(), _ptr(s["idx"]), _ptr(s["lab"]), s["cap"],
            ctypes.byref(n), None, _native.MAX_PASSES,
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream)))
        return [n.value, s["idx"], s["lab"], s["work"]]   # the buffers stay zero past the n spikes
    if kind == "segments":
        segs = [(V, dt, info, dict(m)) for V, dt, info, m in s["segments"]]
        out = pursue_segments(segs, streams=s["streams"], verbose=False)
        for k, (ev, lab, _, _) in enumerate(out):
            s["spikes"][0, k, :len(ev)] = ev
            s["spikes"][1, k, :len(ev)] = lab
        return [[len(r[0]) for r in out], s["spikes"]]
    if kind == "refine":
        T = s["templates"].detach().requires_grad_(True)
        a = s["amplitude"].detach().requires_grad_(True)
        tau = s["shift"].detach().requires_grad_(True)
        E = residual_energy(s["voltage"], T, s["onsets"], s["labels"], a, tau)
        E.backward()
        return [E.detach(), T.grad, a.grad, tau.grad]
    if kind == "inputs":
        np.random.seed(s["seed"])   # the covariance rows come from numpy's global generator
        T, covs = full_binary_pursuit.templates_and_covariances(
            s["probe"], s["voltage"], np.arange(s["chans"]), s["units"], list(CLIP_WIDTH), s["chans"], s["window"],
            s["cov_samples"])
        return [T, covs]
    if kind == "noise":
        m = neuron_separability.compute_separability_metrics(s["templates"], s["covs"], s["info"])
        pair, contamination, misses = neuron_separability.pairwise_separability(m, s["info"])
        return [m["template_SS"], m["neuron_variances"], m["neuron_lower_thresholds"], m["neuron_lower_CI"],
                m["contamination"], m["peak_channel"], pair, contamination, misses]
    return remove_segment_duplicates(s["events"], s["labels"], s["clips"], s["found"], s["tol"])


# --------------------------------------------------------------------------- required work


def _correlation_flops(chans, units, samples, W):
    """All templates against `samples` samples by overlap-save with transforms of 256: the
    fewest operations this framework knows a way to do it in."""
    blocks = samples / (257.0 - W)
    return blocks * ((chans + units) * 0.5 * 5 * 256 * 8 + units * min(chans, 6) * 129 * 8)


def work(case):
    kind, fs = case["kind"], case["fs"]
    W = _window(fs)
    if kind == "segments":
        n = case["segments"] * 0.5 * (case["seconds"] + case["most_seconds"]) * fs
        C, M = 0.5 * (case["chans"] + case["most_chans"]), 0.5 * (case["units"] + case["most_units"])
        return {"bytes": 4 * C * n + 4 * M * C * W, "flops": _correlation_flops(C, M, n, W)}
    C, M = case["chans"], case["units"]
    hz = 1.2 * PROBES[case["probe"]]["rate"][0]
    if kind == "noise":
        lags = 2 * (W // 4) - 1
        return {"bytes": 4 * M * C * W + 8 * C * W * W + 8 * M * M,
                "flops": 2.0 * M * C * W * W + M * M * 2.0 * C * (lags * W + W * W)}
    if kind == "duplicates":
        return {"bytes": 4.0 * case["spikes"] * C * W + 17 * case["spikes"], "flops": 4.0 * case["spikes"] * C * W}
    n = case["seconds"] * fs
    spikes = M * hz * case["seconds"]
    if kind == "refine":
        return {"bytes": 4 * C * n + 8 * M * C * W + 24 * spikes, "flops": 20.0 * spikes * C * W + 2 * C * n}
    if kind == "inputs":
        return {"bytes": 4 * C * n + 4 * M * C * W + 8 * C * W * W,
                "flops": 2.0 * C * W * W * case["cov_samples"] + 8 * spikes * C * W}
    out = 8 * spikes + (4 * spikes * C * W if case["clips"] else 0)
    flops = _correlation_flops(C, M, n, W)
    if case["recheck"]:   # every spike's window against every template
        flops += _correlation_flops(C, M, spikes * (257.0 - W), W)
    return {"bytes": (4 if kind == "host" else 8) * C * n + 4 * M * C * W + out, "flops": flops}


# --------------------------------------------------------------------------- results in 64 bits


def _exact_refine(s):
    V, T = s["voltage"].double(), s["templates"].double()
    a, tau = s["amplitude"].double()[:, None, None], s["shift"].double()[:, None, None]
    M, C, W = T.shape
    N = V.shape[1]
    u = tau.abs()
    right = tau >= 0
    Tp = torch.nn.functional.pad(T, (2, 2))[s["labels"]]        # sample j at column j + 2
    here, before, after = Tp[..., 1:-1], Tp[..., :-2], Tp[..., 2:]   # j = -1 .. W
    other = torch.where(right, before, after)
    moved = (1 - u) * here + u * other
    x = s["onsets"][:, None] + torch.arange(-1, W + 1, device=DEV)
    inside = (x >= 0) & (x < N)
    xc = x.clamp(0, N - 1)
    r = V.clone()
    for c in range(C):
        r[c].index_add_(0, xc.reshape(-1), torch.where(inside, -(a[:, 0] * moved[:, c]), 0.0).reshape(-1))
    near = torch.where(inside, r[:, xc], 0.0).permute(1, 0, 2)   # [n][C][W + 2]
    ga = -2 * (moved * near).sum((1, 2))
    sign = torch.where(right, 1.0, -1.0)[:, 0, 0]
    gs = -2 * a[:, 0, 0] * sign * ((other - here) * near).sum((1, 2))
    mid = near[..., 1:-1]
    g = -2 * a * ((1 - u) * mid + u * torch.where(right, near[..., 2:], near[..., :-2]))
    gT = torch.zeros_like(T).index_add_(0, s["labels"], g)
    return [(r * r).sum(), gT, ga, gs]


def _median(x):
    v = torch.sort(x, dim=0).values
    n = v.shape[0]
    return 0.5 * (v[(n - 1) // 2] + v[n // 2])


def _exact_inputs(s):
    V = s["voltage"].double()
    C, W = s["chans"], s["window"]
    lo = -int(round(-CLIP_WIDTH[0] * s["probe"]["sampling_rate"]))
    taps = torch.arange(lo, lo + W, device=DEV)
    templates, residuals = [], []
    for idx in s["units"]:
        at = torch.from_numpy(idx).to(DEV)
        at = at[(at + lo >= 0) & (at + lo + W <= V.shape[1])]
        x = V[:, at[:, None] + taps].permute(1, 0, 2).reshape(at.numel(), C * W)
        t = x[0]
        if at.numel() > 1:
            med = _median(x)
            mad = _median((x - med).abs()) / 0.6745
            keep = (x > med - mad) & (x < med + mad)
            k = keep.sum(0)
            v = torch.sort(torch.where(keep, x, math.inf), dim=0).values
            pick = lambda i: v.gather(0, i.clamp(min=0)[None])[0]  # noqa: E731
            t = torch.where(k > 0, 0.5 * (pick((k - 1) // 2) + pick(k // 2)), med)
        templates.append(t)
        residuals.append(x - t)
    R = torch.cat(residuals)
    np.random.seed(s["seed"])
    covs = []
    for c in range(C):
        n = s["cov_samples"]
        rows = np.arange(R.shape[0]) if n >= R.shape[0] else np.random.randint(0, R.shape[0], n)
        x = R[torch.from_numpy(rows).to(DEV), c * W:(c + 1) * W]
        x = x - x.mean(0)
        covs.append(x.T @ x / rows.size)
    return [torch.stack(templates), covs]


def _exact_noise(s):
    info = s["info"]
    C, W = info["n_channels"], info["n_samples_per_chan"]
    T = torch.from_numpy(np.vstack(s["templates"])).to(DEV).double()
    K = torch.from_numpy(np.stack(s["covs"])).to(DEV).double()
    M = T.shape[0]
    T3 = T.reshape(M, C, W)
    upper = lambda z: 0.5 * torch.erfc(z / math.sqrt(2.0))  # noqa: E731
    ss = (T * T).sum(1)
    form = lambda D: (torch.einsum("pci,cij->pcj", D, K) * D).sum((1, 2))  # noqa: E731
    var = form(T3)
    sd = var.sqrt()
    thr = -0.5 * ss + info["sigma_bp_noise"] * sd
    ci = 0.5 * ss - info["sigma_bp_CI"] * sd
    noise = upper((thr + 0.5 * ss) / sd)
    most = W // 4 - 1
    L = C * W
    best = torch.full((M, M), -1.0, dtype=torch.float64, device=DEV)
    shift = torch.zeros((M, M), dtype=torch.int64, device=DEV)
    for k in range(-most, most + 1):
        a = T[:, max(k, 0):L + min(k, 0)]
        b = T[:, max(-k, 0):L - max(k, 0)]
        cc = (a @ b.T).abs()
        better = cc > best
        best = torch.where(better, cc, best)
        shift[better] = k
    pair = torch.zeros((M, M), dtype=torch.float64, device=DEV)
    for k in range(-most, most + 1):
        for at in torch.nonzero(shift == k).split(4096):
            if not at.numel():
                continue
            P1, P2 = torch.zeros((2, at.shape[0], C, W), dtype=torch.float64, device=DEV)
            lo, hi = max(k, 0), W + min(k, 0)
            P1[..., lo:hi] = T3[at[:, 0], :, lo:hi]
            P2[..., lo:hi] = T3[at[:, 1], :, lo - k:hi - k]
            v = form(P1 - P2)
            e = 0.5 * ss[at[:, 0]] - ((P1 * P2).sum((1, 2)) - 0.5 * ss[at[:, 1]])
            pair[at[:, 0], at[:, 1]] = torch.where(v > 0, upper(e / v.clamp(min=1e-300).sqrt()), 0.0)
    return [ss, var, thr, ci, noise, None, pair, noise, upper((0.5 * ss - thr) / sd)]


def exact(case, seed):
    # the spikes of a pursuit and the keep mask of the duplicates are whole numbers, and the
    # residual and the clips are what is left of the voltage after them: nothing to add in 64 bits
    if case["kind"] not in ("refine", "inputs", "noise"):
        return None
    s = prepare(case, seed)
    return {"refine": _exact_refine, "inputs": _exact_inputs, "noise": _exact_noise}[case["kind"]](s)
