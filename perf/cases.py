"""The work whose speed counts: pursuits of segments from a tenth of a second
on a tetrode to a hundred seconds on a 384-channel probe, through the calls a
sorting program makes, and the two steps that prepare them.

Kinds of a case:
  call    binary_pursuit() on a host recording (upload, pursuit, spike trains
          and, where asked for, adjusted clips back on the host)
  chunk   fbp_pursuit_chunk() on a recording that is already on the GPU, with
          the caller's own workspace and spike buffers
  batch   segments of mixed sizes submitted at once to a PursuitServer with
          four slots, which the program keeps
  inputs  templates, noise covariance, variances and thresholds of a pursuit
          from the units' spikes (pursuit_templates_and_covariance(),
          compute_separability_metrics())
  whiten  ZCA matrix of a recording and its application

Recordings follow synthetic.py's recipe (band-limited noise, biphasic
templates, Poisson trains), drawn on the GPU so that a long one takes
milliseconds: "dense" templates lie on all channels (tetrodes, shanks),
"probe" ones fall off along a linear probe, "masked" ones cover 16 channels of
a high-density probe.  Spikes are added as integers of 2^-16 noise SD, which
gives the same recording whatever order they are added in.
"""
import ctypes
import math

import numpy as np
import torch

from spikesorting_fullpursuit_b200 import _lib, synthetic

QUANTUM = 65536.0          # template quanta per noise SD in a recording
INT16_SCALE = 16.0         # int16 counts per noise SD


def _case(name, kind, model, chans, seconds, fs, templates, length, **more):
    c = {"name": name, "kind": kind, "model": model, "chans": chans, "seconds": seconds, "fs": fs,
         "templates": templates, "length": length, "dtype": "float32", "precision": "bf16", "overlap": True,
         "clips": False, "production_shift": True}
    c.update(more)
    return c


def listed():
    return [
        # the smallest call: half a second of a tetrode, clips asked for, as an interactive program re-sorts a
        # stretch of a recording; latency and launches
        _case("tetrode_half_second", "call", "dense", 4, 0.5, 40000, 8, 101, clips=True, production_shift=False),
        # a whole tetrode recording with the reference's default shift (half a clip)
        _case("tetrode_30s", "call", "dense", 4, 30.0, 40000, 8, 101, production_shift=False),
        # one ragged segment of a batched sort, int16 as an acquisition system writes it
        _case("ragged_segment", "call", "dense", 17, 3.07, 40000, 23, 77, dtype="int16"),
        # the same without the overlap recheck (do_overlap_recheck=False), short clips
        _case("no_overlap_recheck", "call", "dense", 32, 5.3, 30000, 37, 43, overlap=False),
        # one request of the serving mix: part of a high-density probe, host call
        _case("served_request", "call", "masked", 201, 2.5, 30000, 157, 61),
        # many small segments at once on four slots
        _case("batch_of_12", "batch", "dense", 32, 3.0, 40000, 40, 101, segments=12),
        # the 16-channel probe, 64 units, device-resident: half of its ten-minute recording
        _case("linear16_300s", "chunk", "probe", 16, 300.0, 40000, 64, 101),
        # the 384-channel probe, 300 units: a short stretch and a long one (the long one is the largest case)
        _case("hd384_10s", "chunk", "masked", 384, 10.0, 30000, 300, 61, dtype="int16"),
        _case("hd384_100s", "chunk", "masked", 384, 100.0, 30000, 300, 61, dtype="int16"),
        # the plain FP32 path, chosen where the tensor cores are not wanted
        _case("linear16_10s_fp32", "chunk", "probe", 16, 10.0, 40000, 64, 101, precision="fp32"),
        # what is computed before a pursuit: robust templates, noise covariance, thresholds
        _case("pursuit_inputs", "inputs", "probe", 16, 30.0, 40000, 64, 101),
        # whitening of a shank's recording
        _case("whiten_32ch", "whiten", "dense", 32, 40.0, 30000, 3, 61),
    ]


def _log_uniform(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choices(["call", "chunk", "batch", "inputs", "whiten"], [5, 5, 1, 1, 1])[0]
    if kind == "whiten":
        chans = int(_log_uniform(rng, 4, 129))
        return _case("", kind, "dense", chans, round(min(60.0, _log_uniform(rng, 0.5, 2000.0 / chans)), 3), 30000, 3,
                     61, dtype=rng.choice(["float32", "float32", "int16"]))
    if kind == "batch":
        return _case("", kind, "dense", rng.randint(4, 32), round(_log_uniform(rng, 0.3, 4.0), 3), 40000,
                     rng.randint(2, 40), rng.randint(61, 101), segments=rng.randint(5, 16))
    if kind == "inputs":
        return _case("", kind, "probe", rng.randint(4, 24), round(_log_uniform(rng, 2.0, 30.0), 3), 40000,
                     rng.randint(3, 64), rng.randint(61, 101))
    fp32 = rng.random() < 0.15
    more = {"precision": "fp32" if fp32 else "bf16", "dtype": rng.choice(["float32", "int16"]),
            "overlap": rng.random() < 0.85, "production_shift": rng.random() < 0.7}
    if rng.random() < 0.5:
        chans, templates, length, model, fs = rng.randint(33, 384), rng.randint(4, 300), 61, "masked", 30000
        if rng.random() < 0.3:
            length = rng.randint(41, 90)
        most = 4.0 if fp32 else 60.0
    else:
        chans, templates, model, fs = rng.randint(4, 32), rng.randint(2, 40), "dense", rng.choice([30000, 40000])
        length = rng.randint(31, 101)
        if rng.random() < 0.5:
            model, length = "probe", rng.randint(61, 101)
        most = 20.0 if fp32 else 60.0
    seconds = round(_log_uniform(rng, 0.15, most), 4)
    # adjusted clips of a call: whole clips on every channel, for the short stretches
    more["clips"] = kind == "call" and chans <= 32 and seconds < 2.0 and rng.random() < 0.5
    return _case("", kind, model, chans, seconds, fs, templates, length, **more)


def _autocov(fs, L, f_lo=300.0, f_hi=8000.0):
    """Autocovariance at lags 0..L-1 of unit-variance noise that is flat
    between f_lo and f_hi."""
    lag = np.arange(L) / fs
    with np.errstate(invalid="ignore", divide="ignore"):
        r = (np.sin(2 * np.pi * f_hi * lag) - np.sin(2 * np.pi * f_lo * lag)) / (2 * np.pi * lag * (f_hi - f_lo))
    r[0] = 1.0
    return r


def _templates(rng, case):
    """[K, C, L] in noise SD."""
    C, K, L = case["chans"], case["templates"], case["length"]
    align = int(round(0.4 * (L - 1)))
    T = np.zeros((K, C, L))
    taper = np.exp(-0.5 * ((np.arange(L) - align) / (0.3 * L)) ** 2)
    for k in range(K):
        shape = synthetic.biphasic_waveform(rng, L, align)
        if case["model"] == "masked":
            lo = int(rng.integers(0, C - 16 + 1))
            chans = np.arange(lo, lo + 16)
            gain = np.exp(-np.abs(chans - (lo + rng.integers(16))) / 4.0)
            amp = 6.0 * np.exp(0.35 * rng.standard_normal())
        elif case["model"] == "probe":
            chans = np.arange(C)
            gain = np.exp(-np.abs(chans - rng.integers(C)) / 2.0)
            amp = rng.uniform(3.0, 10.0)
        else:
            chans = np.arange(C)
            gain = rng.uniform(0.15, 1.0, C)
            gain[rng.integers(C)] = 1.0
            amp = rng.uniform(3.0, 10.0)
        jitter = 1.0 + 0.1 * rng.standard_normal((len(chans), L)) * taper
        T[k, chans] = amp * gain[:, None] * shape * jitter
    return T


def _noise(gen, rows, n, fs, dev):
    """Band-limited unit-variance noise, [rows, n]."""
    step = 1 << 17
    nfft = 1 << max(10, (n - 1).bit_length()) if n < (1 << 20) else (n + step - 1) // step * step
    f = torch.fft.rfftfreq(nfft, 1.0 / fs, device=dev)
    keep = ((f >= 300.0) & (f <= 8000.0)).to(torch.float32)
    scale = math.sqrt(nfft / max(1.0, 2.0 * float(keep.sum())))
    x = torch.randn((rows, nfft), generator=gen, device=dev)
    return torch.fft.irfft(torch.fft.rfft(x, dim=1) * (keep * scale), n=nfft, dim=1)[:, :n]


def _recording(case, seed):
    """(voltage [C, n] on the GPU, templates [K, C*L] float32, metrics,
    sort_info, spike starts per unit) of a case and a seed."""
    dev = torch.device("cuda", torch.cuda.current_device())
    rng = np.random.Generator(np.random.PCG64(seed))
    gen = torch.Generator(device=dev)
    gen.manual_seed(int(seed))
    C, K, L, fs = case["chans"], case["templates"], case["length"], case["fs"]
    n = int(round(case["seconds"] * fs))
    T = _templates(rng, case)
    quanta = torch.from_numpy(np.rint(T * QUANTUM).astype(np.int32)).to(dev)
    if case["model"] == "masked":
        rates = rng.uniform(0.5, 100.0, K)
    elif case["model"] == "probe":
        rates = rng.uniform(1.0, 80.0, K)
    else:
        rates = rng.uniform(5.0, 50.0, K)
    starts = []
    for k in range(K):
        s = synthetic.poisson_train(rng, rates[k], n, fs) - int(round(0.4 * (L - 1)))
        s = s[(s >= 0) & (s + L <= n)]
        if case["model"] == "probe" and k > 0 and s.size and starts[k - 1].size:
            # one spike in seven onto a spike of the unit before it, within a millisecond
            m = s.size // 7
            pick = rng.choice(s.size, m, replace=False)
            s[pick] = rng.choice(starts[k - 1], m) + rng.integers(-int(1e-3 * fs), int(1e-3 * fs) + 1, m)
            s = np.unique(np.clip(s, 0, n - L))
        starts.append(s)
    is_int = case["dtype"] == "int16"
    voltage = torch.empty((C, n), dtype=torch.int16 if is_int else torch.float32, device=dev)
    lags = torch.arange(L, device=dev)
    where = [torch.from_numpy(s).to(dev) for s in starts]
    for c0 in range(0, C, 16):
        c1 = min(C, c0 + 16)
        acc = torch.zeros((c1 - c0) * n, dtype=torch.int32, device=dev)
        for k in range(K):
            chans = np.nonzero(np.any(T[k, c0:c1] != 0, axis=1))[0]
            if chans.size == 0 or starts[k].size == 0:
                continue
            lo, hi = int(chans[0]), int(chans[-1]) + 1
            rows = torch.arange(lo, hi, device=dev)
            at = (where[k][:, None, None] + rows[None, :, None] * n + lags).reshape(-1)
            acc.index_add_(0, at, quanta[k, c0 + lo:c0 + hi].expand(where[k].numel(), hi - lo, L).reshape(-1))
        x = _noise(gen, c1 - c0, n, fs, dev) + acc.view(c1 - c0, n) * (1.0 / QUANTUM)
        voltage[c0:c1] = torch.clamp(torch.round(x * INT16_SCALE), -32768, 32767).to(torch.int16) if is_int else x
        del x, acc
    sd = INT16_SCALE if is_int else 1.0
    cov = _autocov(fs, L)[np.abs(np.subtract.outer(np.arange(L), np.arange(L)))] * sd * sd
    templates = (T * sd).astype(np.float32).reshape(K, C * L)
    t64 = templates.astype(np.float64)
    SS = np.sum(t64 ** 2, axis=1)
    rows = t64.reshape(K * C, L)
    var = np.sum((rows @ cov) * rows, axis=1).reshape(K, C).sum(axis=1)
    lower_ci = 0.5 * SS - 4.0 * np.sqrt(var)
    metrics = {"bp_n_samples_per_chan": L, "templates": templates, "template_SS": SS, "neuron_variances": var,
               "neuron_lower_CI": lower_ci,
               "neuron_lower_thresholds": np.maximum(np.maximum(-0.5 * SS + 1.645 * np.sqrt(var), 0.0), lower_ci)}
    info = {"sampling_rate": float(fs), "clip_width": synthetic.clip_width_for(L, 0.4, fs), "n_samples_per_chan": L,
            "n_channels": C, "n_samples": n, "do_overlap_recheck": bool(case["overlap"]),
            "get_adjusted_clips": bool(case["clips"]), "sigma_bp_noise": 1.645, "sigma_bp_CI": 4.0}
    return voltage, templates, metrics, info, starts


def _shift(case):
    return case["length"] - 1 if case["production_shift"] else None


def _batch_cases(case):
    """The batch's segments: uneven sizes up to the case's own."""
    rng = np.random.Generator(np.random.PCG64(case["segments"] * 1009 + case["chans"]))
    out = []
    for i in range(case["segments"]):
        out.append(dict(case, kind="call", chans=int(rng.integers(4, max(5, case["chans"] + 1))),
                        seconds=float(case["seconds"] * rng.uniform(0.05, 1.0)),
                        templates=int(rng.integers(2, max(3, case["templates"] + 1))),
                        length=int(rng.integers(61, max(62, case["length"] + 1)))))
    return out


def _zca_thresholds(voltage, case):
    """Six noise SD, the multiple at which the reference looks for spikes."""
    sd = INT16_SCALE if case["dtype"] == "int16" else 1.0
    return np.full(voltage.shape[0], 6.0 * sd)


def _cov_rows(starts, window, n):
    """Rows of the clip matrix that the covariance is taken over: 20,000 of
    them with replacement, or all when there are no more."""
    total = sum(int(np.sum((s >= 0) & (s + window < n))) for s in starts)
    if total <= 20000:
        return np.arange(total, dtype=np.int64)
    return np.random.Generator(np.random.PCG64(11)).integers(0, total, 20000).astype(np.int64)


_SERVER = []


def _server():
    """The program's server."""
    if not _SERVER:
        from spikesorting_fullpursuit_b200.serving import PursuitServer
        _SERVER.append(PursuitServer(slots=4))
    return _SERVER[0]


def prepare(case, seed):
    kind = case["kind"]
    if kind == "batch":
        segments = []
        for i, c in enumerate(_batch_cases(case)):
            v, _, metrics, info, _ = _recording(c, seed * 131 + i)
            segments.append((v.cpu().numpy(), info, metrics, _shift(c)))
        return {"case": case, "segments": segments, "server": _server(),
                "trains": [_empty_trains(c, s[0], False) for c, s in zip(_batch_cases(case), segments)]}
    voltage, templates, metrics, info, starts = _recording(case, seed)
    state = {"case": case, "info": info, "metrics": metrics}
    if kind == "call":
        state["voltage"] = voltage.cpu().numpy()
        state["trains"] = _empty_trains(case, voltage, case["clips"])
    elif kind == "chunk":
        dev = voltage.device
        L, K, n = case["length"], case["templates"], int(voltage.shape[1])
        nmax = _shift(case)
        nmax = L // 2 if nmax is None else nmax
        precision = _lib.PREC_FP32 if case["precision"] == "fp32" else _lib.PREC_BF16_REFINE
        size = ctypes.c_size_t(0)
        _lib.check(_lib.lib().fbp_pursuit_workspace_bytes(n, case["chans"], K, L, nmax, precision,
                                                          ctypes.byref(size)))
        cap = _spike_room(case, n)
        state.update(
            recording=voltage.to(torch.float32), precision=precision, nmax=nmax, cap=cap,
            templates=torch.from_numpy(templates).to(dev),
            tss=torch.from_numpy(np.float32(-0.5 * metrics["template_SS"])).to(dev),
            thr=torch.from_numpy(np.float32(metrics["neuron_lower_thresholds"])).to(dev),
            workspace=torch.empty(size.value, dtype=torch.uint8, device=dev),
            idx=torch.zeros(cap, dtype=torch.int32, device=dev), lab=torch.zeros(cap, dtype=torch.int32, device=dev))
        state["residual"] = torch.empty_like(state["recording"])
    elif kind == "inputs":
        align = -synthetic.clip_width_for(case["length"], 0.4, case["fs"])[0] * case["fs"]
        state["voltage"] = voltage
        state["events"] = [s + int(round(align)) for s in starts if s.size > 1]
        state["cov_rows"] = _cov_rows([s for s in starts if s.size > 1], case["length"], int(voltage.shape[1]))
        info["n_threshold_crossings"] = np.full(case["chans"], 100, dtype=np.int64)
    elif kind == "whiten":
        state["voltage"] = voltage
        state["thresholds"] = _zca_thresholds(voltage, case)
    return state


def _spike_room(case, n):
    return 32 * ((n + case["length"] - 1) // case["length"]) + 4096


def _empty_trains(case, voltage, clips):
    """The program's own arrays for a pursuit's spike train: [room] events and
    labels, zero past the last spike, and clips."""
    n = int(voltage.shape[1])
    room = _spike_room(case, n)
    out = {"events": np.zeros(room, np.int64), "labels": np.zeros(room, np.int64)}
    if clips:
        most = 8 * ((n + case["length"] - 1) // case["length"]) + 64
        out["clips"] = np.zeros((most, case["chans"] * case["length"]), np.dtype(case["dtype"]))
    return out


def _keep(result, into):
    """Append the 4-tuple of a pursuit to the program's arrays."""
    events, labels, _, clips = result
    m = len(events)
    into["events"][:m] = events
    into["labels"][:m] = labels
    if "clips" in into and m:
        into["clips"][:m] = clips
    return into


def run(state):
    from spikesorting_fullpursuit_b200 import binary_pursuit
    case = state["case"]
    kind = case["kind"]
    if kind == "call":
        v = state["voltage"]
        return _keep(binary_pursuit(v, v.dtype, state["info"], state["metrics"], n_max_shift_inds=_shift(case),
                                    precision=case["precision"]), state["trains"])
    if kind == "chunk":
        v = state["residual"]
        v.copy_(state["recording"])                  # the pursuit turns its voltage into the residual
        found, passes = ctypes.c_uint32(0), ctypes.c_uint32(0)
        stream = _lib.stream_ptr(torch.cuda.current_stream(v.device))
        p = _lib.ptr
        _lib.check(_lib.lib().fbp_pursuit_chunk(
            p(v), int(v.shape[1]), case["chans"], p(state["templates"]), case["templates"], case["length"],
            p(state["tss"]), p(state["thr"]), state["nmax"], int(case["overlap"]), state["precision"],
            _lib.OVERLAP_FAST, 1000000, p(state["workspace"]), state["workspace"].numel(), p(state["idx"]),
            p(state["lab"]), state["cap"], None, ctypes.byref(found), ctypes.byref(passes), 0, None, stream))
        return {"events": state["idx"], "labels": state["lab"], "spikes": int(found.value), "residual": v,
                "passes": int(passes.value)}
    if kind == "batch":
        futures = [state["server"].submit(*segment) for segment in state["segments"]]
        return [_keep(f.result().outputs, t) for f, t in zip(futures, state["trains"])]
    if kind == "inputs":
        from spikesorting_fullpursuit_b200.full_binary_pursuit import pursuit_templates_and_covariance
        from spikesorting_fullpursuit_b200.neuron_separability import compute_separability_metrics, set_bp_threshold
        info = state["info"]
        templates, cov = pursuit_templates_and_covariance(
            state["voltage"], state["events"], info["sampling_rate"], info["clip_width"], len(state["cov_rows"]),
            cov_sample_inds=state["cov_rows"])
        m = set_bp_threshold(compute_separability_metrics(templates, cov, info))
        return {"templates": templates, "covariance": np.stack(cov), "SS": m["template_SS"],
                "variances": m["neuron_variances"], "thresholds": m["neuron_lower_thresholds"]}
    from spikesorting_fullpursuit_b200.preprocessing import get_noise_sampled_zca_matrix, zca_apply
    Z = get_noise_sampled_zca_matrix(state["voltage"], state["thresholds"], 4.0, case["length"])
    return {"matrix": Z, "whitened": zca_apply(Z, state["voltage"], as_tensor=True)}


def work(case):
    if case["kind"] == "batch":
        parts = [work(c) for c in _batch_cases(case)]
        return {k: sum(p[k] for p in parts) for k in ("bytes", "flops")}
    C, K, L = case["chans"], case["templates"], case["length"]
    n = int(round(case["seconds"] * case["fs"]))
    item = 2 if case["dtype"] == "int16" else 4
    on = 16 if case["model"] == "masked" else C
    if case["kind"] == "call":          # the recording in; one likelihood of every sample and template
        return {"bytes": item * C * n, "flops": 2.0 * on * L * K * n}
    if case["kind"] == "chunk":         # the recording in, the residual out
        return {"bytes": 8 * C * n, "flops": 2.0 * on * L * K * n}
    if case["kind"] == "inputs":        # the recording in; the covariance products of the chosen rows
        return {"bytes": item * C * n, "flops": 2.0 * 20000 * C * L * L}
    return {"bytes": 2 * item * C * n, "flops": 3.0 * C * C * n}      # covariance (half of it) and product


def _exact_inputs(case, seed):
    voltage, _, _, info, starts = _recording(case, seed)
    v = voltage.double()
    C, L, n = case["chans"], case["length"], int(voltage.shape[1])
    starts = [s for s in starts if s.size > 1]
    lags = torch.arange(L, device=v.device)

    def median(x):                       # numpy's: the mean of the two middle values
        s = torch.sort(x, dim=0).values
        m = s.shape[0]
        return s[m // 2] if m % 2 else 0.5 * (s[m // 2 - 1] + s[m // 2])

    templates, resid = [], []
    for s in starts:
        s = s[(s >= 0) & (s + L < n)]
        at = torch.from_numpy(s).to(v.device)[:, None] + lags
        clips = v[:, at].permute(1, 0, 2).reshape(len(s), C * L)
        mid = median(clips)
        mad = median((clips - mid).abs()) / 0.6745
        far = (clips < mid - mad) | (clips > mid + mad)
        inside = torch.where(far, torch.full_like(clips, math.inf), clips)
        inside = torch.sort(inside, dim=0).values
        count = (~far).sum(dim=0)
        hi = torch.gather(inside, 0, (count // 2).clamp(max=len(s) - 1)[None])[0]
        lo = torch.gather(inside, 0, ((count - 1) // 2).clamp(min=0)[None])[0]
        t = torch.where(count > 0, 0.5 * (hi + lo), mid)
        templates.append(t)
        resid.append(clips - t)
    rows = torch.from_numpy(_cov_rows(starts, L, n)).to(v.device)
    x = torch.cat(resid)[rows].view(len(rows), C, L).permute(1, 2, 0)
    x = x - x.mean(dim=2, keepdim=True)
    cov = x @ x.transpose(1, 2) / len(rows)
    T = torch.stack(templates)
    SS = (T ** 2).sum(dim=1)
    Tc = T.view(len(templates), C, L)
    var = (torch.einsum("kcl,clm->kcm", Tc, cov) * Tc).sum(dim=(1, 2))
    thr = torch.maximum(torch.maximum(-0.5 * SS + 1.645 * var.sqrt(), torch.zeros_like(SS)), 0.5 * SS - 4.0 * var.sqrt())
    return {"templates": T.cpu().numpy(), "covariance": cov.cpu().numpy(), "SS": SS.cpu().numpy(),
            "variances": var.cpu().numpy(), "thresholds": thr.cpu().numpy()}


def _exact_whiten(case, seed):
    v = _recording(case, seed)[0]
    thr = torch.from_numpy(_zca_thresholds(v, case)).to(v.device)
    x = v.double()
    cushion = case["length"]
    over = (x.abs() > 0.9 * thr[:, None]).to(torch.float32)
    masked = torch.nn.functional.max_pool1d(over[:, None], 2 * cushion + 1, 1, cushion)[:, 0] > 0
    ok = (~masked).double()
    xm = x * ok
    sigma = (xm @ xm.T) / (ok @ ok.T - 1.0)
    count = ok.sum(dim=1)
    centred = (x - (xm.sum(dim=1) / count)[:, None]) * ok
    sigma[range(len(count)), range(len(count))] = (centred ** 2).sum(dim=1) / (count - 1.0)
    U, S, _ = np.linalg.svd(sigma.cpu().numpy())
    Z = U @ np.diag(1.0 / np.sqrt(S + 1e-9)) @ U.T
    Z = Z / np.diag(Z)[:, None]
    out = torch.from_numpy(Z).to(v.device) @ x
    return {"matrix": Z, "whitened": None if case["dtype"] == "int16" else out}


def exact(case, seed):
    """Float64 values of the computed numbers.  A pursuit's answer is its
    spikes, whole numbers; its residual and adjusted clips follow from the
    spikes by float32 subtractions in a fixed order."""
    if case["kind"] == "inputs":
        return _exact_inputs(case, seed)
    if case["kind"] == "whiten":
        return _exact_whiten(case, seed)
    return None
