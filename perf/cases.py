"""Timed cases of the framework: what its users have it do, through its public
entry points.

``listed()`` holds the cases, ``draw(rng)`` gives more of the same ranges,
``prepare`` makes what a program holds before the call (a configured
component, inputs on the GPU), ``run`` is one pass, ``work`` the bytes and
operations that pass cannot do without, and ``exact`` the same outputs in
64-bit torch arithmetic written out here from the formulas.

A case is a dict of plain values; its ``op`` says which entry point runs:

  forward   DepoTransform.forward_device   depos in HBM -> dense frame
  host      DepoTransform.__call__         pinned host depos -> pinned host frame
  fit       depo_transform + backward      frame, dL/d(depos), dL/d(DL, DT, lifetime)
  batch     DepoTransform.forward_batch_device  events in HBM -> frames
  splat     DepoTransform.splat_device     DepoFluxSplat truth frame
  readout   add_noise_device, Digitizer.device  noise on a frame, then its ADC values
  dft       dft_2d_device                  IDFT 2-D transform
"""

import importlib
import math

import numpy as np
import torch

PKG = "wire-cell-toolkit_b200"
wct = importlib.import_module(PKG)
synth = importlib.import_module(PKG + ".synth")

DEV = "cuda"
GEOM_ROWS = {"plane": 960, "apa": 2560}
GEOM_PLANES = {"plane": 1, "apa": 3}


def listed():
    return [
        # one collection plane, point depos: the smallest event, where launches and latency count
        {"name": "plane_2k", "op": "forward", "geom": "plane", "kind": "points", "n": 2000, "nticks": 6000,
         "fluct": False},
        # a few low-energy tracks in a full three-plane APA: the everyday event of a simulation job
        {"name": "apa_20k", "op": "forward", "geom": "apa", "kind": "tracks", "n": 20000, "nticks": 6000,
         "fluct": False},
        # 20 muons at one depo per 0.1 mm: the full-APA event
        {"name": "apa_520k", "op": "forward", "geom": "apa", "kind": "tracks", "n": 520000, "nticks": 6000,
         "fluct": False},
        # tracks with EM showers: patches up to 40 impacts x 200 ticks
        {"name": "apa_shower_200k", "op": "forward", "geom": "apa", "kind": "mixed", "n": 200000, "nticks": 6000,
         "fluct": False},
        # binomial fluctuation of patches and drift on, as production samples are made
        {"name": "apa_fluct_100k", "op": "forward", "geom": "apa", "kind": "tracks", "n": 100000, "nticks": 6000,
         "fluct": True},
        # the IDepoFramer call of a toolkit graph: host buffers in and out
        {"name": "apa_host_100k", "op": "host", "geom": "apa", "kind": "mixed", "n": 100000, "nticks": 6000,
         "fluct": False},
        # one step of a gradient fit of 20k track depos and the drift parameters
        {"name": "fit_20k", "op": "fit", "geom": "apa", "kind": "tracks", "n": 20000, "nticks": 6000},
        # one event's share of a large calibration step: cosmic muons and showers
        {"name": "fit_500k", "op": "fit", "geom": "apa", "kind": "calib", "n": 500000, "nticks": 6000},
        # events of very uneven size in one call
        {"name": "batch_16", "op": "batch", "geom": "apa", "nev": 16, "lo": 500, "hi": 200000, "nticks": 6000},
        # the truth frame that goes with a simulated event
        {"name": "splat_200k", "op": "splat", "geom": "apa", "kind": "mixed", "n": 200000, "nticks": 6000},
        # electronics noise and digitisation of a frame
        {"name": "readout_6000", "op": "readout", "nticks": 6000},
        # the IDFT plugin on an APA frame
        {"name": "dft_2560x6000", "op": "dft", "nrows": 2560, "ncols": 6000, "inverse": False},
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["forward", "forward", "forward", "host", "fit", "batch", "splat", "readout", "dft"])
    nticks = rng.randint(2000, 6000)
    if op == "forward":
        fluct = rng.random() < 0.25
        geom = rng.choice(["plane", "apa", "apa"])
        kind = "points" if geom == "plane" else rng.choice(["tracks", "mixed"])
        n = _logint(rng, 500, 60000 if fluct else 300000)
        return {"op": op, "geom": geom, "kind": kind, "n": n, "nticks": nticks, "fluct": fluct}
    if op == "host":
        return {"op": op, "geom": "apa", "kind": rng.choice(["tracks", "mixed"]), "n": _logint(rng, 1000, 200000),
                "nticks": nticks, "fluct": False}
    if op == "fit":
        return {"op": op, "geom": "apa", "kind": rng.choice(["tracks", "calib"]), "n": _logint(rng, 1000, 200000),
                "nticks": nticks}
    if op == "batch":
        lo = _logint(rng, 500, 5000)
        return {"op": op, "geom": "apa", "nev": rng.randint(2, 16), "lo": lo, "hi": _logint(rng, lo, 100000),
                "nticks": nticks}
    if op == "splat":
        return {"op": op, "geom": "apa", "kind": rng.choice(["tracks", "mixed"]), "n": _logint(rng, 1000, 200000),
                "nticks": nticks}
    if op == "readout":
        # record lengths with a 7-smooth half (the noise spectrum's length)
        return {"op": op, "nticks": rng.choice([2000, 2240, 2400, 2560, 3000, 3200, 3584, 3840, 4096, 4480, 4800, 5120,
                                                 5376, 5600, 5760])}
    # lengths with large prime factors among them
    return {"op": op, "nrows": _logint(rng, 200, 2560), "ncols": _logint(rng, 500, 6000),
            "inverse": rng.random() < 0.5}


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _config(case, seed):
    cfg = (synth.plane1_config if case["geom"] == "plane" else synth.apa_config)(nticks=case["nticks"])
    if case.get("fluct"):
        cfg["fluctuate"] = True
        cfg["seed"] = int(seed)
        cfg["drifter"]["fluctuate"] = True
    return cfg


def _tracks(n, seed, ntracks=20):
    """Straight muon tracks with uniform endpoints, stepped so that they hold n depos."""
    lo = np.array((synth.RESPONSE_X, -3000.0, -1150.0))
    hi = np.array((synth.RESPONSE_X + 2500.0, 3000.0, 1150.0))
    length = 0.0
    for k in range(ntracks):
        rng = np.random.default_rng([seed, k])
        a, b = rng.random(3), rng.random(3)
        length += float(np.linalg.norm((hi - lo) * (b - a)))
    step = length / (n + 2 * ntracks)
    return np.concatenate([synth.track_depos(np.random.default_rng([seed, k]), ntracks=1, step=step, lo=lo, hi=hi)
                           for k in range(ntracks)])[:n]


def _depos(kind, n, seed):
    if kind == "points":
        return synth.plane1_depos(n=n, seed=seed)
    if kind == "tracks":
        return _tracks(n, seed)
    if kind == "calib":
        return synth.calibration_events(1, n, seed=seed)[0]
    return synth.batch_events(1, seed=seed, lo=n, hi=n)[0]


def _events(case, seed):
    return synth.batch_events(case["nev"], seed=seed, lo=case["lo"], hi=case["hi"])


def _fit_inputs(case, seed):
    """float32 leaves of a fit, and the data frame that it is fitted to: noise
    of about 500 electrons (the first step of a fit, the residual as large as
    the signal)."""
    d = torch.from_numpy(_depos(case["kind"], case["n"], seed)).to(DEV).float()
    p = torch.tensor([synth.DRIFT["DL"], synth.DRIFT["DT"], synth.DRIFT["lifetime"]], dtype=torch.float32)
    g = torch.Generator(device=DEV).manual_seed(seed)
    data = torch.randn((GEOM_ROWS[case["geom"]], case["nticks"]), generator=g, device=DEV) * 1e-9
    return d, p, data


SPLAT = dict(tick=synth.TICK, nsigma=3.0, drift_speed=1.6 * synth.mm / synth.us, response_plane=synth.RESPONSE_X,
             smear_long=[3.0, 3.0, 3.0], smear_tran=[0.5, 0.5, 0.5])


def _splat_inputs(case, seed):
    """Drifted depos: at the response plane, with the arrival time and widths
    of their drift."""
    d = _depos(case["kind"], case["n"], seed).copy()
    dt = (d[:, 2] - synth.RESPONSE_X) / synth.DRIFT["drift_speed"]
    d[:, 0] += dt
    d[:, 1] *= np.exp(-dt / synth.DRIFT["lifetime"])
    d[:, 5] = np.sqrt(2 * synth.DRIFT["DL"] * dt + d[:, 5] ** 2)
    d[:, 6] = np.sqrt(2 * synth.DRIFT["DT"] * dt + d[:, 6] ** 2)
    d[:, 2] = synth.RESPONSE_X
    cfg = dict(SPLAT, window_start=0.0, window_duration=case["nticks"] * synth.TICK)
    return d, cfg


READOUT_ROWS = (800, 800, 960)
READOUT_SPECTRA = 10


def _readout_inputs(case, seed):
    """A frame with some signal, ten amplitude spectra (falling with frequency,
    growing with wire length, about 1 mV), the row -> spectrum map."""
    n, rows = case["nticks"], sum(READOUT_ROWS)
    g = torch.Generator(device=DEV).manual_seed(seed)
    frame = torch.randn((rows, n), generator=g, device=DEV) * 5e-9
    f = torch.arange(n, device=DEV, dtype=torch.float32)
    f = torch.minimum(f, n - f) / n
    shape = (f + 0.02) / (0.02 + 40 * f * f)
    amp = torch.linspace(0.5, 1.5, READOUT_SPECTRA, device=DEV)[:, None] * shape[None, :] * 1e-9 * math.sqrt(n)
    spec = torch.randint(0, READOUT_SPECTRA, (rows,), generator=g, device=DEV, dtype=torch.int32)
    chan = torch.arange(rows, device=DEV, dtype=torch.int32)
    return frame, amp.contiguous(), spec, chan


def _dft_input(case, seed):
    g = torch.Generator(device=DEV).manual_seed(seed)
    re, im = (torch.randn((case["nrows"], case["ncols"]), generator=g, device=DEV) for _ in range(2))
    return torch.complex(re, im)


# ---------------------------------------------------------------------------
# the calls
# ---------------------------------------------------------------------------
def _stream():
    """torch's current stream; its default stream by the explicit handle (0
    would select a component's own stream in some of the entry points)."""
    return torch.cuda.current_stream().cuda_stream or wct.CUDA_STREAM_LEGACY


def prepare(case, seed):
    op = case["op"]
    s = {"case": case}
    if op in ("forward", "host", "fit", "batch", "splat"):
        s["dt"] = wct.from_config(_config(case, seed), device=0)
    rows = GEOM_ROWS.get(case.get("geom"))
    if op == "forward":
        s["depos"] = torch.from_numpy(_depos(case["kind"], case["n"], seed)).to(DEV)
        s["frame"] = torch.empty((rows, case["nticks"]), dtype=torch.float32, device=DEV)
    elif op == "host":
        s["pin"] = torch.from_numpy(_depos(case["kind"], case["n"], seed)).pin_memory()
        s["depos"] = s["pin"].numpy()
        s["out"] = torch.empty((rows, case["nticks"]), dtype=torch.float32, pin_memory=True).numpy()
    elif op == "fit":
        s["depos"], s["params"], s["data"] = _fit_inputs(case, seed)
    elif op == "batch":
        ev = _events(case, seed)
        s["offsets"] = np.concatenate([[0], np.cumsum([len(e) for e in ev])]).astype(np.int64)
        s["depos"] = torch.from_numpy(np.concatenate(ev)).to(DEV)
        s["frames"] = torch.empty((len(ev), rows, case["nticks"]), dtype=torch.float32, device=DEV)
    elif op == "splat":
        d, s["cfg"] = _splat_inputs(case, seed)
        s["depos"] = torch.from_numpy(d).to(DEV)
        s["frame"] = torch.empty(s["dt"].splat_shape(**s["cfg"]), dtype=torch.float32, device=DEV)
    elif op == "readout":
        s["frame"], s["spectra"], s["spec"], s["chan"] = _readout_inputs(case, seed)
        s["adc"] = torch.empty_like(s["frame"])
        s["digitizer"] = wct.Digitizer(READOUT_ROWS)
        s["baseline"] = torch.from_numpy(s["digitizer"].row_baseline).to(DEV)
        s["event"] = 0
    else:
        s["x"] = _dft_input(case, seed)
        s["y"] = torch.empty_like(s["x"])
    return s


def run(s):
    case = s["case"]
    op = case["op"]
    if op == "forward":
        s["dt"].forward_device(s["depos"].data_ptr(), s["depos"].shape[0], s["frame"].data_ptr(), stream=_stream())
        return s["frame"]
    if op == "host":
        frame, _, _ = s["dt"](s["depos"], out=s["out"])
        return frame
    if op == "fit":
        d = s["depos"].detach().requires_grad_(True)
        p = s["params"].detach().requires_grad_(True)
        frame = wct.depo_transform(s["dt"], d.double(), p.double())
        ((frame - s["data"]) ** 2).sum().backward()
        return frame.detach(), d.grad, p.grad
    if op == "batch":
        s["dt"].forward_batch_device(s["depos"].data_ptr(), s["offsets"], s["frames"].data_ptr(), stream=_stream())
        return s["frames"]
    if op == "splat":
        s["dt"].splat_device(s["depos"].data_ptr(), s["depos"].shape[0], s["frame"].data_ptr(), stream=_stream(),
                             **s["cfg"])
        return s["frame"]
    if op == "readout":
        f = s["frame"]
        rows, n = f.shape
        wct.add_noise_device(f.data_ptr(), n, rows, n, s["spectra"].data_ptr(), n, s["spec"].data_ptr(),
                             s["chan"].data_ptr(), seed=7, ident=s["event"], model=0, stream=_stream())
        s["digitizer"].device(f.data_ptr(), n, rows, n, s["baseline"].data_ptr(), s["adc"].data_ptr(), n,
                              stream=_stream())
        s["event"] += 1
        return f, s["adc"]
    wct.dft_2d_device(s["x"].data_ptr(), s["y"].data_ptr(), case["nrows"], case["ncols"], inverse=case["inverse"],
                      stream=_stream())
    return s["y"]


def work(case):
    """Inputs read once, outputs written once; the operations of the patches
    (about 150 cells a plane, two groups a cell), of one real transform of the
    charge and the frame, and of the transforms themselves."""
    op = case["op"]
    if op == "dft":
        m = case["nrows"] * case["ncols"]
        return {"bytes": 16 * m, "flops": 5 * m * math.log2(m)}
    if op == "readout":
        m = sum(READOUT_ROWS) * case["nticks"]
        return {"bytes": 12 * m, "flops": 2.5 * m * math.log2(case["nticks"])}
    frame = GEOM_ROWS[case["geom"]] * case["nticks"]
    if op == "batch":
        r = math.log(case["hi"] / case["lo"]) if case["hi"] > case["lo"] else 0.0
        n = case["nev"] * ((case["hi"] - case["lo"]) / r if r else case["lo"])
        frame *= case["nev"]
    else:
        n = case["n"]
    patches = 600.0 * n * GEOM_PLANES[case["geom"]]
    if op == "splat":
        return {"bytes": 56 * n + 4 * frame, "flops": patches / 10}
    fft = 5.0 * frame * math.log2(max(2, case["nticks"]))
    if op == "fit":
        return {"bytes": 2 * 28 * n + 8 * frame, "flops": 3 * (patches + fft)}
    return {"bytes": 56 * n + 4 * frame, "flops": patches + fft}


# ---------------------------------------------------------------------------
# the same in 64 bits
# ---------------------------------------------------------------------------
SQ2 = math.sqrt(2.0)
SQ2PI = math.sqrt(2.0 * math.pi)
CHUNK_CELLS = 12_000_000
FAST_LENGTHS = (33, 35, 40, 42, 44, 56, 64, 66, 70, 77, 80, 96, 98, 100, 112, 121, 128, 140, 143, 160, 168, 169, 200)


def _cdf(u):
    return 0.5 * torch.special.erfc(-u / SQ2)


def _pdf(u):
    return torch.exp(-0.5 * u * u) / SQ2PI


def _drift(d, dr, params):
    """Drifted (t, q, x, y, z, sigma_L, sigma_T) of depos between response plane
    and cathode (x outside it: dropped, as a zero charge)."""
    DL, DT, life = params
    _, resp, cath = dr["xregions"][0]
    ok = (d[:, 2] > resp) & (d[:, 2] < cath)
    dt = ((resp - d[:, 2]) / dr["drift_speed"]).abs()
    q = d[:, 1] - d[:, 1] * (1.0 - torch.exp(-dt / life))
    sL = torch.sqrt(2.0 * DL * dt + d[:, 5] * d[:, 5])
    sT = torch.sqrt(2.0 * DT * dt + d[:, 6] * d[:, 6])
    return d[:, 0] + dt, q, torch.full_like(q, resp), d[:, 3], d[:, 4], sL, sT, ok


def _bins(c, s, lo, hi, nbins, nsigma):
    """(inside, first bin, bins) of a Gaussian on a binning."""
    bs = (hi - lo) / nbins
    inside = ((lo - c) / s <= nsigma) & ((hi - c) / s >= -nsigma)
    b0 = ((c - s * nsigma - lo) / bs).trunc().long().clamp(min=0)
    b1 = (((c + s * nsigma - lo) / bs).trunc().long() + 1).clamp(max=nbins)
    return inside & (b1 > b0), b0, b1 - b0


def _edges(b0, nmax, c, lo, bs):
    """Bin edges from the centre, [n][nmax + 1]."""
    k = torch.arange(nmax + 1, device=c.device)
    return lo + (b0[:, None] + k[None, :]).double() * bs - c[:, None]


class _Plane:
    def __init__(self, cfg, ip):
        pl = cfg["planes"][ip]
        self.nw, self.nimp = pl["nwires"], pl["nimp"]
        region = (pl["pitchmax"] - pl["pitchmin"]) / (self.nw - 1)
        self.lo, self.hi = pl["pitchmin"] - 0.5 * region, pl["pitchmax"] + 0.5 * region
        self.nbins = self.nw * self.nimp
        self.bs = (self.hi - self.lo) / self.nbins
        a = np.array(pl["pitch"], dtype=np.float64)
        self.axis = (a / math.sqrt(float(a @ a))).tolist()
        self.origin = [float(v) for v in pl["origin"]]
        self.G = self.nimp + 1
        self.K = self._response(cfg, cfg["fr"][ip])
        self.npad = (self.K.shape[1] - 1) // 2

    def _response(self, cfg, fr):
        """[group][wire offset + npad][tick]: field response binned on ticks,
        circularly convolved with the electronics over the short window."""
        ns = int(cfg["overall_short_padding"] / cfg["tick"])
        ns = next(v for v in FAST_LENGTHS if v >= ns)
        cur, pos, pitch = np.asarray(fr["current"]), np.asarray(fr["pitchpos"]), fr["pitch"]
        bins = ((fr["tstart"] + (np.arange(cur.shape[1]) + 0.5) * fr["period"]) / cfg["tick"]).astype(int)
        wave = np.zeros((cur.shape[0], ns))
        for b in range(ns):
            wave[:, b] = cur[:, bins == b].sum(axis=1) * fr["period"]
        spec = np.fft.fft(wave, axis=1)
        for e in cfg["short_responses"]:
            w = np.zeros(ns)
            w[:min(ns, len(e))] = e[:ns]
            spec = spec * np.fft.fft(w)[None, :]
        wave = np.real(np.fft.ifft(spec, axis=1)).astype(np.float32).astype(np.float64)  # a response is float data
        half = cur.shape[0] // 6 // 2
        # six paths a wire region, half a pitch below the wire up to it; the other half mirrored
        byw = {}
        for i, p in enumerate(pos):
            byw.setdefault(int(math.ceil((p - 1e-15 * pitch) / pitch)), []).append(i)
        rows = [byw[r] + byw[-r][::-1][1:] for r in range(-half, half + 1)]
        K = np.zeros((self.G, 2 * half + 1, ns))
        for g in range(self.G):
            for j in range(2 * half + 1):  # the charge on group g of a wire seen by the wire j - half above it
                K[g, j] = wave[rows[half - (j - half)][g]]
        return torch.from_numpy(K).to(DEV)


def _centre(P, cfg, drifted):
    """Pitch coordinate and time width of drifted depos on plane P."""
    _, _, x, y, z, sL, _, _ = drifted
    c = P.axis[0] * (x - P.origin[0]) + P.axis[1] * (y - P.origin[1]) + P.axis[2] * (z - P.origin[2])
    return c, sL / cfg["drift_speed"]


def _windows(P, cfg, drifted, nticks):
    t, q, x, y, z, sL, sT, ok = drifted
    c, st = _centre(P, cfg, drifted)
    tin, t0, nt = _bins(t, st, cfg["start_time"], cfg["start_time"] + cfg["readout_time"], nticks, cfg["nsigma"])
    pin, p0, npp = _bins(c, sT, P.lo, P.hi, P.nbins, cfg["nsigma"])
    if "face_bb" in cfg:
        for v, lo, hi in zip((x, y, z), cfg["face_bb"][0], cfg["face_bb"][1]):
            ok = ok & (v >= lo) & (v <= hi)
    return ok & tin & pin, t0, nt, p0, npp


def _cells(P, cfg, drifted, win, T, K, nticks):
    """Charge of the cells of depos with at most T ticks and K impacts: (flat
    index of the lower group's cell in [G][nw][nticks], lower, upper), masked
    cells at index 0 with zero charge."""
    t, q, x, y, z, sL, sT, _ = drifted
    t0, nt, p0, npp = win
    c, st = _centre(P, cfg, drifted)
    tbs = cfg["readout_time"] / nticks
    te = _edges(t0, T, t, cfg["start_time"], tbs) / st[:, None]
    pe = _edges(p0, K, c, P.lo, P.bs)
    u = pe / sT[:, None]
    tm = torch.arange(T, device=t.device)[None, :] < nt[:, None]
    pm = torch.arange(K, device=t.device)[None, :] < npp[:, None]
    # differences on the side of the centre that the bin lies on (no cancellation in the tails)
    F = torch.where(te[:, :-1] > 0, _cdf(-te[:, :-1]) - _cdf(-te[:, 1:]), _cdf(te[:, 1:]) - _cdf(te[:, :-1])) * tm
    p = torch.where(u[:, :-1] > 0, _cdf(-u[:, :-1]) - _cdf(-u[:, 1:]), _cdf(u[:, 1:]) - _cdf(u[:, :-1])) * pm
    f = _pdf(u)
    a = (sT[:, None] * (f[:, 1:] - f[:, :-1]) + pe[:, 1:] * p) / P.bs * pm
    qn = q / (F.sum(1) * p.sum(1))
    tq = F * qn[:, None]
    k = p0[:, None] + torch.arange(K, device=t.device)[None, :]
    w = torch.div(k, P.nimp, rounding_mode="floor")
    cell = ((k - w * P.nimp) * P.nw + w)[:, :, None] * nticks + (t0[:, None] + torch.arange(T, device=t.device))[:, None, :]
    cell = torch.where(pm[:, :, None] & tm[:, None, :], cell, torch.zeros_like(cell))
    return cell, a[:, :, None] * tq[:, None, :], (p - a)[:, :, None] * tq[:, None, :]


def _chunks(nt, npp, sel):
    """Index ranges of `sel`, ordered by patch size, with the padded size of each."""
    order = sel[torch.argsort(nt[sel] * 4096 + npp[sel])]
    i, nt, npp = 0, nt[order].cpu().numpy(), npp[order].cpu().numpy()
    while i < len(nt):
        j, T, K = i, 1, 1
        while j < len(nt):
            m = min(len(nt), j + 256)
            T2, K2 = max(T, int(nt[j:m].max())), max(K, int(npp[j:m].max()))
            if j > i and T2 * K2 * (m - i) > CHUNK_CELLS:
                break
            T, K, j = T2, K2, m
        yield order[i:j], T, K
        i = j


def _take(drifted, idx):
    return tuple(v[idx] for v in drifted)


def _grid(P, cfg, drifted, nticks):
    ok, t0, nt, p0, npp = _windows(P, cfg, drifted, nticks)
    Q = torch.zeros(P.G * P.nw * nticks, dtype=torch.float64, device=DEV)
    up = P.nw * nticks
    for idx, T, K in _chunks(nt, npp, ok.nonzero()[:, 0]):
        cell, lo, hi = _cells(P, cfg, _take(drifted, idx), (t0[idx], nt[idx], p0[idx], npp[idx]), T, K, nticks)
        Q.index_add_(0, cell.reshape(-1), lo.reshape(-1))
        Q.index_add_(0, cell.reshape(-1) + up, hi.reshape(-1))
    return Q.view(P.G, P.nw, nticks)


def _sizes(P, nticks):
    return P.nw + 2 * P.npad, nticks + P.K.shape[2]


def _convolve(P, Q, nticks):
    """Frame of a plane: the linear convolution of every group with its responses."""
    n = _sizes(P, nticks)
    acc = sum(torch.fft.rfft2(Q[g], s=n) * torch.fft.rfft2(P.K[g], s=n) for g in range(P.G))
    return torch.fft.irfft2(acc, s=n)[P.npad:P.npad + P.nw, :nticks]


def _correlate(P, gF, nticks):
    """The transpose: dL/dQ of a frame gradient."""
    n = _sizes(P, nticks)
    pad = torch.zeros((P.nw + 2 * P.npad, nticks), dtype=torch.float64, device=DEV)
    pad[P.npad:P.npad + P.nw] = gF
    G = torch.fft.rfft2(pad, s=n)
    return torch.stack([torch.fft.irfft2(G * torch.fft.rfft2(P.K[g], s=n).conj(), s=n)[:P.nw, :nticks]
                        for g in range(P.G)])


def _params(cfg):
    return tuple(cfg["drifter"][k] for k in ("DL", "DT", "lifetime"))


def _frame(cfg, d, params):
    nticks = int(cfg["readout_time"] / cfg["tick"])
    drifted = _drift(d, cfg["drifter"], params)
    out = []
    for ip in range(len(cfg["planes"])):
        P = _Plane(cfg, ip)
        out.append(_convolve(P, _grid(P, cfg, drifted, nticks), nticks))
    return torch.cat(out)


def _exact_fit(case, seed):
    cfg = _config(case, seed)
    nticks = case["nticks"]
    d, p, data = _fit_inputs(case, seed)
    d, p = d.double(), p.double().to(DEV)
    frame = _frame(cfg, d, tuple(p))
    gF = 2.0 * (frame - data.double())
    gd, gp = torch.zeros_like(d), torch.zeros_like(p)
    drifted = _drift(d, cfg["drifter"], tuple(p))
    row = 0
    for ip in range(len(cfg["planes"])):
        P = _Plane(cfg, ip)
        dQ = _correlate(P, gF[row:row + P.nw], nticks).reshape(-1)
        row += P.nw
        ok, t0, nt, p0, npp = _windows(P, cfg, drifted, nticks)
        up = P.nw * nticks
        for idx, T, K in _chunks(nt, npp, ok.nonzero()[:, 0]):
            for part in idx.split(max(1, len(idx) // 4 + 1)):
                x = d[part].requires_grad_(True)
                q = p.clone().requires_grad_(True)
                dr = _drift(x, cfg["drifter"], tuple(q))
                cell, lo, hi = _cells(P, cfg, dr, (t0[part], nt[part], p0[part], npp[part]), T, K, nticks)
                s = (lo * dQ[cell]).sum() + (hi * dQ[cell + up]).sum()
                gx, gq = torch.autograd.grad(s, (x, q))
                gd[part] += gx
                gp += gq
    return frame, gd, gp.cpu()


def _exact_splat(case, seed):
    geo = _config(case, seed)
    dep, cfg = _splat_inputs(case, seed)
    d = torch.from_numpy(dep).to(DEV)
    nticks = case["nticks"]
    t, q, x, y, z, el, et = d.T
    live = torch.ones_like(t, dtype=torch.bool)
    for v, lo, hi in zip((x, y, z), geo["face_bb"][0], geo["face_bb"][1]):
        live = live & (v >= lo) & (v <= hi)
    t = t + cfg["response_plane"] / cfg["drift_speed"]
    out = []
    for ip, pl in enumerate(geo["planes"]):
        a = np.array(pl["pitch"], dtype=np.float64)
        a = (a / math.sqrt(float(a @ a))).tolist()
        c = sum(a[k] * (v - pl["origin"][k]) for k, v in enumerate((x, y, z)))
        nw = pl["nwires"]
        bs = (pl["pitchmax"] - pl["pitchmin"]) / (nw - 1)
        lo, hi = pl["pitchmin"] - 0.5 * bs, pl["pitchmax"] + 0.5 * bs
        st = torch.sqrt((el / cfg["drift_speed"]) ** 2 + (cfg["smear_long"][ip] * cfg["tick"]) ** 2)
        sp = torch.sqrt(et ** 2 + (cfg["smear_tran"][ip] * bs) ** 2)
        tin, t0, nt = _bins(t, st, 0.0, cfg["window_duration"], nticks, cfg["nsigma"])
        pin, p0, npp = _bins(c, sp, lo, hi, nw, cfg["nsigma"])
        use = live & tin & pin
        live = live & ~(tin & ~pin)  # a depo that misses a plane's wires in pitch skips the planes after it
        acc = torch.zeros(nw * nticks, dtype=torch.float64, device=DEV)
        for idx, T, K in _chunks(nt, npp, use.nonzero()[:, 0]):
            te = _edges(t0[idx], T, t[idx], 0.0, cfg["window_duration"] / nticks) / st[idx][:, None]
            pe = _edges(p0[idx], K, c[idx], lo, (hi - lo) / nw) / sp[idx][:, None]
            kt, kp = torch.arange(T, device=DEV), torch.arange(K, device=DEV)
            tm, pm = kt[None, :] < nt[idx][:, None], kp[None, :] < npp[idx][:, None]
            F, p = torch.diff(_cdf(te)) * tm, torch.diff(_cdf(pe)) * pm
            v = (q[idx] / (F.sum(1) * p.sum(1))).abs()
            cell = (p0[idx][:, None] + kp)[:, :, None] * nticks + (t0[idx][:, None] + kt)[:, None, :]
            cell = torch.where(pm[:, :, None] & tm[:, None, :], cell, torch.zeros_like(cell))
            acc.index_add_(0, cell.reshape(-1), (p[:, :, None] * (F * v[:, None])[:, None, :]).reshape(-1))
        out.append(acc.view(nw, nticks))
    return torch.cat(out)


def _normals(key0, key1, stream, model, index):
    """Standard normals of counters (stream, model, index, 0): Philox-4x32-10, then Box-Muller."""
    low = 0xFFFFFFFF
    c = [stream, torch.full_like(index, model), index, torch.zeros_like(index)]
    k0, k1 = key0, key1
    for _ in range(10):
        m0, m1 = c[0] * 0xD2511F53, c[2] * 0xCD9E8D57
        c = [((m1 >> 32) & low) ^ c[1] ^ k0, m1 & low, ((m0 >> 32) & low) ^ c[3] ^ k1, m0 & low]
        k0, k1 = (k0 + 0x9E3779B9) & low, (k1 + 0xBB67AE85) & low
    u = [((((hi << 32) | lo) >> 11) & ((1 << 53) - 1)).double().add(0.5) * 2.0 ** -53
         for hi, lo in ((c[0], c[1]), (c[2], c[3]))]
    return torch.sqrt(-2.0 * torch.log(u[0])) * torch.cos(2.0 * math.pi * u[1])


def _exact_readout(case, seed):
    frame, amp, spec, chan = _readout_inputs(case, seed)
    rows, n = frame.shape
    h = n // 2
    out = torch.empty((rows, n), dtype=torch.float64, device=DEV)
    for r0 in range(0, rows, 256):
        r = slice(r0, min(rows, r0 + 256))
        i = torch.arange(n + 1, device=DEV)[None, :].expand(chan[r].shape[0], -1)
        z = _normals(7, 0, chan[r].long()[:, None].expand_as(i), 0, i.contiguous())  # the first event's key
        m = amp[spec[r].long()].double()[:, :h + 1] * math.sqrt(2.0 / 3.141592)
        X = torch.complex(m * z[:, :h + 1], m * z[:, h:])
        X[:, 0], X[:, h] = X[:, 0].abs().to(X.dtype), X[:, h].abs().to(X.dtype)
        out[r] = frame[r].double() + torch.fft.irfft(X, n=n)
    g = wct.Digitizer.VOLT
    base = torch.cat([torch.full((k,), b * g, device=DEV) for k, b in zip(READOUT_ROWS, (0.9, 0.9, 0.2))])
    v = out + base.float().double()[:, None]
    adc = torch.floor(v / (2.0 * g) * 4095.0)
    return out, torch.where(v <= 0, torch.zeros_like(adc), torch.where(v >= 2.0 * g, torch.full_like(adc, 4095.0), adc))


def exact(case, seed):
    op = case["op"]
    if op in ("forward", "host"):
        if case["fluct"]:
            return None  # random draws
        cfg = _config(case, seed)
        f = _frame(cfg, torch.from_numpy(_depos(case["kind"], case["n"], seed)).to(DEV), _params(cfg))
        return f.cpu().numpy() if op == "host" else f
    if op == "fit":
        return _exact_fit(case, seed)
    if op == "batch":
        cfg = _config(case, seed)
        return torch.stack([_frame(cfg, torch.from_numpy(e).to(DEV), _params(cfg)) for e in _events(case, seed)])
    if op == "splat":
        return _exact_splat(case, seed)
    if op == "readout":
        return _exact_readout(case, seed)
    x = _dft_input(case, seed).to(torch.complex128)
    return torch.fft.ifft2(x) if case["inverse"] else torch.fft.fft2(x)
