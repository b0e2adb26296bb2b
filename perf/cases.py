"""Workloads of the matched-filtering path whose speed matters to its users.

Each case is one call sequence of a user's program through the public Python
layer: pymflib's host-in / host-out calls, network banks (one signal per
template, shift-and-stack), day-long multi-channel banks with peak finding,
banks of many template lengths, the precision-stress signals, requests served
from a resident bank, the single-channel detector, and DBSCAN association.
Signals are seeded band-passed noise at 100 Hz with scaled template copies
added; templates are Hann-tapered band-passed noise.

listed() and draw() give the cases, prepare() what the program holds before
the call, run() the call, work() the bytes and operations it cannot do
without, exact() the same outputs from plain torch in 64 bits.
"""
import ctypes as C
import math

import numpy as np
import torch

import mflib_gb300 as mf
from mflib_gb300 import _lib, serving

FS = 100.0
SEPARATION = 250  # of peaks, in samples


def listed():
    return [
        # pymflib's own use, double precision: three minutes of one channel, three 10 s templates, samples and
        # coefficients in host arrays; latency counts
        {"name": "pymflib_f64", "kind": "host", "bits": 64, "nt": 3, "L": 1001, "n": 18001},
        # a served detection request: one minute of one three-component station against a bank of 100 templates
        {"name": "request_100", "kind": "request", "nt": 100, "Lmin": 200, "Lmax": 3000, "nch": 3, "n": 6000},
        # a large served request: ten minutes of 24 channels against 2,000 templates
        {"name": "request_2000", "kind": "request", "nt": 2000, "Lmin": 200, "Lmax": 3000, "nch": 24, "n": 60000},
        # the reference's multi-channel layout in double precision (one signal per template: stations x phases),
        # one hour, coefficients shifted and stacked
        {"name": "stack_f64", "kind": "stack", "bits": 64, "nt": 64, "L": 500, "n": 360000},
        # the same layout in single precision, a day's eighth, an odd length
        {"name": "stack_f32", "kind": "stack", "bits": 32, "nt": 72, "L": 733, "n": 1080000},
        # a bank of several template lengths in double precision on shared channels, one hour
        {"name": "bank_f64", "kind": "bank", "bits": 64, "nt": 160, "Lmin": 200, "Lmax": 2000, "nch": 8, "n": 360000,
         "thr": 0.7},
        # short templates (2 s), many per channel, three hours of 24 channels
        {"name": "day_short_f32", "kind": "bank", "bits": 32, "nt": 384, "Lmin": 200, "Lmax": 200, "nch": 24,
         "n": 1080000, "thr": 0.7},
        # the 24-channel day (three hours of it): 192 templates of 500, peaks gathered
        {"name": "day_f32", "kind": "bank", "bits": 32, "nt": 192, "Lmin": 500, "Lmax": 500, "nch": 24, "n": 1080000,
         "thr": 0.5},
        # the bank of 2,000 templates of 200-3,000 samples on 96 channels, one hour
        {"name": "uneven_f32", "kind": "bank", "bits": 32, "nt": 2000, "Lmin": 200, "Lmax": 3000, "nch": 96,
         "n": 360000, "thr": 0.7},
        # precision stress: large offsets and an envelope over six decades, 512 templates of 1,000 on one channel
        {"name": "stress_f32", "kind": "stress", "bits": 32, "nt": 512, "L": 1000, "n": 432000},
        # the single-channel detector over six hours: traces reduced over the templates, peaks, refined times
        {"name": "detector_f32", "kind": "detect", "bits": 32, "nt": 96, "L": 500, "n": 2160000},
        # association: origin times of eight events' detections clustered per event
        {"name": "associate", "kind": "cluster", "nobs": 9500, "nseg": 8, "nf": 1},
    ]


def draw(rng):
    def log(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    kind = rng.choice(["host", "request", "request", "stack", "bank", "bank", "bank", "uneven", "uneven", "stress",
                       "detect", "cluster"])
    if kind == "host":
        L = log(100, 2000)
        return {"kind": "host", "bits": rng.choice([64, 64, 32]), "nt": log(1, 12), "L": L, "n": L + log(3000, 60000)}
    if kind == "request":
        return {"kind": "request", "nt": log(100, 2000), "Lmin": 200, "Lmax": log(1000, 3000), "nch": log(1, 32),
                "n": log(6000, 60000)}
    if kind == "stack":
        bits = rng.choice([32, 64])
        return {"kind": "stack", "bits": bits, "nt": log(8, 96), "L": log(100, 2000),
                "n": log(60000, 1080000 if bits == 32 else 360000)}
    if kind == "bank":
        bits, L = rng.choice([32, 32, 64]), log(150, 2000)
        nch = log(1, 24)
        return {"kind": "bank", "bits": bits, "nt": nch * log(2, 16) + rng.randrange(3), "Lmin": L, "Lmax": L, "nch": nch,
                "n": log(60000, 1080000 if bits == 32 else 240000), "thr": rng.choice([0.5, 0.7])}
    if kind == "uneven":
        bits = rng.choice([32, 32, 64])
        return {"kind": "bank", "bits": bits, "nt": log(40, 1200 if bits == 32 else 200), "Lmin": log(100, 400),
                "Lmax": log(800, 3000), "nch": log(2, 48), "n": log(60000, 360000), "thr": 0.7}
    if kind == "stress":
        return {"kind": "stress", "bits": 32, "nt": log(32, 512), "L": log(300, 1500), "n": log(60000, 432000)}
    if kind == "detect":
        return {"kind": "detect", "bits": 32, "nt": log(8, 96), "L": log(200, 1500), "n": log(60000, 2160000)}
    return {"kind": "cluster", "nobs": log(1000, 40000), "nseg": log(1, 16), "nf": rng.choice([1, 1, 2])}


# ---------------------------------------------------------------------------
# seeded signals and templates
def _gen(seed):
    return torch.Generator(device="cuda").manual_seed(int(seed))


def _band(w, lo, hi):
    """Zero-phase band pass of the rows of w; lo and hi in Hz, numbers or a column per row."""
    n = w.shape[-1]
    f = torch.fft.rfftfreq(n, 1.0 / FS, dtype=torch.float64, device=w.device).clamp_min(1e-9)
    h = ((f * f - lo * hi) / (f * (hi - lo))) ** 8
    return torch.fft.irfft(torch.fft.rfft(w) * (1.0 / torch.sqrt(1.0 + h)), n=n)


def _templates(g, lens, lo, hi):
    """Hann-tapered band-passed noise, row t of lens[t] samples (zeros after them)."""
    lens = torch.as_tensor(lens, device="cuda").reshape(-1, 1)
    m = int(lens.max())
    b = _band(torch.randn(len(lens), m, generator=g, dtype=torch.float64, device="cuda"), lo, hi)
    j = torch.arange(m, device="cuda", dtype=torch.float64)
    return torch.where(j < lens, b * (0.5 - 0.5 * torch.cos(2 * math.pi * j / (lens - 1).clamp_min(1))), 0.0)


def _lengths(case, g):
    lo, hi = case.get("Lmin", case.get("L")), case.get("Lmax", case.get("L"))
    if lo == hi:
        return [lo] * case["nt"]
    lens = torch.randint(lo, hi + 1, (case["nt"],), generator=g, device="cuda").tolist()
    lens[-1] = hi
    return lens


def _channels(case, g):
    """The channel of each template."""
    kind = case["kind"]
    if kind == "stack":
        return list(range(case["nt"]))
    if kind in ("host", "stress", "detect"):
        return [0] * case["nt"]
    if kind == "request":  # template t reads request channel slot % channels
        return [t % serving.N_SLOTS % case["nch"] for t in range(case["nt"])]
    if case["Lmin"] == case["Lmax"]:
        return [t % case["nch"] for t in range(case["nt"])]
    return torch.randint(0, case["nch"], (case["nt"],), generator=g, device="cuda").tolist()


def _data(case, seed):
    """Signals (channels x samples, of the case's type, on the GPU), templates (rows of float64), their lengths and
    channels."""
    g = _gen(seed)
    lens, chan = _lengths(case, g), _channels(case, g)
    nt, n, one = case["nt"], case["n"], len(set(lens)) == 1
    u = torch.rand(2, nt, 1, generator=g, dtype=torch.float64, device="cuda")
    lo = 2.0 if one else 1.0 + 6.0 * u[0]
    hi = 8.0 if one else lo + 2.0 + (13.0 - lo) * u[1]
    b = _templates(g, lens, lo, hi)
    nch = max(chan) + 1 if "nch" not in case else case["nch"]
    x = _band(torch.randn(nch, n, generator=g, dtype=torch.float64, device="cuda"), 1.0, 10.0)
    x /= x.square().mean().sqrt()
    # scaled copies of every template on its channel
    copies = {"host": 2, "request": 2, "detect": 4}.get(case["kind"], 6)
    amp = 1.0 + 2.0 * torch.rand(nt, copies, generator=g, dtype=torch.float64, device="cuda")
    rms = b.square().sum(1) / torch.as_tensor(lens, device="cuda")
    at = torch.rand(nt, copies, generator=g, dtype=torch.float64, device="cuda")
    at = (at * (n - torch.as_tensor(lens, device="cuda").reshape(-1, 1) + 1)).long()
    rows = torch.as_tensor(chan, device="cuda") * n
    j = torch.arange(b.shape[1], device="cuda")
    live = j < torch.as_tensor(lens, device="cuda").reshape(-1, 1)
    for k in range(copies):
        pos = (rows + at[:, k]).reshape(-1, 1) + j
        x.view(-1).index_put_((pos[live],), (b * (amp[:, k] / rms.sqrt()).reshape(-1, 1))[live], accumulate=True)
    if case["kind"] == "stress":
        # piecewise-constant envelope over six decades, a new level every 10 to 20 minutes, on a large offset
        seg = 60000 + int(60000 * float(u[0, 0, 0]))
        lev = 10.0 ** (6.0 * torch.rand(n // seg + 1, generator=g, dtype=torch.float64, device="cuda") - 3.0)
        x = x * lev.repeat_interleave(seg)[:n] + 1e3 * 10.0 ** (2.0 * float(u[1, 0, 0]))
    x = x.to(torch.float32 if case.get("bits", 32) == 32 else torch.float64)
    return x, b, lens, chan


def _shifts(case):
    """Travel time less onset of each template, in samples."""
    return [(37 * t) % 1500 for t in range(case["nt"])]


def _weights(case):
    return [1.0 - 0.5 * (t % 4) / 4 for t in range(case["nt"])]


def _parameters(params, case, b, lens):
    rows = b.cpu().numpy()
    for t, L in enumerate(lens):
        w = mf.WaveformTemplate()
        w.set_signal(rows[t, :L])
        w.set_sampling_rate(FS)
        if case["kind"] == "stack":
            w.set_phase_onset_time_in_signal(0.0)
            w.set_phase_travel_time(_shifts(case)[t] / FS)
            w.set_shift_and_stack_weight(_weights(case)[t])
        params.add_template(w)
    params.set_signal_size(case["n"])
    return params


# ---------------------------------------------------------------------------
class _Rows:
    """Coefficients of an object's last apply where they lie (templates x lags); keeps the object alive."""

    def __init__(self, f, nt, n):
        p, q, nv = C.c_void_p(), C.c_void_p(), C.c_int()
        _lib.call("mfgpu_mf_get_device_signal", f._h, 0, C.byref(p), C.byref(nv))
        _lib.call("mfgpu_mf_get_device_signal", f._h, nt - 1, C.byref(q), C.byref(nv))
        size = f.dtype.itemsize
        self.owner = f
        self.__cuda_array_interface__ = {
            "shape": (nt, n), "strides": ((q.value - p.value) // (nt - 1) if nt > 1 else n * size, size),
            "typestr": f.dtype.str, "data": (p.value, False), "version": 3}


def _device_rows(f, nt, n):
    return torch.as_tensor(_Rows(f, nt, n), device="cuda")


def _kept(s, name, values):
    """Values in a buffer that the program keeps, with room for as many as the peak separation allows; -1 after them."""
    buf, used = s[name]
    buf[:len(values)] = values
    buf[len(values):used] = -1
    s[name] = buf, len(values)
    return buf


def _room(s, most, **types):
    for name, t in types.items():
        s[name] = np.full(most, -1, dtype=t), 0


def prepare(case, seed):
    kind, s = case["kind"], {"case": case}
    if kind == "cluster":
        rng = np.random.default_rng(seed)
        nobs, nseg, nf = case["nobs"], case["nseg"], case["nf"]
        # per event: origins of about 50 shots, seen by several templates within a few samples, and scattered false ones
        seg = np.sort(rng.integers(0, nseg, nobs))
        X = rng.integers(0, 8_640_000, (nseg, 50, nf))[seg, rng.integers(0, 50, nobs)].astype(np.float64)
        X += np.rint(rng.normal(0.0, 8.0, (nobs, nf)))
        stray = rng.random(nobs) < 0.1
        X[stray] = rng.integers(0, 8_640_000, (int(stray.sum()), nf))
        db = mf.DBSCAN()
        db.initialize(50.0, 3)
        s.update(db=db, X=X, off=np.searchsorted(seg, np.arange(nseg + 1)).astype(np.int32))
        return s
    x, b, lens, chan = _data(case, seed)
    dtype = np.float32 if case.get("bits", 32) == 32 else np.float64
    if kind == "request":
        rows = b.cpu().numpy()
        bank = serving.TemplateBank("bank", [rows[t, :L] for t, L in enumerate(lens)], sampling_rate=FS)
        f = serving.GpuExecutor().create(bank, min(v for v in serving.DEFAULT_BUCKETS if v >= case["n"]))
        s.update(f=f, x=x.cpu().numpy(), nfilt=bank.valid_lags(case["n"]))
        _room(s, case["nt"] * (s["nfilt"] // SEPARATION + 1), peaks=np.int32)
        return s
    if kind in ("host", "stress", "detect"):
        f = mf.SingleChannel.MatchedFilter(dtype=dtype)
        f.initialize(_parameters(mf.SingleChannel.MatchedFilterParameters(), case, b, lens))
    else:
        f = mf.MultiChannel.MatchedFilter(dtype=dtype)
        p = _parameters(mf.MultiChannel.MatchedFilterParameters(), case, b, lens)
        if kind == "stack":
            f.initialize(p)
        else:
            f.initialize(p, template_channels=chan, n_channels=case["nch"])
            f.set_peak_threshold(case["thr"])
            f.set_graph(True)
    host = x.cpu().numpy()
    s.update(f=f, nfilt=case["n"] - max(lens) + 1)
    if kind == "host":
        s["x"] = host[0]
    else:
        f.set_channel_signals(host)
    if kind == "bank":
        _room(s, case["nt"] * (s["nfilt"] // SEPARATION + 1), peaks=np.int32)
    if kind == "detect":
        _room(s, s["nfilt"] // SEPARATION + 1, template=np.int32, time=np.float64, refined=np.float64, rho_at=np.float32,
              amplitude=np.float64)
        q = mf.SingleChannel.DetectorParameters()
        q.set_detection_threshold(0.7)
        q.set_minimum_detection_spacing(SEPARATION)
        q.set_matched_filtered_signal_detector_policy(mf.MatchedFilteredSignalDetectorPolicy.reduce)
        s["detector"] = mf.SingleChannel.Detector()
        s["detector"].initialize(q)
    return s


def run(s):
    case = s["case"]
    kind, nt = case["kind"], case.get("nt")
    if kind == "cluster":
        labels, clusters = s["db"].cluster_segments(s["X"], s["off"])
        return {"labels": labels, "clusters": clusters}
    f = s["f"]
    if kind == "request":
        # what the serving loop does with a request on an object of its pool
        f.set_window(s["x"])
        f.apply()
        f.find_peaks(0.7, SEPARATION, s["nfilt"])
        counts, peaks = f.get_all_peaks()
        return {"rho": _device_rows(f, nt, s["nfilt"]), "counts": counts, "peaks": _kept(s, "peaks", peaks)}
    if kind == "host":
        f.set_signal(s["x"])
        f.apply()
        return {"rho": [f.get_matched_filtered_signal(t) for t in range(nt)]}
    f.apply()
    if kind == "stack":
        stack = f.shift_and_stack()
        return {"rho": _device_rows(f, nt, s["nfilt"]), "stack": stack}
    if kind == "bank":
        f.find_peaks(case["thr"], SEPARATION)
        counts, peaks = f.get_all_peaks()
        return {"rho": _device_rows(f, nt, s["nfilt"]), "counts": counts, "peaks": _kept(s, "peaks", peaks)}
    if kind == "detect":
        got = s["detector"].detect(f).get_detections()
        gr = mf.RelativeMagnitudeType.gibbons_ringdal_2006
        return {"rho": _device_rows(f, nt, s["nfilt"]),
                "template": _kept(s, "template", [d.get_template_identifier()[1] for d in got]),
                "time": _kept(s, "time", [d.get_detection_time() for d in got]),
                "refined": _kept(s, "refined", [d.get_interpolated_detection_time() for d in got]),
                "rho_at": _kept(s, "rho_at", [d.get_correlation_coefficient() for d in got]),
                "amplitude": _kept(s, "amplitude", [d.get_amplitude_scaling_factor(gr) for d in got])}
    return {"rho": _device_rows(f, nt, s["nfilt"])}


def work(case):
    """Bytes: samples and template samples read once, coefficients written once (and the stack).  Operations: a real
    transform of each channel's samples, and per coefficient its share of an inverse transform, the product of the
    spectra and the normalisation, at transforms of 4,096 samples.  Association: a sort and a neighbour search."""
    if case["kind"] == "cluster":
        n, nf = case["nobs"], case["nf"]
        return {"bytes": n * (8 * nf + 4), "flops": 4 * n * math.log2(n) * nf}
    size = case.get("bits", 32) // 8
    nt, n = case["nt"], case["n"]
    lo, hi = case.get("Lmin", case.get("L")), case.get("Lmax", case.get("L"))
    nch = {"host": 1, "stress": 1, "detect": 1, "stack": nt}.get(case["kind"]) or case["nch"]
    lags = nt * (n - hi + 1)
    more = {"stack": n * size, "detect": 0}.get(case["kind"], 0)
    return {"bytes": size * (nch * n + lags) + 8 * nt * (lo + hi) // 2 + more, "flops": 30 * nch * n + 46 * lags}


# ---------------------------------------------------------------------------
def _pearson64(x, b, lens, chan, n):
    """Pearson coefficients at the first n lags of every template: products as matrix multiplications, window variances
    from sums over short blocks (or two-pass, `x` with wide amplitude ranges), everything in 64 bits."""
    out = torch.empty(len(lens), n, dtype=torch.float64, device="cuda")
    lt = torch.as_tensor(lens, device="cuda", dtype=torch.float64)
    live = torch.arange(b.shape[1], device="cuda") < lt.reshape(-1, 1)
    u = torch.where(live, b - b.sum(1, keepdim=True) / lt.reshape(-1, 1), 0.0)
    u = u / u.norm(dim=1, keepdim=True)
    for c in sorted(set(chan)):
        mine = [t for t in range(len(lens)) if chan[t] == c]
        m = max(lens[t] for t in mine)
        xc = x[c].double()
        step = max(1024, int(2.0e9 / 8 / m))
        for a in range(0, n, step):
            e = min(n, a + step)
            seg = xc[a:e + m - 1]
            w = (seg - seg.mean()).unfold(0, m, 1).contiguous()
            num = w @ u[mine, :m].T
            for L in sorted({lens[t] for t in mine}):
                if len({lens[t] for t in mine}) == 1:
                    v = (w - w.mean(1, keepdim=True)).square().sum(1)
                else:
                    blk = 512
                    nb = -(-(e - a) // blk)
                    y = torch.nn.functional.pad(seg - seg.mean(), (0, max(0, nb * blk + L - seg.numel())))
                    y = y.unfold(0, blk + L, blk)[:nb]
                    y = y - y.mean(1, keepdim=True)
                    s1 = torch.nn.functional.pad(y.cumsum(1), (1, 0))
                    s2 = torch.nn.functional.pad(y.square().cumsum(1), (1, 0))
                    s1, s2 = s1[:, L:L + blk] - s1[:, :blk], s2[:, L:L + blk] - s2[:, :blk]
                    v = (s2 - s1 * s1 / L).reshape(-1)[:e - a]
                for i, t in enumerate(mine):
                    if lens[t] == L:
                        out[t, a:e] = num[:, i] / v.sqrt()
    return out


def exact(case, seed):
    kind = case["kind"]
    if kind == "cluster":
        return None
    x, b, lens, chan = _data(case, seed)
    nfilt = case["n"] - max(lens) + 1
    rho = _pearson64(x, b, lens, chan, nfilt)
    if kind == "host":
        return {"rho": [rho[t] for t in range(case["nt"])]}
    if kind == "stack":
        sh, w = _shifts(case), _weights(case)
        m = nfilt - max(sh)
        stack = torch.zeros(m, dtype=torch.float64, device="cuda")
        for t in range(case["nt"]):
            stack += w[t] / sum(w) * rho[t, sh[t]:sh[t] + m].abs()
        return {"rho": rho, "stack": stack}
    if kind in ("bank", "request"):
        return {"rho": rho, "counts": None, "peaks": None}
    if kind == "detect":
        return {"rho": rho, "template": None, "time": None, "refined": None, "rho_at": None, "amplitude": None}
    return {"rho": rho}
