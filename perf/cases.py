"""What a user of this framework has it do, as cases that can be timed.

Three kinds of programs call the framework, and each has cases here:

* a program with its own device memory that wants the filter-output plane
  (FOP) of a spectrum: ``fdas_ft_convolution_noalloc`` (kind "conv");
* a search host in the manner of the reference's driver: a handle per
  spectrum length, ``launch`` / ``wait`` on buffer sets A and B, candidate
  lists back in host memory (kinds "search", "loop", "list"), with the
  upstream spectrum made on the GPU where the program starts from a time series
  (kinds "spectrum", "series");
* a pipeline over many dedispersed trials: ``Batch`` when all trials are at
  hand, ``Server`` when they arrive one by one (kinds "batch", "served").

Lengths are those of the repository's workloads (32,768 bins: the emulator
size; 2^21: the full single trial; 2^17 to 2^21: the batch; 2^15 to 2^21: the
server), powers of two and ragged ones; the template bank is the 85-row Fresnel
bank or its 43-row half; planes are 4, 8 or 16; thresholds are those of a
1e-6 false-alarm rate under chi-square noise.  Spectra are unit-power noise
with none to three accelerated signals whose amplitudes follow the repository's
workloads, so candidate counts run from a few (noise) to hundreds of thousands.
"""
import ctypes
import math

import numpy as np
import torch

from fdas_gb300 import _lib
from fdas_gb300.batch import Batch
from fdas_gb300.fdas import FDAS
from fdas_gb300.server import HALF_BANK, Server
from fdas_gb300.templates import template_bank, template_spectra

TILE, OVERLAP, ROWS = 2048, 420, 85
FAR = 1e-6
RECORDS = 1 << 17
BANK = template_bank()


# ------------------------------------------------------------------ the cases
def listed():
    return [
        # a few tiles: the smallest FOP a program asks for, bound by launches
        {"name": "conv_4096", "kind": "conv", "bins": 4096, "templates": 85, "part": 2, "p4": True, "signals": 1},
        # a ragged length, one acceleration sign, natural-order spectra
        {"name": "conv_100003_pos", "kind": "conv", "bins": 100003, "templates": 85, "part": 1, "p4": False,
         "signals": 1},
        # the largest power of two the allocation-free call takes
        {"name": "conv_2p19", "kind": "conv", "bins": 1 << 19, "templates": 85, "part": 2, "p4": True, "signals": 1},
        # the emulator-size search of the reference's tests, one signal, lists back on the host
        {"name": "search_32768", "kind": "search", "bins": 32768, "templates": 85, "planes": 8, "signals": 1,
         "strong": True},
        # an ordinary ragged length, half bank, 16 planes, noise only: what most trials of a survey look like
        {"name": "search_300007_half", "kind": "search", "bins": 300007, "templates": 43, "planes": 16, "signals": 0,
         "strong": False},
        # the full single-trial search: the headline workload, three strong signals
        {"name": "search_2p21", "kind": "search", "bins": 1 << 21, "templates": 85, "planes": 8, "signals": 3,
         "strong": True},
        # the reference driver's loop over sets A and B, four full-size trials of noise
        {"name": "loop_2p21", "kind": "loop", "bins": 1 << 21, "templates": 85, "planes": 8, "signals": 0,
         "strong": False},
        # a search whose every hit is fetched (the wide list), not only the 512 strongest of each plane
        {"name": "list_2p18", "kind": "list", "bins": 1 << 18, "templates": 85, "planes": 8, "signals": 2,
         "strong": False},
        # the upstream step alone: time series on the device to its normalised spectrum on the host, mixed radices
        {"name": "spectrum_1000000", "kind": "spectrum", "bins": 1000000},
        # time series on the device to candidates: the spectrum never leaves the GPU
        {"name": "series_2p21", "kind": "series", "bins": 1 << 21, "templates": 85, "planes": 8, "signals": 1},
        # dedispersed trials of uneven length in one batch
        {"name": "batch_24", "kind": "batch", "trials": 24, "planes": 8, "mix": 4242},
        # requests of mixed length, bank and planes to the server, submitted together
        {"name": "served_8", "kind": "served", "requests": 8, "mix": 17},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    """The largest number of radices 2, 3, 5, 7 that is at most n."""
    while True:
        m = n
        for f in (2, 3, 5, 7):
            while m % f == 0:
                m //= f
        if m == 1:
            return n
        n -= 1


def draw(rng):
    kind = rng.choice(["conv", "conv", "search", "search", "search", "loop", "list", "spectrum", "series", "batch",
                       "served"])
    if kind == "conv":
        return {"kind": kind, "bins": _log(rng, 1024, 1 << 19), "templates": rng.choice([85, 85, 43]),
                "part": rng.choice([2, 2, 1, 0]), "p4": rng.random() < 0.5, "signals": rng.randrange(3)}
    if kind in ("search", "loop"):
        strong = rng.random() < 0.3
        return {"kind": kind, "bins": _log(rng, 1 << 15, 1 << 21), "templates": rng.choice([85, 85, 43]),
                "planes": rng.choice([4, 8, 8] if strong else [4, 8, 8, 16]), "signals": rng.randrange(4),
                "strong": strong}
    if kind == "list":
        return {"kind": kind, "bins": _log(rng, 1 << 15, 1 << 18), "templates": rng.choice([85, 43]),
                "planes": rng.choice([4, 8, 16]), "signals": rng.randrange(3), "strong": False}
    if kind == "spectrum":
        return {"kind": kind, "bins": _smooth(_log(rng, 1 << 15, 1 << 21))}
    if kind == "series":
        return {"kind": kind, "bins": _smooth(_log(rng, 1 << 15, 1 << 21)), "templates": rng.choice([85, 43]),
                "planes": rng.choice([4, 8, 16]), "signals": rng.randrange(3)}
    if kind == "batch":
        return {"kind": kind, "trials": rng.randint(3, 24), "planes": rng.choice([4, 8]), "mix": rng.randrange(10000)}
    return {"kind": kind, "requests": rng.randint(2, 8), "mix": rng.randrange(10000)}


# ------------------------------------------------------------------ inputs
def _thresholds(planes):
    """Power above which the sum of k unit-mean powers lies with probability FAR, k = 1..planes."""
    out = []
    for k in range(1, planes + 1):
        lo, hi = 0.0, 200.0
        for _ in range(100):
            t = 0.5 * (lo + hi)
            term = total = 1.0
            for i in range(1, k):
                term *= t / i
                total += term
            lo, hi = (t, hi) if total * math.exp(-t) > FAR else (lo, t)
        out.append(hi)
    return np.array(out, dtype=np.float32)


def _series(bins, signals, seed, strong=False):
    """2 x bins float32 samples on the GPU: white noise of unit variance plus accelerated periodic signals, of
    0.02 to 0.04 sigma (the full single trial's strength) or of an amplitude that falls with the length (the
    batch's)."""
    rng = np.random.default_rng(seed)
    g = torch.Generator(device="cuda").manual_seed(seed)
    n = 2 * bins
    x = torch.randn(n, device="cuda", generator=g, dtype=torch.float64)
    u = torch.arange(n, device="cuda", dtype=torch.float64) / n
    for _ in range(signals):
        r0, z, harmonics = rng.uniform(0.05, 0.45) * bins, rng.uniform(-42, 42), int(rng.integers(1, 9))
        amp = rng.uniform(0.02, 0.04) if strong else 0.05 * math.sqrt((1 << 16) / n)
        phase = 2 * math.pi * (r0 * u + 0.5 * z * u * u)
        for h in range(1, harmonics + 1):
            x += amp * torch.cos(h * phase)
    return x.float()


def _spectrum(bins, signals, seed, strong=False):
    """bins complex64 values on the GPU, noise of unit mean power."""
    x = _series(bins, signals, seed, strong).double()
    return (torch.fft.rfft(x)[:bins] / math.sqrt(2 * bins)).to(torch.complex64)


def _bank(templates):
    """The full bank, or the contiguous rows of the half bank."""
    first = (ROWS - templates) // 2
    return np.ascontiguousarray(BANK[first:first + templates])


def _p4(spectra):
    """Natural order to the template file's order: position 4 s + j holds bin bitrev2(j) * 512 + s."""
    out = np.empty_like(spectra)
    for j, b in enumerate((0, 2, 1, 3)):
        out[:, j::4] = spectra[:, 512 * b:512 * (b + 1)]
    return out


class _Null:
    def write(self, _line):
        pass


def _handle(case):
    h = FDAS(_Null())
    ok = h.initialise_accelerator(case["bins"], n_templates=case["templates"], n_planes=case["planes"])
    for ab in (FDAS.A, FDAS.B):
        ok = ok and h.upload_templates(_bank(case["templates"]), ab)
    if not ok:
        raise RuntimeError(h.last_error)
    return h


def _pinned(count, dtype):
    """A NumPy array in pinned host memory, which lives as long as the array."""
    return torch.empty(count * np.dtype(dtype).itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(dtype)


def _pinned_spectrum(*args):
    x = _spectrum(*args).cpu().numpy()
    p = _pinned(x.size, np.complex64)
    p[:] = x
    return p


def _mix(kind, count, seed):
    """Lengths (and, for the server, banks and planes) of a mix of trials, spread evenly over the logarithm."""
    rng = np.random.default_rng(seed)
    if kind == "batch":
        return [(int(math.exp(rng.uniform(math.log(1 << 17), math.log(1 << 21)))), int(rng.integers(0, 3)))
                for _ in range(count)]
    return [(int(math.exp(rng.uniform(math.log(1 << 15), math.log(1 << 20)))), int(rng.integers(0, 3)),
             [ROWS, HALF_BANK[1]][int(rng.integers(0, 2))], [4, 8, 16][int(rng.integers(0, 3))])
            for _ in range(count)]


def prepare(case, seed):
    kind = case["kind"]
    s = {"kind": kind}
    if kind == "conv":
        n, rows = case["bins"], case["templates"]
        t = template_spectra(_bank(rows)).astype(np.complex64)
        s.update(bins=n, rows=rows, part=case["part"], stride=(n + 255) // 256 * 256,
                 layout=_lib.TEMPLATES_FFT_P4 if case["p4"] else _lib.TEMPLATES_FFT_NATURAL,
                 x=_spectrum(n, case["signals"], seed), t=torch.from_numpy(_p4(t) if case["p4"] else t).cuda(),
                 status=torch.zeros(1, dtype=torch.int32, device="cuda"))
        s["fop"] = torch.zeros((rows, s["stride"]), dtype=torch.float32, device="cuda")
        return s
    if kind == "batch":
        mix = _mix(kind, case["trials"], case["mix"])
        s["x"] = torch.cat([_spectrum(n, sig, seed * 1000 + i) for i, (n, sig) in enumerate(mix)])
        s["thr"] = _thresholds(case["planes"])
        s["batch"] = Batch(BANK, [n for n, _ in mix], n_planes=case["planes"])
        s["loc"] = np.zeros((len(mix), 512 * case["planes"]), np.uint32)
        s["pwr"] = np.zeros((len(mix), 512 * case["planes"]), np.float32)
        s["trials"] = [s["batch"].trial(i) for i in range(len(mix))]
        for t in s["trials"]:
            t.log = _Null()
        torch.cuda.synchronize()
        s["batch"].set_inputs_device(s["x"].data_ptr())
        s["batch"].run(s["thr"])  # the program's first batch: the plan is made
        return s
    if kind == "served":
        mix = _mix(kind, case["requests"], case["mix"])
        s["server"] = Server(BANK, max_bins=1 << 20)
        s["requests"] = [(_spectrum(n, sig, seed * 1000 + i).cpu().numpy(), _thresholds(planes),
                          (ROWS // 2 - rows // 2, rows)) for i, (n, sig, rows, planes) in enumerate(mix)]
        s["records"] = [_record_arrays() for _ in mix]
        run(s)  # the server has been up for a while: its slots exist
        return s
    n = case["bins"]
    if kind in ("spectrum", "series"):
        s["series"] = _series(n, case.get("signals", 1), seed)
    if kind == "spectrum":
        s["h"] = FDAS(_Null())
        if not s["h"].initialise_accelerator(n):
            raise RuntimeError(s["h"].last_error)
        s["out"] = _pinned(n, np.complex64)
        torch.cuda.synchronize()
        return s
    if kind == "list":
        s["records"] = _record_arrays()
    s.update(h=_handle(case), thr=_thresholds(case["planes"]), scale=1.0 / math.sqrt(2 * n))
    lists = 4 if kind == "loop" else 1
    count = s["h"].get_candidate_list_sz()
    s["loc"] = [_pinned(count, np.uint32) for _ in range(lists)]
    s["pwr"] = [_pinned(count, np.float32) for _ in range(lists)]
    if kind != "series":
        s["x"] = [_pinned_spectrum(n, case["signals"], seed * 10 + i, case["strong"]) for i in range(lists)]
    torch.cuda.synchronize()
    return s


# ------------------------------------------------------------------ one pass
def _ok(done, h):
    if not done:
        raise RuntimeError(h.last_error)


def run(s):
    kind = s["kind"]
    if kind == "conv":
        st = _lib.load().fdas_ft_convolution_noalloc(
            s["x"].data_ptr(), s["bins"], s["t"].data_ptr(), s["layout"], s["rows"], OVERLAP, s["part"],
            s["fop"].data_ptr(), s["stride"], s["status"].data_ptr(),
            ctypes.c_void_p(torch.cuda.current_stream().cuda_stream))
        if st != _lib.OK:
            raise RuntimeError(_lib.STATUS_NAMES[st])
        return {"fop": s["fop"], "status": s["status"]}
    if kind == "batch":
        b = s["batch"]
        b.set_inputs_device(s["x"].data_ptr())
        b.run(s["thr"])
        for t, loc, pwr in zip(s["trials"], s["loc"], s["pwr"]):
            _ok(t.retrieve_candidates(loc, pwr, FDAS.A), t)
        return {"loc": s["loc"], "pwr": s["pwr"]}
    if kind == "served":
        ids = [s["server"].submit(x, thr, rows) for x, thr, rows in s["requests"]]
        return [_records(s["server"].result(i), into) for i, into in zip(ids, s["records"])]
    h = s["h"]
    if kind == "spectrum":
        _ok(h.series_to_spectrum(s["series"], FDAS.A, spectrum=s["out"]), h)
        return s["out"]
    if kind == "series":
        _ok(h.series_to_spectrum(s["series"], FDAS.A, scale=s["scale"]), h)
        _ok(h.launch(None, s["thr"], s["loc"][0], s["pwr"][0], FDAS.AllAccelerations, FDAS.A), h)
        _ok(h.wait(FDAS.A), h)
    else:
        last = len(s["x"]) - 1
        for i, x in enumerate(s["x"]):  # the reference driver's order: launch one set, wait for the other
            _ok(h.launch(x, s["thr"], s["loc"][i], s["pwr"][i], FDAS.AllAccelerations, i & 1), h)
            if i:
                _ok(h.wait(1 - (i & 1)), h)
        _ok(h.wait(last & 1), h)
    out = {"loc": s["loc"], "pwr": s["pwr"]}
    if kind == "list":
        out["all"] = _records(h.retrieve_candidate_list(FDAS.A), s["records"])
    return out


def _record_arrays():
    """Where a program gathers a list's fields; more room than a list of these cases takes."""
    return {"harmonic": np.zeros(RECORDS, np.uint32), "template": np.zeros(RECORDS, np.int32),
            "bin": np.zeros(RECORDS, np.uint32), "power": np.zeros(RECORDS, np.float32)}


def _records(r, into):
    rec, total, dropped = r[0], r[1], r[2]
    for name, field in (("harmonic", "harmonic"), ("template", "template_num"), ("bin", "bin"), ("power", "power")):
        into[name][:rec.size] = rec[field]
    return dict(into, total=total, dropped=dropped)


# ------------------------------------------------------------------ work
def _tiles(n):
    return -(-n // (TILE - OVERLAP))


def _search_flops(n, rows, planes):
    """Forward transforms, products, inverse transforms and powers of the tiles; sums of the planes."""
    fft = 5 * TILE * 11
    return _tiles(n) * (fft + rows * (6 * TILE + fft + 3 * (TILE - OVERLAP))) + rows * n * (planes - 1)


def work(case):
    kind = case["kind"]
    if kind == "conv":
        rows = case["templates"] if case["part"] == 2 else case["templates"] // 2 + 1
        return {"bytes": 8 * case["bins"] + 8 * TILE * rows + 4 * rows * case["bins"],
                "flops": _search_flops(case["bins"], rows, 1)}
    if kind == "spectrum":
        n = case["bins"]
        return {"bytes": 16 * n, "flops": 5 * n * math.log2(n) + 14 * n}
    if kind == "batch":
        mix = _mix(kind, case["trials"], case["mix"])
        return {"bytes": sum(8 * n + 8 * 512 * case["planes"] for n, _ in mix),
                "flops": sum(_search_flops(n, ROWS, case["planes"]) for n, _ in mix)}
    if kind == "served":
        mix = _mix(kind, case["requests"], case["mix"])
        return {"bytes": sum(8 * n for n, _, _, _ in mix),
                "flops": sum(_search_flops(n, rows, planes) for n, _, rows, planes in mix)}
    n, rows, planes = case["bins"], case["templates"], case["planes"]
    lists = 4 if kind == "loop" else 1
    flops = _search_flops(n, rows, planes) + (5 * n * math.log2(n) if kind == "series" else 0)
    return {"bytes": lists * (8 * n + 8 * 512 * planes), "flops": lists * flops}


# ------------------------------------------------------------------ in 64 bits
def _fop64(x, spectra, rows=None):
    """|overlap-save convolution|^2 of complex128 x with each row of spectra; rows not asked for stay zero."""
    n, payload = x.numel(), TILE - OVERLAP
    tiles = _tiles(n)
    padded = torch.zeros(OVERLAP + tiles * payload, dtype=torch.complex128, device=x.device)
    padded[OVERLAP:OVERLAP + n] = x
    f = torch.fft.fft(padded.unfold(0, TILE, payload))
    out = torch.zeros((spectra.shape[0], n), dtype=torch.float64, device=x.device)
    for r in range(spectra.shape[0]) if rows is None else rows:
        y = torch.fft.ifft(f * spectra[r])[:, OVERLAP:].reshape(-1)[:n]
        out[r] = y.real.square() + y.imag.square()
    return out


def _hits64(x, bank, thr):
    """For each plane: (row, bin, power) of the cells above the threshold, sorted by row and bin."""
    spectra = torch.from_numpy(template_spectra(bank)).to(x.device)
    fop = _fop64(x, spectra)
    rows, n = fop.shape
    half = rows // 2
    t = torch.arange(rows, device=x.device) - half
    f = torch.arange(n, device=x.device)
    total, hits = torch.zeros_like(fop), []
    for j in range(1, len(thr) + 1):
        r = half + torch.sign(t) * (t.abs() // j)
        total += fop[r][:, f // j]
        at = (total > float(thr[j - 1])).nonzero()
        hits.append((at[:, 0], at[:, 1], total[at[:, 0], at[:, 1]]))
    return hits


def _list64(hits):
    """Powers of the fixed-size list: the 512 strongest of each plane in location order, -1 where there are fewer."""
    out = torch.full((len(hits), 512), -1.0, dtype=torch.float64)
    for j, (_, _, p) in enumerate(hits):
        p = p.cpu()
        if p.numel() > 512:
            p = p[torch.sort(p, descending=True, stable=True).indices[:512].sort().values]
        out[j, :p.numel()] = p
    return out.reshape(-1)


def _all64(hits):
    """Powers of the wide list, in the order of planes, rows and bins."""
    out = torch.zeros(RECORDS, dtype=torch.float64)
    p = torch.cat([p for _, _, p in hits]).cpu()
    out[:p.numel()] = p
    return {"harmonic": None, "template": None, "bin": None, "power": out, "total": None, "dropped": None}


def exact(case, seed):
    kind = case["kind"]
    if kind == "conv":
        n, rows = case["bins"], case["templates"]
        t = torch.from_numpy(template_spectra(_bank(rows)).astype(np.complex64)).cuda().to(torch.complex128)
        part = {0: range(rows // 2 + 1), 1: range(rows // 2, rows), 2: range(rows)}[case["part"]]
        fop = torch.zeros((rows, (n + 255) // 256 * 256), dtype=torch.float64, device="cuda")
        fop[:, :n] = _fop64(_spectrum(n, case["signals"], seed).to(torch.complex128), t, part)
        return {"fop": fop, "status": None}
    if kind == "batch":
        thr = _thresholds(case["planes"])
        return {"loc": None, "pwr": torch.stack([
            _list64(_hits64(_spectrum(n, sig, seed * 1000 + i).to(torch.complex128), BANK, thr))
            for i, (n, sig) in enumerate(_mix(kind, case["trials"], case["mix"]))])}
    if kind == "served":
        out = []
        for i, (n, sig, rows, planes) in enumerate(_mix(kind, case["requests"], case["mix"])):
            x = _spectrum(n, sig, seed * 1000 + i).to(torch.complex128)
            out.append(_all64(_hits64(x, _bank(rows), _thresholds(planes))))
        return out
    n = case["bins"]
    if kind in ("spectrum", "series"):
        x = _series(n, case.get("signals", 1), seed).double()
    if kind == "spectrum":
        return torch.fft.rfft(x)[:n] / (2 * n)
    if kind == "series":
        xs = [torch.fft.rfft(x)[:n] / math.sqrt(2 * n)]
    else:
        xs = [_spectrum(n, case["signals"], seed * 10 + i, case["strong"]).to(torch.complex128)
              for i in range(4 if kind == "loop" else 1)]
    hits = [_hits64(x, _bank(case["templates"]), _thresholds(case["planes"])) for x in xs]
    out = {"loc": None, "pwr": [_list64(h) for h in hits]}
    if kind == "list":
        out["all"] = _all64(hits[0])
    return out
