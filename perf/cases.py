"""The work that users of this library have it do, as cases that can be timed.

Two programs use the library.  A catalogue run (SGTpsv / SGTsh) holds a
context of one Earth model and asks it for batches of frequency slices; its
records are complex64 in host memory (what the drivers write to files), or
complex128 on the device for a caller that goes on there.  A kernel run
(KernelMaker) holds a catalogue handle per receiver radius and asks for time
series or per-point kernels of the points of its grid.  A third, occasional
use trains the network that predicts angular-order cutoffs.

Every input comes from the seed: the Earth model, the records, the spectra,
the points.  Sizes are those of the repository's benchmark configurations
(psv2048, psv1024, sh256, catalogue, kernels) and tests, with the number of
slices per call small enough that three contexts fit one GPU.
"""
import cmath
import ctypes
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
sys.path.insert(0, os.path.join(ROOT, "dsm-kernel_b200"))

import dsmsgt  # noqa: E402
from dsmsgt import synth  # noqa: E402

PRECISION = {"fp64": dsmsgt.DSM_PREC_FP64, "mixed": dsmsgt.DSM_PREC_MIXED}


# --------------------------------------------------------------- the cases
def listed():
    return [
        # one slice of a coarse model: a quick look at a set-up, the smallest
        # call of the engine, complex128 arrays back in the caller's memory
        dict(name="psv_quicklook", kind="sgt", mode="psv", precision="fp64", output="host", tlen=1638.4, imax=64,
             nfreq=1, rmin=1000.0, rmax=6300.0, rdelta=500.0, thdelta=15.0, depths="300"),
        # the plain FP64 configuration: slices of the 1024-frequency band that
        # the caller keeps on the device
        dict(name="psv_band1024_fp64", kind="sgt", mode="psv", precision="fp64", output="device", tlen=3276.8,
             imax=1024, nfreq=4, rmin=1000.0, rmax=6350.0, rdelta=26.75, thdelta=0.25, depths="300"),
        # the same band as a production catalogue: mixed precision, records
        # to the host
        dict(name="psv_band1024_mixed", kind="sgt", mode="psv", precision="mixed", output="records", tlen=3276.8,
             imax=1024, nfreq=8, rmin=1000.0, rmax=6350.0, rdelta=26.75, thdelta=0.25, depths="300"),
        # the benchmark's band and grid, records to the host: the largest
        # catalogue (orders to 7000, 1441 distances)
        dict(name="psv_band2048_mixed", kind="sgt", mode="psv", precision="mixed", output="records", tlen=3276.8,
             imax=2048, nfreq=3, rmin=1000.0, rmax=6350.0, rdelta=26.75, thdelta=0.125, depths="300"),
        # several source depths of one model in one context, the usual way
        # to build a catalogue for more than one event
        dict(name="psv_depths_mixed", kind="sgt", mode="psv", precision="mixed", output="records", tlen=1638.4,
             imax=256, nfreq=4, rmin=1000.0, rmax=6350.0, rdelta=53.5, thdelta=0.5, depths="10,300,600"),
        # SH catalogue of the reference's CPU configuration
        dict(name="sh_band256_mixed", kind="sgt", mode="sh", precision="mixed", output="records", tlen=1638.4,
             imax=256, nfreq=16, rmin=3500.0, rmax=6321.5, rdelta=28.5, thdelta=0.5, depths="100"),
        # a few SH slices in plain FP64 for a caller on the device
        dict(name="sh_few_fp64", kind="sgt", mode="sh", precision="fp64", output="device", tlen=1638.4, imax=128,
             nfreq=3, rmin=3500.0, rmax=6300.0, rdelta=100.0, thdelta=1.0, depths="100"),
        # time series at the points of a kernel grid from one receiver
        # radius of the large catalogue, all on the device
        dict(name="series_grid", kind="series", num=20, theta_n=1441, theta_delta=0.125, fmax=2048, tlen=3276.8,
             hz=2.0, start=400.0, end=1000.0, window_deg=10.0, slowness=0.0, points=1681, nout=6),
        # a handful of stations from a small catalogue with a reducing
        # slowness: launches and latency
        dict(name="series_stations", kind="series", num=10, theta_n=361, theta_delta=0.5, fmax=256, tlen=1638.4,
             hz=1.0, start=300.0, end=900.0, window_deg=10.0, slowness=8.0, points=37, nout=3),
        # P and S kernels at the points of the grid, spectra on the device
        dict(name="kernels_grid", kind="kernels", fmax=2048, tlen=3276.8, hz=2.0, start=400.0, end=1000.0,
             points=1681, nfilter=0, npoles=4, types=3, filtered=False, radii=4, host=False),
        # one profile of points with three pass bands, spectra in host
        # memory, the filtered series back as well
        dict(name="kernels_profile", kind="kernels", fmax=256, tlen=1638.4, hz=1.0, start=300.0, end=900.0,
             points=41, nfilter=2, npoles=4, types=3, filtered=True, radii=7, host=True),
        # a few epochs of the cutoff network on 64 models x 3 depths x 64
        # frequencies: forward, backward and update
        dict(name="cutoff_training", kind="training", samples=12288, epochs=4, batch=256),
    ]


def draw(rng):
    """One more case of the same ranges: band, grid, depth, batch and points
    spread over theirs, odd sizes among them."""
    def log_int(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    what = rng.choice(["psv", "psv", "psv", "sh", "sh", "series", "series", "kernels", "kernels", "training"])
    if what in ("psv", "sh"):
        precision = rng.choice(["mixed", "mixed", "fp64"])
        top = 1024 if what == "psv" else 256
        if what == "psv" and precision == "mixed":
            top = 2048
        imax = log_int(40, top)
        tlen = 3276.8 if what == "psv" and imax > 256 else 1638.4
        cap = 3 * 2048 if precision == "mixed" else 2048
        nfreq = rng.randint(1, max(1, min(8 if what == "psv" else 16, cap // imax)))
        depths = ",".join(str(d) for d in sorted(rng.sample(range(10, 651, 5), rng.choice([1, 1, 1, 2, 3]))))
        if what == "sh":
            depths = str(rng.randint(20, 500))
        elif imax > 512:
            depths = depths.split(",")[0]
        thdelta = rng.choice([0.25, 0.5, 1.0, 1.5, 3.0])
        rdelta = round(rng.uniform(26.75, 400.0), 2)
        rmin = rng.choice([1000.0, 1000.0, 3600.0]) if what == "psv" else 3500.0
        return dict(kind="sgt", mode=what, precision=precision,
                    output=rng.choice(["host", "device"]) if precision == "fp64" else "records", tlen=tlen,
                    imax=imax, nfreq=nfreq, rmin=rmin, rmax=6300.0, rdelta=rdelta, thdelta=thdelta, depths=depths)
    if what == "training":
        return dict(kind="training", samples=log_int(300, 12288), epochs=rng.randint(1, 4),
                    batch=rng.choice([64, 128, 256]))
    fmax = log_int(60, 2048)
    tlen = 3276.8 if fmax > 512 else 1638.4
    hz = 2.0 if fmax > 512 else 1.0
    start = round(rng.uniform(100.0, 500.0), 1)
    common = dict(fmax=fmax, tlen=tlen, hz=hz, start=start, end=round(start + rng.uniform(100.0, 600.0), 1),
                  points=log_int(5, 1681))
    if what == "series":
        delta = rng.choice([0.125, 0.25, 0.5])
        return dict(kind="series", num=rng.choice([10, 20]), theta_n=int(180 / delta) + 1, theta_delta=delta,
                    window_deg=rng.choice([5.0, 10.0]), slowness=rng.choice([0.0, 8.0]), nout=rng.randint(1, 6),
                    **common)
    return dict(kind="kernels", nfilter=rng.choice([0, 0, 1, 2]), npoles=rng.choice([2, 4, 6]),
                types=rng.choice([1, 2, 3, 3]), filtered=rng.random() < 0.3, radii=rng.randint(1, 9),
                host=rng.random() < 0.3, **common)


# ------------------------------------------------------------- preparation
def _freqs(case):
    """Slices spread evenly over the band."""
    n, imax = case["nfreq"], case["imax"]
    return sorted({max(1, int((j + 0.5) * imax / n)) for j in range(n)})


def _depths(case):
    return [float(d) for d in case["depths"].split(",")]


def _grid(case):
    radii = int(math.floor((case["rmax"] - case["rmin"]) / case["rdelta"] + 1e-9)) + 1
    return radii, int(round(180.0 / case["thdelta"])) + 1


def _prepare_sgt(case, seed):
    model = (synth.psv_earth_model if case["mode"] == "psv" else synth.sh_mantle_model)(seed)
    setups = []
    for d in _depths(case):
        text = synth.param_file(tlen=case["tlen"], rmin=case["rmin"], rmax=case["rmax"], rdelta=case["rdelta"],
                                r0=6371.0 - d, thmin=0.0, thmax=180.0, thdelta=case["thdelta"], imin=0,
                                imax=case["imax"])
        setups.append(dsmsgt.Setup(dsmsgt.Job(text, synth.dsm_config(), model), case["mode"]))
    fl = np.array(_freqs(case), np.int32)
    prec = PRECISION[case["precision"]]
    if len(setups) == 1:
        ctx = dsmsgt.Context(setups[0], precision=prec, freq_batch=len(fl))
    else:
        ctx = dsmsgt.MultiSourceContext(setups, precision=prec, freq_batch=len(fl))
    s = dict(run=_RUN_SGT[case["output"]], ctx=ctx, setups=setups, freqs=fl)
    if case["output"] == "records":
        # the caller's record buffers (pinned, reused from call to call)
        nt, nr, ns = setups[0].num
        R, T = setups[0].r_n, setups[0].theta_n
        s["rec"] = [tuple(torch.empty(shape, dtype=torch.complex64, pin_memory=True) for shape in
                          ((len(fl), R, T, nt), (len(fl), R, T, nr), (len(fl), T, ns))) for _ in setups]
        s["llog"] = [np.zeros(len(fl), np.int32) for _ in setups]
    return s


def _run_host(s):
    if len(s["setups"]) == 1:
        return list(s["ctx"].run(s["freqs"]))
    return [list(x) for x in s["ctx"].run(s["freqs"])]


class _DeviceArray:
    """A device buffer of a context as torch sees it; the tensor made from it
    holds this object, and so the context that owns the memory."""

    def __init__(self, ctx, ptr, shape):
        self.ctx = ctx
        self.__cuda_array_interface__ = {"shape": tuple(shape) + (2,), "typestr": "<f8", "data": (ptr, False),
                                         "version": 3, "strides": None}


def _run_device(s):
    fl, setup = s["freqs"], s["setups"][0]
    if len(s["setups"]) > 1:
        return _run_host(s)
    p = [ctypes.c_void_p() for _ in range(3)]
    llog = np.zeros(len(fl), np.int32)
    ip = ctypes.POINTER(ctypes.c_int)
    rc = dsmsgt.lib().dsm_run_freqs_device(s["ctx"].h, fl.ctypes.data_as(ip), len(fl), *(ctypes.byref(x) for x in p),
                                           llog.ctypes.data_as(ip))
    if rc:
        raise dsmsgt.DsmError("dsm_run_freqs_device failed", rc)
    return [torch.as_tensor(_DeviceArray(s["ctx"], x.value, shape), device="cuda")
            for x, shape in zip(p, setup.out_shapes(len(fl)))] + [llog]


def _run_records(s):
    fl, n = s["freqs"], len(s["setups"])
    outs = (dsmsgt.Out * n)()
    fp, ip = ctypes.POINTER(ctypes.c_float), ctypes.POINTER(ctypes.c_int)
    for o, rec, llog in zip(outs, s["rec"], s["llog"]):
        o.tsgt32, o.rsgt32, o.synn32 = (ctypes.cast(ctypes.c_void_p(x.data_ptr()), fp) for x in rec)
        o.llog = llog.ctypes.data_as(ip)
    L = dsmsgt.lib()
    if n == 1:
        rc = L.dsm_run_freqs(s["ctx"].h, fl.ctypes.data_as(ip), len(fl), outs)
    else:
        rc = L.dsm_run_freqs_multi(s["ctx"].h, fl.ctypes.data_as(ip), len(fl), outs, n)
    if rc:
        raise dsmsgt.DsmError("dsm_run_freqs failed", rc)
    return [list(rec) + [llog] for rec, llog in zip(s["rec"], s["llog"])]


_RUN_SGT = {"host": _run_host, "device": _run_device, "records": _run_records}


def _catalogue_params(case):
    np1, hz, s0, s1 = dsmsgt.cat_np1(case["tlen"], case["fmax"], case["hz"], case["start"], case["end"])
    return dict(num=case.get("num", 20), theta_n=case.get("theta_n", 361), theta_min=0.0,
                theta_delta=case.get("theta_delta", 0.5), fmin=0, fmax=case["fmax"], np1=np1, tlen=case["tlen"],
                omegai=math.log(100.0) / case["tlen"], ipdistance=case.get("window_deg", 10.0),
                c_red_reci=case.get("slowness", 0.0), iwin_start=s0, iwin_end=s1), hz


def _decay(nf):
    """Amplitude of a source spectrum over the band (a smooth low-pass)."""
    x = np.arange(nf) / nf
    return 1.0 / (1.0 + (x / 0.3) ** 4)


def _series_inputs(case, seed):
    p, _ = _catalogue_params(case)
    g = torch.Generator(device="cuda").manual_seed(seed)
    nf = p["fmax"] + 1
    rec = torch.view_as_complex(torch.randn((nf, p["theta_n"], p["num"], 2), generator=g, device="cuda"))
    rec = (rec * torch.from_numpy(_decay(nf)).float().cuda()[:, None, None]).contiguous()
    r = np.random.default_rng(seed)
    dist = np.sort(r.uniform(20.0, 90.0, case["points"]))
    coef = r.standard_normal((case["points"], case["nout"], p["num"]))
    return p, rec, dist, coef


def _prepare_series(case, seed):
    p, rec, dist, coef = _series_inputs(case, seed)
    cat = dsmsgt.Catalogue(p)
    cat.add(rec)
    out = torch.empty((len(dist), case["nout"], cat.nwin), dtype=torch.float64, device="cuda")
    return dict(run=_run_series, cat=cat, rec=rec, dist=dist, coef=coef, out=out)


def _run_series(s):
    # a radius at a time: its records are registered, then read at the points
    s["cat"].clear()
    s["cat"].add(s["rec"])
    return s["cat"].series(s["dist"], s["coef"], out=s["out"])


def _kernel_inputs(case, seed):
    p, hz = _catalogue_params(case)
    nf, n, nwin = p["fmax"] + 1, case["points"], p["iwin_end"] - p["iwin_start"] + 1
    g = torch.Generator(device="cuda").manual_seed(seed)
    shape = torch.from_numpy(_decay(nf)).cuda()
    h = [(torch.randn((n, 6, nf), generator=g, device="cuda", dtype=torch.complex128) * shape).contiguous()
         for _ in range(2)]
    r = np.random.default_rng(seed)
    nfl = case["nfilter"] + 1
    kp = dict(types=case["types"], nfilter=case["nfilter"], fclp=[0.005 * (k + 1) for k in range(nfl)],
              fchp=[0.05 + 0.01 * k for k in range(nfl)], npoles=case["npoles"], sampling_hz=hz,
              nt1=[p["iwin_start"] + nwin // 8 + k for k in range(nfl)],
              nt2=[p["iwin_end"] - nwin // 8 - k for k in range(nfl)],
              coeff=r.standard_normal((nwin, case["radii"], 8, nfl)),
              jacobian=r.standard_normal((nf, case["radii"])) + 1j * r.standard_normal((nf, case["radii"])))
    return p, h[0], h[1], kp, r.integers(0, case["radii"], n).astype(np.int32)


def _prepare_kernels(case, seed):
    p, h3, h4, kp, ir = _kernel_inputs(case, seed)
    cat = dsmsgt.Catalogue(p)
    cat.set_kernel_params(kp["types"], kp["nfilter"], kp["fclp"], kp["fchp"], kp["npoles"], kp["sampling_hz"],
                          kp["nt1"], kp["nt2"], kp["coeff"], kp["jacobian"])
    if case["host"]:
        h3, h4 = h3.cpu().numpy(), h4.cpu().numpy()
    return dict(run=_run_kernels, cat=cat, h3=h3, h4=h4, ir=ir, filtered=case["filtered"])


def _run_kernels(s):
    return s["cat"].kernels(s["ir"], s["h3"], s["h4"], filtered=s["filtered"])


def _prepare_training(case, seed):
    r = np.random.default_rng(seed)
    n = case["samples"]
    X = np.empty((n, dsmsgt.LMAX_NFEAT), np.float32)
    X[:, 0] = np.log1p(r.uniform(1.0, 2048.0, n) * 2 * math.pi / 3276.8 * 6371.0 / 3.2)
    lo = [0.90, 0.995, 0.31, 0.38, 0.31, 0.71, 0.01, 0.25, 1.0, 0.6]
    hi = [0.998, 0.997, 0.33, 0.47, 0.33, 0.74, 0.60, 0.26, 1.0, 0.95]
    X[:, 1:] = r.uniform(lo, hi, (n, 10))
    T = (0.9 * np.exp(-0.6 * X[:, 0]) - 0.04 * X[:, 0] + 0.3 * X[:, 7] + 0.01 * r.standard_normal(n)).astype(np.float32)
    return dict(run=_run_training, X=X, T=T, P=dsmsgt.lmax_init(X, T, seed=seed % 1000), epochs=case["epochs"],
                batch=case["batch"])


def _run_training(s):
    P, losses = dsmsgt.lmax_train(s["X"], s["T"], s["P"], epochs=s["epochs"], batch=s["batch"], lr=1e-3,
                                  weight_decay=1e-3)
    return [P, losses]


_PREPARE = {"sgt": _prepare_sgt, "series": _prepare_series, "kernels": _prepare_kernels,
            "training": _prepare_training}


def prepare(case, seed):
    return _PREPARE[case["kind"]](case, seed)


def run(state):
    return state["run"](state)


# --------------------------------------------------------- necessary work
def work(case):
    kind = case["kind"]
    if kind == "sgt":
        R, T = _grid(case)
        psv = case["mode"] == "psv"
        nt, nr, ns = (20, 10, 10) if psv else (10, 5, 5)
        nsrc, nbytes = len(_depths(case)), 8 if case["output"] == "records" else 16
        flops = bytes_ = 0.0
        vtop = 3.2 if psv else 6.0
        for f in _freqs(case):
            # orders to the cutoff: those of waves at the surface, and the
            # near field of the source
            L = 2 * math.pi * f / case["tlen"] * 6371.0 / vtop + 300.0
            # strains of a receiver and distance: real products of the
            # field rows of 18 (P-SV) or 8 (SH) slots with two basis columns
            flops += nsrc * (576.0 if psv else 96.0) * R * T * L
            # band rows of an order (about 16 nodes a wavelength), one
            # factorisation and the solves of its right-hand sides
            rows = (16.4 if psv else 6.0) * case["imax"] * 3276.8 / case["tlen"]
            flops += L * rows * (124.0 + 144.0 * nsrc if psv else 40.0)
            bytes_ += nsrc * (((nt + nr) * R + ns) * T * nbytes)
        return dict(bytes=bytes_, flops=flops)
    if kind == "training":
        steps = case["epochs"] * case["samples"]
        return dict(bytes=48.0 * case["samples"] + 2 * 4.0 * 34713, flops=6.0 * 34713 * steps)
    p, _ = _catalogue_params(case)
    nf, nwin, n2 = p["fmax"] + 1, p["iwin_end"] - p["iwin_start"] + 1, 2 * p["np1"]
    fft = 2.5 * n2 * math.log2(n2)
    if kind == "series":
        nw = 2 * int(case["window_deg"] / case["theta_delta"] / 2.0) + 1
        n = case["points"]
        used = min(p["theta_n"], int(70.0 / case["theta_delta"]) + nw)
        flops = n * (nf * (4.0 * nw * case["num"] + 4.0 * case["nout"] * case["num"]) + case["nout"] * fft)
        return dict(bytes=8.0 * nf * used * case["num"] + 8.0 * n * case["nout"] * (nwin + case["num"]), flops=flops)
    n, nfl = case["points"], case["nfilter"] + 1
    series = (1 if case["types"] & 1 else 0) + (2 if case["types"] & 2 else 0)
    flops = n * (nf * 80.0 + series * (fft + nfl * nwin * (7.0 * case["npoles"] + 6.0)))
    out = 72.0 * nfl + (8.0 * series * nfl * nwin if case["filtered"] else 0.0)
    return dict(bytes=n * (2 * 6 * 16.0 * nf + out), flops=flops)


# ------------------------------------------------------------- in 64 bits
def exact(case, seed):
    """Series and kernels from their definitions in 64 bits.  An SGT slice has
    no short definition: its value is thousands of band solves and their sum
    over orders, minutes on a host; the training run's depends on the order
    in which the trainer draws its batches."""
    if case["kind"] == "series":
        return _exact_series(case, seed)
    if case["kind"] == "kernels":
        return _exact_kernels(case, seed)
    return None


def _transform(p, spec):
    """Windowed real series of spectra [..., fmax+1]: Hermitian extension,
    unnormalised inverse transform of 2 np1 points, growth and scale."""
    n1, n2 = p["np1"], 2 * p["np1"]
    H = torch.zeros(spec.shape[:-1] + (n2,), dtype=torch.complex128, device=spec.device)
    H[..., :spec.shape[-1]] = spec
    H[..., n1:] = torch.conj(torch.flip(H[..., 1:n1 + 1], dims=(-1,)))
    x = torch.fft.ifft(H, norm="forward").real[..., p["iwin_start"]:p["iwin_end"] + 1]
    t = torch.arange(p["iwin_start"], p["iwin_end"] + 1, dtype=torch.float64, device=spec.device) * p["tlen"] / n2
    return x * torch.exp(p["omegai"] * t) / p["tlen"] * 1e3


def _exact_series(case, seed):
    p, rec, dist, coef = _series_inputs(case, seed)
    dev = rec.device
    nf, T, d = p["fmax"] + 1, p["theta_n"], p["theta_delta"]
    f = torch.arange(nf, dtype=torch.float64, device=dev)
    theta = torch.arange(T, dtype=torch.float64, device=dev) * d
    w = 2.0 * math.pi / p["tlen"] * p["c_red_reci"]
    W = torch.zeros((len(dist), T), dtype=torch.float64)
    half = int(p["ipdistance"] / d / 2.0)
    for k, x in enumerate(dist):
        lo, hi = int(x / d) - half, int(x / d) + half
        if lo < 0:
            lo, hi = 0, hi - lo
        if hi > T - 1:
            lo, hi = max(0, lo - (hi - T + 1)), T - 1
        u = np.sinc((x - lo * d) / d - np.arange(hi - lo + 1))
        W[k, lo:hi + 1] = torch.from_numpy(u / u.sum())
    W, C = W.to(dev), torch.from_numpy(coef).to(dev)
    dd = torch.from_numpy(dist).to(dev)
    spec = torch.empty((len(dist), case["nout"], nf), dtype=torch.complex128, device=dev)
    for k in range(nf):
        a = rec[k].to(torch.complex128) * (1e-21 * torch.polar(torch.ones_like(theta), w * k * theta))[:, None]
        v = W.to(torch.complex128) @ a
        v = v * torch.polar(torch.ones_like(dd), -w * k * dd)[:, None]
        spec[:, :, k] = torch.einsum("pjc,pc->pj", C.to(torch.complex128), v)
    spec[:, :, 0] = 0
    return _transform(p, spec)


def _sections(f1, f2, npoles, dt):
    """Second-order sections of KernelMaker's band-pass, whose poles pass
    through single precision (its complex constants have no kind)."""
    d2 = 2.0 / dt
    w1, w2 = (d2 * math.tan(2.0 * math.pi * f / d2) for f in (f1, f2))
    w0 = 0.5 * (w2 - w1)
    roots = []
    for n in range(1, npoles + 1):
        ph = float(np.float32((2 * n - 1 + npoles) * math.pi / (2 * npoles)))
        t1 = complex(np.float32(math.cos(ph)), np.float32(math.sin(ph))) * float(np.float32(w0))
        t2 = cmath.sqrt(t1 * t1 - float(np.float32(w1 * w2)))
        roots += [t1 + t2, t1 - t2]
    out = []
    for s in roots[:npoles]:
        q = abs(s) ** 2
        f1_ = d2 * d2 - 2.0 * d2 * s.real + q
        out.append((2.0 * d2 * w0 / f1_, 2.0 * (q - d2 * d2) / f1_, (d2 * d2 + 2.0 * d2 * s.real + q) / f1_))
    return out


def _exact_kernels(case, seed):
    p, h3, h4, kp, ir = _kernel_inputs(case, seed)
    dev = h3.device
    irt = torch.from_numpy(ir.astype(np.int64)).to(dev)
    # chunks of points keep the transforms small
    du = []
    for a in range(0, len(ir), 128):
        x, y, spec = h3[a:a + 128], h4[a:a + 128], []
        if kp["types"] & 1:
            spec.append(-(x[:, 0] + x[:, 1] + x[:, 2]) * (y[:, 0] + y[:, 1] + y[:, 2]) * 1e3)
        if kp["types"] & 2:
            shear = x[:, 3] * y[:, 3] + x[:, 4] * y[:, 4] + x[:, 5] * y[:, 5]
            cross = x[:, 0] * (y[:, 1] + y[:, 2]) + x[:, 1] * (y[:, 0] + y[:, 2]) + x[:, 2] * (y[:, 0] + y[:, 1])
            diag = x[:, 0] * y[:, 0] + x[:, 1] * y[:, 1] + x[:, 2] * y[:, 2]
            jac = torch.from_numpy(kp["jacobian"]).to(dev).T[irt[a:a + 128]]
            spec.append((cross - 2.0 * shear) * 1e3)
            spec.append((2.0 / 3.0 * cross - 4.0 * shear - 4.0 / 3.0 * diag) * jac * 1e3)
        du.append(_transform(p, torch.stack(spec, 1)))
    x = torch.cat(du).cpu().numpy()
    nfl, nwin = kp["nfilter"] + 1, x.shape[-1]
    filt = np.empty(x.shape[:2] + (nfl, nwin))
    ker = np.zeros((len(ir), nfl, kp["coeff"].shape[2] + 1))
    uses = ([(1, 3, 4)] if kp["types"] & 1 else []) + ([(5, 7), (8,)] if kp["types"] & 2 else [])
    for f in range(nfl):
        y = x
        for a, b1, b2 in _sections(kp["fclp"][f], kp["fchp"][f], kp["npoles"], 1.0 / kp["sampling_hz"]):
            z = np.zeros_like(y)
            for t in range(nwin):
                z[..., t] = a * (y[..., t] - (y[..., t - 2] if t > 1 else 0.0))
                if t > 0:
                    z[..., t] -= b1 * z[..., t - 1]
                if t > 1:
                    z[..., t] -= b2 * z[..., t - 2]
            y = z
        filt[:, :, f] = y
        t1, t2 = kp["nt1"][f] - p["iwin_start"], kp["nt2"][f] - p["iwin_start"]
        wt = np.zeros(nwin)
        wt[t1:t2 + 1] = 1.0
        wt[t1] -= 0.5
        wt[t2] -= 0.5
        for s, ks in enumerate(uses):
            for k in ks:
                c = kp["coeff"][:, ir, k - 1, f].T
                ker[:, f, k] = (c * wt * y[:, s]).sum(-1)
    return (ker, filt) if case["filtered"] else ker
