"""The work that users of this framework have it do, as cases that can be timed.

Every case goes through the package's public entry points: the stage calls
(channelise, bandpass, the RFI and statistics calls, DedispPlan, boxcar) with
device buffers that a program keeps, and the plan API (Plan) for a whole
observation.  The sizes are those of the package's own configurations:

  * the reference's defaults: 360 MHz, 3908 channels, NAVE 4, bundles of 32 rows;
  * the full band: 384 MHz, 6250 channels, NAVE 10 (1024 rows per second),
    in 1-s chunks (streaming) or blocks of several seconds;
  * the small plain configuration: 7.5-s blocks, DM 0-200 in 201 trials, with
    its FP16 and int8 forms;
  * the full-scale grid: DM 0-1000 in 2048 trials;
  * the two-trial time-series tool: 3840 channels, NAVE 4, DM 0 and 119.3.

listed() names the cases, draw() gives more of the same ranges, prepare() makes
what a program holds before the call, run() is one pass, work() its unavoidable
bytes and operations, exact() the same outputs in 64 bits by plain torch.
"""
import importlib.util
import math
import os
import sys

import numpy as np
import torch

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
N_FFT = 12500          # samples per window
FPS = 25600            # frames per second and polarisation
FRAME, HDR, DATA = 5032, 32, 5000
RATE = 128e6
F32, F16, I8 = 0, 1, 2


def _package():
    """The package (its folder's name holds a hyphen)."""
    if "vlite_frb_b200" not in sys.modules:
        d = os.path.join(ROOT, "vlite-frb_b200")
        spec = importlib.util.spec_from_file_location("vlite_frb_b200", os.path.join(d, "__init__.py"),
                                                      submodule_search_locations=[d])
        m = importlib.util.module_from_spec(spec)
        sys.modules["vlite_frb_b200"] = m
        spec.loader.exec_module(m)
    return sys.modules["vlite_frb_b200"]


def listed():
    return [
        # one bundle at the reference's defaults: what block mode channelises as
        # soon as 32 rows' frames are there (the smallest call, latency counts)
        dict(name="channelise_bundle", kind="channelise", rows=32, nave=4, muos=360.0),
        # 8 s of the full band at once: batch processing of a recording
        dict(name="channelise_8s", kind="channelise", rows=8192, nave=10, muos=384.0),
        # the bandpass of one 7.5-s block, plain FP32 form
        dict(name="bandpass_block_f32", kind="bandpass", rows=7680, nch=6250, storage=F32),
        # the bandpass of one 1-s chunk in streaming, FP16 form with its shifted copy
        dict(name="bandpass_chunk_f16", kind="bandpass", rows=1024, nch=6250, storage=F16),
        # RFI-heavy statistics of one block: whole-block bandpass, zero-DM
        # subtraction, the time-major product, 1-s channel statistics, kurtosis
        dict(name="rfi_stats_block", kind="rfi", rows=7680, nch=6250, ncol=1024),
        # the small plain configuration's block: 201 trials, an odd sample count
        dict(name="dedisp_201_f32", kind="dedisp", ndm=201, dm_max=200.0, nave=10, muos=384.0, nt=5145, storage=F32,
             stats=True),
        # the same block in its int8 form (a weight per channel)
        dict(name="dedisp_201_i8", kind="dedisp", ndm=201, dm_max=200.0, nave=10, muos=384.0, nt=5145, storage=I8,
             stats=True),
        # the full-scale grid over 16 s with per-trial statistics
        dict(name="dedisp_2048_f32", kind="dedisp", ndm=2048, dm_max=1000.0, nave=10, muos=384.0, nt=16384,
             storage=F32, stats=True),
        # one streamed 1-s chunk of the full-scale grid, FP16 form, series only
        dict(name="dedisp_chunk_f16", kind="dedisp", ndm=2048, dm_max=1000.0, nave=10, muos=384.0, nt=1024,
             storage=F16, stats=False),
        # the time-series tool's block: two trials with per-sample channel sigma
        dict(name="series_sigma", kind="sigma", dm=119.3, nt=18211),
        # the candidate search of a 1-s chunk of 2048 series, boxcars to 16 samples
        dict(name="boxcar_chunk", kind="boxcar", ndm=2048, nt=1024, width=16),
        # a whole observation through the plan API, streamed: 4 s of frames
        # already on the device in 1-s pushes, 256 trials, boxcar candidates
        dict(name="plan_stream_4s", kind="plan", seconds=4, ndm=256, dm_max=100.0, width=16),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["channelise", "bandpass", "rfi", "dedisp", "dedisp", "dedisp", "sigma", "boxcar"])
    if kind == "channelise":
        nave, muos = rng.choice([(4, 360.0), (10, 384.0), (10, 360.0), (4, 384.0)])
        return dict(kind=kind, rows=_log(rng, 32, 8192), nave=nave, muos=muos)
    if kind == "bandpass":
        return dict(kind=kind, rows=_log(rng, 128, 8192), nch=rng.choice([3840, 3908, 6250]),
                    storage=rng.choice([F32, F16, I8]))
    if kind == "rfi":
        ncol = rng.choice([512, 1024, 1000])
        return dict(kind=kind, rows=max(ncol, _log(rng, 1024, 8192)), nch=rng.choice([3840, 3908, 6250]), ncol=ncol)
    if kind == "dedisp":
        nave, muos = rng.choice([(4, 360.0), (10, 384.0), (10, 384.0)])
        ndm = _log(rng, 24, 2048)
        nt = _log(rng, 300, 16384)
        return dict(kind=kind, ndm=ndm, dm_max=round(rng.uniform(0.1, 1.0) * min(1000.0, 2.0 * ndm), 1), nave=nave,
                    muos=muos, nt=nt, storage=rng.choice([F32, F32, F16, I8]), stats=rng.random() < 0.5)
    if kind == "sigma":
        return dict(kind=kind, dm=round(rng.uniform(5.0, 300.0), 1), nt=_log(rng, 1000, 40000))
    return dict(kind=kind, ndm=_log(rng, 32, 2048), nt=_log(rng, 300, 16384), width=rng.choice([1, 4, 8, 16, 32, 64]))


# ---- inputs --------------------------------------------------------------------
def _gen(seed, salt=0):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed) * 1009 + salt)
    return g


def _frames(npairs, seed):
    """Frames of both polarisations as a capture writes them: 32-byte headers,
    8-bit noise clip(round(128 + 12 N(0, 1)))."""
    sp = sys.modules.get("vlite_frb_b200_synth")
    if sp is None:
        spec = importlib.util.spec_from_file_location("vlite_frb_b200_synth",
                                                      os.path.join(ROOT, "vlite-frb_b200", "synth.py"))
        sp = importlib.util.module_from_spec(spec)
        sys.modules["vlite_frb_b200_synth"] = sp
        spec.loader.exec_module(sp)
    head = sp._headers(npairs, sp.StreamSpec(duration=npairs / FPS, seed=seed), None)
    out = torch.empty((npairs, 2, FRAME), dtype=torch.uint8, device="cuda")
    out[:, :, :HDR] = torch.from_numpy(head).cuda()
    g = _gen(seed)
    for a in range(0, npairs, 12800):
        b = min(npairs, a + 12800)
        x = torch.randn((b - a, 2, DATA), generator=g, device="cuda") * 12.0 + 128.0
        out[a:b, :, HDR:] = x.round_().clamp_(0, 255).to(torch.uint8)
    return out.view(-1)


def _raw_power(rows, nch, seed, nave=10):
    """A raw time-major filterbank: chi-square power (2 pols x NAVE spectra) on
    a bandpass shape, with the 10-Hz calibration step every 128 rows."""
    g = _gen(seed, 1)
    k = 4.0 * nave
    z = torch.randn((rows, nch), generator=g, device="cuda")
    x = (z.mul_(math.sqrt(2.0 / (9.0 * k))).add_(1.0 - 2.0 / (9.0 * k))).pow_(3)
    base = torch.rand(nch, generator=g, device="cuda") * 100.0 + 250.0
    cal = 1.0 + 0.1 * ((torch.arange(rows, device="cuda") // 128) % 2).float()
    return x.mul_(base).mul_(cal[:, None])


def _delays(dms, nave, muos, fixed=0):
    vf = _package()
    L = vf.layout(nave=nave, muoslowfreq=muos, nchanout_fixed=fixed)
    off, _ = vf.delay_table(L, np.asarray(dms, np.float32))
    return L, off


def _bandpassed(off, nt, seed, align=16):
    """A bandpass-subtracted channel-major filterbank [nchan][rows] of unit
    noise with a few dispersed pulses."""
    ndm, nch = off.shape
    rows = nt + int(off.max())
    g = _gen(seed, 2)
    x = torch.zeros((nch, (rows + align - 1) // align * align), device="cuda")
    x[:, :rows] = torch.randn((nch, rows), generator=g, device="cuda")
    rng = np.random.default_rng(seed)
    c = torch.arange(nch, device="cuda")
    for _ in range(3):
        d, t = int(rng.integers(0, ndm)), int(rng.integers(0, nt))
        x[c, torch.from_numpy(off[d]).cuda().long() + t] += float(rng.uniform(0.1, 0.4))
    return x, rows


def _dedisp_inputs(case, seed):
    dms = np.linspace(0.0, case["dm_max"], case["ndm"]).astype(np.float32)
    _, off = _delays(dms, case["nave"], case["muos"])
    x, rows = _bandpassed(off, case["nt"], seed)
    kw = {}
    if case["storage"] == F16:
        x = x.half()
        x1 = torch.zeros_like(x)
        x1[:, :-1] = x[:, 1:]
        kw = dict(uniform_scale=3.7, fb_shift1=x1)
    elif case["storage"] == I8:
        x = (x * 16.0).round_().clamp_(-127, 127).to(torch.int8)
        w = torch.rand(x.shape[0], generator=_gen(seed, 3), device="cuda") * 2.0 + 2.0
        kw = dict(chan_scale=w / 16.0)
    return off, x, rows, kw


def prepare(case, seed):
    vf = _package()
    kind = case["kind"]
    if kind == "channelise":
        npairs = (case["rows"] * case["nave"] * N_FFT + DATA - 1) // DATA
        L = vf.layout(nave=case["nave"], muoslowfreq=case["muos"])
        idx = torch.arange(npairs, dtype=torch.int64, device="cuda") * (2 * FRAME) + HDR
        return dict(kind=kind, frames=_frames(npairs, seed), s0=idx, s1=idx + FRAME, rows=case["rows"], L=L,
                    out=torch.empty((case["rows"], L.nchanout), device="cuda"))
    if kind == "bandpass":
        raw = _raw_power(case["rows"], case["nch"], seed)
        st = dict(kind=kind, raw=raw, storage=case["storage"], inv=None, out1=None)
        dt = {F32: torch.float32, F16: torch.float16, I8: torch.int8}[case["storage"]]
        st["out"] = torch.zeros((case["nch"], (case["rows"] + 15) // 16 * 16), dtype=dt, device="cuda")
        if case["storage"] == F16:
            st["out1"] = torch.zeros_like(st["out"])
        if case["storage"] != F32:
            st["inv"] = 1.0 / raw[:128].std(dim=0)
        return st
    if kind == "rfi":
        rows, nch = case["rows"], case["nch"]
        return dict(kind=kind, raw=_raw_power(rows, nch, seed), rows=rows, ncol=case["ncol"], nblk=rows // case["ncol"],
                    cm=torch.zeros((nch, (rows + 15) // 16 * 16), device="cuda"),
                    tm=torch.empty((rows, nch), device="cuda"))
    if kind == "dedisp":
        off, x, rows, kw = _dedisp_inputs(case, seed)
        plan = vf.DedispPlan(off)
        return dict(kind=kind, plan=plan, x=x, rows=rows, kw=kw, nt=case["nt"], storage=case["storage"],
                    stats=case["stats"], out=torch.empty((case["ndm"], case["nt"]), device="cuda"),
                    ws=torch.empty(max(1, plan.workspace_bytes(case["nt"])), dtype=torch.uint8, device="cuda"))
    if kind == "sigma":
        _, off = _delays([0.0, case["dm"]], 4, 360.0, 3840)
        x, rows = _bandpassed(off, case["nt"], seed)
        return dict(kind=kind, plan=vf.DedispPlan(off), x=x, rows=rows, nt=case["nt"],
                    out=torch.empty((2, case["nt"]), device="cuda"), sig=torch.empty((2, case["nt"]), device="cuda"))
    if kind == "boxcar":
        x = _series(case, seed)
        return dict(kind=kind, x=x, ave=x.mean(dim=1), sig=x.std(dim=1), width=case["width"])
    dms = np.linspace(0.0, case["dm_max"], case["ndm"]).astype(np.float32)
    plan = vf.Plan(dms, nave=10, muoslowfreq=384.0, mode=vf.MODE_STREAM, nstreams=0, chunk_seconds=1.0,
                   ring_seconds=2.0, outputs=vf.OUT_DEDISP | vf.OUT_DMSTATS | vf.OUT_CANDS, cand_snr=7.0,
                   boxcar_max=case["width"])
    return dict(kind=kind, plan=plan, frames=_frames(case["seconds"] * FPS, seed))


def _series(case, seed):
    g = _gen(seed, 4)
    x = torch.randn((case["ndm"], case["nt"]), generator=g, device="cuda") * 0.013
    d = torch.arange(0, case["ndm"], 17, device="cuda")
    x[d, (d * 31) % case["nt"]] += 0.1
    return x


# ---- one pass --------------------------------------------------------------------
def run(s):
    vf = _package()
    kind = s["kind"]
    if kind == "channelise":
        return vf.channelise(s["frames"], s["s0"], s["s1"], 0, s["rows"], s["L"], out=s["out"])
    if kind == "bandpass":
        vf.bandpass(s["raw"], storage=s["storage"], out=s["out"], inv_scale=s["inv"], out_shift1=s["out1"])
        return dict(out=s["out"], out1=s["out1"])
    if kind == "rfi":
        cm, rows = s["cm"], s["rows"]
        vf.bandpass(s["raw"], out=cm, subtract_mode=1)
        vf.subtract_bp_full(cm, nrows=rows)
        vf.subtract_zero(cm, nrows=rows)
        vf.fb_to_time_major(cm, nrows=rows, out=s["tm"])
        ave, sig, outlier = vf.chan_stats(cm, rows, s["ncol"], s["nblk"])
        sk = vf.chan_sk(s["raw"], s["ncol"], s["nblk"], 20)
        return dict(cm=cm, tm=s["tm"], ave=ave, sig=sig, outlier=outlier, sk=sk)
    if kind == "dedisp":
        out, st = s["plan"](s["x"], s["nt"], storage=s["storage"], nrows_valid=s["rows"], out=s["out"],
                            stats=s["stats"], workspace=s["ws"], **s["kw"])
        return dict(out=out, **st)
    if kind == "sigma":
        s["plan"](s["x"], s["nt"], nrows_valid=s["rows"], out=s["out"], sigma_out=s["sig"], stats=False)
        return dict(out=s["out"], sigma=s["sig"])
    if kind == "boxcar":
        snr, start, width = vf.boxcar(s["x"], s["ave"], s["sig"], s["width"])
        return dict(snr=snr, start=start, width=width)
    plan, frames = s["plan"], s["frames"]
    sid = plan.open_stream()
    got = []
    piece = 2 * FPS * FRAME
    for a in range(0, frames.numel(), piece):
        plan.push(sid, frames[a:a + piece])
        while (r := plan.poll(wait=False)) is not None:
            got.append(r)
    plan.push(sid, None)
    got += plan.drain()
    plan.close_stream(sid)
    keys = ("dd", "ave", "sigma", "peak", "frb", "argmax", "box_snr", "box_start", "box_width")
    return [{k: r[k] for k in keys} for r in got]


# ---- what a pass cannot do without ---------------------------------------------------
def _nch(muos):
    n = int((muos - 320.0) / (64.0 / 6250)) + 1
    n += n % 2
    return min(n, 6250)


def work(case):
    kind = case["kind"]
    if kind == "channelise":
        win = 2 * case["rows"] * case["nave"]
        return {"bytes": win * N_FFT + 4 * case["rows"] * _nch(case["muos"]),
                "flops": win * 2.5 * N_FFT * math.log2(N_FFT)}
    if kind == "bandpass":
        n = case["rows"] * case["nch"]
        return {"bytes": n * (4 + {F32: 4, F16: 4, I8: 1}[case["storage"]]), "flops": 10 * n}
    if kind == "rfi":
        n = case["rows"] * case["nch"]
        return {"bytes": 12 * n, "flops": 30 * n}  # raw read, cm and tm written
    if kind == "dedisp":
        nch = _nch(case["muos"])
        rows = case["nt"] + _sweep(case["dm_max"], case["nave"], nch)
        eb = {F32: 4, F16: 2, I8: 1}[case["storage"]]
        return {"bytes": nch * rows * eb + 4 * case["ndm"] * case["nt"], "flops": nch * case["ndm"] * case["nt"]}
    if kind == "sigma":
        rows = case["nt"] + _sweep(case["dm"], 4, 3840)
        return {"bytes": 4 * 3840 * rows + 16 * case["nt"], "flops": 6 * 3840 * case["nt"]}
    if kind == "boxcar":
        n = case["ndm"] * case["nt"]
        return {"bytes": 4 * n, "flops": 4 * n * (1 + int(math.log2(case["width"])))}
    rows = 1024 * case["seconds"]
    win = 2 * rows * 10
    return {"bytes": win * N_FFT, "flops": win * 2.5 * N_FFT * math.log2(N_FFT) + 6250 * case["ndm"] * rows}


def _sweep(dm, nave, nch):
    """Largest delay in rows: the dispersion sweep over the band."""
    hi = 320.0 + nch * 64.0 / 6250
    return int(4.148808e3 * dm * (320.0 ** -2 - hi ** -2) / (nave * N_FFT / RATE))


# ---- the same in 64 bits ---------------------------------------------------------------
def _channelise64(frames, rows, nave, nch, nskip):
    pol = frames.view(-1, 2, FRAME)[:, :, HDR:]
    p = [pol[:, i].reshape(-1)[:rows * nave * N_FFT].view(rows, nave, N_FFT) for i in (0, 1)]
    out = torch.empty((rows, nch), dtype=torch.float64, device="cuda")
    step = max(1, 2048 // nave)
    for a in range(0, rows, step):
        acc = 0.0
        for x in p:
            f = torch.fft.rfft(x[a:a + step].double() - 128.0, dim=2)
            acc = acc + (f.real ** 2 + f.imag ** 2)[:, :, nskip:nskip + nch].mean(dim=1)
        out[a:a + step] = acc / (N_FFT // 2 + 1)
    return out


def _bandpass64(raw):
    out = torch.empty_like(raw, dtype=torch.float64)
    for a in range(0, raw.shape[0], 128):
        x = raw[a:a + 128].double()
        ave = x.mean(dim=0)
        var = x.var(dim=0)
        keep = (x < ave + 3.0 * var) & (x > ave - 3.0 * var)
        out[a:a + 128] = x - (x * keep).sum(dim=0) / keep.sum(dim=0).clamp(min=1)
    return out


def _dedisperse64(x, off, nt, scale):
    """(1/nchan) sum_c scale_c x[c][t + off[d][c]] for x [nchan][rows]."""
    ndm, nch = off.shape
    o = torch.from_numpy(np.ascontiguousarray(off.T)).cuda().long()
    out = torch.zeros((ndm, nt), dtype=torch.float64, device="cuda")
    for c in range(nch):
        win = (x[c].double() * scale[c]).unfold(0, nt, 1)
        out += win[o[c]]
    return out / nch


def _stats64(dd):
    ave, sig = dd.mean(dim=1), dd.std(dim=1)
    return dict(ave=ave, sigma=sig, peak=((dd.max(dim=1).values - ave) / sig).clamp(min=0.0))


def _boxcar64(dd, ave, sig, width):
    cs = torch.cat([torch.zeros((dd.shape[0], 1), dtype=torch.float64, device="cuda"), dd.cumsum(dim=1)], dim=1)
    best, w = None, 1
    while w <= min(width, dd.shape[1]):
        s = (((cs[:, w:] - cs[:, :-w]) - w * ave[:, None]) / (sig[:, None] * math.sqrt(w))).max(dim=1).values
        best = s if best is None else torch.maximum(best, s)
        w *= 2
    return best


def exact(case, seed):
    kind = case["kind"]
    if kind == "channelise":
        npairs = (case["rows"] * case["nave"] * N_FFT + DATA - 1) // DATA
        nch = _nch(case["muos"])
        return _channelise64(_frames(npairs, seed), case["rows"], case["nave"], nch, N_FFT // 2 - nch + 1)
    if kind == "bandpass":
        raw = _raw_power(case["rows"], case["nch"], seed)
        if case["storage"] == I8:
            return None  # whole numbers
        y = torch.zeros((case["nch"], (case["rows"] + 15) // 16 * 16), dtype=torch.float64, device="cuda")
        y[:, :case["rows"]] = _bandpass64(raw).t()
        if case["storage"] == F32:
            return dict(out=y, out1=None)
        y *= (1.0 / raw[:128].std(dim=0)).double()[:, None]
        y1 = torch.zeros_like(y)
        y1[:, :-1] = y[:, 1:]
        return dict(out=y, out1=y1)
    if kind == "rfi":
        rows, nch, ncol = case["rows"], case["nch"], case["ncol"]
        raw = _raw_power(rows, nch, seed)
        x = raw.double().t().contiguous()
        ave = x.sum(dim=1) / nch
        d = x - ave[:, None]
        var = ((d * d).sum(dim=1) - d.sum(dim=1) ** 2 / rows) / (rows - 1)
        keep = (d.abs() < 3.0 * var[:, None])
        x = x - ((x * keep).sum(dim=1) / keep.sum(dim=1))[:, None]
        del d, keep
        m, v = x.mean(dim=0), x.var(dim=0)
        keep = (x - m).abs() < 3.0 * v
        x = x - (x * keep).sum(dim=0) / keep.sum(dim=0).clamp(min=1)
        del keep
        nblk = rows // ncol
        b = x[:, :nblk * ncol].reshape(nch, nblk, ncol)
        a, s = b.mean(dim=2), b.var(dim=2)
        outl = torch.div((b > (a + 5.0 * s)[:, :, None]).sum(dim=2), ncol, rounding_mode="floor").double()
        r = raw[:nblk * ncol].double().view(nblk, ncol, nch)
        s1, s2 = r.sum(dim=1), (r * r).sum(dim=1)
        sk = (ncol * 20 + 1.0) / (ncol - 1.0) * (ncol * s2 / (s1 * s1) - 1.0)
        cm = torch.zeros((nch, (rows + 15) // 16 * 16), dtype=torch.float64, device="cuda")
        cm[:, :rows] = x
        return dict(cm=cm, tm=x.t().contiguous(), ave=a.t().contiguous(), sig=s.t().contiguous(),
                    outlier=outl.t().contiguous(), sk=sk)
    if kind == "dedisp":
        off, x, _, kw = _dedisp_inputs(case, seed)
        w = kw.get("chan_scale")
        scale = w.double() if w is not None else torch.full((x.shape[0],), float(np.float32(kw.get(
            "uniform_scale", 1.0))), dtype=torch.float64, device="cuda")
        dd = _dedisperse64(x, off, case["nt"], scale)
        return dict(out=dd, **(_stats64(dd) if case["stats"] else {}))
    if kind == "sigma":
        _, off = _delays([0.0, case["dm"]], 4, 360.0, 3840)
        x, _ = _bandpassed(off, case["nt"], seed)
        one = torch.ones(3840, dtype=torch.float64, device="cuda")
        m = _dedisperse64(x, off, case["nt"], one)
        q = _dedisperse64(x.double() ** 2, off, case["nt"], one)
        return dict(out=m, sigma=torch.sqrt((q - m * m) / (3840 - 1)))
    if kind == "boxcar":
        x = _series(case, seed)
        return dict(snr=_boxcar64(x.double(), x.mean(dim=1).double(), x.std(dim=1).double(), case["width"]),
                    start=None, width=None)
    rows = 1024 * case["seconds"]
    dms = np.linspace(0.0, case["dm_max"], case["ndm"]).astype(np.float32)
    _, off = _delays(dms, 10, 384.0)
    y = _bandpass64(_channelise64(_frames(case["seconds"] * FPS, seed), rows, 10, 6250, 1).float())
    nt = rows - int(off.max())
    dd = _dedisperse64(y.t().contiguous(), off, nt, torch.ones(6250, dtype=torch.float64, device="cuda"))
    got = []
    for a in range(0, nt, 1024):
        part = dd[:, a:a + 1024].contiguous()
        st = _stats64(part)
        got.append(dict(dd=part, **st, box_snr=_boxcar64(part, st["ave"], st["sigma"], case["width"])))
    return got
