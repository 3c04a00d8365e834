"""Workloads of the FRB search, each one call sequence of a user's program.

A case is one of five kinds:
  plan    hdd_execute_adv / hdd_execute_guru on device pointers: dedispersion
          alone, as a program that uses the dedisp-shaped plan API calls it;
  search  one gulp of a single- or multi-beam context (hella_process_gulp):
          flagging, dedispersion, smoothing and peak finding of one beam after
          another, to the candidate list;
  batch   one gulp of every beam of a batched context
          (hella_batch_process_gulp: one CUDA graph);
  stream  the serving loop's step: submit a gulp, poll the one before it, two
          in flight, beams being slots that can join and leave;
  step    one gradient step of the candidate refinement (forward + adjoint);
  fit     a whole Adam fit of a set of candidates.

Inputs are on the device: u8 filterbank gulps (or fp16 channel-major ones),
Gaussian noise with narrowband RFI, broadband impulses and dispersed bursts;
cutouts of dispersed bursts in unit noise.  The gulp loops feed the same gulp
again and again, its bursts painted periodically, so that every searched
window holds the same samples and a pass gives the same candidates.
"""
import math
import sys
from pathlib import Path

import numpy as np
import torch

sys.path.insert(0, str(Path(__file__).resolve().parent.parent / "casm-hella_gb300"))

import hella_gb300 as hg  # noqa: E402

F0, FLO = 468.75, 375.0  # MHz: channel 0 and the band's lower edge
K_DM = 4.148808e3        # s MHz^2 per unit DM
FWHM = 2.0 * math.sqrt(2.0 * math.log(2.0))
LR = (0.5, 0.2, 0.05, 0.05, 0.05)  # Adam rates of (dm, t0, width, amp, index)


def listed():
    return [
        # dedispersion of a short ragged block: 128 channels, 1501 output samples
        dict(name="plan_small", kind="plan", nchan=128, tsamp=1e-3, dm_max=150.0, ti_us=40.0, nout=1501,
             rows=0, first=0, kill=0.0, pad=0),
        # the plain configuration's gulp through the plan API, channel by channel (its default)
        dict(name="plan_plain", kind="plan", nchan=512, tsamp=1.048576e-3, dm_max=500.0, ti_us=500.0, nout=16448,
             rows=0, first=0, kill=0.0, pad=0),
        # a beam of the multi-beam configuration: killed channels, padded input rows, an odd
        # sample count, rows of channel quads
        dict(name="plan_rows", kind="plan", nchan=1024, tsamp=1.048576e-3, dm_max=1500.0, ti_us=40.0, nout=32831,
             rows=4, first=0, kill=0.06, pad=16),
        # the smallest gulps that a search is run on, on the default tile shape
        dict(name="search_small", kind="search", nchan=128, nbeam=1, gulp=2048, tsamp=1.048576e-3, dm_max=400.0,
             ti_us=500.0, wmax=64, snr=7.0, mode=0, dada=False, scrunch=0),
        # plain single beam: 512 channels, gulps of 16384, DM 0-500, widths 1-32, pair rows
        dict(name="search_plain", kind="search", nchan=512, nbeam=1, gulp=16384, tsamp=1.048576e-3, dm_max=500.0,
             ti_us=500.0, wmax=64, snr=7.0, mode=5, dada=False, scrunch=0),
        # two beams one after another, a ragged gulp, wide pulses (widths 1-256), default tile shape
        dict(name="search_wide", kind="search", nchan=256, nbeam=2, gulp=10016, tsamp=0.524288e-3, dm_max=600.0,
             ti_us=40.0, wmax=512, snr=7.0, mode=0, dada=False, scrunch=0),
        # full single beam: 2048 channels, gulps of 65536, DM 0-2000, widths 1-256, quad rows
        dict(name="search_full", kind="search", nchan=2048, nbeam=1, gulp=65536, tsamp=0.524288e-3, dm_max=2000.0,
             ti_us=40.0, wmax=512, snr=7.0, mode=6, dada=False, scrunch=0),
        # fp16 channel-major gulps (the DADA input) with a SCRUNCH flagging entry
        dict(name="search_dada", kind="search", nchan=512, nbeam=1, gulp=8192, tsamp=1.048576e-3, dm_max=500.0,
             ti_us=500.0, wmax=64, snr=7.0, mode=5, dada=True, scrunch=1),
        # multi-beam batch: 1024 channels, gulps of 32768, uneven DM ceilings and killmasks
        dict(name="batch_beams", kind="batch", nchan=1024, nbeam=8, gulp=32768, tsamp=1.048576e-3, dm_max=2000.0,
             ti_us=40.0, wmax=64, snr=7.0, mode=6, kill=0.1),
        # serving loop: short gulps (the latency end) of 16 slots, two gulps in flight
        dict(name="stream_beams", kind="stream", nchan=1024, nbeam=16, gulp=8192, tsamp=1.048576e-3, dm_max=2000.0,
             ti_us=40.0, wmax=64, snr=7.0, mode=5, kill=0.0),
        # one gradient step on a gulp's worth of candidates
        dict(name="refine_step", kind="step", ncut=64, nchan=1024, nsamp=2048, steps=1),
        # the whole refinement of those candidates
        dict(name="refine_fit", kind="fit", ncut=64, nchan=1024, nsamp=2048, steps=50),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def draw(rng):
    kind = rng.choice(["plan", "plan", "search", "search", "search", "batch", "stream", "step", "fit"])
    if kind in ("step", "fit"):
        ncut = max(1, int(_log(rng, 1, 96)))
        return dict(kind=kind, ncut=ncut, nchan=16 * int(_log(rng, 4, 64.99)), nsamp=128 * int(_log(rng, 2, 16.99)),
                    steps=1 if kind == "step" else rng.randint(5, 60))
    tsamp = rng.choice([1.048576e-3, 0.524288e-3])
    ti = rng.choice([40.0, 500.0])
    if kind == "plan":
        c = dict(kind=kind, nchan=int(_log(rng, 64, 2048)), tsamp=tsamp, dm_max=round(_log(rng, 100, 2000), 1),
                 ti_us=ti, nout=int(_log(rng, 500, 66048)), rows=rng.choice([0, 0, 2, 4]), first=rng.choice([0, 0, 11]),
                 kill=rng.choice([0.0, 0.05, 0.2]), pad=rng.choice([0, 0, 7, 16]))
        size = "nout"
    else:
        c = dict(kind=kind, nchan=32 * int(_log(rng, 2, 64.99)), nbeam=1, gulp=32 * int(_log(rng, 32, 2048.99)),
                 tsamp=tsamp, dm_max=round(_log(rng, 200, 2000), 1), ti_us=ti, wmax=64, snr=7.0,
                 mode=rng.choice([0, 5, 6]))
        if kind == "search":
            c.update(nbeam=rng.choice([1, 1, 2]), wmax=rng.choice([16, 64, 256, 512]), dada=rng.random() < 0.25,
                     scrunch=rng.choice([0, 0, 1]))
        else:
            c.update(nbeam=rng.randint(2, 16), kill=rng.choice([0.0, 0.1]))
            if kind == "stream":
                c["gulp"] = min(c["gulp"], 16384)
        size = "gulp"
    # no more adds than a third of the full beam's, no more input than its gulp
    while _adds(c) > 1.0e11 or c.get("nbeam", 1) * c["nchan"] * c[size] > 1.0e8:
        if c[size] <= 1024 and c.get("nbeam", 1) > 1:
            c["nbeam"] //= 2
        elif kind == "plan":
            c[size] //= 2
        else:
            c[size] = max(256, c[size] // 64 * 32)
    return c


# ------------------------------------------------------------- plan geometry

def _df(c):
    return -(F0 - FLO) / c["nchan"]


def _dm_list(c):
    """DM trials of the smearing tolerance 1.25 (Cordes & McLaughlin 2003), in 64 bits, kept in 32."""
    f32 = lambda v: float(np.float32(v))  # noqa: E731
    n, ts, ti, tol2 = c["nchan"], f32(c["tsamp"]) * 1e6, f32(c["ti_us"]), f32(1.25) ** 2
    adf, f0 = abs(f32(_df(c))), f32(F0)
    f = (f0 - (n * 0.5 - 0.5) * adf) * 1e-3
    a = 8.3 * adf / (f * f * f)
    a2 = a * a
    b2 = a2 * n * n / 16.0
    k0 = (ts * ts + ti * ti) * (tol2 - 1.0)
    dm, out = 0.0, [0.0]
    while dm < f32(c["dm_max"]):
        k = k0 + tol2 * a2 * dm * dm
        dm = (b2 * dm + math.sqrt(-a2 * b2 * dm * dm + (a2 + b2) * k)) / (a2 + b2)
        out.append(dm)
    return np.array(out, np.float32)


def _tab(nchan, tsamp):
    """Delay of each channel per unit DM, samples (the fp32 table)."""
    adf, f0, dt = abs(float(np.float32(-(F0 - FLO) / nchan))), float(np.float32(F0)), float(np.float32(tsamp))
    fc = f0 - np.arange(nchan) * adf
    return (K_DM / dt * (1.0 / (fc * fc) - 1.0 / (f0 * f0))).astype(np.float32)


def _delays(c):
    p = _dm_list(c)[:, None] * _tab(c["nchan"], c["tsamp"])[None, :]
    return (p + np.float32(0.5)).astype(np.int64)


def _killmask(c, seed, nbeam=None):
    rng = np.random.default_rng([seed, 77])
    shape = c["nchan"] if nbeam is None else (nbeam, c["nchan"])
    if not c.get("kill"):
        return None
    frac = c["kill"] if nbeam is None else rng.uniform(0.0, c["kill"], nbeam)[:, None]
    return (rng.random(shape) >= frac).astype(np.int32)


# ---------------------------------------------------------------- the inputs

def _gulp(c, n, rng, out):
    """Fills `out` (u8 [n][nchan], CUDA) with one beam: noise, 1 % RFI
    channels, three impulses and two bursts painted periodically in n."""
    nchan = c["nchan"]
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(rng.integers(1 << 60)))
    x = torch.randn((n, nchan), generator=gen, device="cuda")
    sd = np.full(nchan, 20.0, np.float32)
    sd[rng.choice(nchan, max(1, nchan // 100), replace=False)] = 80.0
    gain = 128.0 * (1.0 + 0.2 * (np.arange(nchan) / max(1, nchan - 1) - 0.5))
    x.mul_(torch.from_numpy(sd).cuda()).add_(torch.from_numpy(gain.astype(np.float32)).cuda())
    for _ in range(3):
        t = int(rng.integers(0, n - 5))
        x[t:t + 5] += 60.0
    tab = _tab(nchan, c["tsamp"]).astype(np.float64)
    for _ in range(2):
        dm, fwhm = rng.uniform(0.2, 0.9) * c["dm_max"], float(np.exp(rng.uniform(np.log(1.0), np.log(8.0))))
        sig = max(1.0, fwhm / FWHM / (c["tsamp"] * 1e3))
        amp = rng.uniform(20.0, 40.0) * 20.0 / math.sqrt(nchan * sig * math.sqrt(math.pi))
        hw = int(math.ceil(4 * sig))
        at = int(rng.integers(0, n)) + np.rint(dm * tab).astype(np.int64)
        t = (at[:, None] + np.arange(-hw, hw + 1)[None, :]) % n
        v = np.broadcast_to(amp * np.exp(-0.5 * (np.arange(-hw, hw + 1) / sig) ** 2)[None, :], t.shape)
        ch = np.broadcast_to(np.arange(nchan)[:, None], t.shape)
        idx = (torch.from_numpy(t.copy()).cuda(), torch.from_numpy(ch.copy()).cuda())
        x.index_put_(idx, torch.from_numpy(v.astype(np.float32)).cuda(), accumulate=True)
    out.copy_(x.round_().clamp_(0, 255))


def _gulps(c, seed):
    """Every beam's gulp: u8 [nbeam][gulp][nchan], or fp16 [nbeam][nchan][gulp]."""
    rng = np.random.default_rng(seed)
    x = torch.empty((c["nbeam"], c["gulp"], c["nchan"]), dtype=torch.uint8, device="cuda")
    for b in range(c["nbeam"]):
        _gulp(c, c["gulp"], rng, x[b])
    return x.transpose(1, 2).contiguous().half() if c.get("dada") else x


def _plan_input(c, seed):
    nsamp = c["nout"] + int(_delays(c).max())
    x = torch.zeros((nsamp, c["nchan"] + c["pad"]), dtype=torch.uint8, device="cuda")
    _gulp(c, nsamp, np.random.default_rng(seed), x[:, :c["nchan"]])
    return x


def _cutouts(c, seed):
    """Cutouts of bursts in unit noise, their detection DMs and the grid
    points (nearest trial, nearest boxcar, detection sample) a fit starts from."""
    rng = np.random.default_rng(seed)
    n, nchan, nsamp, tsamp = c["ncut"], c["nchan"], c["nsamp"], 1.048576e-3
    tab, lnf = _tab(nchan, tsamp).astype(np.float64), np.log(1.0 - np.arange(nchan) * (F0 - FLO) / nchan / F0)
    dm, width = rng.uniform(100.0, 2000.0, n), rng.uniform(0.5, 20.0, n)
    idx, snr = rng.uniform(-3.0, 3.0, n), rng.uniform(6.0, 40.0, n)
    step = 2.0 * 1024 / nchan
    dm_ref = (np.round(dm / step) * step).astype(np.float32)
    sig = width / (FWHM * tsamp * 1e3)
    amp = snr / np.sqrt(np.exp(2.0 * idx[:, None] * lnf).sum(1) * sig * math.sqrt(math.pi))
    t0 = nsamp / 2 + rng.uniform(-8.0, 8.0, n)
    t_det = np.round(t0 + ((dm - dm_ref)[:, None] * tab).mean(1))
    k = np.clip(np.round(np.log2(np.maximum(width / (tsamp * 1e3), 1.0))), 0, 5)
    theta0 = np.stack([dm_ref, t_det, 2.0 ** k * tsamp * 1e3, amp * rng.uniform(0.7, 1.3, n), np.zeros(n)], 1)
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(rng.integers(1 << 60)))
    cut = torch.randn((n, nchan, nsamp), generator=gen, device="cuda")
    off = np.floor(dm_ref[:, None] * _tab(nchan, tsamp) + np.float32(0.5)).astype(np.float64)
    mu = torch.from_numpy((t0[:, None] + dm[:, None] * tab - off).astype(np.float32)).cuda()
    a = torch.from_numpy((amp[:, None] * np.exp(idx[:, None] * lnf)).astype(np.float32)).cuda()
    t = torch.arange(nsamp, device="cuda", dtype=torch.float32)
    for i in range(n):
        u = (t[None, :] - mu[i][:, None]) / float(sig[i])
        cut[i] += a[i][:, None] * torch.exp(-0.5 * u * u)
    f = lambda v: torch.from_numpy(v.astype(np.float32)).cuda()  # noqa: E731
    return cut, f(dm_ref), f(theta0), f(rng.uniform(0.5, 1.5, n))


# -------------------------------------------------------------- the passes

def _params(c):
    p = dict(nchan=c["nchan"], nbeam=c["nbeam"], gulp=c["gulp"], tsamp=c["tsamp"], plan_dt=c["tsamp"], f0_mhz=F0,
             df_mhz=_df(c), dm_min=0.0, dm_max=c["dm_max"], dm_tol=1.25, ti_us=c["ti_us"], width_min=1,
             width_max=c["wmax"], snr=c["snr"], input_format=1 if c.get("dada") else 0)
    if c.get("scrunch"):
        p["scrunches"] = [(4, 2, 3.0, 1)]
    return hg.default_params(**p)


def _tuning(c):
    return hg.HellaTuning(16, 4, 16, 0, 4 if c["mode"] == 6 else 8, c["mode"])


def prepare(case, seed):
    c, kind = case, case["kind"]
    if kind == "plan":
        plan = hg.Plan(c["nchan"], c["tsamp"], F0, _df(c))
        plan.generate_dm_list(0.0, c["dm_max"], c["ti_us"], 1.25)
        plan.set_killmask(_killmask(c, seed))
        plan.set_pair_rows(c["rows"])
        x = _plan_input(c, seed)
        out = torch.empty((plan.dm_count - c["first"], c["nout"]), dtype=torch.float32, device="cuda")
        return dict(c=c, plan=plan, x=x, out=out)
    if kind in ("step", "fit"):
        cut, dm_ref, theta, g = _cutouts(c, seed)
        r = hg.Refine(c["ncut"], c["nchan"], c["nsamp"], 1.048576e-3, F0, _df(c))
        return dict(c=c, r=r, cut=cut, dm_ref=dm_ref, theta=theta, g=g)
    gulp = _gulps(c, seed)
    torch.cuda.synchronize()  # the batched contexts read it on their own streams
    if kind == "search":
        s = hg.Search(_params(c))
        if c["mode"]:
            s.set_tuning(_tuning(c))
        searched = False
        while not searched:  # fills the ring
            _, searched = s.process_gulp(gulp, on_device=True)
        return dict(c=c, s=s, gulp=gulp)
    rng = np.random.default_rng([seed, 78])
    ceil = rng.uniform(0.5 * c["dm_max"], c["dm_max"], c["nbeam"]).astype(np.float32)
    ceil[0] = c["dm_max"]
    b = hg.Batch(_params(c), dm_max=ceil, killmask=_killmask(c, seed, c["nbeam"]), dynamic=kind == "stream",
                 inflight=2 if kind == "stream" else 1)
    if c["mode"]:
        b.set_tuning(_tuning(c))
    while not b.process_gulp(gulp, on_device=True)[2].all():  # fills the rings
        pass
    if kind == "stream":
        b.submit(gulp, on_device=True)
    return dict(c=c, b=b, gulp=gulp)


def _cands(cand, c):
    """The candidate list as a program that keeps fixed-size records holds it: the count, then one array a
    field of the list's full capacity."""
    n, cap = len(cand), c["nbeam"] * hg.HELLA_MAX_GIANTS
    out = {"n": n}
    for k in ("beam", "dm_idx", "width", "samp", "snr"):
        out[k] = np.zeros(cap, cand.dtype[k])
        out[k][:n] = cand[k]
    return out


def run(state):
    c, kind = state["c"], state["c"]["kind"]
    if kind == "plan":
        x, out, first = state["x"], state["out"], c["first"]
        if first:
            state["plan"].execute_guru(x.shape[0], x, x.stride(0), out, 4 * c["nout"], first, out.shape[0],
                                       hg.HDD_DEVICE_POINTERS)
        else:
            state["plan"].execute_adv(x.shape[0], x, x.stride(0), out, 4 * c["nout"], hg.HDD_DEVICE_POINTERS)
        return out
    if kind == "step":
        r, theta = state["r"], state["theta"]
        chi2, grad = torch.empty_like(state["g"]), torch.empty_like(theta)
        r.forward(state["cut"], state["dm_ref"], theta, chi2)
        r.adjoint(state["cut"], state["dm_ref"], theta, state["g"], grad)
        return {"chi2": chi2, "grad": grad}
    if kind == "fit":
        theta, chi2 = state["theta"].clone(), torch.empty_like(state["g"])
        state["r"].fit(state["cut"], state["dm_ref"], theta, c["steps"], LR, chi2)
        return {"theta": theta, "chi2": chi2}
    if kind == "search":
        return _cands(state["s"].process_gulp(state["gulp"], on_device=True)[0], c)
    if kind == "batch":
        cand, counts, _ = state["b"].process_gulp(state["gulp"], on_device=True)
    else:
        state["b"].submit(state["gulp"], on_device=True)
        cand, counts = state["b"].poll()[:2]
    return dict(_cands(cand, c), counts=counts)


# ---------------------------------------------------------- work and exact

def _adds(c):
    nout = c["nout"] if c["kind"] == "plan" else c["gulp"] + c["wmax"]
    return float(len(_dm_list(c)) - c.get("first", 0)) * c["nchan"] * nout * c.get("nbeam", 1)


def work(case):
    """bytes: the inputs once and the outputs once.  flops: dedispersion, the
    sums channel by channel, and the smoothing's multiply-adds; refinement,
    about 16 operations an element of each pass.  A search's outputs are its
    few candidates."""
    c, kind = case, case["kind"]
    if kind in ("step", "fit"):
        n = float(c["ncut"]) * c["nchan"] * c["nsamp"]
        return dict(bytes=4.0 * n, flops=16.0 * n * (2 if kind == "step" else c["steps"]))
    ndm, md = len(_dm_list(c)) - c.get("first", 0), int(_delays(c).max())
    if kind == "plan":
        return dict(bytes=float(c["nout"] + md) * c["nchan"] + 4.0 * ndm * c["nout"], flops=_adds(c))
    taps, w = 0, 1
    while w < c["wmax"]:
        taps, w = taps + 2 * w + 1, 2 * w
    size = 2.0 if c.get("dada") else 1.0
    share = 0.75 if kind in ("batch", "stream") else 1.0  # the beams' DM ceilings
    return dict(bytes=size * c["nbeam"] * c["gulp"] * c["nchan"],
                flops=share * (_adds(c) + 2.0 * taps * ndm * c["gulp"] * c["nbeam"]))


def _exact_plan(c, seed):
    x = _plan_input(c, seed)
    delays = torch.from_numpy(_delays(c)[c["first"]:]).cuda()
    keep = _killmask(c, seed)
    acc = torch.zeros((delays.shape[0], c["nout"]), dtype=torch.int32, device="cuda")
    for ch in range(c["nchan"]):
        if keep is None or keep[ch]:
            acc += x[:, ch].contiguous().unfold(0, c["nout"], 1)[delays[:, ch]]
    return acc.double()


def _exact_pass(c, cut, dm_ref, th):
    """chi2 and its gradient in 64 bits at th [n][5]."""
    tab = torch.from_numpy(_tab(c["nchan"], 1.048576e-3)).cuda()
    lnf = torch.from_numpy(np.log(1.0 - np.arange(c["nchan"]) * (F0 - FLO) / c["nchan"] / F0)).cuda()
    off = (dm_ref[:, None] * tab + 0.5).to(torch.int64).double()
    tab = tab.double()
    t = torch.arange(c["nsamp"], device="cuda", dtype=torch.float64)
    c_w = 1.0 / (FWHM * 1.048576)
    chi2, grad = torch.empty(len(th), dtype=torch.float64, device="cuda"), torch.empty_like(th)
    for i in range(len(th)):
        dm, t0, w, amp, idx = (th[i, k] for k in range(5))
        sig, s = w * c_w, torch.exp(idx * lnf)
        u = (t[None, :] - (t0 + dm * tab - off[i])[:, None]) / sig
        e = torch.exp(-0.5 * u * u)
        r = cut[i].double() - (amp * s)[:, None] * e
        chi2[i] = (r * r).sum()
        re = r * e
        s1, s2, s3 = re.sum(1), (re * u).sum(1), (re * u * u).sum(1)
        g = -2.0 * amp * s * s2 / sig
        grad[i] = torch.stack([(tab * g).sum(), g.sum(), (-2.0 * amp * s * s3 / sig * c_w).sum(),
                               (-2.0 * s * s1).sum(), (-2.0 * amp * s * lnf * s1).sum()])
    return chi2, grad


def exact(case, seed):
    c, kind = case, case["kind"]
    if kind == "plan":
        return _exact_plan(c, seed)
    if kind in ("step", "fit"):
        cut, dm_ref, theta, g = _cutouts(c, seed)
        th = theta.double()
        if kind == "step":
            chi2, grad = _exact_pass(c, cut, dm_ref, th)
            return {"chi2": chi2, "grad": grad * g.double()[:, None]}
        if float(cut.numel()) * c["steps"] > 7.5e9:
            return None
        m, v, lr = torch.zeros_like(th), torch.zeros_like(th), torch.tensor(LR, device="cuda", dtype=torch.float64)
        for k in range(1, c["steps"] + 1):
            chi2, grad = _exact_pass(c, cut, dm_ref, th)
            m, v = 0.9 * m + 0.1 * grad, 0.999 * v + 0.001 * grad * grad
            th = th - lr * (m / (1 - 0.9 ** k)) / (torch.sqrt(v / (1 - 0.999 ** k)) + 1e-8)
            th[:, 0].clamp_(min=0.0)
            th[:, 2].clamp_(min=0.05)
        return {"theta": th, "chi2": chi2}
    # candidates: indices that have to stay equal, and S/Ns that rest on the flagger's fp16 steps
    return None
