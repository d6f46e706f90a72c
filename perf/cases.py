"""Performance cases: what a user of this framework has it do.

A survey's night goes through these steps, each a public entry point of
``prestozl_b200.jerk``: subband blocks are downsampled and dedispersed into DM
trials (``downsample_subbands``, ``Dedisperser``), each trial's series becomes
a whitened, zapped spectrum (``spectrum_from_timeseries``, ``zap_birdies``),
the spectra are searched (``JerkPlan.search``, or ``JerkServer`` for a stream
of them), and the candidates that remain are looked at and polished
(``JerkPlan.volume``, ``volume_static``, ``Polisher``).  The named geometries
(zmax, wmax, numharm), lengths and thresholds are the workloads of the tests
and the benchmark.

A case is a dict of plain values; ``kind`` says which step it is.
"""

from __future__ import annotations

import math

import numpy as np
import torch

from prestozl_b200 import jerk

DEV = "cuda"
LN2 = math.log(2.0)


# ---------------------------------------------------------------------------
# the cases

def listed():
    return [
        # one subharmonic's plane of one rstep by the allocation-free call: the
        # smallest call there is (a real-time loop that looks at one block)
        dict(name="static_z20", kind="static", fftlen=2048, zmax=20, wmax=0, bins=1 << 16),
        # the ffdot volume around a candidate, for plotting
        dict(name="plane_z100w60", kind="plane", fftlen=2048, zmax=100, wmax=60, bins=1 << 18),
        # the CPU-runnable plain jerk search: a whole 2^20-sample spectrum from
        # host memory, the drop-in's default batch
        _search("search_small", 1 << 20, 64e-6, 20, 60, 8, 2.0, batch=8, host=True, pulsars=1),
        # plain acceleration search (no jerk) of a 2^22-sample trial
        _search("search_accel", 1 << 22, 64e-6, 100, 0, 16, 3.0, batch=32, pulsars=2),
        # small jerk search of the mixed batch
        _search("search_jerk", 1 << 22, 64e-6, 50, 150, 8, 3.0, batch=32, pulsars=2),
        # the paper-scale geometry on a 2^25-sample spectrum: one GPU's share of
        # its rsteps (a spectrum split over GPUs), batches as tuned
        _search("search_paper", 1 << 25, 54.6e-6, 200, 300, 16, 3.0, batch=64, rsteps=512,
                first=2000, pulsars=4),
        # the memory-heavy geometry (fftlen 4096), a few batches of its rsteps
        _search("search_heavy", 1 << 25, 54.6e-6, 300, 600, 2, 4.0, batch=16, rsteps=48,
                first=500, pulsars=2),
        # a stream of dedispersed trials through the server
        dict(name="served_trials", kind="served", N=1 << 21, dt=64e-6, zmax=50, wmax=150,
             numharm=8, sigma=3.0, trials=6, batch=16),
        # a paper-scale trial: series to whitened and zapped spectrum
        dict(name="series_2p25", kind="series", N=1 << 25, birds=20),
        # a short trial of a length that is no power of two
        dict(name="series_short", kind="series", N=3 << 18, birds=3),
        # one block of a DM range: downsampled 4x and dedispersed to 512 trials
        dict(name="dedisp_64x512", kind="dedisp", worklen=65536, nsub=64, numdms=512, bs=4,
             ddm=0.5, dt=64e-6),
        # a paper-scale 16-harmonic candidate polished (z and w of the candidate
        # are the fundamental's: the sixteenth part of what was searched)
        dict(name="polish_h16", kind="polish", bins=1 << 22, numharm=16, z=9.5, w=-14.0),
    ]


def _search(name, N, dt, zmax, wmax, numharm, sigma, batch, rsteps=0, first=0, host=False,
            pulsars=1):
    return dict(name=name, kind="search", N=N, dt=dt, zmax=zmax, wmax=wmax, numharm=numharm,
                sigma=sigma, batch=batch, rsteps=rsteps, first=first, host=host, pulsars=pulsars)


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


# series lengths that the device real FFT takes: 2 R1 R2 over its block sizes
def _series_len(rng, lo, hi):
    sizes = [128, 192, 256, 384, 512, 768, 1024, 1280, 2048, 4096]
    while True:
        n = 2 * rng.choice(sizes) * rng.choice(sizes)
        if lo <= n <= hi:
            return n


def draw(rng):
    kind = rng.choice(["static", "plane", "search", "search", "search", "search", "served",
                       "series", "series", "dedisp", "polish"])
    if kind == "static":
        return dict(kind=kind, fftlen=rng.choice([1024, 1280, 2048, 4096]),
                    zmax=2 * rng.randint(2, 70), wmax=20 * rng.randint(0, 4),
                    bins=_logint(rng, 1 << 15, 1 << 20))
    if kind == "plane":
        return dict(kind=kind, fftlen=rng.choice([1024, 1280, 2048, 4096]),
                    zmax=2 * rng.randint(5, 60), wmax=20 * rng.randint(0, 5),
                    bins=_logint(rng, 1 << 15, 1 << 20))
    if kind == "search":
        zmax = 2 * _logint(rng, 5, 150)
        wmax = rng.choice([0, 20 * rng.randint(1, 15)])
        numharm = rng.choice([1, 2, 4, 8, 16]) if zmax * max(wmax, 20) < 20000 else 2
        N = _series_len(rng, 1 << 18, 1 << 24)
        return _search("", N, rng.choice([54.6e-6, 64e-6, 81.92e-6]), zmax, wmax, numharm,
                       rng.choice([2.0, 3.0, 4.0]), batch=rng.choice([8, 16, 27, 32]),
                       rsteps=rng.randint(40, 300), host=rng.random() < 0.3,
                       pulsars=rng.randint(1, 3))
    if kind == "served":
        return dict(kind=kind, N=_series_len(rng, 1 << 19, 1 << 21), dt=64e-6,
                    zmax=2 * rng.randint(5, 50), wmax=rng.choice([0, 60, 100]),
                    numharm=rng.choice([4, 8]), sigma=rng.choice([3.0, 4.0]),
                    trials=rng.randint(2, 6), batch=rng.choice([8, 16]))
    if kind == "series":
        return dict(kind=kind, N=_series_len(rng, 1 << 16, 1 << 25), birds=rng.randint(0, 20))
    if kind == "dedisp":
        return dict(kind=kind, worklen=_logint(rng, 8192, 65536), nsub=rng.choice([32, 64, 96, 51]),
                    numdms=_logint(rng, 16, 300), bs=rng.choice([1, 2, 4]),
                    ddm=rng.choice([0.1, 0.5, 1.0]), dt=64e-6)
    numharm = rng.choice([1, 2, 4, 8, 16])
    return dict(kind=kind, bins=_logint(rng, 1 << 20, 1 << 22), numharm=numharm,
                z=rng.uniform(-180.0, 180.0) / numharm, w=rng.uniform(-280.0, 280.0) / numharm)


# ---------------------------------------------------------------------------
# inputs

def _gen(seed):
    g = torch.Generator(device=DEV)
    g.manual_seed(seed)
    return g


def _uniform(g, n, lo, hi):
    return (lo + (hi - lo) * torch.rand(n, generator=g, device=DEV, dtype=torch.float64)).tolist()


def _pulse_train(N, r, z, w, snr, nharm):
    """A pulsar of average frequency r bins, f-dot z and f-dot-dot w over the
    series (PRESTO's phase convention): nharm harmonics of amplitude ~ 1/k."""
    u = torch.arange(N, device=DEV, dtype=torch.float64) / N
    phi = u * ((r - 0.5 * z + w / 12.0) + u * (0.5 * (z - 0.5 * w) + u * (w / 6.0)))
    phi -= torch.floor(phi)
    scale = snr / math.sqrt(sum(1.0 / k ** 2 for k in range(1, nharm + 1)) * N / 4.0)
    x = torch.zeros(N, device=DEV, dtype=torch.float32)
    for k in range(1, nharm + 1):
        x += (scale / k * torch.cos(2.0 * math.pi * k * phi)).float()
    return x


def _spectrum_of(ts):
    X = torch.fft.rfft(ts)
    spec = X[: ts.numel() // 2].contiguous()
    spec[0] = complex(1.0, 1.0)
    return spec


def _noise_spectrum(g, bins):
    x = torch.randn((bins, 2), generator=g, device=DEV, dtype=torch.float32)
    return torch.view_as_complex(x)


# ---------------------------------------------------------------------------
# a caller's own kernels (static and plane cases): one subharmonic, the
# fundamental, rows of f-dot z and f-dot-dot w

def _halfwidth(z, w):
    return int(1.1 * (0.5 * abs(z) + abs(w) / 12.0)) + 16


def _grid(case):
    zs = [-case["zmax"] + 2 * j for j in range(case["zmax"] + 1)]
    ws = [-case["wmax"] + 20 * i for i in range(case["wmax"] // 10 + 1)]
    return zs, ws


def _kernels(case):
    """[numw][numz][fftlen] complex64: the FFT of each row's Fourier response at
    half-bin steps, cut at the row's own half width and wrapped around."""
    N, npts = case["fftlen"], 8192
    zs, ws = _grid(case)
    u = (torch.arange(npts, device=DEV, dtype=torch.float64) + 0.5) / npts
    out = torch.empty((len(ws), len(zs), N), device=DEV, dtype=torch.complex64)
    for i, w in enumerate(ws):
        for j, z in enumerate(zs):
            hw = _halfwidth(z, w)
            phi = u * ((-0.5 * z + w / 12.0) + u * (0.5 * (z - 0.5 * w) + u * (w / 6.0)))
            x = torch.polar(torch.full_like(u, 1.0 / npts), 2.0 * math.pi * phi)
            F = torch.fft.fft(x, n=2 * npts)  # value at q half bins: index q mod 2 npts
            q = torch.arange(-2 * hw, 2 * hw, device=DEV)
            F = F[q % (2 * npts)] * torch.exp(-0.5j * math.pi * q / npts)  # midpoint samples
            row = torch.zeros(N, device=DEV, dtype=torch.complex128)
            row[q % N] = F
            out[i, j] = torch.fft.fft(row).to(torch.complex64)
    return out


def _own_geometry(case):
    """uselen, halfwidth and first bin of a one-subharmonic search whose good
    bins fill the FFT length."""
    hw = _halfwidth(case["zmax"], case["wmax"])
    uselen = case["fftlen"] - 4 * hw
    uselen -= uselen % 2
    return uselen, hw, float(case["bins"] // 3)


# ---------------------------------------------------------------------------
# prepare / run

def prepare(case, seed):
    g = _gen(seed)
    st = {"kind": case["kind"], "case": dict(case)}
    kind = case["kind"]
    if kind == "static":
        uselen, hw, r = _own_geometry(case)
        zs, ws = _grid(case)
        st["spec"] = _noise_spectrum(g, case["bins"])
        st["spec"][int(r) + uselen // 4] += 30.0
        st["kern"] = _kernels(case)
        st["sub"] = dict(numharm=1, harmnum=1, zmax=case["zmax"], wmax=case["wmax"], numz=len(zs),
                         numw=len(ws), fftlen=case["fftlen"], halfwidth=hw)
        st["uselen"], st["r"] = uselen, r
        st["vol"] = torch.zeros((len(ws), len(zs), uselen), device=DEV, dtype=torch.float32)
    elif kind == "plane":
        uselen, hw, r = _own_geometry(case)
        zs, ws = _grid(case)
        st["spec"] = _noise_spectrum(g, case["bins"])
        st["spec"][int(r) + uselen // 4] += 30.0
        o = jerk.Obs()
        o.numbins, o.lobin, o.highestbin = case["bins"], 0, case["bins"] - 1
        o.rlo, o.zlo, o.wlo = r, -case["zmax"], -case["wmax"]
        o.corr_uselen, o.numz, o.numw = uselen, len(zs), len(ws) if case["wmax"] else 0
        o.numharmstages = 1
        o.numindep[0], o.powcut[0] = case["bins"], 40.0
        sub = dict(numharm=1, harmnum=1, zmax=case["zmax"], wmax=case["wmax"], numz=len(zs),
                   numw=len(ws), fftlen=case["fftlen"], halfwidth=hw,
                   kern=_kernels(case).cpu().numpy())
        st["plan"] = jerk.JerkPlan(o, [sub], batch=1)
    elif kind == "search":
        N = case["N"]
        obs, fftlen, _ = jerk.obs_from_params(N // 2, N, case["dt"], case["zmax"], case["wmax"],
                                              case["numharm"], case["sigma"],
                                              wmax_given=case["wmax"] > 0)
        subs = jerk.subharm_sizes(obs, fftlen)
        ts = torch.randn(N, generator=g, device=DEV, dtype=torch.float32)
        T, span = N * case["dt"], obs.corr_uselen // 2
        r0 = obs.rlo + case["first"] * span
        r1 = r0 + case["rsteps"] * span if case["rsteps"] else min(500.0 * T, N / 8.0)
        r1 = min(r1, N / 4.0)
        for _ in range(case["pulsars"]):
            r, z, w, snr, h = _uniform(g, 5, 0.0, 1.0)
            ts += _pulse_train(N, r0 + r * (r1 - r0), 0.9 * case["zmax"] * (2 * z - 1),
                               0.9 * case["wmax"] * (2 * w - 1), 10.0 + 10.0 * snr, 1 + int(4 * h))
        spec = _spectrum_of(ts)
        st["bank"] = jerk.DeviceBank(subs)
        st["plan"] = jerk.JerkPlan(obs, subs, batch=case["batch"],
                                   device_bank=st["bank"].ptr.value)
        st["spec"] = spec.cpu().numpy() if case["host"] else spec
    elif kind == "served":
        st["server"] = jerk.JerkServer(max_active=case["trials"], batch=case["batch"])
        st["series"] = []
        T = case["N"] * case["dt"]
        r, z, w = _uniform(g, 3, 0.0, 1.0)
        for k in range(case["trials"]):
            ts = torch.randn(case["N"], generator=g, device=DEV, dtype=torch.float32)
            ts += _pulse_train(case["N"], (50.0 + 200.0 * r) * T, 0.9 * case["zmax"] * (2 * z - 1),
                               0.9 * case["wmax"] * (2 * w - 1), 4.0 + 3.0 * k, 4)
            st["series"].append(ts)
    elif kind == "series":
        N = case["N"]
        # white noise with slow baseline wander, as dedispersed data have it
        ts = torch.randn(N, generator=g, device=DEV, dtype=torch.float32)
        walk = torch.cumsum(torch.randn(1024, generator=g, device=DEV, dtype=torch.float32), 0)
        ts += 0.3 * torch.nn.functional.interpolate(walk.view(1, 1, -1), size=N, mode="linear").view(-1)
        st["ts"] = ts
        st["out"] = torch.empty(N // 2, device=DEV, dtype=torch.complex64)
        st["birds"] = _birds(case)
    elif kind == "dedisp":
        raw = (case["worklen"] * case["bs"], case["nsub"])
        st["raw"] = torch.randn(raw, generator=g, device=DEV, dtype=torch.float32)
        st["last"] = torch.randn((case["worklen"], case["nsub"]), generator=g, device=DEV,
                                 dtype=torch.float32)
        st["ds"] = torch.empty_like(st["last"])
        st["out"] = torch.empty((case["numdms"], case["worklen"]), device=DEV, dtype=torch.float32)
        st["dd"] = jerk.Dedisperser(case["worklen"], case["nsub"], _offsets(case))
    elif kind == "polish":
        st["spec"] = _noise_spectrum(g, case["bins"])
        r = _polish_r(case)
        for k in range(1, case["numharm"] + 1):
            st["spec"][int(round(r * k))] += 12.0 / math.sqrt(k)
        st["polisher"] = jerk.Polisher()
    torch.cuda.synchronize()
    return st


MOST_CANDS = 8192


def _table(cands):
    """The candidate list as a survey's table keeps it: its columns, in list
    order, in a table of fixed length (zeros after the last candidate)."""
    if len(cands) > MOST_CANDS:
        raise ValueError("more candidates than the table holds")
    out = {}
    for k in ("power", "sigma", "numharm", "r", "z", "w"):
        out[k] = np.zeros(MOST_CANDS, dtype=cands[k].dtype)
        out[k][: len(cands)] = cands[k]
    return out


def run(state):
    kind, case = state["kind"], state["case"]
    if kind == "static":
        stream = torch.cuda.current_stream().cuda_stream
        jerk.volume_static(state["spec"].data_ptr(), case["bins"], 0, state["sub"],
                           state["kern"].data_ptr(), state["r"], state["uselen"], 0.0,
                           state["vol"].data_ptr(), stream)
        return state["vol"]
    if kind == "plane":
        return state["plan"].volume(state["spec"], 0, 0)[0]
    if kind == "search":
        return _table(state["plan"].search(state["spec"], case["first"], case["rsteps"]))
    if kind == "served":
        srv = state["server"]
        tags = [srv.submit(ts, case["N"], case["dt"], case["zmax"], case["wmax"], case["numharm"],
                           case["sigma"], wmax_given=case["wmax"] > 0, timeseries=True)
                for ts in state["series"]]
        done = {}
        while len(done) < len(tags):
            got = srv.poll(10000)
            if got is not None:
                done[got[0]] = got[1]
        return [_table(done[t]) for t in tags]
    if kind == "series":
        out = jerk.spectrum_from_timeseries(state["ts"], state["out"])
        lo, hi = state["birds"]
        return jerk.zap_birdies(out, case["N"], lo, hi) if len(lo) else out
    if kind == "dedisp":
        cur = jerk.downsample_subbands(state["raw"], case["bs"], state["ds"])
        return {"block": cur, "trials": state["dd"](cur, state["last"], state["out"])}
    rzw, derivs, locpow = state["polisher"].optimize(state["spec"], case["numharm"],
                                                     _polish_r(case), case["z"], case["w"])
    return {"rzw": np.array(rzw), "locpow": locpow, "pow": np.ascontiguousarray(derivs["pow"]),
            "phs": np.ascontiguousarray(derivs["phs"])}


def _polish_r(case):
    return 0.037 * case["bins"] + 0.25


def _birds(case):
    """Single-line birdies, three bins wide, over the band."""
    n, M = case["birds"], case["N"] // 2
    lo = np.array([M * (k + 1.5) / (n + 2.0) - 1.0 for k in range(n)])
    return lo, lo + 3.0


def _offsets(case):
    """Cold-plasma delays over 1200-1600 MHz relative to the top subband, in
    samples after downsampling; DMs from 0 in steps of ddm."""
    f = np.linspace(1200.0, 1600.0, case["nsub"], endpoint=False)
    delay = 4.148808e3 * (1.0 / f ** 2 - 1.0 / 1600.0 ** 2)  # s per unit DM
    dms = case["ddm"] * np.arange(case["numdms"])
    off = np.rint(dms[:, None] * delay[None, :] / (case["dt"] * case["bs"]))
    return np.minimum(off, case["worklen"]).astype(np.int32)


# ---------------------------------------------------------------------------
# the work of one pass

def _geometry_rows(case, N):
    obs, fftlen, _ = jerk.obs_from_params(N // 2, N, case.get("dt", 64e-6), case["zmax"],
                                          case["wmax"], case["numharm"], 3.0,
                                          wmax_given=case["wmax"] > 0)
    return obs, [(s["numw"] * s["numz"], s["fftlen"], s["harmnum"] / s["numharm"])
                 for s in jerk.subharm_sizes(obs, fftlen)]


def _corr_flops(rows, fftlen, numrs):
    """rows kernels against one chunk: the product with the kernel, two
    transforms of fftlen/2 points (even and odd half bins) and the powers."""
    half = fftlen / 2
    return rows * (2 * (5.0 * half * math.log2(half) + 6.0 * half) + 3.0 * numrs)


def work(case):
    kind = case["kind"]
    if kind in ("static", "plane"):
        uselen, _, _ = _own_geometry(case)
        zs, ws = _grid(case)
        rows, N = len(zs) * len(ws), case["fftlen"]
        return {"bytes": rows * (8.0 * N + 4.0 * uselen) + 4.0 * N,
                "flops": _corr_flops(rows, N, uselen)}
    if kind in ("search", "served"):
        N = case["N"]
        obs, subs = _geometry_rows(case, N)
        total = max(1, int((min(obs.highestbin, N // 2) - obs.rlo) // (obs.corr_uselen // 2)))
        steps = min(case["rsteps"], total) if case.get("rsteps") else total
        flops = 0.0
        for rows, fftlen, hf in subs:
            flops += steps * _corr_flops(rows, fftlen, hf * obs.corr_uselen)
        flops += steps * subs[0][0] * obs.corr_uselen * len(subs)
        bank = 8.0 * sum(rows * fftlen for rows, fftlen, _ in subs)
        trials = case.get("trials", 1)
        series = (5.0 * (N / 2) * math.log2(N / 2) + 4.0 * N) if kind == "served" else 0.0
        return {"bytes": bank + trials * 4.0 * obs.corr_uselen * steps,
                "flops": trials * (flops + series)}
    if kind == "series":
        N = case["N"]
        return {"bytes": 8.0 * N, "flops": 2.5 * N * math.log2(N) + 6.0 * N}
    if kind == "dedisp":
        block = case["worklen"] * case["nsub"]
        return {"bytes": 4.0 * (block * case["bs"] + 2 * block + case["numdms"] * case["worklen"]),
                "flops": float(block) * (case["bs"] + case["numdms"])}
    # polish: per harmonic 17 x 17 kernels of a few thousand points
    flops = 0.0
    for k in range(1, case["numharm"] + 1):
        n = 2.0 ** math.ceil(math.log2(16.0 * (_halfwidth(k * case["z"], k * case["w"]) + 8)))
        flops += 289 * 2 * 5.0 * n * math.log2(n)
    return {"bytes": 8.0 * 2048 * case["numharm"], "flops": flops}


# ---------------------------------------------------------------------------
# the same results in 64 bits

def exact(case, seed):
    kind = case["kind"]
    if kind in ("static", "plane"):
        return _exact_volume(case, seed)
    if kind == "series":
        return _exact_series(case, seed)
    if kind == "dedisp":
        return _exact_dedisp(case, seed)
    # searches pick cells (and the polisher grid points) by comparisons
    return None


def _exact_volume(case, seed):
    uselen, hw, r = _own_geometry(case)
    N = case["fftlen"]
    g = _gen(seed)
    spec = _noise_spectrum(g, case["bins"])
    spec[int(r) + uselen // 4] += 30.0
    lo = int(r) - hw
    d = spec[lo:lo + N // 2].to(torch.complex128)
    if d.numel() < N // 2:
        d = torch.nn.functional.pad(d, (0, N // 2 - d.numel()))
    p = (d.real ** 2 + d.imag ** 2).sort().values
    d = d / torch.sqrt(p[(N // 2 - 1) // 2] / LN2)
    D = torch.fft.fft(d).repeat(2)  # the chunk spread to even half bins
    K = _kernels(case).to(torch.complex128)
    y = torch.fft.ifft(D * K.conj(), dim=-1)[..., 2 * hw:2 * hw + uselen]
    v = y.real ** 2 + y.imag ** 2
    return v.cpu().numpy() if case["kind"] == "plane" else v


def _exact_series(case, seed):
    st = prepare(case, seed)
    N, M = case["N"], case["N"] // 2
    x = torch.fft.rfft(st["ts"].double())[:M]
    p = x.real ** 2 + x.imag ** 2
    # whitening blocks: 6 ln(start) bins from bin 1 on, at most 200
    starts, lens = [1], [6]
    while True:
        b = starts[-1] + lens[-1]
        n = min(200, int(6 * math.log(b)))
        if b + n >= M:
            break
        starts.append(b)
        lens.append(n)
    starts, lens = np.array(starts), np.array(lens)
    level = torch.empty(len(starts), device=DEV, dtype=torch.float64)
    for n in np.unique(lens):  # medians, blocks of one length together
        k = torch.from_numpy(np.flatnonzero(lens == n)).to(DEV)
        s = torch.from_numpy(starts[lens == n]).to(DEV)
        blk = p[s[:, None] + torch.arange(int(n), device=DEV)[None, :]]
        level[k] = blk.sort(dim=1).values[:, (int(n) - 1) // 2] / LN2
    # between block middles the level runs linearly; the last slope goes on
    mid = torch.from_numpy(starts + lens // 2).to(DEV)
    dl = (level[1:] - level[:-1]) / torch.from_numpy(0.5 * (lens[1:] + lens[:-1])).to(DEV)
    slope = torch.cat([dl, dl[-1:]]) if len(starts) > 1 else torch.ones_like(level)
    i = torch.arange(M, device=DEV)
    seg = torch.searchsorted(mid, i, right=True) - 1
    c = seg.clamp(min=0)
    lv = torch.where(seg < 0, level[0], level[c] + slope[c] * (i - mid[c]))
    # the whitening's inverse square root: bit-level guess, one Newton step
    y = (0x5f3759df - (lv.float().view(torch.int32) >> 1)).view(torch.float32).double()
    x = x * (y * (1.5 - 0.5 * lv * y * y))
    x[0] = complex(1.0, 1.0)
    for lo, hi in zip(*_birds(case)):
        if not lo - 300.0 > 1:
            continue
        med = []
        for first in (int(lo - 300), int(hi - 100)):
            v = torch.zeros(200, device=DEV, dtype=torch.float64)
            s = x[first:min(M, first + 200)]
            v[: s.numel()] = s.real ** 2 + s.imag ** 2
            med.append(v.sort().values[99])
        amp = torch.sqrt(0.5 * (med[0] + med[1]) / LN2)
        x[math.floor(lo):min(M, math.ceil(hi))] = torch.complex(amp, torch.zeros_like(amp))
    return x


def _exact_dedisp(case, seed):
    st = prepare(case, seed)
    W, bs, nsub = case["worklen"], case["bs"], case["nsub"]
    cur = st["raw"].double().view(W, bs, nsub).mean(1)
    x = torch.cat([st["last"].double(), cur]).t().contiguous()
    off = torch.from_numpy(_offsets(case)).to(DEV).long()
    t = torch.arange(W, device=DEV)
    out = torch.zeros((case["numdms"], W), device=DEV, dtype=torch.float64)
    for s in range(nsub):
        out += x[s][t[None, :] + off[:, s:s + 1]]
    return {"block": cur, "trials": out}
