"""Work that users of this framework have it do, as cases to measure.

A case is one call (or one short chain of calls) through the public entry
points on data that is already where a user's program holds it: spectra, time
series and filterbank blocks in device memory, candidates in host lists.
Geometries are those of the benchmark workloads and the tests (N = 2^16 to
2^23 samples, zmax 0 to 600, wmax 0 to 300, 1 to 16 harmonics) and what lies
between them; the synthetic data are the benchmark's recipes (unit Gaussian
noise, a few accelerated pulsars) made on the device.
"""
import ctypes as C
import math

import numpy as np
import torch

import presto_b200 as pb
from presto_b200 import accel

DT = 64e-6                        # sampling time of the benchmark workloads (s)
LOFREQ, BANDWIDTH = 1400.0, 256.0  # MHz, the dedispersion benchmark's band
MAXCANDS = 4096                   # records of the buffer that a search fills


def listed():
    return [
        # the f-fdot planes of one block as a program on the accel.h functions
        # asks for them, harmonic by harmonic: the smallest calls there are
        dict(name="planes_block", kind="planes", N=262144, zmax=50, wmax=0, numharm=4),
        # a quick look without acceleration at a short observation
        dict(name="search_zmax0", kind="search", N=1 << 19, zmax=0, wmax=-1, numharm=16, locpow=False),
        # the ordinary acceleration search of one DM trial (plane in memory)
        dict(name="search_plain", kind="search", N=1 << 20, zmax=200, wmax=-1, numharm=8, locpow=False),
        # a series of FFT-friendly but not power-of-two length, standard mode,
        # normalised by the local power
        dict(name="search_locpow", kind="search", N=3628800, zmax=300, wmax=-1, numharm=8, locpow=True),
        # the larger acceleration search, the benchmark's headline
        dict(name="search_large", kind="search", N=1 << 23, zmax=600, wmax=-1, numharm=16, locpow=False),
        # the jerk search: r, z and w
        dict(name="search_jerk", kind="search", N=1 << 22, zmax=200, wmax=300, numharm=8, locpow=False),
        # a dedispersed series made into a de-reddened spectrum: a power of two
        # and a 2^a 3^b 5^c 7^d length
        dict(name="series_pow2", kind="series", n=1 << 23),
        dict(name="series_smooth", kind="series", n=6048000),
        # filterbank spectra to a batch of DM trials
        dict(name="dedisperse", kind="dedisperse", nspec=1 << 19, nchan=1024, nsub=64, ndm=128,
             dmmax=300.0, downsamp=1),
        # filterbank spectra to the candidates of every trial
        dict(name="pipeline", kind="pipeline", nspec=(1 << 18) + 77, nchan=256, nsub=32, ndm=8,
             dmmax=100.0, downsamp=1, zmax=50, numharm=8),
        # the candidates of a search polished: acceleration and jerk
        dict(name="polish_accel", kind="polish", N=1 << 23, ncand=160, zmax=600, wmax=-1, numharm=16),
        dict(name="polish_jerk", kind="polish", N=1 << 21, ncand=48, zmax=200, wmax=300, numharm=8),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _smooth(n):
    """The largest 2^a 3^b 5^c 7^d below or at n that is a multiple of 64."""
    m = n // 64
    while True:
        k = m
        for p in (2, 3, 5, 7):
            while k % p == 0:
                k //= p
        if k == 1:
            return 64 * m
        m -= 1


def _length(rng, lo, hi):
    """A series length as programs choose them: a power of two, a smooth
    length, or any even number."""
    n = _logint(rng, lo, hi)
    how = rng.choice(("pow2", "smooth", "even"))
    if how == "pow2":
        return 1 << (n.bit_length() - 1)
    return _smooth(n) if how == "smooth" else n // 2 * 2


def draw(rng):
    while True:
        kind = rng.choice(("planes", "search", "search", "search", "jerk", "series", "dedisperse",
                           "pipeline", "polish", "polish"))
        if kind == "planes":
            c = dict(kind=kind, N=_length(rng, 1 << 17, 1 << 22), zmax=2 * rng.randint(0, 150),
                     wmax=rng.choice((-1, 0)), numharm=rng.choice((1, 2, 4, 8)))
        elif kind == "search":
            c = dict(kind=kind, N=_length(rng, 1 << 18, 1 << 23), zmax=2 * rng.randint(0, 300), wmax=-1,
                     numharm=rng.choice((1, 2, 4, 8, 16)), locpow=rng.random() < 0.2)
        elif kind == "jerk":
            c = dict(kind="search", N=_length(rng, 1 << 18, 1 << 22), zmax=2 * rng.randint(5, 100),
                     wmax=20 * rng.randint(1, 15), numharm=rng.choice((1, 2, 4, 8)), locpow=False)
        elif kind == "series":
            c = dict(kind=kind, n=_length(rng, 1 << 17, 1 << 24))
        elif kind == "dedisperse":
            nsub = rng.choice((16, 32, 64))
            c = dict(kind=kind, nspec=_logint(rng, 1 << 16, 1 << 19), nchan=nsub * rng.choice((4, 8, 12, 16)),
                     nsub=nsub, ndm=rng.randint(8, 128), dmmax=round(rng.uniform(20.0, 300.0), 1),
                     downsamp=rng.choice((1, 1, 2, 3)))
        elif kind == "pipeline":
            c = dict(kind=kind, nspec=_logint(rng, 1 << 17, 1 << 19), nchan=rng.choice((128, 256, 512)),
                     nsub=32, ndm=rng.randint(2, 10), dmmax=round(rng.uniform(20.0, 200.0), 1),
                     downsamp=rng.choice((1, 2)), zmax=2 * rng.randint(0, 50), numharm=rng.choice((4, 8)))
        else:
            jerk = rng.random() < 0.5
            c = dict(kind=kind, N=1 << rng.randint(19, 21 if jerk else 23), ncand=rng.randint(4, 48 if jerk else 160),
                     zmax=200 if jerk else 2 * rng.randint(10, 300), wmax=20 * rng.randint(1, 15) if jerk else -1,
                     numharm=rng.choice((1, 2, 4, 8)) if jerk else rng.choice((1, 2, 4, 8, 16)))
        if _cost(c) <= 1.0:
            return c


def _cost(c):
    """A case's size over the largest listed one of its kind."""
    if c["kind"] == "search":
        a, b = accel.algorithmic_counts(_obs(c)), accel.algorithmic_counts(_obs(listed()[5]))
        return max(a["corr_flops"] / b["corr_flops"], a["harmsum_min_bytes"] / b["harmsum_min_bytes"])
    if c["kind"] == "polish" and c["wmax"] >= 0:
        return c["ncand"] * c["numharm"] / (48 * 8.0)
    return 0.5


def _obs(c, N=None, dt=DT):
    wmax = c.get("wmax", -1)
    N = N or c["N"]
    return pb.obs_init(pb.make_params(N, dt, N // 2, zmax=c["zmax"], wmax=wmax if wmax >= 0 else None,
                                      numharm=c["numharm"], sigma=2.0, locpow=c.get("locpow", False)))


# ---------------------------------------------------------------------------
# inputs
# ---------------------------------------------------------------------------
def _pulsars(g, N, zmax, wmax, count, nharm, power):
    """count pulsars of nharm harmonics, each of about `power` times the mean
    noise power: r in bins log-uniform over 2 to 700 Hz, z and w uniform."""
    T = N * DT
    out = []
    for _ in range(count):
        f = math.exp(g.uniform(math.log(2.0), math.log(700.0)))
        out.append(dict(r=f * T, z=g.uniform(-0.8, 0.8) * zmax, w=g.uniform(-0.8, 0.8) * max(wmax, 0),
                        amp=math.sqrt(4.0 * power / N), phases=[g.uniform(0, 2 * math.pi) for _ in range(nharm)]))
    return out


def _series(n, seed, pulsars):
    """Unit Gaussian noise plus the pulsars' harmonics (phases by the mean
    r, z, w of the observation, evaluated in FP64), on the device."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    x = torch.randn(n, generator=gen, device="cuda", dtype=torch.float32)
    if pulsars:
        u = torch.arange(n, device="cuda", dtype=torch.float64) / n
        for p in pulsars:
            r0, z0 = p["r"] - p["z"] / 2.0 + p["w"] / 12.0, p["z"] - p["w"] / 2.0
            base = u * (u * (u * (p["w"] / 6.0) + z0 / 2.0) + r0)
            for k, phs in enumerate(p["phases"], start=1):
                x += (p["amp"] * torch.cos(2.0 * math.pi * torch.frac(k * base) + phs)).float()
    return x


def _spectrum(x):
    """The series' packed spectrum (bin 0 = DC and Nyquist) at unit mean noise
    power, complex64 on the device."""
    n = x.numel()
    X = torch.fft.rfft(x.double()) / math.sqrt(n)
    out = X[:n // 2].clone()
    out[0] = torch.complex(X[0].real, X[n // 2].real)
    return out.to(torch.complex64).contiguous()


def _filterbank(c, seed):
    """8-bit-like filterbank spectra [nspec][nchan] as floats: Gaussian noise
    of sigma 16 about 96 and a dispersed 7 ms pulsar in the middle of the DM range."""
    gen = torch.Generator(device="cuda").manual_seed(int(seed))
    g = np.random.default_rng(seed)
    nspec, nchan = c["nspec"], c["nchan"]
    width = BANDWIDTH / nchan
    x = torch.empty(nspec, nchan, device="cuda", dtype=torch.float32)
    t = torch.arange(nspec, device="cuda", dtype=torch.float64)[:, None] * DT
    freq = LOFREQ + width * torch.arange(nchan, device="cuda", dtype=torch.float64)
    delay = 0.5 * c["dmmax"] / (0.000241 * freq * freq)
    period, phase = float(g.uniform(0.006, 0.008)), float(g.uniform(0, 1))
    step = max(1, (1 << 27) // nchan)
    for a in range(0, nspec, step):
        b = min(nspec, a + step)
        x[a:b].normal_(96.0, 16.0, generator=gen)
        for q in range(a, b, 1 << 15):                 # the pulse: 1/16 of a turn, a fifth of the noise
            e = min(b, q + (1 << 15))
            turn = torch.frac((t[q:e] - delay) / period + phase + 1000.0)
            x[q:e] += 3.2 * (turn < 0.0625)
        x[a:b].round_().clamp_(0.0, 255.0)
    return x


def _dms(c):
    return np.linspace(0.0, c["dmmax"], c["ndm"])


def prepare(case, seed):
    g = np.random.default_rng(seed)
    kind = case["kind"]
    ctx = pb.Context(0)
    s = dict(case=case, ctx=ctx)
    if kind in ("planes", "search", "polish"):
        N, wmax = case["N"], case.get("wmax", -1)
        ps = _search_pulsars(g, case) if kind != "polish" else _polish_pulsars(g, case)
        s["fft"] = _spectrum(_series(N, seed, ps))
        s["buf"] = (accel.Cand * MAXCANDS)()
        s["obs"] = _obs(case)
        if kind != "polish":
            ctx.prepare(s["obs"])                      # template banks: kept by a program between spectra
        if kind == "planes":
            ctx.set_spectrum(s["obs"], s["fft"].cpu().numpy())
            s["block"] = _block(case)
        if kind == "polish":
            s["cands"] = _candidates(g, case, ps)
    elif kind == "series":
        n = case["n"]
        x = _series(n, seed, _pulsars(g, n, 20, 0, 2, 4, 100.0))
        walk = torch.randn(n // 4096 + 2, device="cuda", generator=torch.Generator(device="cuda").manual_seed(int(seed) + 1))
        red = torch.cumsum(walk, 0) * 0.2              # receiver drift: red noise for the de-reddening
        s["x"] = x + torch.repeat_interleave(red, 4096)[:n]
        s["out"] = torch.empty(n // 2, device="cuda", dtype=torch.complex64)
    else:
        s["x"] = _filterbank(case, seed)
        s["dms"] = _dms(case)
        s["width"] = BANDWIDTH / case["nchan"]
        if kind == "dedisperse":
            s["out"] = torch.empty(case["ndm"], case["nspec"] // case["downsamp"], device="cuda")
        else:
            ds = case["downsamp"]
            s["obs"] = _obs(case, case["nspec"] // ds & ~1, DT * ds)
            ctx.prepare(s["obs"])
            s["buf"], s["first"] = (accel.Cand * MAXCANDS)(), (C.c_longlong * (case["ndm"] + 1))()
    torch.cuda.synchronize()                           # the framework works on streams of its own
    return s


def _search_pulsars(g, case):
    """Pulsars as bright as those a survey finds: 40 times the noise power in a harmonic."""
    wmax = case.get("wmax", -1)
    return _pulsars(g, case["N"], case["zmax"], wmax, 2 if wmax > 0 else 3, 8 if case["numharm"] >= 8 else 4, 40.0)


def _polish_pulsars(g, case):
    """Their drifts in the fundamental: a search's zmax and wmax bound the highest harmonic's."""
    nh = case["numharm"]
    return _pulsars(g, case["N"], case["zmax"] / nh, case["wmax"] / nh, 4, 8, 100.0)


def _candidates(g, case, pulsars):
    """Search-grid candidates, half of them at the injected pulsars and their second harmonics and half on noise:
    (power, sigma, numharm, r, z, w) tuples as a search returns them."""
    N, wmax = case["N"], max(case["wmax"], 0)
    out = []
    for k in range(case["ncand"]):
        nh = 1 << k // 2 % case["numharm"].bit_length()
        zm, wm = case["zmax"] / nh, wmax / nh
        if k % 2 == 0:
            p, m = pulsars[k // 2 % len(pulsars)], 1 + k // 4 % 2
            r, z, w = p["r"] * m + g.uniform(-0.2, 0.2), p["z"] * m, p["w"] * m
        else:
            r, z, w = g.uniform(0.002, 0.47) * N / nh, g.uniform(-zm, zm), g.uniform(-wm, wm)
        while r * nh > 0.47 * N:
            r *= 0.5
        z, w = max(-zm, min(zm, z)), max(-wm, min(wm, w))
        out.append((40.0, 6.0, nh, round(r * 2 * nh) / (2.0 * nh), 2.0 * round(z * nh / 2) / nh,
                    20.0 * round(w * nh / 20) / nh))
    return out


# ---------------------------------------------------------------------------
# one pass
# ---------------------------------------------------------------------------
def _harmonics(numharm):
    out, m = [(1, 1)], 2
    while m <= numharm:
        out += [(m, h) for h in range(1, m, 2)]
        m *= 2
    return out


def _records(buf, n):
    """The n records of a filled buffer (zeros behind them); r, z and w as the whole grid steps they are."""
    a = np.frombuffer(buf, dtype=np.dtype(dict(names=("power", "sigma", "numharm", "r", "z", "w"),
                                               formats=("f4", "f4", "i4", "f8", "f8", "f8"),
                                               offsets=(0, 4, 8, 16, 24, 32), itemsize=C.sizeof(accel.Cand))))[:n]
    out = {k: np.zeros(MAXCANDS, np.float32) for k in ("power", "sigma")}
    out.update({k: np.zeros(MAXCANDS, np.int32) for k in ("numharm", "r", "z", "w")})
    for k in ("power", "sigma", "numharm"):
        out[k][:n] = a[k]
    for k, step in (("r", 0.5), ("z", 2.0), ("w", 20.0)):
        out[k][:n] = np.rint(a[k] * a["numharm"] / step)
    return out


def _ok(ctx, rc):
    if rc:
        raise RuntimeError(f"error {rc}: {ctx.L.ab_ctx_last_error(ctx.ptr)}")


def run(s):
    c, ctx = s["case"], s["ctx"]
    kind = c["kind"]
    if kind == "planes":
        lo = s["block"]
        hi = lo + s["obs"].rstep - 0.5
        banks = _harmonics(c["numharm"]) if not s["obs"].inmem else [(1, 1)]
        return [ctx.subharm_fderivs_vol(s["obs"], m, h, lo, hi)[1] for m, h in banks]
    if kind == "search":
        n = C.c_longlong()
        _ok(ctx, ctx.L.ab_search(ctx.ptr, C.byref(s["obs"]), s["fft"].data_ptr(), 1, 0, -1, s["buf"], MAXCANDS, C.byref(n)))
        return _records(s["buf"], n.value)
    if kind == "series":
        _ok(ctx, ctx.L.ab_series_to_fft(ctx.ptr, s["x"].data_ptr(), c["n"], DT, 1, s["out"].data_ptr(), 1))
        return s["out"]
    if kind == "dedisperse":
        ctx.dedisperse(None, LOFREQ, s["width"], DT, c["nsub"], s["dms"], c["downsamp"],
                       device_ptr=s["x"].data_ptr(), nspec=c["nspec"], nchan=c["nchan"],
                       out_ptr=s["out"].data_ptr())
        return s["out"]
    if kind == "pipeline":
        _ok(ctx, ctx.L.ab_search_dedispersed(
            ctx.ptr, s["x"].data_ptr(), 1, c["nspec"], c["nchan"], LOFREQ, s["width"], DT, c["nsub"],
            s["dms"].ctypes.data, c["ndm"], c["downsamp"], C.byref(s["obs"]), s["buf"], MAXCANDS, s["first"]))
        first = np.array(s["first"][:])
        return dict(_records(s["buf"], int(first[-1])), first=first)
    pol = ctx.optimize_cands(s["obs"], None, s["cands"], device_ptr=s["fft"].data_ptr())
    return dict(pows=np.concatenate([p["pows"] for p in pol]), r=np.concatenate([p["hirs"] for p in pol]),
                z=np.concatenate([p["hizs"] for p in pol]), w=np.concatenate([p["hiws"] for p in pol]),
                derivs=np.concatenate([p["derivs"] for p in pol]))


# ---------------------------------------------------------------------------
# what a pass cannot do without
# ---------------------------------------------------------------------------
def _search_work(obs):
    a = accel.algorithmic_counts(obs)
    # spectrum in; template products and inverse transforms at the reference's
    # lengths, one addition per harmonic and cell
    adds = a["cells"] / obs.numharmstages * 2 ** (obs.numharmstages - 1)
    return 8.0 * obs.numbins, a["corr_flops"] + adds


def _series_work(n):
    m = n // 2
    return 4.0 * n + 8.0 * m, 5.0 * m * math.log2(m) + 16.0 * m


def _dedisperse_work(c):
    nout = c["nspec"] // c["downsamp"]
    return (4.0 * c["nspec"] * c["nchan"] + 4.0 * c["ndm"] * nout,
            1.0 * c["nspec"] * c["nchan"] + 1.0 * nout * c["nsub"] * c["ndm"])


def work(case):
    kind = case["kind"]
    if kind == "planes":
        obs = _obs(case)
        banks = accel.bank_geometry(obs)
        flops = sum(b["nz"] * (5.0 * b["fftlen_ref"] * math.log2(b["fftlen_ref"]) + 8.0 * b["fftlen_ref"]) for b in banks)
        return dict(bytes=sum(4.0 * b["nz"] * b["numrs_max"] + 4.0 * b["fftlen_ref"] for b in banks), flops=flops)
    if kind == "search":
        b, f = _search_work(_obs(case))
    elif kind == "series":
        b, f = _series_work(case["n"])
    elif kind == "dedisperse":
        b, f = _dedisperse_work(case)
    elif kind == "pipeline":
        ds = case["downsamp"]
        n = case["nspec"] // ds & ~1
        b, f = _dedisperse_work(case)
        b -= 4.0 * case["ndm"] * (case["nspec"] // ds)   # the trials stay inside
        f += case["ndm"] * (_series_work(n)[1] + _search_work(_obs(case, n, DT * ds))[1])
    else:
        # amplitudes of every harmonic: about 80 simplex evaluations of
        # 2 * halfwidth points in an acceleration search, a 17 x 17 x 24 volume
        # of correlations in a jerk search; 8 operations per point
        nh = 0.5 * (case["numharm"] + 1)
        hw = 16 + 0.55 * case["zmax"] * nh
        points = 24.0 * 289 * 2 * hw if case["wmax"] > 0 else 80.0 * 2 * hw
        b, f = case["ncand"] * nh * 16.0 * hw, case["ncand"] * nh * 8.0 * points
    return dict(bytes=float(b), flops=float(f))


def tolerance(case):
    kind = case["kind"]
    if kind == "planes":
        return dict(rel=2e-6, max=1e-4)
    if kind == "series":
        return dict(rel=4e-6, max=4e-4)
    if kind == "dedisperse":
        # sums of whole numbers below 2^24: exact in any order but for the
        # division of the downsampling
        return "exact" if case["downsamp"] in (1, 2) else dict(rel=1e-6)
    if kind == "polish":
        # the optimum of a flat peak: its place is known to the square root of
        # the rounding (3e-4 bins), a phase may wrap
        return dict(rel=1e-3, max=0.2)
    # powers are 32-bit sums; a tie of two neighbouring cells may fall either way
    return dict(rel=1e-5, max=4e-4, differ=0.01)


# ---------------------------------------------------------------------------
# the same in 64 bits, where one pass has computed numbers as its answer
# ---------------------------------------------------------------------------
def _block(case):
    """Start bin of the block whose planes are asked for: one in the middle of the search's block grid."""
    obs = _obs(case)
    return obs.rlo + obs.rstep * (pb.num_blocks(obs) // 3)


def _halfwidth(z):
    return int(0.5 * 1.1 * abs(z)) + 16


def _response(z, q):
    """The amplitude at q bins from a signal's mean frequency when it drifts by z bins: the integral over the
    observation u = 0..1 of exp(2 pi i (q u + z (u^2 - u) / 2)), by Gauss-Legendre quadrature."""
    u, wt = np.polynomial.legendre.leggauss(3 * int(abs(z) + np.max(np.abs(q))) + 96)
    u, wt = 0.5 * (u + 1.0), 0.5 * wt
    return np.exp(2j * np.pi * q[:, None] * u[None, :]) @ (wt * np.exp(1j * np.pi * z * (u * u - u)))


def _good_length(n):
    for g in (128, 192, 256, 384, 512, 768, 1024, 1280, 2048, 4096, 5120, 7680, 10240):
        if n <= g:
            return g


def _exact_planes(case, seed):
    ps = _search_pulsars(np.random.default_rng(seed), case)
    fft = _spectrum(_series(case["N"], seed, ps)).cpu().numpy().astype(np.complex128)
    obs = _obs(case)
    lo = _block(case)
    hi = lo + obs.rstep - 0.5
    kern = 4 * _halfwidth(case["zmax"])
    reflen = max(2048, next(n for lim, n in ((6, 128), (52, 256), (67, 512), (378, 1024), (664, 2048), (1672, 4096)) if kern < lim))
    uselen = reflen - kern
    out = []
    for m, h in (_harmonics(case["numharm"]) if not obs.inmem else [(1, 1)]):
        f = h / m
        zmax = 2 * int(math.floor(0.5 * case["zmax"] * f + 0.5))
        hw = _halfwidth(zmax)
        rlo = int(math.floor(np.rint(2 * lo * f) / 2))
        rhi = int(math.ceil(np.rint(2 * hi * f) / 2))
        numrs = uselen if m == 1 else (2 * (rhi - rlo) + 2) // 2 * 2
        if m > 1:
            reflen = _good_length(math.ceil(uselen * f) + 2 + 4 * hw)
        first = rlo - hw
        d = np.zeros(reflen // 2, np.complex128)
        a, b = max(first, 0), min(first + d.size, fft.size)
        d[a - first:b - first] = fft[a:b]
        d /= math.sqrt(np.median(np.abs(d) ** 2) / math.log(2.0))
        if 4 * hw + numrs - 1 > reflen:
            out.append(None)                           # the window wraps round into these cells
            continue
        dev = torch.from_numpy(d).cuda()
        plane = np.empty((1, zmax + 1, numrs))
        for i in range(zmax + 1):
            z = -zmax + 2 * i
            n = _halfwidth(z)
            j = np.arange(-2 * n, 2 * n)
            k = np.zeros(2 * d.size, np.complex128)    # taps on the half-bin grid, tap 0 first
            # bin b sees a signal of mean frequency r as the response at r - b
            np.add.at(k, j % k.size, _response(z, -j / 2.0))
            K = torch.from_numpy(k).cuda()
            x = torch.zeros(2 * d.size, dtype=torch.complex128, device="cuda")
            x[::2] = dev
            y = torch.fft.ifft(torch.fft.fft(x) * torch.conj(torch.fft.fft(K)))
            plane[0, i] = (y.abs() ** 2)[2 * hw:2 * hw + numrs].cpu().numpy()
        out.append(plane)
    return out


def _fast_invsqrt(x):
    """The 32-bit inverse square root with one Newton step that the de-reddening is defined by."""
    x = np.float32(x)
    y = (np.int32(0x5f3759df) - (x.view(np.int32) >> 1)).view(np.float32)
    return y * (np.float32(1.5) - np.float32(0.5) * x * y * y)


def _exact_series(case, seed):
    s = prepare(case, seed)
    n = case["n"]
    X = torch.fft.rfft(s["x"].double()).cpu().numpy()
    spec = X[:n // 2].copy()
    spec[0] = complex(X[0].real, X[n // 2].real)
    power = np.abs(spec) ** 2
    # blocks of 6 ln(bin) bins up to 200; a line through the mid-points of
    # neighbouring blocks' medians / ln 2
    starts, lens, pos, width = [], [], 1, 6
    Tf, endf = np.float32(DT * n), 0.5 / DT
    while pos < spec.size:
        w = min(width, spec.size - pos)
        starts.append(pos)
        lens.append(w)
        pos += w
        if len(starts) == 1 or float(np.float32(pos) / Tf) < endf:
            width = min(200, int(6 * math.log(pos)))
        else:
            width = 200
    means = np.array([np.median(power[a:a + w]) / math.log(2.0) for a, w in zip(starts, lens)])
    norm = np.empty(spec.size)
    for k, (a, w) in enumerate(zip(starts, lens)):
        if k == 0:
            norm[a:a + w // 2] = means[0]
        end = starts[k + 1] + lens[k + 1] // 2 if k + 1 < len(starts) else a + w
        mid = a + w // 2
        if k + 1 < len(starts):
            slope = (means[k + 1] - means[k]) / (0.5 * (w + lens[k + 1]))
        elif k:
            slope = (means[k] - means[k - 1]) / (0.5 * (w + lens[k - 1]))
        else:
            slope = 1.0
        norm[mid:end] = means[k] + slope * np.arange(end - mid)
    spec[1:] *= _fast_invsqrt(norm[1:].astype(np.float32)).astype(np.float64)
    spec[0] = 1.0
    return spec


def _exact_dedisperse(case, seed):
    x = _filterbank(case, seed)
    nspec, nchan, nsub, ds = case["nspec"], case["nchan"], case["nsub"], case["downsamp"]
    cps, width, dms = nchan // nsub, BANDWIDTH / nchan, _dms(case)
    nout = nspec // ds
    delay = lambda dm, f: dm / (0.000241 * f * f)      # noqa: E731
    top = LOFREQ + (cps - 1) * width                   # the first subband's highest channel
    subs = torch.zeros(nsub, nout, device="cuda", dtype=torch.float64)
    mean = float(np.sum(dms) / len(dms))
    for c in range(nchan):
        s = c // cps
        d = int(math.floor((delay(mean, LOFREQ + c * width) - delay(mean, top + s * cps * width)) / DT + 0.5))
        col = torch.zeros(nspec, device="cuda", dtype=torch.float64)
        col[:max(0, nspec - d)] = x[d:, c].double()
        subs[s] += col[:nout * ds].reshape(nout, ds).sum(1) / ds
    out = torch.zeros(case["ndm"], nout, device="cuda", dtype=torch.float64)
    for k, dm in enumerate(dms):
        ref = delay(dm, top + (nsub - 1) * cps * width)
        for s in range(nsub):
            d = int(math.floor((delay(dm, top + s * cps * width) - ref) / (DT * ds) + 0.5))
            if d < nout:
                out[k, :nout - d] += subs[s, d:]
    return out


def exact(case, seed):
    if case["kind"] == "planes" and case["zmax"] <= 120:
        return _exact_planes(case, seed)
    if case["kind"] == "series" and case["n"] <= 1 << 23:
        return _exact_series(case, seed)
    if case["kind"] == "dedisperse":
        return _exact_dedisperse(case, seed)
    # candidate lists and optima: what is kept depends on comparisons along the way
    return None
