"""Measured cases of the library's transforms.

Each case is one call of a public entry point as a user's program makes it:
device tensors and a plan (or the reference interface's filter storage) in
hand, new results out.  `listed()` gives the fixed cases, `draw(rng)` one more
of the same ranges, `prepare` / `run` one pass, `work` what a pass cannot do
without, `exact` the same results by 64-bit torch arithmetic of its own.

Kinds:
  plan       AdjointNFFT: one light curve, or several value channels at once
  bootstrap  AdjointNFFT.bootstrap: resamples with replacement of one curve
  batch      BatchAdjointNFFT: many series of uneven length in one call
  grad       autograd through BatchedAdjointNFFT (series of one length) or, for
             one series, adjoint_nfft: the spectra and both gradients
  ls         lomb_scargle: floating-mean periodogram with uncertainties
  compat     the reference library's interface: filter coefficients and
             transform (or bootstrap) of one light curve
"""
import math
import random

import numpy as np
import torch

from cunfft_adjoint_gb300 import cuna
from cunfft_adjoint_gb300.autograd import BatchedAdjointNFFT, adjoint_nfft
from cunfft_adjoint_gb300.lombscargle import lomb_scargle
from cunfft_adjoint_gb300.nfft import AdjointNFFT, BatchAdjointNFFT

F32, F64 = "float32", "float64"


def listed():
    return [
        # a short light curve, one look at it: latency and launches
        dict(name="plan_f32_n1000_nf2048", kind="plan", dtype=F32, n=1000, nf=2048, R=2, m=8, chan=1, sorted=True),
        # an ordinary light curve
        dict(name="plan_f32_n10000_nf16384", kind="plan", dtype=F32, n=10_000, nf=1 << 14, R=2, m=8, chan=1,
             sorted=True),
        # a long survey light curve, float32 and float64
        dict(name="plan_f32_n1000000_nf1048576", kind="plan", dtype=F32, n=1_000_000, nf=1 << 20, R=4, m=12, chan=1,
             sorted=False),
        dict(name="plan_f64_n1000000_nf1048576", kind="plan", dtype=F64, n=1_000_000, nf=1 << 20, R=4, m=12, chan=1,
             sorted=False),
        # significance of a peak: 1024 resamples of one light curve
        dict(name="bootstrap_f32_n5000_x1024_nf32768", kind="bootstrap", dtype=F32, n=5000, nf=32768, R=2, m=8,
             nbs=1024),
        # a survey's light curves in one call
        dict(name="batch_f32_x4096_uneven", kind="batch", dtype=F32, series=4096, lo=100, hi=100_000, nfcap=1 << 18,
             R=2, m=8, lengths=4),
        # training steps through the transform: many long series, many short
        # ones, and one in float64
        dict(name="grad_f32_x64_n200000_nf262144", kind="grad", dtype=F32, series=64, n=200_000, nf=1 << 18, R=2,
             m=10),
        dict(name="grad_f32_x48_n3001_nf4096", kind="grad", dtype=F32, series=48, n=3001, nf=4096, R=2, m=8),
        dict(name="grad_f64_x1_n200000_nf262144", kind="grad", dtype=F64, series=1, n=200_000, nf=1 << 18, R=2, m=10),
        # a period search of one light curve with uncertainties
        dict(name="ls_f32_n5003_nfreq50000", kind="ls", dtype=F32, n=5003, nfreq=50_000, R=2, m=8),
        # programs written against the reference's interface, its float and
        # double builds
        dict(name="compat_f32_n1000000_ng4194304", kind="compat", dtype=F32, n=1_000_000, ng=1 << 22, nbs=0),
        dict(name="compat_f64_n100003_ng524288", kind="compat", dtype=F64, n=100_003, ng=1 << 19, nbs=0),
    ]


def _logint(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["plan", "plan", "bootstrap", "batch", "grad", "grad", "ls", "compat"])
    dtype = rng.choice([F32, F32, F64])
    # filter widths of the configurations: float ones reach 1e-6, double 1e-9 and below
    R, m = rng.choice([(2, 8), (2, 10), (4, 6), (4, 12)] if dtype == F32 else [(2, 10), (2, 12), (4, 12)])
    if kind == "plan":
        chan = rng.choice([1, 1, 1, 2, 5])
        n = _logint(rng, 200, 1_000_000 // chan)
        # from as many outputs as samples to several times as many
        nf = 1 << max(9, min(20 if R == 4 else 21, round(math.log2(n * rng.uniform(0.7, 4.5)))))
        while nf * R * chan > 1 << 22 and nf > 512:
            nf //= 2
        return dict(kind=kind, dtype=dtype, n=n, nf=nf, R=R, m=m, chan=chan, sorted=rng.random() < 0.6)
    if kind == "bootstrap":
        nf = 1 << rng.randint(10, 15)
        n = _logint(rng, 300, 12_000)
        cap = min(1024 if dtype == F32 else 256, (1 << 26) // (nf * R), 5_000_000 // n)
        return dict(kind=kind, dtype=dtype, n=n, nf=nf, R=R, m=m, nbs=_logint(rng, 20, cap))
    if kind == "batch":
        series = _logint(rng, 24, 1500 if dtype == F32 else 300)
        return dict(kind=kind, dtype=dtype, series=series, lo=100, hi=_logint(rng, 2000, 100_000), nfcap=1 << 18,
                    R=2, m=max(8, m), lengths=rng.randrange(1 << 30))
    if kind == "grad":
        n = _logint(rng, 500, 200_000)
        nf = 1 << max(9, min(18, round(math.log2(n * rng.uniform(0.7, 2.0)))))
        series = _logint(rng, 1, max(1, min(64, 12_000_000 // n) // (1 if dtype == F32 else 8)))
        return dict(kind=kind, dtype=dtype, series=series, n=n, nf=nf, R=2, m=10 if dtype == F64 else m)
    if kind == "ls":
        return dict(kind=kind, dtype=dtype, n=_logint(rng, 300, 200_000), nfreq=_logint(rng, 1000, 400_000), R=R, m=m)
    if rng.random() < 0.3:  # bootstrap of the reference interface
        n, ng = _logint(rng, 300, 8000), 1 << rng.randint(11, 16)
        cap = min(1024 if dtype == F32 else 128, (1 << 25) // ng, 3_000_000 // n)
        return dict(kind=kind, dtype=dtype, n=n, ng=ng, nbs=_logint(rng, 8, cap))
    n = _logint(rng, 500, 1_000_000 if dtype == F32 else 250_000)
    ng = 1 << max(10, min(22 if dtype == F32 else 20, round(math.log2(n * rng.uniform(2.0, 6.0)))))
    return dict(kind=kind, dtype=dtype, n=n, ng=ng, nbs=0)


def _dt(case):
    return torch.float32 if case["dtype"] == F32 else torch.float64


def _lengths(case):
    """Samples and outputs per series of a batch case (part of the case, like
    the plan's, not of the inputs)."""
    r = random.Random(case["lengths"])
    n = [_logint(r, case["lo"], case["hi"]) for _ in range(case["series"])]
    nf = [min(case["nfcap"], 1 << max(6, math.ceil(math.log2(4 * v)))) for v in n]
    T = [math.exp(r.uniform(math.log(10.0), math.log(3000.0))) for _ in n]
    return np.array(n), np.array(nf), np.array(T)


def _series(n, T, g, order):
    """Sample times in [0, T) and values of one light curve."""
    if n >= 500_000 and not order:  # ten observing seasons
        w = torch.randint(0, 10, (n,), generator=g, device="cuda")
        t = (w + torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * (200.0 / 365.0)) * (T / 10.0)
    else:
        t = torch.rand(n, generator=g, device="cuda", dtype=torch.float64) * T
        if order:
            t = t.sort().values
    y = (torch.sin(2 * math.pi * t * 1.43) + 0.3 * torch.sin(2 * math.pi * t / 3.3)
         + torch.randn(n, generator=g, device="cuda", dtype=torch.float64))
    return t, y


_SPAN = {"plan": 3650.0, "bootstrap": 100.0, "grad": 500.0, "ls": 400.0}


def _inputs(case, seed):
    """The tensors a program has before the call."""
    g = torch.Generator(device="cuda").manual_seed(seed)
    dt, kind = _dt(case), case["kind"]
    if kind == "plan":
        t, y = _series(case["n"], _SPAN[kind], g, case["sorted"])
        if case["chan"] == 1:
            return dict(t=t, y=y.to(dt))
        # further bands at the same times, the last one the window function
        Y = torch.randn((case["chan"], case["n"]), generator=g, device="cuda", dtype=torch.float64)
        Y[0] = y
        Y[-1] = 1.0
        return dict(t=t, y=Y.to(dt))
    if kind == "bootstrap":
        t, y = _series(case["n"], _SPAN[kind], g, False)
        return dict(t=t, y=y.to(dt), seed=seed & 0xFFFFFF)
    if kind == "batch":
        n, _, T = _lengths(case)
        Tr = torch.as_tensor(np.repeat(T, n), device="cuda")
        tot = int(n.sum())
        return dict(t=torch.rand(tot, generator=g, device="cuda", dtype=torch.float64) * Tr,
                    y=torch.randn(tot, generator=g, device="cuda", dtype=dt))
    if kind == "grad":
        B, n, nf = case["series"], case["n"], case["nf"]
        t = (torch.rand((B, n), generator=g, device="cuda", dtype=torch.float64) * _SPAN[kind]).sort(dim=1).values
        y = torch.randn((B, n), generator=g, device="cuda", dtype=dt)
        G = torch.complex(torch.randn((B, nf), generator=g, device="cuda", dtype=dt),
                          torch.randn((B, nf), generator=g, device="cuda", dtype=dt))
        if B == 1:
            t, y, G = t[0], y[0], G[0]
        return dict(t=t, y=y, G=G)
    if kind == "ls":
        t, y = _series(case["n"], _SPAN[kind], g, True)
        dy = 0.3 + 0.5 * torch.rand(case["n"], generator=g, device="cuda", dtype=torch.float64)
        return dict(t=t, y=y.to(dt), dy=dy.to(dt))
    # positions in [-1/2, 1/2), as scale_x leaves them
    t, y = _series(case["n"], 1.0, g, True)
    return dict(x=(t - 0.5).to(dt), y=y.to(dt), seed=seed & 0xFFFFFF)


def prepare(case, seed):
    st = _inputs(case, seed)
    kind, dt = case["kind"], _dt(case)
    st["case"] = case
    if kind in ("plan", "bootstrap"):
        st["plan"] = AdjointNFFT(case["nf"], case["R"], case["m"], dt)
    elif kind == "batch":
        n, nf, T = _lengths(case)
        st["plan"] = BatchAdjointNFFT(n, nf, case["R"], case["m"], np.zeros(len(n)), T, dt)
    elif kind == "grad":
        st["t"].requires_grad_(True)
        st["y"].requires_grad_(True)
        if case["series"] == 1:
            st["plan"] = AdjointNFFT(case["nf"], case["R"], case["m"], dt)
        else:
            B = case["series"]
            st["plan"] = BatchedAdjointNFFT(B, case["n"], case["nf"], case["R"], case["m"], [0.0] * B,
                                            [_SPAN[kind]] * B, dt)
    elif kind == "compat":
        st["filter"] = cuna.FilterProperties(case["n"], dt, "cuda")
        shape = (case["nbs"], case["ng"]) if case["nbs"] else (case["ng"],)
        st["f_hat"] = torch.zeros(shape, dtype=torch.complex64 if dt == torch.float32 else torch.complex128,
                                  device="cuda")
    return st


def run(st):
    case = st["case"]
    kind = case["kind"]
    if kind == "plan":
        if case["chan"] == 1:
            return st["plan"](st["t"], st["y"], 0.0, _SPAN[kind])
        return st["plan"].multi(st["t"], st["y"], 0.0, _SPAN[kind])
    if kind == "bootstrap":
        return st["plan"].bootstrap(st["t"], st["y"], case["nbs"], st["seed"], 0.0, _SPAN[kind])
    if kind == "batch":
        return st["plan"](st["t"], st["y"])
    if kind == "grad":
        if case["series"] == 1:
            F = adjoint_nfft(st["t"], st["y"], st["plan"], 0.0, _SPAN[kind])
        else:
            F = st["plan"](st["t"], st["y"])
        gt, gy = torch.autograd.grad(F, (st["t"], st["y"]), st["G"])
        return F.detach(), gt, gy
    if kind == "ls":
        return lomb_scargle(st["t"], st["y"], st["dy"], nfreq=case["nfreq"], df=1.0 / (5.0 * _SPAN[kind]), t0=0.0,
                            R=case["R"], m=case["m"])
    f_hat, fp, n, ng = st["f_hat"], st["filter"], case["n"], case["ng"]
    s = torch.cuda.current_stream()
    f_hat.zero_()  # the call accumulates
    cuna.generate_pinned_filter_properties(st["x"], n, ng, fp, s)
    if case["nbs"]:
        cuna.cunfft_adjoint_raw_async_bootstrap(st["x"], st["y"], f_hat, n, ng, case["nbs"], fp, s, st["seed"])
    else:
        cuna.cunfft_adjoint_raw_async(st["x"], st["y"], f_hat, n, ng, fp, s)
    return f_hat


def _fft_flops(ng):
    return 2.5 * ng * math.log2(ng)  # a real transform of ng points


def work(case):
    e = 4 if case["dtype"] == F32 else 8
    kind = case["kind"]
    if kind == "plan":
        n, nf, c = case["n"], case["nf"], case["chan"]
        return {"bytes": 8 * n + c * (e * n + 2 * e * nf),
                "flops": c * (6.0 * case["m"] * n + _fft_flops(nf * case["R"]))}
    if kind == "bootstrap":
        n, nf, b = case["n"], case["nf"], case["nbs"]
        return {"bytes": (8 + e) * n + 2 * e * nf * b, "flops": b * (6.0 * case["m"] * n + _fft_flops(nf * case["R"]))}
    if kind == "batch":
        n, nf, _ = _lengths(case)
        return {"bytes": float((8 + e) * n.sum() + 2 * e * nf.sum()),
                "flops": 6.0 * case["m"] * float(n.sum()) + sum(_fft_flops(int(v) * case["R"]) for v in nf)}
    if kind == "grad":
        n, nf, b = case["n"], case["nf"], case["series"]
        # forward: t, y -> F; backward: t, y, G -> dL/dt, dL/dy
        return {"bytes": b * (2 * (8 + e) * n + 4 * e * nf + (8 + e) * n),
                "flops": b * (14.0 * case["m"] * n + 2 * _fft_flops(nf * case["R"]))}
    if kind == "ls":
        n, k = case["n"], case["nfreq"]
        return {"bytes": (8 + 2 * e) * n + e * k,
                "flops": 2 * (6.0 * case["m"] * n + _fft_flops(4 * k * case["R"])) + 40.0 * k}
    n, ng, b = case["n"], case["ng"], max(1, case["nbs"])
    rf = 6 if e == 4 else 12
    return {"bytes": 2 * e * n + 2 * e * ng * b, "flops": b * (8.0 * rf * n + 5.0 * ng * math.log2(ng))}


# ---------------------------------------------------------------------------
# the same results in 64 bits: sums over samples through a Gaussian of 28
# cells on a four times oversampled grid (error below 1e-16 of the spectrum),
# grid positions with the division's remainder carried
# ---------------------------------------------------------------------------
_XR, _XM = 4, 14
_XTAU = _XM * _XR / (4.0 * math.pi * (_XR - 0.5))


def _split(a):
    c = a * 134217729.0
    h = c - (c - a)
    return h, a - h


def _cells(t, T, ng):
    """(cell, fraction) of ng * (t / T mod 1) for t in [0, T)."""
    q = t / T
    qh, ql = _split(q)
    Th, Tl = _split(T)
    p = q * T
    err = ((qh * Th - p) + qh * Tl + ql * Th) + ql * Tl  # q T = p + err exactly
    r = ((t - p) - err) / T
    s = q * ng
    c = torch.floor(s)
    f = (s - c) + r * ng
    return torch.remainder(c, ng).to(torch.int64), f


def _decon(nf, ng):
    k = torch.arange(-(nf // 2), nf // 2, device="cuda", dtype=torch.float64)
    s = torch.exp(4 * math.pi ** 2 * _XTAU * (k / ng) ** 2) / math.sqrt(4 * math.pi * _XTAU)
    return torch.where(k.to(torch.int64) % 2 == 0, s, -s)


def _sums(t, y, T, nf, row, rows):
    """F[row, k + nf/2] = sum over that row's samples of y e^{2 pi i k (t/T - 1/2)}."""
    ng = _XR * nf
    c, f = _cells(t, T, ng)
    grid = torch.zeros(rows * ng, device="cuda", dtype=torch.float64)
    for d in range(-_XM + 1, _XM + 1):
        grid.index_add_(0, row * ng + torch.remainder(c + d, ng), y * torch.exp(-(d - f) ** 2 / (4 * _XTAU)))
    h = torch.fft.rfft(grid.view(rows, ng))[:, :nf // 2 + 1].conj()
    F = torch.cat([h[:, 1:].conj().flip(1), h[:, :nf // 2]], dim=1)
    return F * _decon(nf, ng)


def _fields(G, t, T, nf):
    """Re sum_k conj(G_k) e^{2 pi i k (t/T - 1/2)} at every t, one row of G per row of t."""
    ng = _XR * nf
    k = torch.arange(-(nf // 2), nf // 2, device="cuda", dtype=torch.int64)
    z = torch.zeros((G.shape[0], ng), device="cuda", dtype=torch.complex128)
    z[:, torch.remainder(k, ng)] = G.conj() * _decon(nf, ng)
    r = (torch.fft.ifft(z) * ng).real
    c, f = _cells(t, T, ng)
    out = torch.zeros_like(t)
    for d in range(-_XM + 1, _XM + 1):
        out += torch.gather(r, 1, torch.remainder(c + d, ng)) * torch.exp(-(d - f) ** 2 / (4 * _XTAU))
    return out


def _draws(n, nbs, seed):
    """The reference's bootstrap draw stream: xorshift32(wang_hash(seed + i)) mod n."""
    M = 0xFFFFFFFF
    s = (torch.arange(n * nbs, device="cuda", dtype=torch.int64) + seed) & M
    s = (s ^ 61) ^ (s >> 16)
    s = (s * 9) & M
    s = s ^ (s >> 4)
    s = (s * 0x27d4eb2d) & M
    s = s ^ (s >> 15)
    s = s ^ ((s << 13) & M)
    s = s ^ (s >> 17)
    s = s ^ ((s << 5) & M)
    return (s % n).view(nbs, n)


def _rows_in_chunks(fn, rows, per):
    return torch.cat([fn(a, min(rows, a + per)) for a in range(0, rows, per)])


def _exact_compat(case, a):
    x32, y = a["x"], a["y"].double()
    n, ng, b_ = case["n"], case["ng"], case["nbs"]
    rf = 6 if case["dtype"] == F32 else 12
    Rr = ng / n
    b = 2 * Rr / (2 * Rr - 1) * (rf / math.pi)
    x = x32.double()
    u = torch.trunc(ng * x32 - rf).double()  # the origin in the sample's own precision
    eps = ng * x - u
    E1, E2 = torch.exp(-eps * eps / b) / math.sqrt(math.pi * b), torch.exp(2 * eps / b)
    j = torch.trunc((x + 0.5) * (ng - 1)).to(torch.int64).clamp(0, ng - 1)
    rows = max(1, b_)
    if b_:
        d = _draws(n, b_, a["seed"])
        E1, E2, y, j = E1[d], E2[d], y[d], j.expand(b_, n)
    grid = torch.zeros(rows * ng, device="cuda", dtype=torch.float64)
    base = torch.arange(rows, device="cuda").view(-1, 1) * ng
    E1, E2, y, j = E1.reshape(rows, n), E2.reshape(rows, n), y.reshape(rows, n), j.reshape(rows, n)
    for m in range(-rf + 1, rf):
        c = j + m
        ok = (c >= 0) & (c < ng)
        w = torch.where(ok, y * E1 * E2 ** m * math.exp(-m * m / b), torch.zeros((), device="cuda", dtype=torch.float64))
        grid.index_add_(0, (base + c.clamp(0, ng - 1)).reshape(-1), w.reshape(-1))
    K = torch.arange(ng, device="cuda", dtype=torch.float64) / ng
    F = torch.fft.ifft(grid.view(rows, ng)) * ng * (math.sqrt(2 * math.pi) * torch.exp(K * K * b * 0.25))
    return F if b_ else F[0]


def exact(case, seed):
    a = _inputs(case, seed)
    kind = case["kind"]
    if kind == "compat":
        return _exact_compat(case, a)
    if kind == "batch":
        n, nf, T = _lengths(case)
        off, foff = np.concatenate([[0], np.cumsum(n)]), np.concatenate([[0], np.cumsum(nf)])
        out = torch.empty(int(foff[-1]), device="cuda", dtype=torch.complex128)
        for v in np.unique(nf):
            ids = np.nonzero(nf == v)[0]
            per = max(1, (1 << 27) // (_XR * int(v)))
            for c0 in range(0, len(ids), per):
                part = ids[c0:c0 + per]
                at = torch.as_tensor(np.concatenate([np.arange(off[s], off[s + 1]) for s in part]), device="cuda")
                row = torch.as_tensor(np.repeat(np.arange(len(part)), n[part]), device="cuda")
                Ts = torch.as_tensor(np.repeat(T[part], n[part]), device="cuda")
                F = _sums(a["t"][at], a["y"][at].double(), Ts, int(v), row, len(part))
                for i, s in enumerate(part):
                    out[foff[s]:foff[s + 1]] = F[i]
        return out
    T = torch.full((), 5.0 * _SPAN[kind] if kind == "ls" else _SPAN[kind], device="cuda", dtype=torch.float64)
    t, y = a["t"], a["y"].double()
    n = case["n"]
    if kind == "plan":
        zero = torch.zeros(n, device="cuda", dtype=torch.int64)
        F = torch.cat([_sums(t, v, T, case["nf"], zero, 1) for v in y.view(case["chan"], n)])
        return F[0] if case["chan"] == 1 else F
    if kind == "bootstrap":
        d = _draws(n, case["nbs"], a["seed"])

        def part(lo, hi):
            dd = d[lo:hi].reshape(-1)
            row = torch.arange(hi - lo, device="cuda").repeat_interleave(n)
            return _sums(t[dd], y[dd], T, case["nf"], row, hi - lo)
        return _rows_in_chunks(part, case["nbs"], max(1, (1 << 27) // (_XR * case["nf"])))
    if kind == "grad":
        B, nf = case["series"], case["nf"]
        t, y, G = t.view(B, n), y.view(B, n), a["G"].to(torch.complex128).view(B, nf)
        k = torch.arange(-(nf // 2), nf // 2, device="cuda", dtype=torch.float64)
        per = max(1, (1 << 26) // (_XR * nf))

        def fwd(lo, hi):
            row = torch.arange(hi - lo, device="cuda").repeat_interleave(n)
            return _sums(t[lo:hi].reshape(-1), y[lo:hi].reshape(-1), T, nf, row, hi - lo)
        F = _rows_in_chunks(fwd, B, per)
        gy = _rows_in_chunks(lambda lo, hi: _fields(G[lo:hi], t[lo:hi], T, nf), B, per)
        # conj(Gk) 2 pi i k / T = conj(-2 pi i k Gk / T)
        gt = _rows_in_chunks(lambda lo, hi: _fields(G[lo:hi] * (-2j * math.pi / _SPAN[kind]) * k, t[lo:hi], T, nf),
                             B, per) * y
        return (F, gt, gy) if B > 1 else (F[0], gt[0], gy[0])
    # ls
    w = 1.0 / a["dy"].double() ** 2
    w = w / w.sum()
    yc = y - (w * y).sum()
    K = case["nfreq"]
    nf = 1 << math.ceil(math.log2(4 * K + 4))
    zero = torch.zeros(n, device="cuda", dtype=torch.int64)
    A = _sums(t, w * yc, T, nf, zero, 1)[0][nf // 2:]
    Bw = _sums(t, w, T, nf, zero, 1)[0][nf // 2:]
    q = torch.arange(1, K + 1, device="cuda")
    YC, YS, C, S = A[q].real, A[q].imag, Bw[q].real, Bw[q].imag
    C2, S2 = Bw[2 * q].real, Bw[2 * q].imag
    CC, SS, CS = (1 + C2) / 2 - C * C, (1 - C2) / 2 - S * S, S2 / 2 - C * S
    return (SS * YC * YC + CC * YS * YS - 2 * CS * YC * YS) / ((w * yc * yc).sum() * (CC * SS - CS * CS))
