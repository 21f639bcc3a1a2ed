"""GPU tests of the kernels' size-dependent paths, at the sizes where a rule
switches and at the edges of tiles and windows, against the oracle.

Tolerances (relative L2, derived): the compared programs evaluate the same
sums in the same precision; double paths differ by a few roundings per term
(an exponent of E2^m amplifies one ulp of E2 at most 11 times, about 3e-15,
and the FFT adds log2(ng) 1e-16), so 1e-13.
"""
import numpy as np
import pytest
import torch

from conftest import rel_l2

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def mods(native_built):
    from cunfft_adjoint_gb300 import cuna, nfft
    return cuna, nfft


@pytest.mark.parametrize("n,ng", [(1, 1 << 14), (777, 1 << 14), (40_001, 1 << 17), (70_000, 1 << 21)])
def test_compat_double_powers_and_factors(mods, oracle_lib, n, ng):
    """E2^m by running products (many and few tiles per SM) and the row
    pass's deconvolution factors between exps, with samples on both ends of
    the grid and on tile boundaries."""
    cuna, _ = mods
    rng = np.random.default_rng(n)
    x = rng.uniform(-0.5, 0.5, n)
    edge = np.array([-0.5, 0.5, np.nextafter(0.5, 0), (4096 - 0.5) / (ng - 1) - 0.5, 4096.5 / (ng - 1) - 0.5])
    x[:min(n, len(edge))] = edge[:min(n, len(edge))]
    y = rng.normal(0, 1, n)
    xd, yd = torch.as_tensor(x, device="cuda"), torch.as_tensor(y, device="cuda")
    fp = cuna.generate_filter_properties(xd, n, ng)
    f_hat = torch.zeros(ng, dtype=torch.complex128, device="cuda")
    cuna.cunfft_adjoint_raw(xd, yd, f_hat, n, ng, fp)
    assert rel_l2(f_hat.cpu().numpy(), oracle_lib.compat_adjoint(x, y, ng, "d")) < 1e-13


@pytest.mark.parametrize("dtype,tol", [(torch.float32, 2e-5), (torch.float64, 1e-9)])
@pytest.mark.parametrize("R,m,nf,ns", [(2, 1, 1 << 15, 1), (2, 12, 1 << 15, 2), (4, 13, 1 << 14, 1), (8, 16, 1 << 13, 3),
                                       (4, 6, 256, 2)])
def test_backward_windows(mods, dtype, tol, R, m, nf, ns):
    """The backward's windows at every alignment and over the grid's seam, for
    narrow and wide filters, one and several series, against the exact
    adjointness relation: <G, F(y)> = <dL/dy, y> for the plan's own forward,
    whose gridding and FFT passes are other kernels (relative to the norms:
    one plan precision's rounding of sums, 2e-5 and 1e-9)."""
    _, nfft = mods
    rng = np.random.default_rng(m)
    n, T = 1001, 7.0
    ng = R * nf
    t = rng.uniform(0, T, (ns, n))
    cells = np.concatenate([np.arange(20), ng - 1 - np.arange(20), rng.integers(0, ng, 160)])
    t[:, :200] = (cells + rng.uniform(0.01, 0.99, 200)) / ng * T
    y = rng.normal(0, 1, (ns, n))
    G = rng.normal(0, 1, (ns, nf)) + 1j * rng.normal(0, 1, (ns, nf))
    plan = nfft.AdjointNFFT(nf, R, m, dtype)
    td, yd = torch.as_tensor(t, device="cuda"), torch.as_tensor(y, dtype=dtype, device="cuda")
    Gd = torch.as_tensor(G, dtype=plan.cdtype, device="cuda")
    gy, gt = plan.backward_batch(td, yd, Gd, 0.0, T)
    for s in range(ns):
        F = plan(td[s], yd[s], 0.0, T).to(torch.complex128)
        Gs = Gd[s].to(torch.complex128)
        lhs = float((Gs.conj() * F).real.sum())
        rhs = float((gy[s].double() * yd[s].double()).sum())
        assert abs(lhs - rhs) < tol * float(Gs.abs().square().sum().sqrt() * F.abs().square().sum().sqrt())
        # dL/dt_j = dL/ds_j of moving one sample's time, by the same relation on
        # the sample's own spectrum: y_j * d/dt of the field; its sum over all
        # samples moved together is the derivative of <G, F> under a shift,
        # which multiplies F_k by exp(2 pi i k dt / T)
        k = torch.arange(-nf // 2, nf // 2, device="cuda", dtype=torch.float64)
        dF = F * (2j * np.pi / T) * k
        lhs = float((Gs.conj() * dF).real.sum())
        rhs = float(gt[s].sum())
        bound = float(Gs.abs().square().sum().sqrt() * dF.abs().square().sum().sqrt())
        kernel = np.exp(-np.pi * m * np.sqrt(1 - 1 / R))
        assert abs(lhs - rhs) < (tol + 20 * kernel) * bound


@pytest.mark.parametrize("n,nf,R,m", [(0, 64, 2, 8), (1, 4, 4, 4), (3, 8, 4, 2), (40, 64, 2, 8), (33, 16, 2, 7),
                                      (1000, 2048, 2, 8), (2049, 2048, 4, 12), (5000, 512, 2, 3), (300, 4096, 2, 16)])
def test_small_gather(mods, oracle_lib, n, nf, R, m):
    """One-CTA float transforms: windows wider than a third of the grid (the
    gather's periodic images), one and several chunks of records, samples on
    the seam, empty input; against the oracle's double restatement of the same
    sums (float rounding of about 2m n terms, 2e-6)."""
    _, nfft = mods
    rng = np.random.default_rng(n + nf)
    t = rng.uniform(0, 3.0, n)
    t[:2] = [0.0, np.nextafter(3.0, 0)][:min(n, 2)]
    y = rng.normal(0, 1, n).astype(np.float32)
    plan = nfft.AdjointNFFT(nf, R, m, torch.float32)
    F = plan(torch.as_tensor(t, device="cuda"), torch.as_tensor(y, device="cuda"), 0.0, 3.0).cpu().numpy()
    if n == 0:
        assert not F.any()
        return
    assert rel_l2(F, oracle_lib.accurate_adjoint(t, y.astype(np.float64), 0.0, 3.0, nf, R, m)) < 2e-6


def _sums_extended(t, y, T, ks):
    """F_k by direct summation in extended precision (numpy longdouble)."""
    x = t.astype(np.longdouble) / np.longdouble(T) - np.longdouble(0.5)
    tau = 2 * np.arctan2(np.longdouble(0), np.longdouble(-1))
    out = np.zeros(len(ks), np.clongdouble)
    for i, k in enumerate(ks):
        ph = int(k) * x
        ph -= np.rint(ph)
        out[i] = np.sum(y * np.cos(tau * ph)) + 1j * np.sum(y * np.sin(tau * ph))
    return out


@pytest.mark.parametrize("nf,R,m", [(1 << 13, 4, 12), (1 << 15, 2, 16), (1 << 17, 2, 10), (1 << 17, 8, 16), (1 << 19, 4, 12)])
def test_float_float_passes_lengths(mods, nf, R, m):
    """Float-float FFT passes at lengths of every leading radix (2, 4, 8) in
    either pass, against direct sums in extended precision on 200 bins.  (The
    oracle's double restatement carries its own phase rounding, 2 pi k 1e-16
    per sample, up to 7e-12 here.)  Bound: ten times the Gaussian kernel's
    exp(-pi m sqrt(1 - 1/R)) plus the passes' rounding, 2^-46 per operation over
    log2(ng) stages amplified by the deconvolution (at most 70): 1e-11."""
    if np.finfo(np.longdouble).nmant < 60:
        pytest.skip("no extended precision")
    _, nfft = mods
    rng = np.random.default_rng(nf + R)
    n = 3000
    t = rng.uniform(0, 50.0, n)
    y = rng.normal(0, 1, n)
    plan = nfft.AdjointNFFT(nf, R, m, torch.float64)
    F = plan(torch.as_tensor(t, device="cuda"), torch.as_tensor(y, device="cuda"), 0.0, 50.0).cpu().numpy()
    ks = np.concatenate([[-nf // 2, -nf // 2 + 1, -1, 0, 1, nf // 2 - 1], rng.integers(-nf // 2, nf // 2, 194)])
    D = _sums_extended(t, y, 50.0, ks).astype(np.complex128)
    assert rel_l2(F[ks + nf // 2], D) < 1e-11 + 10 * np.exp(-np.pi * m * np.sqrt(1 - 1 / R))


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n,nf", [(1, 1 << 15), (8, 1 << 15), (511, 1 << 20), (2049, 1 << 18), (16384, 1 << 16), (16385, 1 << 16)])
def test_binning_in_one_launch(mods, oracle_lib, dt, n, nf):
    """Short series binned by one cluster launch (up to 16384 samples; the next
    size takes the two-launch sort), few and many tiles, samples on tile edges
    and the grid's seam: every tile's records equal the oracle's integer steps,
    as sets."""
    import test_gpu_integer_steps as steps
    from cunfft_adjoint_gb300 import _lib, nfft
    rng = np.random.default_rng(n)
    R, m, T = 2, 8, 5.0
    t = np.sort(rng.uniform(0, T, n))
    edges = np.array([0.0, 2048.0, 4096.0, 2047.99, R * nf - 0.01]) / (R * nf) * T
    t[:min(n, 5)] = edges[:min(n, 5)]
    y = rng.normal(0, 1, n).astype(dt)
    plan = nfft.AdjointNFFT(nf, R, m, torch.float32 if dt == np.float32 else torch.float64)

    class Lib:
        check, core = staticmethod(_lib.check), staticmethod(_lib.core)
    log_tile, offs, recs = steps._plan_bins_device(Lib, plan, t, y, 0.0, T)
    _, cell, _, _ = oracle_lib.phases(t, 0.0, T, plan.ng)
    ta, tb = oracle_lib.accurate_tiles(cell, plan.ng, m, log_tile)
    want = sorted([(int(a), int(cell[i]), i) for i, a in enumerate(ta)]
                  + [(int(b), int(cell[i]), i) for i, b in enumerate(tb) if b != ta[i] and b >= 0])
    tile = np.repeat(np.arange(len(offs) - 1), np.diff(offs))
    assert sorted(zip(tile.tolist(), recs["cell"].tolist(), recs["p"].tolist())) == want


@pytest.mark.parametrize("scale", [1e-30, 1.0, 1e18])
@pytest.mark.parametrize("n,nfreq", [(65, 700), (20000, 5000)])
def test_lomb_scargle_scales(mods, scale, n, nfreq):
    """The float periodogram does not depend on the data's scale: sums beside the
    one-launch binning and after the two-launch one, one and many partial sums,
    against the double plan on the same float values.  Weighted sums of the
    float plan carry a few 1e-7, amplified where CC SS - CS^2 is small: 1e-4, the
    bound of the float periodogram against direct sums."""
    from cunfft_adjoint_gb300.lombscargle import lomb_scargle
    rng = np.random.default_rng(n)
    t = np.sort(rng.uniform(0, 100.0, n))
    y = np.sin(2 * np.pi * t / 2.1) + rng.normal(0, 1, n)
    dy = rng.uniform(0.2, 0.6, n)
    td = torch.as_tensor(t, device="cuda")
    y32 = torch.as_tensor((y * scale).astype(np.float32), device="cuda")
    dy32 = torch.as_tensor(dy.astype(np.float32), device="cuda")
    P = lomb_scargle(td, y32, dy32, nfreq=nfreq, df=1 / 500.0, t0=0.0)
    D = lomb_scargle(td, y32.double() / scale, dy32.double(), nfreq=nfreq, df=1 / 500.0, t0=0.0, R=4, m=12)
    assert rel_l2(P.cpu().numpy(), D.cpu().numpy()) < 1e-4


@pytest.mark.parametrize("R,m", [(8, 1), (4, 4), (2, 5), (2, 8), (2, 16)])
@pytest.mark.parametrize("cnt", [0, 1, 256, 257, 512, 513, 1024, 1025, 2600])
def test_fixed_point_own_values(mods, cnt, R, m):
    """Float fixed-point tiles of one transform, which read their records twice
    (the first two of a thread kept in registers), against the same records
    staged in shared memory, as a channel of a multi-channel transform runs:
    equal bits.  cnt samples fall into one tile, some at its edges, few into
    the others.  Against the double plan of the same filter: 2e-6 (2^-22 of
    each weight's exp2 and 2^-30 of a tile's bound per tap)."""
    from cunfft_adjoint_gb300 import _lib
    _, nfft = mods
    rng = np.random.default_rng(cnt + m)
    nf, T = (1 << 17) // R, 3.0
    ng = R * nf
    pos = np.concatenate([4096 * 5 + rng.uniform(m, 4096 - m, cnt), rng.uniform(0, ng, 50),
                          4096 * 5 + rng.uniform(-m, m, min(cnt, 4)), rng.uniform(0, m, 3), ng - rng.uniform(0, m, 3)])
    t = torch.as_tensor(pos / ng * T, device="cuda")
    y = torch.as_tensor(rng.normal(0, 1, pos.size), device="cuda")
    plan = nfft.AdjointNFFT(nf, R, m)
    plan.set_schedule(12, _lib.GRID_FIXED)
    F = plan(t, y.float(), 0.0, T).clone()
    assert torch.equal(plan.multi(t, torch.stack([y.float(), -y.float()]), 0.0, T)[0], F)
    D = nfft.AdjointNFFT(nf, R, m, torch.float64)(t, y.float().double(), 0.0, T)
    assert rel_l2(F.cpu().numpy(), D.cpu().numpy()) < 2e-6


@pytest.mark.parametrize("n,log_tile", [(0, 9), (1, 9), (5000, 9), (5000, 11)])
def test_scan_of_many_tiles(mods, n, log_tile):
    """8192 and 2048 tiles: one CTA's scan of the counts (above 4096 tiles) and
    the scatter pass's own, against the double plan (float rounding, 2e-6)."""
    from cunfft_adjoint_gb300 import _lib
    _, nfft = mods
    rng = np.random.default_rng(n)
    nf, T = 1 << 21, 2.0
    t = torch.as_tensor(rng.uniform(0, T, n), device="cuda")
    y = torch.as_tensor(rng.normal(0, 1, n), device="cuda")
    plan = nfft.AdjointNFFT(nf, 2, 8)
    plan.set_schedule(log_tile, _lib.GRID_GATHER)
    F = plan(t, y.float(), 0.0, T)
    if n == 0:
        assert not F.abs().any()
        return
    D = nfft.AdjointNFFT(nf, 2, 8, torch.float64)(t, y.float().double(), 0.0, T)
    assert rel_l2(F.cpu().numpy(), D.cpu().numpy()) < 2e-6


@pytest.mark.parametrize("kind", ["uniform", "runs", "burst"])
@pytest.mark.parametrize("n,nf,R,m", [(0, 1 << 12, 2, 8), (1, 1 << 12, 2, 1), (9, 1 << 13, 2, 16), (3001, 1 << 12, 4, 12),
                                      (4097, 1 << 12, 8, 8), (9999, 1 << 14, 4, 5), (16384, 1 << 16, 2, 8),
                                      (16384, 1 << 12, 2, 8), (16385, 1 << 14, 2, 8), (2049, 16, 4, 8), (2049, 1 << 11, 2, 16),
                                      (16384, 1 << 9, 2, 3), (9000, 1 << 8, 8, 8), (8192, 1 << 14, 4, 8),
                                      (8193, 1 << 14, 4, 8)])
def test_short_series_in_one_cluster(mods, kind, n, nf, R, m):
    """The whole short transform in one cluster launch, the grid's FFT spread
    over its CTAs or, where it is small, in one (and one sample more, which
    takes the tiled path): samples uniform, at the edges of the eight
    CTAs' runs of cells and the period's seam, and all inside one run, whose
    list then overflows for n > 4096 (grids of fewer than 16 cells per run: the
    single-CTA path).  Against the double plan of the same
    filter, one and three channels, and against the tiled path, which a chosen
    schedule takes.  Tolerances: float rounding with 2^-22 per weight, 2e-6; a
    burst adds up to n random terms per cell in sequence, eps sqrt(n), 2e-5."""
    from cunfft_adjoint_gb300 import _lib
    _, nfft = mods
    rng = np.random.default_rng(n + m)
    T, ng = 5.0, R * nf
    if kind == "uniform":
        pos = rng.uniform(0, ng, n)
    elif kind == "runs":
        pos = (ng // 8 * rng.integers(0, 8, n) + rng.uniform(-m - 1, m + 1, n)) % ng
    else:
        pos = 3 * ng // 8 + rng.uniform(0, 60, n)
    tol = 2e-6 if kind == "uniform" else 2e-5
    t = torch.as_tensor(pos / ng * T, device="cuda")
    Y = torch.as_tensor(rng.normal(0, 1, (3, n)), device="cuda").float()
    plan = nfft.AdjointNFFT(nf, R, m)
    F = plan(t, Y[0].contiguous(), 0.0, T).clone()
    if n == 0:
        assert not F.abs().any()
        return
    M = plan.multi(t, Y, 0.0, T).clone()
    plan.set_schedule(min(11, ng.bit_length() - 1), _lib.GRID_GATHER)
    G = plan(t, Y[0].contiguous(), 0.0, T)
    ref = nfft.AdjointNFFT(nf, R, m, torch.float64)
    for c in range(3):
        D = ref(t, Y[c].double(), 0.0, T).cpu().numpy()
        assert rel_l2(M[c].cpu().numpy(), D) < tol
        if c == 0:
            assert rel_l2(F.cpu().numpy(), D) < tol
            assert rel_l2(G.cpu().numpy(), D) < tol


@pytest.mark.parametrize("m", [2, 8])
@pytest.mark.parametrize("n,dense", [(1, False), (20_000, False), (20_000, True)])
@pytest.mark.parametrize("chan", [2, 4, 5, 9, 33])
def test_channels_in_groups(mods, chan, n, dense, m):
    """Channels gridded four at a time, their values fetched a group ahead
    (tiles of at most 1024 records) or per chunk of records (one dense tile):
    full and partial groups, one and several per CTA, with and without tap
    masks, against the double plan (float rounding, 2e-6; a dense tile adds up
    to some 40 terms per cell, 4e-6)."""
    _, nfft = mods
    rng = np.random.default_rng(chan)
    nf, T = 1 << 17, 2.0
    pos = rng.uniform(0, 1, n)
    if dense:
        pos[: n // 2] = 0.4 + pos[: n // 2] * 0.004
    t = torch.as_tensor(pos * T, device="cuda")
    Y = torch.as_tensor(rng.normal(0, 1, (chan, n)), device="cuda").float()
    M = nfft.AdjointNFFT(nf, 2, m).multi(t, Y, 0.0, T)
    ref = nfft.AdjointNFFT(nf, 2, m, torch.float64)
    for c in {0, 1, chan // 2, chan - 1}:
        D = ref(t, Y[c].double(), 0.0, T)
        assert rel_l2(M[c].cpu().numpy(), D.cpu().numpy()) < (4e-6 if dense else 2e-6)


@pytest.mark.parametrize("e", [-86, -60, 60, 100])
@pytest.mark.parametrize("n,nf,R,dense", [(300, 1 << 14, 2, False), (20_000, 1 << 17, 2, False), (60_000, 1 << 20, 4, False),
                                          (20_000, 1 << 17, 2, True), (60_000, 1 << 20, 4, True)])
def test_double_scales(mods, e, n, nf, R, dense):
    """Double transforms do not depend on the scale of their values: F(2^e y) /
    2^e against F(y), single, two channels and bootstrap; tiles of 1024 and of
    256 threads, split sums and (dense: 5000 samples in one cell) 64-bit ones.
    A power of two changes no rounding until a float-float pair's low part
    falls below the float range: 2^-150 per operation, 2^-64 of values near
    2^-86; its random sum over 2^22 cells and some 220 operations each,
    deconvolved (7), is 1e-14 of one value, of spectra of sqrt(n) values 1e-15.
    Bound: 1e-14."""
    _, nfft = mods
    rng = np.random.default_rng(n)
    T, s = 3.0, 2.0 ** e
    pos = rng.uniform(0, 1, n)
    if dense:
        pos[:5000] = (12345.0 + rng.uniform(0.1, 0.9, 5000)) / (R * nf)
    t = torch.as_tensor(pos * T, device="cuda")
    Y = torch.as_tensor(rng.normal(0, 1, (2, n)), device="cuda")
    plan = nfft.AdjointNFFT(nf, R, 12, torch.float64)
    for call in (lambda v: plan(t, v[0].contiguous(), 0.0, T), lambda v: plan.multi(t, v, 0.0, T),
                 lambda v: plan.bootstrap(t, v[0].contiguous(), 2, 5, 0.0, T)):
        F, G = call(Y).clone(), call(Y * s) / s
        assert float((G - F).abs().square().sum().sqrt() / F.abs().square().sum().sqrt()) < 1e-14


@pytest.mark.parametrize("e", [-86, -60, 60, 100])
def test_double_lomb_scargle_scales(mods, e):
    """The double periodogram of 2^e y is that of y: as above, but the weighted
    values are 1 / n of the data, 2^-50 per operation at 2^-86 and n = 20000
    (5000 frequencies, 2^16 cells): 2e-13.  Bound: 1e-12."""
    from cunfft_adjoint_gb300.lombscargle import lomb_scargle
    rng = np.random.default_rng(7)
    n = 20_000
    t = torch.as_tensor(np.sort(rng.uniform(0, 100.0, n)), device="cuda")
    y = torch.as_tensor(np.sin(2 * np.pi * t.cpu().numpy() / 2.1) + rng.normal(0, 1, n), device="cuda")
    dy = torch.as_tensor(rng.uniform(0.2, 0.6, n), device="cuda")
    P, Q = (lomb_scargle(t, v, dy, nfreq=5000, df=1 / 500.0, t0=0.0, R=4, m=12) for v in (y, y * 2.0 ** e))
    assert rel_l2(Q.cpu().numpy(), P.cpu().numpy()) < 1e-12


def _direct(t, y, T, nf):
    """F_k, k = -nf/2 .. nf/2 - 1, of one series by 64-bit sums."""
    x = t / T - 0.5
    k = torch.arange(-(nf // 2), nf // 2, device="cuda", dtype=torch.float64)
    ph = k[:, None] * x[None, :]
    return (y.double() * torch.exp(2j * np.pi * (ph - ph.round()))).sum(dim=1)


@pytest.mark.parametrize("n,nf,R,m,bound", [(1000, 2048, 2, 8, 2.13e-7), (500, 512, 2, 8, 2.11e-7), (700, 1024, 4, 6, 1.43e-7),
                                            (300, 2048, 4, 12, 1.38e-7), (2000, 1024, 4, 12, 1.39e-7),
                                            (3001, 4096, 2, 8, 2.24e-7)])
def test_short_float_error(mods, n, nf, R, m, bound):
    """Mean relative error of short float transforms against 64-bit sums over
    16 uniform series: one CTA or one cluster each, in a batch of 16 (an SM
    each) and of 160 (SMs shared; R = 4: gathered and scattered).  Bounds: the
    mean of 32 series by the scatter with running products and full twiddle
    tables, and two standard errors of this mean (2.5 %)."""
    _, nfft = mods
    T, B, S = 5.0, 160, 16
    plan = nfft.AdjointNFFT(nf, R, m)
    rng = np.random.default_rng(n)
    ts = [torch.as_tensor(np.sort(rng.uniform(0, T, n)), device="cuda") for _ in range(S)]
    ys = [torch.as_tensor(rng.normal(0, 1, n), device="cuda").float() for _ in range(S)]
    X = [_direct(t, y, T, nf) for t, y in zip(ts, ys)]

    def error(F):
        return np.mean([float((f.to(torch.complex128) - x).abs().square().sum().sqrt() / x.abs().square().sum().sqrt())
                        for f, x in zip(F, X)])

    def batch(B):
        p = nfft.BatchAdjointNFFT(np.full(B, n), np.full(B, nf), R, m, np.zeros(B), np.full(B, T))
        return p(torch.cat(ts * (B // S)), torch.cat(ys * (B // S))).view(B, nf)[:S]
    for F in ([plan(t, y, 0.0, T) for t, y in zip(ts, ys)], batch(S), batch(B)):
        assert error(F) < 1.025 * bound


def test_short_float_burst_error(mods):
    """10000 samples in 60 of 2^15 cells, a thousand and more terms per cell:
    mean error of 16 series against 64-bit sums.  Bound: the tiled gather's, which
    adds up chunks of at most 1024 records, 4.9e-7 (standard deviation of one
    series 1.2e-7; one sum per cell gives 8e-7)."""
    _, nfft = mods
    n, nf, T = 10_000, 1 << 14, 5.0
    plan = nfft.AdjointNFFT(nf, 2, 8)
    e = []
    for seed in range(16):
        rng = np.random.default_rng(seed)
        t = torch.as_tensor((0.375 + rng.uniform(0, 60, n) / (2 * nf)) * T, device="cuda")
        y = torch.as_tensor(rng.normal(0, 1, n), device="cuda").float()
        X = _direct(t, y, T, nf)
        F = plan(t, y, 0.0, T).to(torch.complex128)
        e.append(float((F - X).abs().square().sum().sqrt() / X.abs().square().sum().sqrt()))
    assert np.mean(e) < 4.9e-7


@pytest.mark.parametrize("dt", [np.float32, np.float64])
@pytest.mark.parametrize("n", [2047, 2048, 2049])
def test_compat_filter_at_half_the_samples(mods, oracle_lib, dt, n):
    """Filter coefficients around ng = n / 2, where the reference's b changes sign
    through infinity: E1 and E2 as the reference's expressions give them (NaN
    for a negative b, 0 and 1 for an infinite one).  Tolerances of the filter's
    parity test: 3e-5 and 1e-14."""
    cuna, _ = mods
    x = np.random.default_rng(n).uniform(-0.5, 0.5, n).astype(dt)
    fp = cuna.generate_filter_properties(torch.as_tensor(x, device="cuda"), n, 1024)
    _, _, _, E1, E2, _ = oracle_lib.compat_filter(x, 1024, "f" if dt == np.float32 else "d")
    for got, want in ((fp.E1, E1), (fp.E2, E2)):
        np.testing.assert_allclose(got[:n].cpu().numpy(), want, rtol=3e-5 if dt == np.float32 else 1e-14)


def _stages(plan, t, y, T):
    import ctypes
    from cunfft_adjoint_gb300 import _lib
    F = torch.empty(plan.nf, dtype=torch.complex64, device="cuda")
    ms, names, k = (ctypes.c_float * 16)(), (ctypes.c_char_p * 16)(), ctypes.c_int()
    _lib.check(_lib.core().cuna2_plan_profile(plan._h, t.data_ptr(), y.data_ptr(), F.data_ptr(), t.numel(), 0.0, T, None,
                                              ms, names, 16, ctypes.byref(k)))
    return [names[i].decode() for i in range(k.value)]


def test_autotune_leaves_short_series_their_path(mods):
    """The one-launch path runs by the number of samples: tuning on a long series
    chooses among the others and leaves short ones on it, also after a chosen
    schedule or the local sort had turned it off; spectra of both against the
    double plan (float rounding, 2e-6)."""
    from cunfft_adjoint_gb300 import _lib
    _, nfft = mods
    rng = np.random.default_rng(3)
    nf, T = 1 << 14, 5.0
    (ts, ys), (tl, yl) = (((torch.as_tensor(rng.uniform(0, T, n), device="cuda"),
                            torch.as_tensor(rng.normal(0, 1, n), device="cuda").float())) for n in (9000, 40_000))
    plan, ref = nfft.AdjointNFFT(nf, 2, 8), nfft.AdjointNFFT(nf, 2, 8, torch.float64)

    def check(cluster):
        assert ("nfft_cluster" in _stages(plan, ts, ys, T)) == cluster
        assert "nfft_cluster" not in _stages(plan, tl, yl, T)
        for t, y in ((ts, ys), (tl, yl)):
            assert rel_l2(plan(t, y, 0.0, T).cpu().numpy(), ref(t, y.double(), 0.0, T).cpu().numpy()) < 2e-6
    check(True)
    plan.autotune(tl, yl, 0.0, T, reps=2)
    check(True)
    plan.set_schedule(11, _lib.GRID_GATHER)
    check(False)
    plan.autotune(tl, yl, 0.0, T, reps=2)
    check(True)
    plan.binning = 1
    check(False)
    plan.binning = 0
    check(True)


_MASKS_SCRIPT = """
import sys
import numpy as np, torch
sys.path.insert(0, sys.argv[1])
from cunfft_adjoint_gb300 import nfft
t = torch.tensor([1.2345], dtype=torch.float64, device="cuda")
y = torch.ones(1, device="cuda")
out = {}
for nf, m in ((2048, 8), (2048, 5), (1 << 14, 8)):
    out["plan_%d_%d" % (nf, m)] = nfft.AdjointNFFT(nf, 2, m)(t, y, 0.0, 3.0).cpu().numpy()
b = nfft.BatchAdjointNFFT(np.ones(2, int), np.full(2, 2048), 2, 8, np.zeros(2), np.full(2, 3.0))
out["batch_2048_8"] = b(t.repeat(2), y.repeat(2)).cpu().numpy()
np.savez(sys.argv[2], **out)
"""


def test_masks_switch_reaches_every_gather(tmp_path, native_built):
    """CUNA2_GATHER_MASKS=1 keeps the tap masks in the one-CTA, cluster and batch
    gathers too: one sample's spectrum (no order of sums) differs in some bits
    from that of whole cell groups, whose cells beyond the window hold below 1e-8
    of the peak (m = 8), and by no more than float rounding; m = 5 keeps the
    masks either way."""
    import os
    import subprocess
    import sys
    root = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))
    script = tmp_path / "masks.py"
    script.write_text(_MASKS_SCRIPT)
    res = []
    for v in "01":
        out = tmp_path / ("masks%s.npz" % v)
        r = subprocess.run([sys.executable, str(script), root, str(out)], env={**os.environ, "CUNA2_GATHER_MASKS": v},
                           capture_output=True, text=True, timeout=600)
        assert r.returncode == 0, r.stderr[-2000:]
        res.append(np.load(out))
    for key in res[0].files:
        assert rel_l2(res[0][key], res[1][key]) < 1e-6, key
        assert np.array_equal(res[0][key], res[1][key]) == key.endswith("_5"), key


@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
@pytest.mark.parametrize("dtype,n,nf,R,m", [(torch.float32, 300, 512, 2, 8), (torch.float32, 500, 1024, 4, 6),
                                            (torch.float32, 2000, 2048, 2, 8), (torch.float32, 9000, 1 << 14, 2, 8),
                                            (torch.float32, 20_000, 1 << 17, 2, 8), (torch.float64, 800, 1 << 11, 2, 10),
                                            (torch.float64, 9000, 1 << 15, 2, 10)])
def test_non_finite_values(mods, bad, dtype, n, nf, R, m):
    """A non-finite value spreads over the spectrum of its own series and no
    other's: one transform (one CTA, one cluster, tiled), the other channel, the
    other series of a batch (an SM each and shared); its gradients stay with
    the sample or the series it belongs to, the others keep their bits or, where
    the order of sums is free, float rounding."""
    _, nfft = mods
    rng = np.random.default_rng(n)
    T, B = 5.0, 3
    t = torch.as_tensor(rng.uniform(0, T, (B, n)), device="cuda")
    y = torch.as_tensor(rng.normal(0, 1, (B, n)), device="cuda").to(dtype)
    w = y.clone()
    w[1, n // 2] = bad
    plan = nfft.AdjointNFFT(nf, R, m, dtype)

    def lost(F):
        return bool((~torch.isfinite(torch.view_as_real(F)).all(dim=-1)).all())

    def near(a, b):
        return rel_l2(a.cpu().numpy(), b.cpu().numpy()) < (1e-6 if dtype == torch.float32 else 1e-13)
    assert lost(plan(t[1], w[1], 0.0, T))
    F, M = plan(t[1], y[2], 0.0, T).clone(), plan.multi(t[1], w[1:], 0.0, T)
    assert lost(M[0]) and near(M[1], F)
    for reps in (1, 60):
        batch = nfft.BatchAdjointNFFT(np.full(B * reps, n), np.full(B * reps, nf), R, m, np.zeros(B * reps),
                                      np.full(B * reps, T), dtype)
        G, H = (batch(t.repeat(reps, 1), v.repeat(reps, 1)).view(-1, nf) for v in (y, w))
        assert lost(H[1]) and near(H[0], G[0]) and near(H[2], G[2])
    g = torch.as_tensor(rng.normal(0, 1, (B, nf)) + 1j * rng.normal(0, 1, (B, nf)), device="cuda").to(plan.cdtype)
    gy, gt = plan.backward_batch(t, y, g, 0.0, T)
    hy, ht = plan.backward_batch(t, w, g, 0.0, T)
    assert torch.equal(gy, hy) and not torch.isfinite(ht[1, n // 2])
    ok = torch.isfinite(ht)
    assert int((~ok).sum()) == 1 and torch.equal(ht[ok], gt[ok])
    g[1, 3] = bad
    hy, ht = plan.backward_batch(t, y, g, 0.0, T)
    assert not torch.isfinite(hy[1]).any() and not torch.isfinite(ht[1]).any()
    assert torch.equal(hy[::2], gy[::2]) and torch.equal(ht[::2], gt[::2])
