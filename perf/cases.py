"""The work that a user of the engine has it do, as cases that can be timed.

`listed()` names twelve of them, `draw()` gives more of the same ranges,
`prepare()` builds what a sampler has in hand before the call (bank, plan,
device tensors), `run()` makes one pass through `glass_gb300.Engine`, and
`exact()` states what the pass should return, in FP64, in plain torch and
numpy and without the engine.

Kinds of case:

* ``dlogl``: delta log-likelihood of a batch of proposals around tempered
  chains, on segments of NFFT bins around one injected source each;
* ``global_fit``: the same on the wide segments of a Galactic population
  (several sources per segment, frequencies from 0.1 mHz up, updates and
  births, template sizes up to 4096);
* ``grad_fisher``: gradient and Fisher matrix of a batch of proposals;
* ``wdm``: the WDM wavelet transform, time series to coefficients or back;
* ``wavelet``: wavelet-domain waveform and sparse-pixel likelihood;
* ``fstat``: F-statistic of a patch of the proposal grid;
* ``noise``: noise-model likelihood, XYZ frequency bins;
* ``noise_wavelet``: the same on coarse-grained wavelet cells.

Sizes are those of the repository's benchmark, tests and reference
configurations.  Every array is made from the seed alone.
"""
import math

import numpy as np
import torch

import glass_gb300 as gg
from glass_gb300 import workloads as wl

T = wl.T_YEAR
PI2 = wl.PI2
CLIGHT, LARM, FSTAR = wl.CLIGHT, wl.LARM, wl.FSTAR
YEAR = 3.15581497632e7
AU = 1.49597870700e11
SQ3 = 1.73205080757
VEARTH = 0.00010103671
DT = 15.0  # sampling cadence of the time series, s

_DEV = torch.device("cuda" if torch.cuda.is_available() else "cpu")
_PREC = {"fp64": gg.PREC_FP64, "mixed": gg.PREC_MIXED}


# --------------------------------------------------------------- the cases
def listed():
    return [
        # one chain evaluating one proposal at a time through host arrays: the
        # reference's own calling pattern, all latency
        dict(name="one_proposal_fp64", kind="dlogl", nseg=1, NFFT=1024, n=1, precision="fp64", entry="host"),
        # one short parallel-tempering ladder on one segment: the batch a
        # single analysis segment has per step, odd in number
        dict(name="ladder_mixed_host", kind="dlogl", nseg=1, NFFT=512, n=21, precision="mixed", entry="host"),
        # the sampler's step at full load: 64 segments, 256 chains x 12
        # temperatures, default (mixed, 1e-3) precision, data on the device
        dict(name="tempered_mixed", kind="dlogl", nseg=64, NFFT=1024, n=3072, precision="mixed", entry="device"),
        # the same step in plain FP64, the parity mode
        dict(name="tempered_fp64", kind="dlogl", nseg=64, NFFT=1024, n=3072, precision="fp64", entry="device"),
        # one move per source of a Galactic population on wide segments
        dict(name="global_fit_mixed", kind="global_fit", nseg=128, NFFT=8192, n=2500, precision="mixed"),
        # Fisher matrices of a batch of chains, for the Fisher-jump proposal
        dict(name="grad_fisher", kind="grad_fisher", nseg=64, NFFT=1024, n=4096, mode=0),
        # a year of 15 s samples to the 1024 x 2048 wavelet grid
        dict(name="wdm_forward", kind="wdm", NF=1024, NT=2048, nx=4.0, direction="forward", precision="fp64"),
        # coefficients of the reference's default grid (1536 x 4096) back to time
        dict(name="wdm_inverse", kind="wdm", NF=1536, NT=4096, nx=6.0, direction="inverse", precision="fp64"),
        # wavelet-domain likelihood of a batch of sources, default precision
        dict(name="wavelet_fp64", kind="wavelet", n=4096, precision="fp64"),
        # a slab of the F-statistic proposal's frequency x sky grid
        dict(name="fstat_grid", kind="fstat", NFFT=1024, f0=3.2e-3, n_f=128, n_theta=20, n_phi=20),
        # the noise sampler's batch, instrument and foreground, 0.1 mHz up
        dict(name="noise_xyz", kind="noise", qmin=3145, N=15360, n=1024, foreground=True),
        # the same in the wavelet domain, foreground modulated over the year
        dict(name="noise_wavelet", kind="noise_wavelet", lmin=10, layers=460, Q=16, n=1024, mode=2),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(["dlogl", "dlogl", "global_fit", "grad_fisher", "wdm", "wavelet", "fstat", "noise",
                       "noise_wavelet"])
    if kind == "dlogl":
        return dict(kind=kind, nseg=_log_int(rng, 1, 64), NFFT=rng.choice([256, 512, 1024, 2048]),
                    n=_log_int(rng, 1, 3072), precision=rng.choice(["fp64", "mixed", "mixed"]),
                    entry=rng.choice(["device", "host"]))
    if kind == "global_fit":
        return dict(kind=kind, nseg=_log_int(rng, 16, 128), NFFT=rng.choice([4096, 8192]),
                    n=_log_int(rng, 100, 2500), precision=rng.choice(["mixed", "mixed", "fp64"]))
    if kind == "grad_fisher":
        return dict(kind=kind, nseg=_log_int(rng, 1, 64), NFFT=rng.choice([512, 1024, 2048]),
                    n=_log_int(rng, 16, 4096), mode=rng.choice([0, 1]))
    if kind == "wdm":
        # NT of the form 2^a 3^b up to 4096; NF likewise, up to the default grid's product
        NT = rng.choice([256, 384, 512, 768, 1024, 1536, 2048, 4096])
        NF = rng.choice([64, 96, 128, 256, 512, 768, 1024, 1536])
        return dict(kind=kind, NF=NF, NT=NT, nx=rng.choice([4.0, 6.0]), direction=rng.choice(["forward", "inverse"]),
                    precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "wavelet":
        return dict(kind=kind, n=_log_int(rng, 16, 4096), precision=rng.choice(["fp64", "fp64", "mixed"]))
    if kind == "fstat":
        return dict(kind=kind, NFFT=rng.choice([512, 1024]), f0=math.exp(rng.uniform(math.log(0.8e-3), math.log(8e-3))),
                    n_f=_log_int(rng, 2, 64), n_theta=rng.choice([10, 15, 20]), n_phi=rng.choice([10, 20]))
    if kind == "noise":
        return dict(kind=kind, qmin=_log_int(rng, 3145, 100000), N=_log_int(rng, 500, 15360), n=_log_int(rng, 1, 1024),
                    foreground=rng.random() < 0.7)
    return dict(kind=kind, lmin=rng.randint(3, 60), layers=_log_int(rng, 20, 400), Q=rng.choice([8, 16, 32, 64]),
                n=_log_int(rng, 1, 512), mode=rng.choice([0, 1, 2, 2]))


# ------------------------------------------- Fourier-domain template (torch)
def _floor_pow2_above(v):
    """2^((int)log2(v) + 1) for v > 1; smaller values end at the caller's minimum."""
    return 2.0 ** (np.floor(np.log2(np.maximum(v, 1.0))) + 1)


def _aenoise(f):
    """The A/E noise of the bandwidth rule's analytic SNR (utils/src/glass_lisa.c:1188-1198)."""
    x = f / FSTAR
    red = 1.0 + 16.0 * ((2.0e-5 / f) ** 10 + (1.0e-4 / f) ** 2)
    return ((16.0 / 3.0) * np.sin(x) ** 2 * ((2.0 + np.cos(x)) * (8.321e-23 + 2.89e-24)
            + 2.0 * (3.0 + 2.0 * np.cos(x) + np.cos(2.0 * x)) * (2.89e-24 / 2.0 + 9.0e-30 / (PI2 * f) ** 4 * red))
            / (2.0 * LARM) ** 2)


def _half_bandwidth(f, fdot, costh, amp, NFFT):
    """ucb_bandwidth (ucb/src/glass_ucb_waveform.c:698-725); templates hold twice this."""
    nmax = 2 ** int(math.log2(NFFT // 2))
    bw = 2 * T * ((4.0 + PI2 * f * (AU / CLIGHT) * np.sin(np.arccos(costh))) / YEAR + np.abs(fdot) * T)
    ds = np.clip(_floor_pow2_above(bw - 1), 16, nmax)
    ss = np.clip(_floor_pow2_above(amp * math.sqrt(T) * np.sin(f / FSTAR) / np.sqrt(_aenoise(f)) - 1), 16, nmax)
    return np.maximum(ds, ss).astype(np.int64)


def _sizes(p, NFFT):
    return 2 * _half_bandwidth(p[:, 0] / T, p[:, 7] / T / T, p[:, 1], np.exp(p[:, 3]), NFFT)


def _positions(t):
    """Analytic spacecraft positions [..., 3 spacecraft, 3] (utils/src/glass_lisa.c:77-124)."""
    ecc = LARM / (2.0 * SQ3 * AU)
    R = AU * ecc
    al = PI2 * t / YEAR
    sa, ca = torch.sin(al), torch.cos(al)
    rows = []
    for sb, cb in ((0.0, 1.0), (0.866025403784439, -0.5), (-0.866025403784438, -0.5)):
        rows.append(torch.stack([AU * ca + R * (sa * ca * sb - (1.0 + sa * sa) * cb),
                                 AU * sa + R * (sa * ca * cb - (1.0 + ca * ca) * sb),
                                 -SQ3 * R * (ca * cb + sa * sb)], -1))
    return torch.stack(rows, -2)


def _sky(costh, phi):
    """Polarisation tensors e+, ex [n, 3, 3] and the propagation vector k [n, 3]."""
    sth, cp, sp = torch.sqrt(1.0 - costh * costh), torch.cos(phi), torch.sin(phi)
    u = torch.stack([costh * cp, costh * sp, -sth], -1)
    v = torch.stack([sp, -cp, torch.zeros_like(sp)], -1)
    k = torch.stack([-sth * cp, -sth * sp, -costh], -1)
    ep = v[:, :, None] * v[:, None, :] - u[:, :, None] * u[:, None, :]
    ec = u[:, :, None] * v[:, None, :] + v[:, :, None] * u[:, None, :]
    return ep, ec, k


def _templates(p, N):
    """ucb_waveform's A and E templates of N bins [n, N] complex, and the
    carrier bins q [n] (ucb/src/glass_ucb_waveform.c:738-1001 and the
    fractional-frequency TDI of utils/src/glass_lisa.c:645-710)."""
    f0, costh, phi, cosi = p[:, 0] / T, p[:, 1], p[:, 2], p[:, 4]
    amp, psi, phi0, fdot = torch.exp(p[:, 3]), p[:, 5], p[:, 6], p[:, 7] / (T * T)
    q = torch.floor((f0 * T).detach())
    ap, ac = amp * (1.0 + cosi * cosi) * 0.5, -amp * cosi
    c2p, s2p = torch.cos(2.0 * psi), torch.sin(2.0 * psi)
    dpr, dpi, dcr, dci = ap * c2p, -ac * s2p, -ap * s2p, -ac * c2p
    ep, ec, k = _sky(costh, phi)
    t = T * torch.arange(N, dtype=torch.float64, device=p.device) / N
    x = _positions(t)
    col = lambda v: v[:, None]  # noqa: E731
    arms, dp, dc, kr = ((0, 1), (0, 2), (1, 2)), {}, {}, {}
    for i, j in arms:
        r = (x[:, j] - x[:, i]) / LARM
        dp[i, j] = dp[j, i] = torch.einsum("ta,tb,nab->nt", r, r, ep)
        dc[i, j] = dc[j, i] = torch.einsum("ta,tb,nab->nt", r, r, ec)
        kr[i, j] = torch.einsum("ta,na->nt", r, k)
        kr[j, i] = -kr[i, j]
    df = PI2 * (q / T)
    d = {}
    for i in range(3):
        kdotx = (x[:, i, 0] * k[:, :1] + x[:, i, 1] * k[:, 1:2] + x[:, i, 2] * k[:, 2:]) / CLIGHT
        xi = t - kdotx
        fonfs = (col(f0) + col(fdot) * xi) / FSTAR
        arg2 = col(PI2 * f0) * xi - col(phi0) - col(df) * t + math.pi * col(fdot) * xi * xi
        aevol = 1.0 + 0.66666666666666666666 * col(fdot / f0) * xi
        for j in range(3):
            if i != j:
                arg1 = 0.5 * fonfs * (1.0 + kr[i, j])
                s = 0.25 * torch.sin(arg1) / arg1 * aevol
                a = dp[i, j] * col(dpr) + dc[i, j] * col(dcr)
                b = dp[i, j] * col(dpi) + dc[i, j] * col(dci)
                c, e = torch.cos(arg1 - arg2), torch.sin(arg1 - arg2)
                z = torch.complex(s * (a * c + b * e), s * (b * c - a * e))
                d[i, j] = torch.fft.fftshift(torch.fft.fft(z, dim=-1), dim=-1) / (2.0 * N)
    f = (col(q) + torch.arange(N, dtype=torch.float64, device=p.device) - N // 2) / T
    w = f / FSTAR
    e1, e2 = torch.polar(torch.ones_like(w), -w), torch.polar(torch.ones_like(w), -2.0 * w)
    pref = f * (4.0 / FSTAR * math.sqrt(T)) * torch.sin(w)
    X, Y, Z = (pref * ((d[i, j] - d[i, k_]) * e2 + (d[j, i] - d[k_, i]) * e1)
               for i, j, k_ in ((0, 1, 2), (1, 2, 0), (2, 0, 1)))
    return (Z - X) * math.sqrt(0.5), (X - 2 * Y + Z) * 0.408248290463863, q


def _by_size(N, budget=1 << 19):
    """Index sets of equal template size, of at most `budget` samples each."""
    for size in np.unique(N):
        idx = np.nonzero(N == size)[0]
        step = max(1, budget // int(size))
        for a in range(0, len(idx), step):
            yield int(size), idx[a:a + step]


def _dev(a):
    return torch.from_numpy(np.ascontiguousarray(a)).to(_DEV)


def _bins(bank, seg, q, N):
    """Segment bins under each template: index, mask, whitening weights, residuals."""
    j = q.long()[:, None] - N // 2 - bank["qmin"][seg][:, None] + torch.arange(N, device=q.device)
    ok = (j >= 0) & (j < bank["NFFT"])
    j = j.clamp(0, bank["NFFT"] - 1) + (seg * bank["NFFT"])[:, None]
    wA, wE = bank["invCA"].reshape(-1)[j] * ok, bank["invCE"].reshape(-1)[j] * ok
    return j, wA, wE, bank["dA"].reshape(-1)[j], bank["dE"].reshape(-1)[j]


def _abs2(z):
    return z.real * z.real + z.imag * z.imag


def _terms(bank, seg, p):
    """(term, (h|h)) of each proposal in FP64: the residual form of the delta log-likelihood."""
    term, hh = np.empty(len(p)), np.empty(len(p))
    dbank = {k: _dev(v) if isinstance(v, np.ndarray) else v for k, v in bank.items()}
    for N, idx in _by_size(_sizes(p, bank["NFFT"])):
        A, E, q = _templates(_dev(p[idx]), N)
        _, wA, wE, rA, rE = _bins(dbank, _dev(seg[idx]).long(), q, N)
        s = (_abs2(rA - A) - _abs2(rA)) * wA + (_abs2(rE - E) - _abs2(rE)) * wE
        term[idx] = -s.sum(-1).cpu().numpy()
        hh[idx] = 2.0 * (_abs2(A) * wA + _abs2(E) * wE).sum(-1).cpu().numpy()
    return term, hh


def _make_bank(rng, nseg, NFFT, qmin, src, seg):
    """Segments of A/E noise (scirdv1) from bin qmin with every source injected."""
    f = (qmin[:, None] + np.arange(NFFT)) / T
    C = wl.aenoise_ff(f)
    sig = np.sqrt(C / 2.0)
    dA, dE = (sig * (rng.standard_normal((nseg, NFFT)) + 1j * rng.standard_normal((nseg, NFFT))) for _ in "AE")
    for N, idx in _by_size(_sizes(src, NFFT)):
        A, E, q = _templates(_dev(src[idx]), N)
        A, E, q = A.cpu().numpy(), E.cpu().numpy(), q.cpu().numpy().astype(np.int64)
        for r, i in enumerate(idx):
            i0 = q[r] - N // 2 - qmin[seg[i]]
            lo, hi = max(0, i0), min(NFFT, i0 + N)
            if hi > lo:
                dA[seg[i], lo:hi] += A[r, lo - i0:hi - i0]
                dE[seg[i], lo:hi] += E[r, lo - i0:hi - i0]
    return dict(NFFT=NFFT, qmin=qmin.astype(np.int64), dA=dA, dE=dE, invCA=1.0 / C, invCE=1.0 / C)


def _engine_bank(bank):
    return wl.SegmentBank(T=T, NFFT=bank["NFFT"], qmin=bank["qmin"].astype(np.int32), dA=bank["dA"], dE=bank["dE"],
                          invCA=bank["invCA"], invCE=bank["invCE"])


def _tempered_sources(case, rng):
    """One source per segment (f0 0.5-15 mHz, amplitude 1e-23 - 1e-21, both
    log-uniform), and the segment and temperature of each proposal's chain."""
    src = np.array([wl.draw_source(rng, 10 ** rng.uniform(math.log10(0.5e-3), math.log10(15e-3)),
                                   10 ** rng.uniform(-23.0, -21.0)) for _ in range(case["nseg"])])
    item = np.arange(case["n"])
    return src, (item // 12 % case["nseg"]).astype(np.int32), 1.5 ** (item % 12)


def _jumped(rng, x, snr, temp):
    """One Gaussian jump from each state, of about a Fisher sigma widened by sqrt(temperature)."""
    scale = np.array([wl.jump_scales(x[i], max(snr[i], 5.0)) for i in range(len(x))])
    jump = rng.standard_normal(x.shape) * scale * np.sqrt(temp)[:, None]
    y = x + jump
    for k in (1, 4):
        bad = np.abs(y[:, k]) >= 1.0
        y[bad, k] = x[bad, k] - jump[bad, k]
        bad = np.abs(y[:, k]) >= 1.0
        y[bad, k] = x[bad, k]
    return y


def _galactic_sources(case, rng):
    """A Galactic population: f0 log-uniform over 0.1-10 mHz, chirps and
    amplitudes from chirp masses 0.2-0.8 Msun at 1-15 kpc, each in the nearest
    of the segments (log-spaced centres).  Sources between the segments, and
    those whose template would exceed the engine's 4096 bins, are drawn again."""
    n, nseg, NFFT = case["n"], case["nseg"], case["NFFT"]
    centre = np.maximum(np.exp(np.linspace(math.log(1.3e-4), math.log(9.7e-3), nseg)), (NFFT // 2 + 16) / T)
    src, seg = np.empty((0, 8)), np.empty(0, np.int32)
    while len(src) < n:
        f = 10 ** rng.uniform(-4.0, -2.0, 2 * n)
        mc = rng.uniform(0.2, 0.8, 2 * n) * 4.925491025543576e-06
        dist = rng.uniform(1.0, 15.0, 2 * n) * 3.0856775814913673e19
        amp = 2.0 * mc ** (5.0 / 3.0) * (math.pi * f) ** (2.0 / 3.0) * CLIGHT / dist
        fdot = 96.0 / 5.0 * math.pi ** (8.0 / 3.0) * mc ** (5.0 / 3.0) * f ** (11.0 / 3.0)
        new = np.array([wl.draw_source(rng, f[i], amp[i], fdot[i]) for i in range(2 * n)])
        s = np.clip(np.searchsorted((centre[1:] + centre[:-1]) / 2, f), 0, nseg - 1).astype(np.int32)
        ok = (_sizes(new, NFFT) <= 4096) & (np.abs(f - centre[s]) * T < 0.48 * NFFT)
        src, seg = np.concatenate([src, new[ok]]), np.concatenate([seg, s[ok]])
    return src[:n], seg[:n], (centre * T).astype(np.int64) - NFFT // 2


def _fourier_inputs(case, seed):
    """Bank, segment of each proposal, parameters, and the cached term of each chain's state."""
    rng = np.random.default_rng(seed)
    if case["kind"] == "global_fit":
        src, seg, qmin = _galactic_sources(case, rng)
        bank = _make_bank(rng, case["nseg"], case["NFFT"], qmin, src, seg)
        tx, hh = _terms(bank, seg, src)
        p = _jumped(rng, src, np.sqrt(hh), 1.5 ** (np.arange(len(src)) % 16))
        birth = rng.random(len(src)) < 0.2  # a prior draw in the source's segment instead
        q = bank["qmin"][seg] + rng.uniform(0.1, 0.9, len(src)) * case["NFFT"]
        new = np.array([wl.draw_source(rng, f / T, 10 ** rng.uniform(-23, -21), 0.0) for f in q])
        ok = (_sizes(new, case["NFFT"]) <= 4096) & birth
        p[ok], tx[ok] = new[ok], 0.0
        big = _sizes(p, case["NFFT"]) > 4096
        p[big] = src[big]
        return dict(bank=bank, seg=seg, p=p, tx=tx)
    src, seg, temp = _tempered_sources(case, rng)
    qmin = src[:, 0].astype(np.int64) - case["NFFT"] // 2
    bank = _make_bank(rng, case["nseg"], case["NFFT"], qmin, src, np.arange(case["nseg"]))
    term, hh = _terms(bank, np.arange(case["nseg"], dtype=np.int32), src)
    return dict(bank=bank, seg=seg, p=_jumped(rng, src[seg], np.sqrt(hh)[seg], temp), tx=term[seg])


def _fourier_sizes(case):
    rng = np.random.default_rng(0)
    if case["kind"] == "global_fit":
        return _sizes(_galactic_sources(case, rng)[0], case["NFFT"])
    src, seg, _ = _tempered_sources(case, rng)
    return _sizes(src, case["NFFT"])[seg]


def _exact_grad(case, x):
    """Gradient of the term and Fisher matrix by forward-mode differentiation of the FP64 template."""
    import torch.autograd.forward_ad as fwd

    bank, seg, p = x["bank"], x["seg"], x["p"]
    n, NFFT = len(p), bank["NFFT"]
    dbank = {k: _dev(v) if isinstance(v, np.ndarray) else v for k, v in bank.items()}
    term, grad, F = np.empty(n), np.empty((n, 8)), np.empty((n, 8, 8))
    for N, idx in _by_size(_sizes(p, NFFT), 1 << 18):
        pt, st = _dev(p[idx]), _dev(seg[idx]).long()
        dA, dE = [], []
        for k in range(8):
            with fwd.dual_level():
                v = torch.zeros_like(pt)
                v[:, k] = 1.0
                A, E, q = _templates(fwd.make_dual(pt, v), N)
                (A, tA), (E, tE) = fwd.unpack_dual(A), fwd.unpack_dual(E)
                dA.append(tA), dE.append(tE)
        _, wA, wE, rA, rE = _bins(dbank, st, q, N)
        term[idx] = -((_abs2(rA - A) - _abs2(rA)) * wA + (_abs2(rE - E) - _abs2(rE)) * wE).sum(-1).cpu().numpy()
        dA, dE = torch.stack(dA, 1), torch.stack(dE, 1)  # [n, 8, N]
        grad[idx] = 2.0 * (((rA - A).conj()[:, None] * dA).real * wA[:, None]
                           + ((rE - E).conj()[:, None] * dE).real * wE[:, None]).sum(-1).cpu().numpy()
        if case["mode"] == 1:  # the reference's indexing: template bin i with the noise of segment bin i
            fA, fE = (dbank[c][st][:, :N] for c in ("invCA", "invCE"))
        else:
            fA, fE = wA, wE
        F[idx] = 2.0 * (torch.einsum("nki,nli,ni->nkl", dA.conj(), dA, fA.to(dA.dtype)).real
                        + torch.einsum("nki,nli,ni->nkl", dE.conj(), dE, fE.to(dE.dtype)).real).cpu().numpy()
    return term, grad, F


# ----------------------------------------------------------------- F-statistic
def _fstat_inputs(case, seed):
    """One segment holding one source (A = 3e-22) and the grid cells of n_f bins x the sky."""
    rng = np.random.default_rng(seed)
    src = wl.draw_source(rng, case["f0"], 3e-22)[None]
    qmin = src[:, 0].astype(np.int64) - case["NFFT"] // 2
    bank = _make_bank(rng, 1, case["NFFT"], qmin, src, np.zeros(1, np.int64))
    first = int(src[0, 0]) - case["n_f"] // 2
    i, j, k = np.meshgrid(np.arange(case["n_f"]), np.arange(case["n_theta"]), np.arange(case["n_phi"]), indexing="ij")
    costh = -1.0 + (j + 0.5) * 2.0 / case["n_theta"]
    cells = np.stack([(first + i + 0.5) / T, np.zeros(i.shape), np.arccos(costh),
                      (k + 0.5) * PI2 / case["n_phi"]], -1).reshape(-1, 4)
    return dict(bank=bank, cells=cells)


def _exact_fstat(case, x):
    """get_Fstat_logL of each cell (ucb/src/glass_ucb_fstatistic.c:231-697): four filters, their products, the fit."""
    bank = {k: _dev(v) if isinstance(v, np.ndarray) else v for k, v in x["bank"].items()}
    bank["invCE"] = bank["invCA"]  # both channels weighted with the A noise, as the reference does
    cells = x["cells"]
    out = np.empty((len(cells), 5))
    N_all = _half_bandwidth(cells[:, 0], cells[:, 1], np.cos(cells[:, 2]), 1e-22, case["NFFT"])
    for N, idx in _by_size(N_all):
        c = cells[idx]
        h = []
        for psi, phase in ((0.0, 0.0), (math.pi / 4, math.pi), (0.0, 1.5 * math.pi), (math.pi / 4, 0.5 * math.pi)):
            one = np.ones(len(c))
            p = np.stack([c[:, 0] * T, np.cos(c[:, 2]), c[:, 3], math.log(2.0) * one, math.cos(math.pi / 2) * one,
                          psi * one, phase * one, c[:, 1] * T * T], -1)
            h.append(_templates(_dev(p), N))
        q = h[0][2]
        j, w, _, dA, dE = _bins(bank, torch.zeros(len(c), dtype=torch.int64, device=_DEV), q, N)
        w = w * (j > 0)
        A, E = torch.stack([v[0] for v in h], 1), torch.stack([v[1] for v in h], 1)
        Nv = 4.0 * (((dA.conj()[:, None] * A).real + (dE.conj()[:, None] * E).real) * w[:, None]).sum(-1)
        wc = w.to(A.dtype)
        M = 4.0 * (torch.einsum("nfi,ngi,ni->nfg", A.conj(), A, wc) + torch.einsum("nfi,ngi,ni->nfg", E.conj(), E, wc)).real
        a = _dev(np.linalg.solve(M.cpu().numpy(), Nv[:, :, None].cpu().numpy())[:, :, 0])
        logl = 0.5 * (Nv * a).sum(-1)
        a1, a2, a3, a4 = a.unbind(-1)
        s1 = torch.sqrt((a1 + a4) ** 2 + (a2 - a3) ** 2)
        s2 = torch.sqrt((a1 - a4) ** 2 + (a2 + a3) ** 2)
        ap, ac = s1 + s2, s1 - s2
        psi = 0.5 * torch.atan2(ap * a4 - ac * a1, -(ac * a2 + ap * a3))
        sg = torch.sign(torch.sin(2.0 * psi))
        root = torch.sqrt(ap * ap - ac * ac)
        phase = torch.atan2(sg * (ap * a4 - ac * a1), -sg * (ac * a3 + ap * a2))
        out[idx] = torch.stack([logl, 0.5 * (ap + root), torch.acos(-ac / (ap + root)), psi, phase], -1).cpu().numpy()
    return out[:, 0], out[:, 1:]


# ------------------------------------------------------------------------ WDM
def _window(Nf, Nt, nx):
    """The Meyer window of the forward transform (utils/src/glass_wavelet.c:305-349), integer nx."""
    dom = math.pi / Nf
    x = np.arange(Nt // 2 + 1) / (Nt / 2)
    n, total, term = int(nx), np.zeros_like(x), np.ones_like(x)
    for k in range(n):  # the incomplete beta function's terminating series
        total = total + term / (n + k)
        term = term * x * (k + 1 - n) / (k + 1)
    beta = x ** n * total * math.gamma(2 * n) / math.gamma(n) ** 2
    w = np.where(x < 1.0, np.cos(beta * math.pi / 2) / math.sqrt(dom), 0.0)
    norm = math.sqrt((2.0 * (w * w).sum() - w[0] ** 2) * 2 * dom / Nt / math.pi) * Nf / 2.0
    return w / norm


def _wdm_inputs(case, seed):
    """Time series: A-channel noise with 100 slowly chirping sources; or coefficients of such noise."""
    g = torch.Generator(device=_DEV).manual_seed(seed)
    ND = case["NF"] * case["NT"]
    if case["direction"] == "inverse":
        return 1e-20 * torch.randn(ND, dtype=torch.float64, device=_DEV, generator=g)
    f = np.arange(ND // 2 + 1) / (ND * DT)
    amp = _dev(np.sqrt(wl.aenoise_ff(np.maximum(f, f[1])) * ND * DT / 4))
    X = torch.complex(*(torch.randn(ND // 2 + 1, dtype=torch.float64, device=_DEV, generator=g) for _ in "ri")) * amp
    x = torch.fft.irfft(X, n=ND) / DT
    t = DT * torch.arange(ND, dtype=torch.float64, device=_DEV)
    rng = np.random.default_rng(seed)
    for f0 in 10 ** rng.uniform(math.log10(0.5e-3), math.log10(15e-3), 100):
        a, ph, fdot = 10 ** rng.uniform(-23, -21), rng.uniform(0, PI2), 1e-17
        x += a * torch.cos(PI2 * (f0 * t + 0.5 * fdot * t * t) + ph)
    return x


def _exact_wdm(case, x):
    NF, NT = case["NF"], case["NT"]
    ND = NF * NT
    win = _dev(_window(NF, NT, case["nx"]))
    m = torch.arange(NF + 1, device=_DEV)[:, None]
    if case["direction"] == "forward":
        F = torch.fft.rfft(x)
        j = torch.arange(-NT // 2, NT // 2, device=_DEV)
        idx = m * (NT // 2) + j
        w = torch.where(j == -NT // 2, 0.0, win[j.abs()]) * ((idx >= 0) & (idx <= ND // 2))
        w[0, NT // 2] *= 0.5
        w[NF, NT // 2] *= 0.5
        z = torch.fft.ifft(F[idx.clamp(0, ND // 2)] * w, dim=-1)
        n = torch.arange(NT, device=_DEV)
        sgn = 1.0 - 2.0 * (m % 2)
        out = torch.where((n + m) % 2 == 0, z.real, sgn * z.imag)[:NF].clone()
        out[0, 0::2] = z[0, 0::2].real * math.sqrt(2.0)
        out[0, 1::2] = z[NF, 0::2].real * math.sqrt(2.0)
        return out.reshape(-1)
    w = x.reshape(NF, NT)
    n = torch.arange(NT, device=_DEV)
    pre = torch.zeros((NF + 1, NT), dtype=torch.complex128, device=_DEV)
    even = (n + m[:NF]) % 2 == 0
    pre[:NF] = torch.complex(torch.where(even, w, 0.0), torch.where(even, 0.0, -w))
    pre[0] = (w[0][(2 * n) % NT] * math.sqrt(0.5)).to(pre.dtype)
    pre[NF] = (w[0][(2 * n) % NT + 1] * math.sqrt(0.5)).to(pre.dtype)
    res = torch.fft.fft(pre, dim=-1)
    X = torch.zeros(ND // 2 + 1, dtype=torch.complex128, device=_DEV)
    for par in (0, 1):  # layers of one parity have disjoint supports
        mm = torch.arange(par, NF + 1, 2, device=_DEV)[:, None]
        i = mm * (NT // 2) - NT // 2 + n
        src = torch.where((mm == 0) | (mm == NF), (2 * i) % NT, i % NT)
        v = torch.gather(res[mm[:, 0]], 1, src) * (win[(i - mm * (NT // 2)).abs()] * (NF / 2))
        ok = (i >= 0) & (i <= ND // 2)
        X[i[ok]] += v[ok]
    X[0], X[-1] = X[0].real.to(X.dtype), X[-1].real.to(X.dtype)
    return torch.fft.irfft(X, n=ND)


# -------------------------------------------------------------------- wavelet
WV_NF, WV_NT, WV_NX, WV_LMIN, WV_LMAX = 1024, 2048, 4.0, 10, 470
WV_DT = DT * WV_NF
WV_DF = 1.0 / (2.0 * WV_DT)


class _Spline:
    """Natural cubic splines of y [..., n] over the nodes x [n] (utils/src/glass_math.c:101-175)."""

    def __init__(self, x, y, even):
        n, self.x, self.even = len(x), x, even
        h = x[1:] - x[:-1]
        xs, i = x.cpu().numpy(), np.arange(1, n - 1)
        A = np.eye(n)
        A[i, i - 1], A[i, i], A[i, i + 1] = xs[1:-1] - xs[:-2], 2.0 * (xs[2:] - xs[:-2]), xs[2:] - xs[1:-1]
        r = torch.zeros_like(y)
        s = (y[..., 1:] - y[..., :-1]) / h
        r[..., 1:-1] = 3.0 * (s[..., 1:] - s[..., :-1])
        c2 = _dev(np.linalg.solve(A, r.reshape(-1, n).T.cpu().numpy()).T).reshape(y.shape)
        self.c0, self.c2 = y[..., :-1], c2[..., :-1]
        self.c1 = s - h * (c2[..., 1:] + 2.0 * c2[..., :-1]) / 3.0
        self.c3 = (c2[..., 1:] - c2[..., :-1]) / (3.0 * h)

    def __call__(self, v):
        """At v: of one shape with the splines but for the last axis, or [m] for all."""
        n = len(self.x)
        if self.even:
            j = torch.floor((v - self.x[0]) / (self.x[1] - self.x[0])).long().clamp(0, n - 2)
        else:
            j = (torch.searchsorted(self.x, v.contiguous(), right=True) - 1).clamp(0, n - 2)
        d = v - self.x[j]
        pick = (lambda c: c[..., j]) if v.dim() == 1 else (lambda c: torch.gather(c, -1, j))  # noqa: E731
        return pick(self.c0) + d * (pick(self.c1) + d * (pick(self.c2) + d * pick(self.c3)))


def _wv_orbit():
    """The interpolated analytic orbit: node times and position splines [3 spacecraft, 3, nodes]."""
    n = max(20, int(200 * T / YEAR))
    buf = T / (n - 1)
    k = torch.arange(n, dtype=torch.float64, device=_DEV)
    t = k * ((T + 2.0 * buf) / (n - 1)) - buf
    return t, _Spline(t, _positions(t).permute(1, 2, 0).contiguous(), False)


def _wv_layers(p):
    """ucb_wavelet_layers: first layer and number of layers (ucb/src/glass_ucb_waveform.c:1003-1042)."""
    fa, fb = p[:, 0] / T, p[:, 0] / T + p[:, 7] / T / T
    lo, hi = np.minimum(fa, fb) * (1.0 - VEARTH), np.maximum(fa, fb) * (1.0 + VEARTH)
    j = np.rint(lo / WV_DF).astype(np.int64)
    jmin, jmax = np.where(lo < j * WV_DF, j - 1, j), np.where(hi > j * WV_DF, j + 1, j)
    return jmin, jmax - jmin + 1


def _wv_amp_phase(M, Mf, ref):
    """Amplitude with sign flips at zero crossings, and unwrapped phase relative to ref
    (extract_amplitude_and_phase and unwrap_phase, utils/src/glass_math.c:1034-1052, 1244-1308)."""
    a = torch.sqrt(M * M + Mf * Mf)
    n = a.shape[-1]
    up, dn, mid = a[..., 2:], a[..., :-2], a[..., 1:-1]
    low = (mid < dn) & (mid < up)
    d1 = up + dn - 2.0 * mid
    c2 = low & (((-up + dn - 2.0 * mid) / d1).abs() < 0.1)
    c3 = low & (((-up + dn + 2.0 * mid) / d1).abs() < 0.1)
    flip, skip = [torch.zeros_like(a[..., 0])], torch.zeros_like(low[..., 0])
    forced = skip
    for i in range(1, n - 1):
        # half-turns so far; a step just past node i - 1 was already taken at node i
        here = flip[-1] + forced.to(a.dtype)
        t2, t3 = c2[..., i - 1] & ~forced, c3[..., i - 1] & ~forced & ~c2[..., i - 1]
        flip.append(here + t3.to(a.dtype))
        forced = t2
    flip.append(flip[-1])
    turns = torch.stack(flip, -1)
    v = ref - PI2 * torch.round(ref / PI2)
    ph = -torch.atan2(Mf, M) + math.pi * turns - v
    out, last = [ph[..., 0]], ph[..., 0]
    for i in range(1, n):
        u = ph[..., i]
        k = torch.round((u - last).abs() / PI2)
        last = u + torch.where(last > u, k, -k) * PI2
        out.append(last)
    return a * (1.0 - 2.0 * (turns % 2)), torch.stack(out, -1)


def _wv_coefficients(p, nl, jmin):
    """ucb_waveform_wavelet's X, Y, Z of sources with nl layers from jmin
    [n, 3, NT, nl] (ucb/src/glass_ucb_waveform.c:1061-1240)."""
    n = len(p)
    torb, orbit = _wv_orbit()
    ns = len(torb)
    pt = _dev(p)
    col = lambda v: v[:, None]  # noqa: E731
    f0, fdot, cosi = pt[:, 0] / T, pt[:, 7] / T / T, pt[:, 4]
    ph = -col(pt[:, 6]) + PI2 * (col(f0) * torb + 0.5 * col(fdot) * torb * torb)
    am = col(torch.exp(pt[:, 3])) * (1.0 + 2.0 / 3.0 * col(fdot / f0) * torb)
    phase, amp = _Spline(torb, ph, True), _Spline(torb, am, True)
    ep, ec, k = _sky(pt[:, 1], pt[:, 2])
    tn = torch.arange(ns, dtype=torch.float64, device=_DEV) * (T / (ns - 1))

    def at_spacecraft(t):  # the barycentre time of spacecraft 1's signal at t
        r = orbit(t)[0] / CLIGHT
        return t - (k[:, :1] * r[0] + k[:, 1:2] * r[1] + k[:, 2:] * r[2])

    x = orbit(tn) / CLIGHT  # [3, 3, ns]
    arm = torch.stack([x[1] - x[2], x[2] - x[0], x[0] - x[1]])
    L = torch.sqrt((arm * arm).sum(1))
    arm = arm / L[:, None]
    kr, kn = torch.einsum("na,sat->snt", k, x), torch.einsum("na,sat->snt", k, arm)
    dp, dc = (torch.einsum("sat,sbt,nab->snt", arm, arm, e) for e in (ep, ec))
    App, Apm, Acp, Acm = dp / (1.0 + kn), dp / (1.0 - kn), dc / (1.0 + kn), dc / (1.0 - kn)
    ap, ac, c2p, s2p = (col(v) for v in (0.5 * (1.0 + cosi * cosi), -cosi, torch.cos(2.0 * pt[:, 5]),
                                         torch.sin(2.0 * pt[:, 5])))
    ref = phase(at_spacecraft(tn))
    nds = WV_NT * (nl + 1)
    tds = torch.arange(nds, dtype=torch.float64, device=_DEV) * (WV_DT / (nl + 1))
    carrier = phase(at_spacecraft(tds)) - PI2 * col((_dev(jmin).double() - 1.0) * WV_DF) * tds
    win = _dev(_window(nl + 1, WV_NT, WV_NX))
    j = torch.arange(-WV_NT // 2, WV_NT // 2, device=_DEV)
    w = torch.where(j == -WV_NT // 2, 0.0, win[j.abs()])
    out = torch.empty((n, 3, WV_NT, nl), dtype=torch.float64, device=_DEV)
    for ch, (a, b, c) in enumerate(((0, 1, 2), (1, 2, 0), (2, 0, 1))):
        M = Mf = 0.0
        for delay, plus, minus in ((kr[a] + 2 * L[c] + 2 * L[b], (Apm[b], Acm[b]), (App[c], Acp[c])),
                                   (kr[b] + L[c] + 2 * L[b], (App[c], Acp[c]), (Apm[c], Acm[c])),
                                   (kr[c] + L[b] + 2 * L[c], (App[b], Acp[b]), (Apm[b], Acm[b])),
                                   (kr[a] + 2 * L[b], (Apm[c], Acm[c]), (Apm[b], Acm[b])),
                                   (kr[a] + 2 * L[c], (App[c], Acp[c]), (App[b], Acp[b])),
                                   (kr[c] + L[b], (Apm[b], Acm[b]), (App[b], Acp[b])),
                                   (kr[b] + L[c], (Apm[c], Acm[c]), (App[c], Acp[c])),
                                   (kr[a], (App[b], Acp[b]), (Apm[c], Acm[c]))):
            t = tn - delay
            A, P = amp(t), phase(t)
            cp, sp = torch.cos(P), torch.sin(P)
            hp, hc = A * (ap * c2p * cp + ac * s2p * sp), A * (ac * c2p * sp - ap * s2p * cp)
            hpf, hcf = A * (ac * s2p * cp - ap * c2p * sp), A * (ac * c2p * cp + ap * s2p * sp)
            gp, gc = plus[0] - minus[0], plus[1] - minus[1]
            M, Mf = M + hp * gp + hc * gc, Mf + hpf * gp + hcf * gc
        ra, rp = _wv_amp_phase(M, Mf, ref)
        wave = _Spline(tn, ra, False)(tds) * torch.cos(_Spline(tn, rp, False)(tds) + carrier)
        F = torch.fft.rfft(wave, dim=-1)
        for l in range(nl):
            idx = (l + 1) * (WV_NT // 2) + j
            z = torch.fft.ifft(F[:, idx] * w, dim=-1)
            m = _dev(jmin + l)[:, None]
            i = torch.arange(WV_NT, device=_DEV)
            v = torch.where((i + m) % 2 == 0, z.real, (1.0 - 2.0 * (m % 2)) * z.imag)
            out[:, ch, :, l] = v * (math.sqrt(WV_NF) / (nl + 1.0))
    return out


def _wv_groups(p, step=128):
    jmin, nl = _wv_layers(p)
    for size in np.unique(nl):
        idx = np.nonzero(nl == size)[0]
        for a in range(0, len(idx), step):
            i = idx[a:a + step]
            yield i, int(size), jmin[i], _wv_coefficients(p[i], int(size), jmin[i])


def _wv_pixels(jmin, nl):
    """Segment pixel of each coefficient [n, NT, nl] (every layer lies inside the segment)."""
    lay = _dev(jmin)[:, None, None] + torch.arange(nl, device=_DEV)
    return torch.arange(WV_NT, device=_DEV)[:, None] + (lay - WV_LMIN) * WV_NT


def _wavelet_inputs(case, seed):
    """Noise of the segment's covariance at a level that gives the sources a
    median SNR near 20, up to 100 of them injected, and one jump from each."""
    rng = np.random.default_rng(seed)
    amp = 10 ** rng.uniform(-23, -21, case["n"])
    src = np.array([wl.draw_source(rng, 10 ** rng.uniform(math.log10(0.5e-3), math.log10(15e-3)), a) for a in amp])
    inj = src[:100]
    N = (WV_LMAX - WV_LMIN) * WV_NT
    unit = wl.wavelet_invC(N, WV_NT, WV_LMIN * WV_NT, 1.0)
    du = _dev(unit)
    add, snr = torch.zeros((3, N), dtype=torch.float64, device=_DEV), np.empty(len(inj))
    for i, nl, jmin, h in _wv_groups(inj):
        pix = _wv_pixels(jmin, nl).reshape(len(i), -1)
        h = h.reshape(len(i), 3, -1)
        C = du[:, :, pix]
        snr[i] = torch.sqrt(torch.einsum("nap,abnp,nbp->n", h, C, h)).cpu().numpy()
        for r in range(len(i)):
            add[:, pix[r]] += h[r]
    scale = float(np.median(snr)) / 20.0
    base = np.full((3, 3), -0.45) + np.eye(3) * 1.45
    s = unit[0, 0] / np.linalg.inv(base)[0, 0]
    data = (np.linalg.cholesky(base) @ rng.standard_normal((3, N))) * (scale / np.sqrt(s)) + add.cpu().numpy()
    level = 20.0 * amp / np.median(amp)  # rough SNR of each source, for the jump widths
    p = _jumped(rng, src, level, np.ones(case["n"]))
    return dict(data=data, invC=unit / scale ** 2, p=p)


def _exact_wavelet(case, x):
    d, C = _dev(x["data"]), _dev(x["invC"])
    term, hh = np.empty(len(x["p"])), np.empty(len(x["p"]))
    for i, nl, jmin, h in _wv_groups(x["p"]):
        pix = _wv_pixels(jmin, nl).reshape(len(i), -1)
        h = h.reshape(len(i), 3, -1)
        Ch = torch.einsum("abnp,nbp->nap", C[:, :, pix], h)
        dh = (d[:, pix].permute(1, 0, 2) * Ch).sum((1, 2))
        h2 = (h * Ch).sum((1, 2))
        hh[i], term[i] = h2.cpu().numpy(), (h2 - 2.0 * dh).cpu().numpy()
    return -0.5 * term, term, hh


# ---------------------------------------------------------------------- noise
def _noise_cov(f, inst, sgal):
    """Instrument covariance [..., 6] = xx, yy, zz, xy, xz, yz at f for link
    levels inst [..., 12], and the foreground's diagonal (noise/src/
    glass_noise_model.c:389-546, 612-654; utils/src/glass_galaxy.c:40-44)."""
    x = f / FSTAR
    cx, s2 = np.cos(x), np.sin(x) ** 2
    acc = np.where(f < 0.01, 2.81837551648e-19 / f ** 2 * (1.0 + (0.4e-3 / f) ** 2) * (1.0 + (f / 8.0e-3) ** 4), 0.0)
    oms = 4.39256635604e-16 * f ** 2 * (1.0 + (2.0e-3 / f) ** 4)
    cx, s2, acc, oms = (_dev(v) for v in (cx, s2, acc, oms))
    A = [inst[:, k:k + 1] * acc for k in range(6)]  # 12, 21, 23, 32, 13, 31
    O = [inst[:, 6 + k:7 + k] * oms for k in range(6)]
    c2 = cx * cx
    dia = [0.25 * (O[0] + O[1] + O[4] + O[5]) + (A[0] + A[4]) + (A[1] + A[5]) * c2,
           0.25 * (O[2] + O[3] + O[1] + O[0]) + (A[2] + A[1]) + (A[3] + A[0]) * c2,
           0.25 * (O[5] + O[4] + O[3] + O[2]) + (A[5] + A[3]) + (A[4] + A[2]) * c2]
    off = [0.5 * (O[0] + O[1]) + 2.0 * (A[0] + A[1]), 0.5 * (O[4] + O[5]) + 2.0 * (A[4] + A[5]),
           0.5 * (O[3] + O[2]) + 2.0 * (A[3] + A[2])]
    C = [4.0 * s2 * v for v in dia] + [-2.0 * s2 * cx * v for v in off]
    if sgal is None:
        return C, 0.0
    g = [v[:, None] for v in (torch.exp(sgal[:, 0]), torch.exp(sgal[:, 1]), sgal[:, 2], torch.exp(sgal[:, 3]),
                              torch.exp(sgal[:, 4]))]
    df = _dev(f)
    S = g[0] * df ** (-7.0 / 3.0) * torch.exp(-(df / g[1]) ** g[2]) * 0.5 * (1.0 + torch.tanh((g[3] - df) / g[4]))
    return C, _dev(x ** 2) * s2 * torch.where(df > 10.0 * g[1], torch.zeros_like(S), S)


def _gauss(C, P):
    """tr(C^-1 P) and log det C for symmetric 3 x 3 C, P given as six entries."""
    xx, yy, zz, xy, xz, yz = C
    d2 = yy - xy * xy / xx
    t = yz - xy * xz / xx
    d3 = (zz - xz * xz / xx) - t * t / d2
    i = 1.0 / (xx * d2 * d3)
    chi = ((yy * zz - yz * yz) * P[0] + (zz * xx - xz * xz) * P[1] + (xx * yy - xy * xy) * P[2]
           + 2.0 * ((xz * yz - zz * xy) * P[3] + (xy * yz - xz * yy) * P[4] + (xy * xz - xx * yz) * P[5])) * i
    return chi, torch.log(xx) + torch.log(d2) + torch.log(d3)


def _noise_models(case, rng):
    inst0, sgal0 = wl.default_noise_params(T)
    inst = inst0 * np.exp(rng.uniform(-0.3, 0.3, (case["n"], 12)))
    return inst0, sgal0, inst, sgal0 + rng.uniform(-0.2, 0.2, (case["n"], 5))


def _noise_inputs(case, seed):
    """XYZ data of the starting model's covariance, and models around it."""
    rng = np.random.default_rng(seed)
    inst0, sgal0, inst, sgal = _noise_models(case, rng)
    f = (case["qmin"] + np.arange(case["N"])) / T
    C, g = _noise_cov(f, _dev(inst0[None]), _dev(sgal0[None]))
    C6 = torch.stack([c + g for c in C[:3]] + [c - 0.5 * g for c in C[3:]], -1)[0].cpu().numpy()
    return dict(xyz=wl.xyz_from_covariance(rng, C6), inst=inst, sgal=sgal if case["foreground"] else None, f=f)


def _exact_noise(case, x):
    z = x["xyz"][:, 0::2] + 1j * x["xyz"][:, 1::2]
    pair = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
    P = [_dev((z[a] * z[b].conj()).real) for a, b in pair]
    out = []
    for a in range(0, case["n"], 64):
        sg = None if x["sgal"] is None else _dev(x["sgal"][a:a + 64])
        C, g = _noise_cov(x["f"], _dev(x["inst"][a:a + 64]), sg)
        chi, ld = _gauss([c + g for c in C[:3]] + [c - 0.5 * g for c in C[3:]], P)
        out.append((-chi - ld).sum(-1) - 3.0 * case["N"] * math.log(2.0 * math.pi))
    return torch.cat(out)


def _noise_wavelet_inputs(case, seed):
    rng = np.random.default_rng(seed)
    inst0, sgal0, inst, sgal = _noise_models(case, rng)
    f = (case["lmin"] + np.arange(case["layers"])) * WV_DF
    C, _ = _noise_cov(f, _dev(inst0[None]), None)
    C6 = torch.stack(C, -1)[0].cpu().numpy() / (WV_NF * WV_NT)
    return dict(xyz=wl.wavelet_noise_data(rng, C6, WV_NT), inst=inst, sgal=sgal if case["mode"] else None, f=f,
                mod=wl.galaxy_modulation_like(WV_NT // case["Q"]))


def _exact_noise_wavelet(case, x):
    NL, Q = case["layers"], case["Q"]
    w = x["xyz"].reshape(3, NL, WV_NT // Q, Q)
    pair = ((0, 0), (1, 1), (2, 2), (0, 1), (0, 2), (1, 2))
    P = [_dev((w[a] * w[b]).mean(-1)) for a, b in pair]  # [layers, cells]
    mod = _dev(x["mod"])
    out = []
    for a in range(0, case["n"], 16):
        sg = None if x["sgal"] is None else _dev(x["sgal"][a:a + 16])
        C, g = _noise_cov(x["f"], _dev(x["inst"][a:a + 16]), sg)
        C = [c[:, :, None] / (WV_NF * WV_NT) for c in C]
        if case["mode"]:
            g = g[:, :, None] / (WV_NF * WV_NT)
            m = mod if case["mode"] == 2 else _dev(np.array([1.0, 1.0, 1.0, -0.5, -0.5, -0.5]))[:, None]
            C = [c + g * m[e] for e, c in enumerate(C)]
        chi, ld = _gauss(C, P)
        s = -0.5 * Q * (chi + ld)
        out.append(s.expand(-1, -1, WV_NT // Q).sum((1, 2)) - 1.5 * NL * WV_NT * math.log(2.0 * math.pi))
    return torch.cat(out)


# ------------------------------------------------------------ the entry points
_STREAM = []


def _engine():
    """An engine on the one stream that the program works on."""
    if not _STREAM:
        _STREAM.append(torch.cuda.Stream())
    eng = gg.Engine(0)
    eng.set_stream(_STREAM[0].cuda_stream)
    return eng


def _out(*shape):
    return torch.empty(shape, dtype=torch.float64, device=_DEV)


def prepare(case, seed):
    kind = case["kind"]
    st = dict(case=case, eng=_engine())
    eng = st["eng"]
    if kind in ("dlogl", "global_fit", "grad_fisher"):
        x = _fourier_inputs(case, seed)
        n = len(x["p"])
        eng.upload(_engine_bank(x["bank"]))
        if case.get("entry") == "host":
            hb = eng.host_batch(n)
            hb.item_seg[:], hb.params[:], hb.term_x[:] = x["seg"], x["p"], x["tx"]
            st.update(batch=hb)
        else:
            st.update(seg=_dev(x["seg"]), p=_dev(x["p"]), tx=_dev(x["tx"]), dl=_out(n), ty=_out(n), hh=_out(n),
                      status=torch.zeros(n, dtype=torch.int32, device=_DEV))
            if kind == "grad_fisher":
                st.update(grad=_out(n, 8), fisher=_out(n, 8, 8))
    elif kind == "wdm":
        x = _wdm_inputs(case, seed)
        st.update(x=x, y=torch.empty_like(x))
    elif kind == "wavelet":
        x = _wavelet_inputs(case, seed)
        n = len(x["p"])
        eng.wavelet_setup(T, 0.0, WV_NF, WV_NT, WV_DT, WV_DF, WV_LMIN * WV_NT, WV_LMAX * WV_NT, nx=WV_NX)
        eng.wavelet_set_data(x["data"], x["invC"])
        st.update(p=_dev(x["p"]), dl=_out(n), ty=_out(n), hh=_out(n),
                  status=torch.zeros(n, dtype=torch.int32, device=_DEV))
    elif kind == "fstat":
        x = _fstat_inputs(case, seed)
        n = len(x["cells"])
        eng.upload(_engine_bank(x["bank"]))
        st.update(seg=torch.zeros(n, dtype=torch.int32, device=_DEV), cells=_dev(x["cells"]), logl=_out(n),
                  fp=_out(n, 4), status=torch.zeros(n, dtype=torch.int32, device=_DEV))
    else:
        if kind == "noise":
            x = _noise_inputs(case, seed)
            eng.noise_setup(T, case["qmin"], *x["xyz"])
        else:
            x = _noise_wavelet_inputs(case, seed)
            eng.noise_wavelet_setup(WV_NF, WV_NT, WV_DF, case["lmin"], case["Q"], *x["xyz"],
                                    x["mod"] if case["mode"] == 2 else None)
        st.update(inst=_dev(x["inst"]), sgal=None if x["sgal"] is None else _dev(x["sgal"]), logl=_out(case["n"]))
    torch.cuda.synchronize()
    return st


def run(s):
    case, eng = s["case"], s["eng"]
    kind, prec = case["kind"], _PREC[case.get("precision", "fp64")]
    if "batch" in s:
        b = s["batch"]
        b.run(prec)
        return dict(dlogl=b.dlogl, term=b.term_y, hh=b.hh, status=b.status)
    if kind in ("dlogl", "global_fit"):
        eng.dlogl_device(s["seg"], s["p"], s["dl"], s["ty"], s["hh"], s["status"], s["tx"], prec)
        return dict(dlogl=s["dl"], term=s["ty"], hh=s["hh"], status=s["status"])
    if kind == "grad_fisher":
        eng.grad_fisher_device(s["seg"], s["p"], s["ty"], s["grad"], s["fisher"], s["status"], case["mode"])
        return dict(term=s["ty"], grad=s["grad"], fisher=s["fisher"], status=s["status"])
    if kind == "wdm":
        go = eng.wdm_forward_device if case["direction"] == "forward" else eng.wdm_inverse_device
        go(case["NF"], case["NT"], s["x"], s["y"], prec, nx=case["nx"])
        return s["y"]
    if kind == "wavelet":
        eng.wavelet_dlogl_device(s["p"], s["dl"], s["ty"], s["hh"], s["status"], precision=prec)
        return dict(dlogl=s["dl"], term=s["ty"], hh=s["hh"], status=s["status"])
    if kind == "fstat":
        eng.fstat_device(s["seg"], s["cells"], s["logl"], s["fp"], s["status"])
        return dict(logl=s["logl"], fit=s["fp"], status=s["status"])
    if kind == "noise":
        eng.noise_logl_device(s["inst"], s["logl"], s["sgal"])
    else:
        eng.noise_wavelet_logl_device(s["inst"], s["logl"], s["sgal"], case["mode"])
    return s["logl"]


def exact(case, seed):
    kind = case["kind"]
    if kind in ("dlogl", "global_fit"):
        x = _fourier_inputs(case, seed)
        term, hh = _terms(x["bank"], x["seg"], x["p"])
        return dict(dlogl=term - x["tx"], term=term, hh=hh, status=None)
    if kind == "grad_fisher":
        term, grad, F = _exact_grad(case, _fourier_inputs(case, seed))
        return dict(term=term, grad=grad, fisher=F, status=None)
    if kind == "wdm":
        return _exact_wdm(case, _wdm_inputs(case, seed))
    if kind == "wavelet":
        dl, term, hh = _exact_wavelet(case, _wavelet_inputs(case, seed))
        return dict(dlogl=dl, term=term, hh=hh, status=None)
    if kind == "fstat":
        logl, fit = _exact_fstat(case, _fstat_inputs(case, seed))
        return dict(logl=logl, fit=fit, status=None)
    if kind == "noise":
        return _exact_noise(case, _noise_inputs(case, seed))
    return _exact_noise_wavelet(case, _noise_wavelet_inputs(case, seed))


def work(case):
    """Bytes: each input read and each output written once (a template's bins
    with the bank, a source's pixels with the data).  Flops: the arithmetic of
    the method in its most economical known form, transcendentals as 20."""
    kind, n = case["kind"], case.get("n", 0)
    if kind in ("dlogl", "global_fit", "grad_fisher"):
        N = _fourier_sizes(case).astype(np.float64)
        log2 = np.log2(N)
        bank = min(48.0 * case["nseg"] * case["NFFT"], 48.0 * N.sum())
        if kind == "grad_fisher":  # 24 series, 8 derivatives, 36 products per bin
            return dict(bytes=float(bank) + n * (68.0 + 588.0), flops=float((N * (900.0 + 120.0 * log2 + 500.0)).sum()))
        return dict(bytes=float(bank) + n * (76.0 + 28.0), flops=float((N * (312.0 + 20.0 * log2 + 120.0)).sum()))
    if kind == "wdm":
        ND = float(case["NF"] * case["NT"])
        return dict(bytes=16.0 * ND, flops=ND * (2.5 * math.log2(ND) + 2.5 * math.log2(case["NT"]) + 4.0))
    if kind == "wavelet":
        nds = 3.0 * WV_NT  # two layers is the usual case
        pix = 2.0 * WV_NT
        data = min(n * pix, float((WV_LMAX - WV_LMIN) * WV_NT)) * 8.0 * (3 + 9)
        return dict(bytes=data + n * (64.0 + 28.0),
                    flops=n * (940.0 * 199 + 85.0 * nds + 7.5 * nds * math.log2(nds)
                               + 7.5 * pix * math.log2(WV_NT) + 54.0 * pix))
    if kind == "fstat":
        cells = float(case["n_f"] * case["n_theta"] * case["n_phi"])
        N = float(_half_bandwidth(np.array([case["f0"]]), 0.0, np.array([0.0]), 1e-22, case["NFFT"])[0])
        return dict(bytes=48.0 * case["NFFT"] + cells * (36.0 + 44.0),
                    flops=cells * (4.0 * N * (150.0 + 20.0 * math.log2(N) + 60.0) + 112.0 * N + 200.0))
    if kind == "noise":
        fg = case["foreground"]
        return dict(bytes=case["N"] * 48.0 + n * (104.0 + (40.0 if fg else 0.0)),
                    flops=n * case["N"] * (110.0 + (70.0 if fg else 0.0)))
    cells = float(case["layers"] * (WV_NT // case["Q"]))
    inv = cells if case["mode"] == 2 else float(case["layers"])
    return dict(bytes=cells * 48.0 + n * (104.0 + (40.0 if case["mode"] else 0.0)),
                flops=n * (inv * 90.0 + case["layers"] * 150.0))
