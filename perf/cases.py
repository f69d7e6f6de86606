"""Measured work of the framework: the calls its users make, over their real range.

A case names one call through the public surface (``get_transformer`` and the
differentiable ``autograd.gclm2lenmap``) with its band limit, spin, accuracy and
data types.  Inputs are seeded Gaussian fields: C_l = 1e3 / (l + 10)^2 (E modes
at a tenth of it), a lensing potential of spectrum 4e-7 (l + 20)^-4 rescaled to
2.5 arcmin rms deflection, white-noise maps for the adjoint direction.

``exact`` restates every call in plain torch FP64: spin-weighted harmonics by the
normalised three-term recursion, the nuFFT on a twice oversampled torus with a
14-tap exponential-of-semicircle kernel (error below 1e-12).
"""
from __future__ import annotations

import functools
import math

import numpy as np
import torch

import cunusht_gb300 as cu
from cunusht_gb300 import autograd as cu_autograd

C128, C64 = torch.complex128, torch.complex64


def listed():
    return [
        # the smallest solve: spin-0 lensing, lmax 255 on 256 x 511 rings, complex128, default
        # precision at eps 1e-7 (FP64) -- interactive use, latency and launches
        dict(name="lens_l255_s0_f64", op="lens", lmax=255, nphi=511, spin=0, eps=1e-7, precision="auto", single=False),
        # single-precision delensing of a small map (quick-look pipelines): complex64 / float32, eps 1e-5
        dict(name="delens_l511_s0_f32", op="delens", lmax=511, nphi=0, spin=0, eps=1e-5, precision="auto", single=True),
        # served launch of the smallest bucket: eight spin-2 requests at lmax 511, eps 1e-5
        dict(name="lens_batch8_l511_s2", op="lens_batch", lmax=511, nphi=0, spin=2, eps=1e-5, precision="mixed", nreq=8),
        # differentiable lensing, float64 at lmax 1023: loss gradient for the field and the deflection
        dict(name="grad_l1023_s0_f64", op="grad", lmax=1023, nphi=0, spin=0, eps=1e-7, precision="auto"),
        # plain transforms of the SHT mode (FP64), an odd band limit and its odd ring count: map -> alm
        dict(name="map2alm_l1400_s0_f64", op="map2alm", lmax=1400, nphi=0, spin=0),
        # pointing for a HEALPix map (rings of 4 to 2048 pixels): deflection and rotation angle only
        dict(name="pointing_hpx512_l1000", op="pointing", lmax=1000, nside=512, eps=1e-5, precision="auto", single=True),
        # type-1 nuSHT of a spin-2 field at given points, ragged count, tight accuracy (FP64)
        dict(name="nusht2d1_l767_s2_f64", op="nusht2d1", lmax=767, spin=2, eps=1e-10, precision="auto", npts=777777),
        # type-2 nuSHT at given points at the size of the published notebook timing, single precision
        dict(name="nusht2d2_l3087_s0_f32", op="nusht2d2", lmax=3087, spin=0, eps=1e-7, precision="mixed", npts=19068400, single=True),
        # the headline: one served launch of eight lmax 2047 spin-2 lensing requests, eps 1e-7, mixed precision
        dict(name="lens_batch8_l2047_s2", op="lens_batch", lmax=2047, nphi=4095, spin=2, eps=1e-7, precision="mixed", nreq=8),
        # the adjoint direction, served: four delensing requests of the same configuration
        dict(name="delens_batch4_l2047_s2", op="delens_batch", lmax=2047, nphi=4095, spin=2, eps=1e-7, precision="mixed", nreq=4),
        # the plain FP64 single-request solve the headline is compared with
        dict(name="lens_l2047_s2_f64", op="lens", lmax=2047, nphi=4095, spin=2, eps=1e-7, precision="fp64", single=False),
        # the largest: lmax 4095 spin 2, gradient + curl deflection, prime 8191-pixel rings, complex64 -> float32
        dict(name="lens_l4095_s2_f32", op="lens", lmax=4095, nphi=8191, spin=2, eps=1e-5, precision="auto", single=True, curl=True),
    ]


def _log_int(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    op = rng.choice(["lens", "lens", "delens", "lens_batch", "lens_batch", "delens_batch", "nusht2d2", "nusht2d1", "grad",
                     "map2alm", "alm2map", "pointing"])
    if op in ("map2alm", "alm2map"):
        return dict(op=op, lmax=_log_int(rng, 63, 2047), nphi=0, spin=rng.choice([0, 0, 2]))
    if op == "grad":
        return dict(op=op, lmax=_log_int(rng, 63, 1200), nphi=0, spin=0, eps=1e-7, precision="auto")
    if op == "pointing":
        nside = rng.choice([64, 128, 256, 512, 1024])
        return dict(op=op, lmax=rng.randrange(nside, 2 * nside + 1), nside=nside, eps=rng.choice([1e-5, 1e-7]),
                    precision="mixed", single=rng.random() < 0.5)
    if op in ("lens_batch", "delens_batch"):
        lmax = _log_int(rng, 255, 2047)
        return dict(op=op, lmax=lmax, nphi=rng.choice([0, 2 * lmax + 1]), spin=rng.choice([0, 2]), eps=rng.choice([1e-5, 1e-7]),
                    precision="mixed", nreq=rng.randrange(1, 9) if op == "lens_batch" else rng.randrange(1, 5))
    # single calls: FP64 plans with 64-bit arrays, mixed plans with single-precision arrays
    single = rng.random() < 0.5
    lmax = _log_int(rng, 63, 3087 if single else 2047)
    eps = rng.choice([1e-5, 1e-6, 1e-7]) if single else rng.choice([1e-7, 1e-8, 1e-10])
    case = dict(op=op, lmax=lmax, spin=rng.choice([0, 2]), eps=eps, precision="mixed" if single else "auto", single=single)
    if op in ("nusht2d1", "nusht2d2"):
        case["npts"] = rng.randrange(lmax * lmax // 2, 2 * lmax * lmax + 1)
    else:
        case["nphi"] = rng.choice([0, 2 * lmax + 1])
    return case


# ----------------------------------------------------------------- inputs
def _nalm(lmax):
    return (lmax + 1) * (lmax + 2) // 2


def _lm(lmax, dev="cuda"):
    """(l, m) of every entry of the m-major layout."""
    m = torch.repeat_interleave(torch.arange(lmax + 1, device=dev), torch.arange(lmax + 1, 0, -1, device=dev))
    return torch.arange(_nalm(lmax), device=dev) - m * (2 * lmax + 1 - m) // 2, m


def _grad_factor(lmax):
    """sqrt(l (l + 1)) of every entry, the gradient of a scalar field."""
    l = _lm(lmax)[0].double()
    return torch.sqrt(l * (l + 1.0))


def _gauss_alm(cl, lmax, gen):
    l, m = _lm(lmax)
    z = torch.randn((2, _nalm(lmax)), dtype=torch.float64, device="cuda", generator=gen)
    a = torch.complex(z[0], z[1] * (m > 0)) * torch.sqrt(0.5 * cl[l])
    return torch.where(m > 0, a, a * math.sqrt(2.0))


def _field(lmax, spin, gen):
    """(ncomp, nalm) complex128: T, or E with B = 0."""
    l = torch.arange(lmax + 1, dtype=torch.float64, device="cuda")
    cl = 1e3 / (l + 10.0) ** 2
    if spin == 0:
        return _gauss_alm(cl, lmax, gen)[None]
    e = _gauss_alm(0.1 * cl, lmax, gen)
    return torch.stack([e, torch.zeros_like(e)])


def _potential(lmax, gen, curl=False):
    """phi_lm (and the curl potential) at 2.5 arcmin rms deflection."""
    l = torch.arange(lmax + 1, dtype=torch.float64, device="cuda")
    cl = 4e-7 * (l + 20.0) ** -4
    p = _gauss_alm(cl, lmax, gen)
    power = torch.sum((p.real ** 2 + p.imag ** 2) * _grad_factor(lmax) ** 2 * torch.where(_lm(lmax)[1] > 0, 2.0, 1.0)) / (4 * math.pi)
    scale = (2.5 / 60.0 * math.pi / 180.0) / torch.sqrt(power)
    return p * scale, (_gauss_alm(0.1 * cl, lmax, gen) * scale if curl else None)


def _noise_map(spin, npix, gen):
    return torch.randn((2, npix) if spin else (npix,), dtype=torch.float64, device="cuda", generator=gen)


def _points(lmax, npts, gen):
    """(npts, 2) colatitude / longitude: the pixels of an iso-latitude map of npts pixels, ring by
    ring, displaced by 2.5 arcmin."""
    nring = lmax + 1
    i = torch.arange(npts, dtype=torch.float64, device="cuda")
    per = npts / nring
    ring = torch.clamp(torch.floor(i / per), max=nring - 1)
    th = math.pi * (ring + 0.5) / nring
    ph = 2 * math.pi * (i / per - ring)
    z = torch.randn((2, npts), dtype=torch.float64, device="cuda", generator=gen) * (2.5 / 60.0 * math.pi / 180.0 / math.sqrt(2.0))
    th2 = torch.clamp(th + z[0], 1e-6, math.pi - 1e-6)
    return torch.stack([th2, torch.remainder(ph + z[1] / torch.sin(th), 2 * math.pi)], dim=1).contiguous()


def _npix(case):
    if "nside" in case:
        return 12 * case["nside"] ** 2
    return (case["lmax"] + 1) * _nphi(case)


def _nphi(case):
    return case["nphi"] or cu.good_size(2 * case["lmax"] + 1, True)


def _inputs(case, seed):
    """The arrays of one call, from the seed alone."""
    gen = torch.Generator(device="cuda")
    gen.manual_seed(int(seed))
    op, lmax, spin = case["op"], case["lmax"], case.get("spin", 0)
    single = case.get("single", False)
    alm_t, map_t = (C64, torch.float32) if single else (C128, torch.float64)
    s = {}
    if op in ("lens_batch", "delens_batch"):
        n = case["nreq"]
        s["d"] = torch.stack([_potential(lmax, gen)[0] for _ in range(n)])
        if op == "lens_batch":
            s["g"] = torch.stack([_field(lmax, spin, gen) for _ in range(n)])
        else:
            s["map"] = torch.stack([_noise_map(spin, _npix(case), gen) for _ in range(n)])
        return s
    if op in ("lens", "delens", "grad", "pointing"):
        d, c = _potential(lmax, gen, case.get("curl", False))
        s["d"] = d.to(alm_t)
        s["c"] = None if c is None else c.to(alm_t)
    if op in ("lens", "grad", "nusht2d2", "alm2map"):
        g = _field(lmax, spin, gen).to(alm_t)
        s["g"] = g if spin else g[0]
    if op in ("delens", "map2alm", "grad"):
        s["map"] = _noise_map(spin, _npix(case), gen).to(map_t)
    if op in ("nusht2d1", "nusht2d2"):
        s["loc"] = _points(lmax, case["npts"], gen)
    if op == "nusht2d1":
        s["map"] = _noise_map(spin, case["npts"], gen).to(map_t)
    return s


@functools.lru_cache(maxsize=1)
def _transformer(op, lmax, nphi, nside, spin, eps, precision, nreq):
    """The handle a program keeps: one transformer per configuration, inputs come and go."""
    geom = ("healpix", {"nside": nside, "lmax": lmax}) if nside else ("gl", {"lmax": lmax, "nphi": nphi})
    if op in ("map2alm", "alm2map"):
        return cu.get_transformer("GPU", mode="SHT")(geom, max_spin=2)
    t = cu.get_transformer("GPU")(geom, nuFFTtype=1 if op in ("delens", "delens_batch", "nusht2d1") else 2, epsilon=eps,
                                  precision=precision, max_spin=spin)
    if nreq:
        t.reserve_batch(nreq)
    return t


def prepare(case, seed):
    s = _inputs(case, seed)
    s["case"] = case
    s["t"] = _transformer(case["op"], case["lmax"], _nphi(case) if "nphi" in case else None, case.get("nside"), case.get("spin", 0),
                          case.get("eps"), case.get("precision"), case.get("nreq"))
    if case["op"] == "grad":
        s["g"].requires_grad_(True)
        s["d"].requires_grad_(True)
    return s


def run(state):
    case, t = state["case"], state["t"]
    op, lmax, spin = case["op"], case["lmax"], case.get("spin", 0)
    if op == "lens":
        return t.gclm2lenmap(state["g"], lmax, lmax, dlm_scaled=state["d"], dclm_scaled=state["c"], spin=spin, verbose=0)
    if op == "delens":
        like = torch.empty(0, dtype=state["d"].dtype, device="cuda")  # the alm type wanted back
        return t.lenmap2gclm(state["map"], state["d"], like, lmax, lmax, dclm_scaled=state["c"], spin=spin, verbose=0)
    if op == "lens_batch":
        return t.lensing_batch(state["g"], state["d"], spin)
    if op == "delens_batch":
        return t.delensing_batch(state["map"], state["d"], spin)
    if op == "pointing":
        ptg = t.dlm2pointing(state["d"], lmax, dclm_scaled=state["c"])
        return {"ptg": ptg, "gamma": t.gamma}
    if op == "nusht2d2":
        return t.nusht2d2(lmax, lmax, state["g"], state["loc"], spin=spin,
                          out_dtype=torch.float32 if case.get("single") else torch.float64)
    if op == "nusht2d1":
        return t.nusht2d1(lmax, lmax, state["map"], state["loc"], spin=spin, alm_dtype=C64 if case.get("single") else C128)
    if op == "alm2map":
        return t.alm2map(state["g"], spin=spin)
    if op == "map2alm":
        return t.map2alm(state["map"], spin=spin)
    g, d = state["g"], state["d"]
    out = cu_autograd.gclm2lenmap(t, g, d, spin)
    loss = torch.sum((out - state["map"]) ** 2)
    gg, gd = torch.autograd.grad(loss, (g, d))
    return {"lenmap": out.detach(), "grad_g": gg, "grad_d": gd}


def work(case):
    """Inputs read once, outputs written once; flops: Legendre contractions (8 per (l, m, ring) and
    component, 4 for spin 0), torus FFTs, kernel taps."""
    op, lmax, spin = case["op"], case["lmax"], case.get("spin", 0)
    n, b = case.get("nreq", 1), 4 if case.get("single") else 8
    nalm, ncomp = _nalm(lmax), 2 if spin else 1
    npts = case["npts"] if "npts" in case else _npix(case)
    leg = (16 if spin else 4) * nalm * (lmax + 1)
    ptg = 8 * nalm * (lmax + 1) if op in ("lens", "delens", "lens_batch", "delens_batch", "grad", "pointing") else 0
    grid = (2 * lmax + 2) ** 2
    taps = math.ceil(math.log10(10 / case["eps"])) ** 2 if "eps" in case else 0
    nufft = 5 * grid * math.log2(grid) * ncomp / 2 + npts * taps * 2 * ncomp
    alm_b, map_b = 2 * b * ncomp * nalm, b * ncomp * npts
    if op == "pointing":
        return {"bytes": 2 * b * nalm + 24 * npts, "flops": ptg}
    if op in ("map2alm", "alm2map"):
        return {"bytes": alm_b + map_b, "flops": leg}
    if op in ("nusht2d1", "nusht2d2"):
        return {"bytes": alm_b + map_b + 16 * npts, "flops": leg + nufft}
    if op == "grad":
        return {"bytes": 4 * alm_b + 2 * map_b, "flops": 2 * (leg + nufft) + 2 * ptg}
    return {"bytes": n * (alm_b + map_b + 2 * b * nalm * (2 if case.get("curl") else 1)), "flops": n * (leg + ptg + nufft)}


# ----------------------------------------------------------------- the same in plain torch, 64 bits
@functools.lru_cache(maxsize=4)
def _gl(n):
    """Gauss-Legendre colatitudes and weights, Newton on P_n."""
    x = np.cos(np.pi * (np.arange(1, n + 1) - 0.25) / (n + 0.5))
    for _ in range(8):
        p0, p1 = np.ones_like(x), x.copy()
        for j in range(2, n + 1):
            p0, p1 = p1, ((2 * j - 1) * x * p1 - (j - 1) * p0) / j
        dp = n * (x * p1 - p0) / (x * x - 1.0)
        dx = p1 / dp
        x = x - dx
        if np.max(np.abs(dx)) < 1e-15:
            break
    return torch.as_tensor(np.arccos(x), device="cuda"), torch.as_tensor(2.0 / ((1.0 - x * x) * dp * dp), device="cuda")


def _rings(case):
    """(theta, phi0, nph) of the geometry's rings."""
    if "nside" not in case:
        n = case["lmax"] + 1
        return _gl(n)[0], np.zeros(n), np.full(n, _nphi(case))
    ns = case["nside"]
    i = np.arange(1, 4 * ns)
    ip = np.minimum(i, 4 * ns - i)
    cap = 2.0 * np.arcsin(np.minimum(ip / (np.sqrt(6.0) * ns), 1.0))
    belt = np.arccos(np.clip(4.0 / 3.0 - 2.0 * i / (3.0 * ns), -1, 1))
    th = np.where(ip < ns, np.where(i < ns, cap, np.pi - cap), belt)
    ph = np.where(ip < ns, np.pi / (4.0 * ip), np.pi / (2.0 * ns) * (1.0 - 0.5 * ((i - ns + 1) % 2)))
    return torch.as_tensor(th, device="cuda"), ph, np.where(ip < ns, 4 * ip, 4 * ns)


def _lambda_blocks(lmax, s, theta, kb):
    """Yields (l0, lam[m, k, ring]) for l = l0 + k: the spin-s harmonics sY_lm(theta, 0), m >= 0.
    Mantissas and a power-of-two exponent per entry keep the sin^m start from underflowing."""
    f = dict(dtype=torch.float64, device="cuda")
    nm = lmax + 1
    m = torch.arange(nm, **f)
    x = torch.cos(theta)[None]
    ls, lc = torch.log2(torch.sin(0.5 * theta))[None], torch.log2(torch.cos(0.5 * theta))[None]
    l0 = torch.clamp(m, min=s)
    lg = 0.5 * (torch.log((2 * l0 + 1) / (4 * math.pi)) + torch.lgamma(2 * l0 + 1) - torch.lgamma(m + s + 1)
                - torch.lgamma((m - s).abs() + 1)) / math.log(2.0)
    a, b = (m + s)[:, None], (m - s).abs()[:, None]
    lg = lg[:, None] + torch.where(a > 0, a * ls, 0.0) + torch.where(b > 0, b * lc, 0.0)
    e = torch.where(torch.isfinite(lg), 200.0 * torch.floor(lg / 200.0), -1e6)
    start = torch.where(torch.isfinite(lg), torch.exp2(lg - e), 0.0) * (1.0 - 2.0 * (m % 2))[:, None]
    scale = torch.exp2(e)
    cur, prev = torch.zeros_like(start), torch.zeros_like(start)
    lam = None
    for l in range(lmax + 1):
        k = l % kb
        if k == 0:
            lam = torch.zeros((nm, min(kb, lmax + 1 - l), theta.numel()), **f)
        if l == s:
            cur[:l + 1] = start[:l + 1]
        elif l > s:
            cur[l] = start[l]
        if l >= s:
            n = l + 1
            torch.mul(cur[:n], scale[:n], out=lam[:n, k])
            lp = l + 1
            mm = m[:n]
            den = torch.sqrt((lp * lp - mm * mm) * (lp * lp - s * s))
            al = lp * math.sqrt((2 * l + 1) * (2 * l + 3)) / den
            ga = al * mm * s / (l * lp) if l else torch.zeros_like(al)
            t = torch.addcmul(ga[:, None], al[:, None], x)
            t *= cur[:n]
            if l:
                be = (lp / l) * math.sqrt((2 * l + 3) / (2 * l - 1)) * torch.sqrt((l * l - mm * mm) * (l * l - s * s)) / den
                t -= be[:, None] * prev[:n]
            prev[:n] = cur[:n]
            cur[:n] = t
            if l % 8 == 7:
                big = (cur[:n].abs() > 2.0 ** 200) & (e[:n] < 0)
                down = torch.where(big, torch.full_like(t, 2.0 ** -200), torch.ones_like(t))
                cur[:n] *= down
                prev[:n] *= down
                e[:n] += torch.where(big, 200.0, 0.0)
                scale[:n] = torch.exp2(e[:n])
        if k == kb - 1 or l == lmax:
            yield l - k, lam


def _dense(alm, lmax):
    """(..., nalm) -> (..., m, l) with zeros for l < m."""
    l, m = _lm(lmax)
    out = torch.zeros(alm.shape[:-1] + (lmax + 1, lmax + 1), dtype=C128, device="cuda")
    out[..., m, l] = alm.to(C128)
    return out


def _block(lmax, nring):
    return max(8, min(64, int(3e9 / (8.0 * (lmax + 1) * nring))))


def _legendre(alm, lmax, s, theta):
    """alm (R, ncomp, nalm) -> columns (R, 2 lmax + 1, ring), m = -lmax .. lmax, of Q + iU = sum s_a_lm sY_lm
    with s_a_lm = -(G + iC) (spin 0: a_lm).  The rings are symmetric about the equator."""
    R, nr = alm.shape[0], theta.numel()
    ga = _dense(alm[:, 0], lmax)
    cc = _dense(alm[:, 1], lmax) if alm.shape[1] > 1 else torch.zeros_like(ga)
    plus = (ga if s == 0 else -(ga + 1j * cc)).permute(1, 0, 2)  # (m, R, l)
    minus = (ga.conj() if s == 0 else -(-1) ** s * (ga.conj() + 1j * cc.conj())).permute(1, 0, 2)
    i = torch.arange(lmax + 1, device="cuda")
    minus = minus * (1.0 - 2.0 * ((i[:, None] + i[None]) % 2))[:, None]
    w = torch.cat([plus.real, plus.imag, minus.real, minus.imag], dim=1).contiguous()
    acc = torch.zeros((lmax + 1, 4 * R, nr), dtype=torch.float64, device="cuda")
    for l0, lam in _lambda_blocks(lmax, s, theta, _block(lmax, nr)):
        acc.baddbmm_(w[:, :, l0:l0 + lam.shape[1]].contiguous(), lam)
    hp = torch.complex(acc[:, :R], acc[:, R:2 * R]).permute(1, 0, 2)
    hm = torch.complex(acc[:, 2 * R:3 * R], acc[:, 3 * R:]).permute(1, 0, 2).flip(2)
    return torch.cat([hm[:, 1:].flip(1), hp], dim=1)


def _legendre_adjoint(h, lmax, s, theta, ncomp):
    """The adjoint of _legendre: (R, 2 lmax + 1, ring) -> (R, ncomp, nalm)."""
    R, nr = h.shape[0], theta.numel()
    hp = h[:, lmax:].permute(1, 0, 2)                       # (m, R, ring)
    hm = h[:, :lmax + 1].flip(1).flip(2).permute(1, 0, 2)   # order -m, rings mirrored
    w = torch.cat([hp.real, hp.imag, hm.real, hm.imag], dim=1).contiguous()
    out = torch.zeros((lmax + 1, 4 * R, lmax + 1), dtype=torch.float64, device="cuda")
    for l0, lam in _lambda_blocks(lmax, s, theta, _block(lmax, nr)):
        out[:, :, l0:l0 + lam.shape[1]] = torch.bmm(w, lam.transpose(1, 2))
    i = torch.arange(lmax + 1, device="cuda")
    par = (1.0 - 2.0 * ((i[:, None] + i[None]) % 2))[:, None]
    p = torch.complex(out[:, :R], out[:, R:2 * R])
    q = (torch.complex(out[:, 2 * R:3 * R], out[:, 3 * R:]) * par).conj()
    if s == 0:
        res = [p]
    else:
        q = (-1) ** s * q
        g, c = -0.5 * (p + q), 0.5j * (p - q)
        g[0], c[0] = -p[0].real + 0j, -p[0].imag + 0j
        res = [g, c][:ncomp]
    l, m = _lm(lmax)
    return torch.stack([r.permute(1, 0, 2)[..., m, l] for r in res], dim=1)


def _ring_phase(lmax, ph0):
    m = torch.arange(-lmax, lmax + 1, dtype=torch.float64, device="cuda")
    return torch.exp(1j * m[:, None] * torch.as_tensor(ph0, device="cuda")[None])


def _ring_synth(h, case):
    """Columns -> pixels, complex (R, npix)."""
    lmax, (_, ph0, nph) = case["lmax"], _rings(case)
    h = h * _ring_phase(lmax, ph0)
    m = torch.arange(-lmax, lmax + 1, device="cuda")
    start = np.concatenate([[0], np.cumsum(nph)])
    out = torch.empty((h.shape[0], int(start[-1])), dtype=C128, device="cuda")
    for n in np.unique(nph):
        which = np.nonzero(nph == n)[0]
        bins = torch.zeros((h.shape[0], int(n), which.size), dtype=C128, device="cuda")
        bins.index_add_(1, m % int(n), h[:, :, torch.as_tensor(which, device="cuda")])
        z = torch.fft.ifft(bins, dim=1, norm="forward").transpose(1, 2)
        px = torch.as_tensor(start[which], device="cuda")[:, None] + torch.arange(int(n), device="cuda")
        out[:, px] = z
    return out


def _ring_adjoint(z, case, weight=None):
    """The adjoint of _ring_synth for rings of one length."""
    lmax, (_, ph0, nph) = case["lmax"], _rings(case)
    f = torch.fft.fft(z.reshape(z.shape[0], nph.size, int(nph[0])), dim=2)
    m = torch.arange(-lmax, lmax + 1, device="cuda")
    h = f[:, :, m % int(nph[0])].transpose(1, 2) * _ring_phase(lmax, ph0).conj()
    return h if weight is None else h * weight


_W, _BETA = 14, 2.30 * 14


def _torus(lmax):
    n = 2 * lmax + 2
    while not _smooth(n):
        n += 2
    return n


def _smooth(n):
    for p in (2, 3, 5, 7):
        while n % p == 0:
            n //= p
    return n == 1


def _deconv(lmax, n):
    """1 / kernel transform at the frequencies -lmax .. lmax of an n-point axis."""
    z, wz = np.polynomial.legendre.leggauss(200)
    k = 2 * np.pi * np.arange(-lmax, lmax + 1) / n
    psi = wz * np.exp(_BETA * (np.sqrt(1 - z * z) - 1))
    return torch.as_tensor(1.0 / (0.5 * _W * (np.cos(np.outer(k, 0.5 * _W * z)) @ psi)), device="cuda")


def _taps(t, n):
    """First grid index and the weights of each point on an n-point periodic axis."""
    x = t * (n / (2 * math.pi))
    i0 = torch.ceil(x - 0.5 * _W)
    z = (i0[:, None] + torch.arange(_W, device="cuda") - x[:, None]) * (2.0 / _W)
    w = torch.exp(_BETA * (torch.sqrt(torch.clamp(1 - z * z, min=0)) - 1))
    idx = (i0.long()[:, None] + torch.arange(_W, device="cuda")) % n
    return idx, w


_CHUNK = 1 << 19


def _type2(h, lmax, s, theta, phi):
    """Columns (2 lmax + 1, nt / 2 + 1) on the rings 2 pi k / nt -> complex values at the points."""
    nt, n = _torus(lmax), 2 * _torus(lmax)
    m = torch.arange(-lmax, lmax + 1, device="cuda")
    sg = (1.0 - 2.0 * ((m + s) % 2))[:, None]
    c = torch.fft.fft(torch.cat([h, sg * h[:, 1:-1].flip(1)], dim=1), dim=1, norm="forward")
    d = _deconv(lmax, n)
    c = c[:, m % nt] * d[:, None] * d[None]
    spec = torch.zeros((n, n), dtype=C128, device="cuda")
    spec[(m % n)[:, None], (m % n)[None]] = c.T.contiguous()
    u = torch.fft.ifft2(spec, norm="forward").reshape(-1)
    del spec, c
    out = torch.empty(theta.numel(), dtype=C128, device="cuda")
    for a in range(0, theta.numel(), _CHUNK):
        it, wt = _taps(theta[a:a + _CHUNK], n)
        ip, wp = _taps(phi[a:a + _CHUNK], n)
        v = u[(it[:, :, None] * n + ip[:, None, :])]
        out[a:a + _CHUNK] = torch.einsum("pi,pij,pj->p", wt.to(C128), v, wp.to(C128))
    return out


def _type1(z, lmax, s, theta, phi):
    """The adjoint of _type2."""
    nt, n = _torus(lmax), 2 * _torus(lmax)
    m = torch.arange(-lmax, lmax + 1, device="cuda")
    u = torch.zeros((2, n * n), dtype=torch.float64, device="cuda")
    for a in range(0, theta.numel(), _CHUNK):
        it, wt = _taps(theta[a:a + _CHUNK], n)
        ip, wp = _taps(phi[a:a + _CHUNK], n)
        at = (it[:, :, None] * n + ip[:, None, :]).reshape(-1)
        w = wt[:, :, None] * wp[:, None, :]
        for k, v in enumerate((z.real, z.imag)):
            u[k].index_add_(0, at, (w * v[a:a + _CHUNK, None, None]).reshape(-1))
    f = torch.fft.fft2(torch.complex(u[0], u[1]).reshape(n, n))
    d = _deconv(lmax, n)
    c = f[(m % n)[:, None], (m % n)[None]].T * d[:, None] * d[None]
    spec = torch.zeros((2 * lmax + 1, nt), dtype=C128, device="cuda")
    spec[:, m % nt] = c
    g = torch.fft.ifft(spec, dim=1)
    h = g[:, :nt // 2 + 1].clone()
    sg = (1.0 - 2.0 * ((m + s) % 2))[:, None]
    h[:, 1:-1] += sg * g[:, nt // 2 + 1:].flip(1)
    return h


def _cc_theta(lmax):
    nt = _torus(lmax)
    return 2 * math.pi * torch.arange(nt // 2 + 1, dtype=torch.float64, device="cuda") / nt


def _synth_at(alm, lmax, s, theta, phi):
    return _type2(_legendre(alm[None], lmax, s, _cc_theta(lmax))[0], lmax, s, theta, phi)


def _adjoint_at(z, lmax, s, theta, phi, ncomp):
    return _legendre_adjoint(_type1(z, lmax, s, theta, phi)[None], lmax, s, _cc_theta(lmax), ncomp)[0]


def _pixels(case):
    th, ph0, nph = _rings(case)
    th = torch.repeat_interleave(th, torch.as_tensor(nph, device="cuda"))
    start = np.concatenate([[0], np.cumsum(nph)])[:-1]
    p = torch.arange(th.numel(), device="cuda") - torch.repeat_interleave(torch.as_tensor(start, device="cuda"), torch.as_tensor(nph, device="cuda"))
    rep = lambda v: torch.repeat_interleave(torch.as_tensor(v, dtype=torch.float64, device="cuda"), torch.as_tensor(nph, device="cuda"))  # noqa: E731
    return th, rep(ph0) + 2 * math.pi * p.double() / rep(nph)


def _move(th, ph, dth, dph):
    """End point of the geodesic of length |d| from (th, ph) along (dth, dph)."""
    a = torch.sqrt(dth * dth + dph * dph)
    sinc, cosa, st, ct = torch.sin(a) / a, torch.cos(a), torch.sin(th), torch.cos(th)
    nx, ny, nz = st * cosa + ct * dth * sinc, -dph * sinc, ct * cosa - st * dth * sinc
    p = ph - torch.atan2(ny, nx)
    return torch.atan2(torch.sqrt(nx * nx + ny * ny), nz), torch.where(p >= 2 * math.pi, p - 2 * math.pi, p)


def _deflection(d, c, case):
    """(dth, dph) of R requests on the geometry's pixels."""
    lmax = case["lmax"]
    f = _grad_factor(lmax)
    alm = d.to(C128)[:, None] * f
    if c is not None:
        alm = torch.cat([alm, c.to(C128)[:, None] * f], dim=1)
    z = _ring_synth(_legendre(alm, lmax, 1, _rings(case)[0]), case)
    return z.real, z.imag


def _gamma(th, dth, dph):
    a = torch.sqrt(dth * dth + dph * dph)
    return torch.atan2(dph, dth) - torch.atan2(dph, a * torch.sin(a) / torch.tan(th) + dth * torch.cos(a))


def _map_of(z, spin):
    return torch.stack([z.real, z.imag]) if spin else z.real


def exact(case, seed):
    s = _inputs(case, seed)
    op, lmax, spin = case["op"], case["lmax"], case.get("spin", 0)
    ncomp = 2 if spin else 1
    if op in ("nusht2d2", "nusht2d1"):
        th, ph = s["loc"].T.contiguous()
        if op == "nusht2d2":
            return _map_of(_synth_at(s["g"].reshape(ncomp, -1), lmax, spin, th, ph), spin)
        m = s["map"].double()
        r = _adjoint_at(torch.complex(m[0], m[1]) if spin else m.to(C128), lmax, spin, th, ph, ncomp)
        return r if spin else r[0]
    if op in ("alm2map", "map2alm"):
        theta, w = _gl(lmax + 1)
        n = _nphi(case)
        if op == "alm2map":
            z = _ring_synth(_legendre(s["g"].reshape(1, ncomp, -1), lmax, spin, theta), case)[0]
            return _map_of(z.reshape(lmax + 1, n).T.reshape(-1), spin)
        m = s["map"].reshape(ncomp, n, lmax + 1).transpose(1, 2).reshape(ncomp, -1)
        z = (torch.complex(m[0], m[1]) if spin else m[0].to(C128))[None]
        return _legendre_adjoint(_ring_adjoint(z, case, w * (2 * math.pi / n)), lmax, spin, theta, ncomp)[0]
    batch = op in ("lens_batch", "delens_batch")
    th, ph = _pixels(case)
    d = s["d"] if batch else s["d"][None]
    dth, dph = _deflection(d, None if s.get("c") is None else s["c"][None], case)
    if op == "pointing":
        return {"ptg": torch.stack(_move(th, ph, dth[0], dph[0])), "gamma": _gamma(th, dth[0], dph[0])}
    if op == "grad":
        return _exact_grad(s, case, th, ph, dth[0], dph[0])
    if op in ("lens", "lens_batch"):
        h = _legendre((s["g"] if batch else s["g"][None]).reshape(d.shape[0], ncomp, -1), lmax, spin, _cc_theta(lmax))
    res = []
    for r in range(d.shape[0]):
        t, p = _move(th, ph, dth[r], dph[r])
        rot = torch.exp(1j * spin * _gamma(th, dth[r], dph[r]))
        if op in ("lens", "lens_batch"):
            res.append(_map_of(_type2(h[r], lmax, spin, t, p) * rot, spin))
        else:
            m = (s["map"][r] if batch else s["map"]).double()
            z = torch.complex(m[0], m[1]) * rot.conj() if spin else m.to(C128)
            res.append(_type1(z, lmax, spin, t, p))
    if op in ("delens", "delens_batch"):
        res = _legendre_adjoint(torch.stack(res), lmax, spin, _cc_theta(lmax), ncomp)
        return res if batch else (res[0] if spin else res[0, 0])
    return torch.stack(res) if batch else res[0]


def _exact_grad(s, case, th, ph, dth, dph):
    """lenmap and the gradients (dL/dRe + i dL/dIm) of sum (lenmap - map)^2."""
    lmax = case["lmax"]
    _, m = _lm(lmax)
    f = _grad_factor(lmax)
    t, p = _move(th, ph, dth, dph)
    g = s["g"].detach().reshape(1, -1)
    out = _synth_at(g, lmax, 0, t, p).real
    v = 2.0 * (out - s["map"])

    def grad_of(a):
        a = a * torch.where(m > 0, 2.0, 1.0)
        return torch.where(m > 0, a, a.real + 0j)

    gg = grad_of(_adjoint_at(v.to(C128), lmax, 0, t, p, 1)[0])
    slope = _synth_at(g * f, lmax, 1, t, p)  # (d/dtheta, 1/sin d/dphi) at the moved points
    x, y = dth.clone().requires_grad_(True), dph.clone().requires_grad_(True)
    with torch.enable_grad():
        t2, p2 = _move(th, ph, x, y)
        gx, gy = torch.autograd.grad((t2, p2), (x, y), (v * slope.real, v * slope.imag * torch.sin(t)))
    h = _ring_adjoint(torch.complex(gx, gy)[None], case)
    gd = grad_of(_legendre_adjoint(h, lmax, 1, _rings(case)[0], 1)[0, 0] * f)
    return {"lenmap": out, "grad_g": gg, "grad_d": gd}
