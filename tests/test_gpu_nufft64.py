"""FP64 plans: kernel weights from double-float arithmetic (widths up to 12,
eps >= 1e-10) and from FP64 functions (above), against the exact direct sum;
pointing increments from their series and from atan2.

Tolerances: the nuFFT's eps (its kernel width is one above the rule for eps);
pointing 4 ulp of 2 pi, divided by sin(theta') for the longitude."""
import numpy as np
import pytest

import oracle
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("eps", [1e-3, 1e-7, 1e-10, 9e-11, 1e-12])
@pytest.mark.parametrize("spin", [0, 2])
def test_weights_both_sides_of_the_width_limit(built_lib, eps, spin):
    import cunusht_gb300 as cu
    lmax = 24
    rng = np.random.default_rng(4)
    th = np.concatenate([rng.uniform(0, np.pi, 995), [0.0, np.pi, 1e-9, np.pi / 2, 1.0]])
    ph = np.concatenate([rng.uniform(0, 2 * np.pi, 995), [0.0, 0.0, 6.283185307179586, np.pi, -3.0]])
    alm, _ = orc.make_inputs(lmax, spin, seed=9)
    t = cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=eps, precision="fp64")
    loc = torch.as_tensor(np.stack([th, ph], 1), device="cuda")
    a = torch.as_tensor(alm if spin else alm[0], device="cuda")
    got = t.nusht2d2(lmax, lmax, a, loc, spin=spin).cpu().numpy()
    ref = oracle.synth_points_c(lmax, spin, alm if spin else alm[0], th, ph)
    assert np.linalg.norm(got - ref) <= eps * np.linalg.norm(ref)
    v = rng.standard_normal((2, th.size) if spin else th.size)
    got = t.nusht2d1(lmax, lmax, torch.as_tensor(v, device="cuda"), loc, spin=spin).cpu().numpy()
    ref = orc.adjoint_synth_points(lmax, spin, v, th, ph)
    assert np.linalg.norm(got - ref) <= eps * np.linalg.norm(ref)


@pytest.mark.parametrize("rms", [1e-6, 7e-4, 0.05, 0.4])
def test_pointing_series_and_large_angles(built_lib, rms):
    """Deflections below and above the series limits, rings next to the poles included."""
    import cunusht_gb300 as cu
    lmax = 96
    t = cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=1e-10, precision="fp64")
    gen = np.random.default_rng(int(rms * 1e7))
    n = t.nalm
    p = gen.standard_normal(n) + 1j * gen.standard_normal(n)
    p[:lmax + 1] = p[:lmax + 1].real
    ll = np.arange(lmax + 1.0)
    p = orc.almxfl(p, rms / (ll + 1.0) ** 2, lmax)
    th, ph = t.geom.pixels()
    d = t.synthesis(torch.as_tensor(orc.almxfl(p, np.sqrt(ll * (ll + 1)), lmax)[None], device="cuda"), spin=1).cpu().numpy()
    got = t.dlm2pointing(torch.as_tensor(p, device="cuda"), lmax).cpu().numpy()
    gam = t.gamma.cpu().numpy()
    rt, rp = orc.pointing(th, ph, d[0], d[1])
    ulp = 4 * np.spacing(2 * np.pi)
    assert np.max(np.abs(got[0] - rt)) < ulp
    dp = np.remainder(got[1] - rp + np.pi, 2 * np.pi) - np.pi
    assert np.max(np.abs(dp) * np.sin(rt)) < 4 * ulp
    g = orc.rotation_gamma(th, d[0], d[1])
    dg = np.remainder(gam - g + np.pi, 2 * np.pi) - np.pi
    # the two arctangents of the reference formula cancel where gamma is small
    assert np.max(np.abs(dg) * np.sin(th)) < 32 * ulp


@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("eps", [1e-6, 1e-7])
@pytest.mark.parametrize("step", [0.0, 0.7, 1.0, 2.0, 2.6])
def test_mixed_strip_spreading(built_lib, eps, spin, step):
    """Strips of a mixed plan with an FP64 grid: neighbours ``step`` fine cells apart (repeated
    points, odd and even columns, the wrap of the longitude), a partial last warp and values of
    very different size, zero and both signs included (every way a strip cell is added to the grid).

    Tolerance: eps, and four roundings of FP32 (the two weights, their products)."""
    import cunusht_gb300 as cu
    lmax, n = 24, 32 * 9 + 5
    rng = np.random.default_rng(12)
    k = np.arange(n)
    th = 1.1 + 0.01 * (k // 96) + 0.002 * np.sin(k)
    ph = np.remainder(6.2 + k * step * 2 * np.pi / 108, 2 * np.pi)
    v = rng.standard_normal((2, n) if spin else n)
    v = v * 10.0 ** rng.integers(-14, 1, v.shape)
    v[..., 5::17] = 0.0
    t = cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=eps, precision="mixed")
    loc = torch.as_tensor(np.stack([th, ph], 1), device="cuda")
    got = t.nusht2d1(lmax, lmax, torch.as_tensor(v, device="cuda"), loc, spin=spin).cpu().numpy()
    ref = orc.adjoint_synth_points(lmax, spin, v, th, ph)
    assert np.linalg.norm(got - ref) <= (eps + 4 * 2.0 ** -24) * np.linalg.norm(ref)
