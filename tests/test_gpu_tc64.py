"""Legendre stages of FP64 plans on the tensor cores (legendre_tc64.cu) against
the FP64 CUDA-core kernels (cunusht_plan_set_tensor_cores(plan, 0)).

Tolerance: the CUDA-core start values carry |log2 start| ln 2 2^-53 with
|log2| up to about 3 lmax where the functions matter, and the recursion adds
2^-53 sqrt(lmax) of the bounds: 8 (lmax + 16) 2^-53 covers both."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _tol(lmax):
    return 8.0 * (lmax + 16) * 2.0 ** -53


def _plan(lmax, geom=None, max_spin=2, eps=1e-10):
    import cunusht_gb300 as cu
    return cu.get_transformer("GPU")(geom or ("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=eps, precision="fp64",
                                     max_spin=max_spin)


def _alm(lmax, mmax, spin, seed):
    import cunusht_gb300 as cu
    gen = torch.Generator(device="cuda").manual_seed(seed)
    n = cu.Alm.getsize(lmax, mmax)
    a = torch.randn((2, n) if spin else (n,), dtype=torch.complex128, device="cuda", generator=gen)
    a[..., :lmax + 1] = a[..., :lmax + 1].real + 0j
    return a


def _both(t, fn):
    """fn() on the tensor cores and on the CUDA cores; the device status stays 0."""
    from cunusht_gb300 import _lib
    out = []
    for on in (1, 0):
        _lib.check(t._lib.cunusht_plan_set_tensor_cores(t._plan, on))
        out.append(fn())
        st = ctypes.c_int(-1)
        _lib.check(t._lib.cunusht_plan_device_status(t._plan, ctypes.byref(st)))
        assert st.value == 0
    return out


def _rel(a, b):
    return float((a - b).norm() / b.norm())


# windows of 128 l, chunks of 8 and 16 l, blocks of 256 / 512 ring pairs and tails of fewer than 32
SIZES = [3, 7, 8, 9, 127, 128, 130, 300, 515, 1030]


@pytest.mark.parametrize("lmax", SIZES)
@pytest.mark.parametrize("spin", [0, 1, 2])
def test_synthesis(built_lib, lmax, spin):
    t = _plan(lmax)
    a = _alm(lmax, lmax, spin, lmax)
    x, y = _both(t, lambda: t.synthesis(a, spin=spin))  # Gauss-Legendre rings
    assert _rel(x, y) < _tol(lmax)
    loc = t.get_grid_uniform().t().contiguous()[:20001]
    x, y = _both(t, lambda: t.nusht2d2(lmax, lmax, a, loc, spin=spin))  # Clenshaw-Curtis rings, pole pair
    assert _rel(x, y) < _tol(lmax)


@pytest.mark.parametrize("spin,mmax", [(0, 17), (0, 0), (1, 0), (2, 1), (2, 120)])
def test_synthesis_truncated_m(built_lib, spin, mmax):
    lmax = 300
    t = _plan(lmax)
    a = _alm(lmax, mmax, spin, 3)
    x, y = _both(t, lambda: t.synthesis(a, lmax=lmax, mmax=mmax, spin=spin))
    assert _rel(x, y) < _tol(lmax)


def test_synthesis_healpix_and_missing_start_table(built_lib):
    """HEALPix rings; and a spin above the plan's (GL start states not stored:
    the kernel evaluates the starts itself)."""
    t = _plan(200, ("healpix", {"nside": 128, "lmax": 200}))
    for spin in (0, 2):
        a = _alm(200, 200, spin, 5)
        x, y = _both(t, lambda: t.synthesis(a, spin=spin))
        assert _rel(x, y) < _tol(200)
    t = _plan(260, max_spin=0)
    a = _alm(260, 260, 2, 6)
    x, y = _both(t, lambda: t.synthesis(a, spin=2))
    assert _rel(x, y) < _tol(260)


@pytest.mark.parametrize("scale", [1e-290, 1e-40, 1e250])
def test_synthesis_scales(built_lib, scale):
    """The digit exponents follow the alm over the FP64 range."""
    t = _plan(150)
    a = _alm(150, 150, 2, 7) * scale
    x, y = _both(t, lambda: t.synthesis(a, spin=2))
    assert _rel(x / scale, y / scale) < _tol(150)


def test_synthesis_zero_and_not_finite(built_lib):
    t = _plan(150)
    a = _alm(150, 150, 0, 8)
    assert float(t.synthesis(torch.zeros_like(a)).abs().max()) == 0.0
    for bad in (float("nan"), float("inf")):
        b = a.clone()
        b[40] = bad
        assert bool(torch.isnan(t.synthesis(b)).any())


@pytest.mark.parametrize("lmax", SIZES)
@pytest.mark.parametrize("spin", [0, 1, 2])
def test_adjoint(built_lib, lmax, spin):
    t = _plan(lmax)
    gen = torch.Generator(device="cuda").manual_seed(lmax)
    n = t.npix()
    v = torch.randn((2, n) if spin else (n,), dtype=torch.float64, device="cuda", generator=gen)
    x, y = _both(t, lambda: t.adjoint_synthesis(v, spin=spin))
    assert _rel(x, y) < _tol(lmax)
    loc = t.get_grid_uniform().t().contiguous()
    x, y = _both(t, lambda: t.nusht2d1(lmax, lmax, v, loc, spin=spin))  # Clenshaw-Curtis rings, pole pair
    assert _rel(x, y) < _tol(lmax)
    if spin:  # gradient alm alone
        x, y = _both(t, lambda: t.adjoint_synthesis(v, spin=spin, ncomp=1))
        assert _rel(x, y) < _tol(lmax)


@pytest.mark.parametrize("spin,mmax", [(0, 17), (0, 0), (1, 0), (2, 1), (2, 120)])
def test_adjoint_truncated_m(built_lib, spin, mmax):
    lmax = 300
    t = _plan(lmax)
    gen = torch.Generator(device="cuda").manual_seed(4)
    n = t.npix()
    v = torch.randn((2, n) if spin else (n,), dtype=torch.float64, device="cuda", generator=gen)
    x, y = _both(t, lambda: t.adjoint_synthesis(v, lmax=lmax, mmax=mmax, spin=spin))
    assert _rel(x, y) < _tol(lmax)


def test_adjoint_healpix_scales_zero_not_finite(built_lib):
    t = _plan(200, ("healpix", {"nside": 128, "lmax": 200}))
    gen = torch.Generator(device="cuda").manual_seed(5)
    for spin in (0, 2):
        v = torch.randn((2, t.npix()) if spin else (t.npix(),), dtype=torch.float64, device="cuda", generator=gen)
        for scale in (1e-290, 1.0, 1e250):
            x, y = _both(t, lambda: t.adjoint_synthesis(v * scale, spin=spin))
            assert _rel(x / scale, y / scale) < _tol(200)
        assert float(t.adjoint_synthesis(torch.zeros_like(v), spin=spin).abs().max()) == 0.0
        v.reshape(-1)[1000] = float("nan")
        assert bool(torch.isnan(t.adjoint_synthesis(v, spin=spin).real).any())
