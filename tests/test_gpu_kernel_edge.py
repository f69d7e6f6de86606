"""Points that lie exactly on the fine grid: a tap at |z| = 1 has weight and
derivative 0 (the kernel's support is open), in double-float as in FP64.  phi = 0
is a grid column for every size; the tap at the edge exists for even widths w
(eps 1e-4, 1e-8, 1e-10: w = 6, 10, 12)."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _plan(lmax, eps, precision="fp64"):
    import cunusht_gb300 as cu
    return cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=eps, precision=precision, max_spin=2)


def _alm(lmax, seed):
    import cunusht_gb300 as cu
    gen = torch.Generator(device="cuda").manual_seed(seed)
    a = torch.randn(cu.Alm.getsize(lmax, lmax), dtype=torch.complex128, device="cuda", generator=gen)
    a[:lmax + 1] = a[:lmax + 1].real + 0j
    return a


def _grad(t, lmax):
    from cunusht_gb300 import autograd
    g = _alm(lmax, 1).requires_grad_(True)
    d = torch.zeros_like(g).requires_grad_(True)
    target = torch.cos(torch.arange(t.npix(), dtype=torch.float64, device="cuda"))
    loss = torch.sum(autograd.gclm2lenmap(t, g, d, 0) * target)
    return torch.autograd.grad(loss, d)[0]


@pytest.mark.parametrize("lmax", [20, 64, 130])
@pytest.mark.parametrize("eps", [1e-4, 1e-8, 1e-10])
def test_deflection_gradient_at_zero_deflection(built_lib, lmax, eps):
    """The first pixel of every ring stays at phi = 0.  Against width 15 (FP64
    weights); the derivative of the kernel carries its error times beta and the
    grid's spacing against the field's, below 100 eps."""
    x, ref = _grad(_plan(lmax, eps), lmax), _grad(_plan(lmax, 1e-13), lmax)
    assert float((x - ref).norm() / ref.norm()) < 100 * eps


@pytest.mark.parametrize("eps", [1e-4, 1e-8, 1e-10])
@pytest.mark.parametrize("spin", [0, 2])
def test_spreading_from_grid_columns(built_lib, eps, spin):
    """Strips (double-float weights, 2.4e-14) against the bin-sorted method (FP64
    weights) for points at phi = 0: e^-beta, 1e-6 at w = 6, were the edge tap to count."""
    lmax = 40
    t = _plan(lmax, eps)
    n = 300
    loc = torch.zeros((n, 2), dtype=torch.float64, device="cuda")
    loc[:, 0] = torch.linspace(0.01, 3.13, n, dtype=torch.float64, device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(2)
    v = torch.randn((2, n) if spin else (n,), dtype=torch.float64, device="cuda", generator=gen)
    x = t.nusht2d1(lmax, lmax, v, loc, spin=spin).clone()
    t.set_spreading("bins", max_points=n)
    y = t.nusht2d1(lmax, lmax, v, loc, spin=spin)
    assert float((x - y).norm() / y.norm()) < 1e-12


# rings whose pixels all lie on grid columns, up to rounding
@pytest.mark.parametrize("geom", [("gl", {"lmax": 63, "nphi": 128}), ("healpix", {"nside": 32, "lmax": 64}),
                                  ("f1", {"ntheta": 70, "nphi": 128, "lmax": 63})])
@pytest.mark.parametrize("eps", [1e-4, 1e-6, 1e-8, 1e-10, 1e-12])
def test_deflection_gradient_on_aligned_rings(built_lib, geom, eps):
    """Zero deflection: every pixel stays on a column, its edge tap within the
    rounding of phi of |z| = 1 (widths 6 to 14; the last has FP64 weights)."""
    import cunusht_gb300 as cu
    lmax = geom[1]["lmax"]
    x, ref = [_grad(cu.get_transformer("GPU")(geom, nuFFTtype=2, epsilon=e, precision="fp64", max_spin=2), lmax)
              for e in (eps, 1e-13)]
    assert float((x - ref).norm() / ref.norm()) < 100 * eps
