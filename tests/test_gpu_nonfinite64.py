"""FP64 plans: values that are not finite, on the tensor cores and on the CUDA
cores.  Rings and l that a block of rings skips (functions below 2^-64 of their
bound) take part in the product on the CUDA cores down to 2^-312, so whatever is
not finite there must not be finite on the tensor cores either."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _both(t, fn):
    from cunusht_gb300 import _lib
    out = []
    for on in (1, 0):
        _lib.check(t._lib.cunusht_plan_set_tensor_cores(t._plan, on))
        out.append(~torch.isfinite(fn()))
    return out


def _plan(lmax):
    import cunusht_gb300 as cu
    return cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=1e-10, precision="fp64", max_spin=2)


# one, two to three, and five blocks of rings
@pytest.mark.parametrize("lmax", [200, 530, 1030])
@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_map(built_lib, lmax, spin, bad):
    t = _plan(lmax)
    n = t.npix()
    for pixel in (5, n // 4, n // 2):  # first ring, mid-latitude, equator
        v = torch.ones((2, n) if spin else (n,), dtype=torch.float64, device="cuda")
        v[..., pixel] = bad
        x, y = _both(t, lambda: t.adjoint_synthesis(v, spin=spin))
        assert bool(y.any()) and bool((x | ~y).all())


@pytest.mark.parametrize("lmax", [200, 530, 1030])
@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("bad", [float("nan"), float("inf")])
def test_alm(built_lib, lmax, spin, bad):
    import cunusht_gb300 as cu
    t = _plan(lmax)
    for l, m in ((lmax, lmax), (lmax, lmax // 2), (lmax // 2 + 9, lmax // 2), (3, 2)):
        a = torch.ones((2, cu.Alm.getsize(lmax, lmax)) if spin else (cu.Alm.getsize(lmax, lmax),), dtype=torch.complex128,
                       device="cuda")
        a[..., m * (2 * lmax + 1 - m) // 2 + l] = bad
        x, y = _both(t, lambda: t.synthesis(a, spin=spin))
        assert bool(y.any()) and bool((x | ~y).all())
