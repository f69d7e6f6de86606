"""Adjoint ring transform of uniform rings by mixed radices (csrc/ring_mr.cu)
against the Bluestein form of the same plan: rings shorter and longer than
2 lmax + 1, weights (map2alm's analysis), every spin.  The two differ only in
the rounding of FP64 transforms: 1e-12 relative."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("lmax,nphi", [(31, 33), (31, 64), (31, 105), (40, 81), (200, 450), (300, 1024)])
@pytest.mark.parametrize("spin", [0, 1, 2])
def test_adjoint_matches_bluestein(built_lib, lmax, nphi, spin):
    import cunusht_gb300 as cu
    from cunusht_gb300 import _lib
    t = cu.get_transformer("GPU", mode="SHT")(("gl", {"lmax": lmax, "nphi": nphi}))
    gen = torch.Generator(device="cuda").manual_seed(nphi)
    m = torch.randn((2, t.npix()) if spin else (t.npix(),), dtype=torch.float64, device="cuda", generator=gen)
    assert t._lib.cunusht_plan_ring_transform(t._plan) == 0
    calls = (lambda: t.map2alm(m, spin=spin),
             lambda: cu.get_transformer("GPU").adjoint_synthesis(t, m, lmax=lmax, mmax=lmax, spin=spin))
    got = [f() for f in calls]
    _lib.check(t._lib.cunusht_plan_set_ring_transform(t._plan, 1))
    for x, f in zip(got, calls):
        y = f()
        assert float((x - y).norm() / y.norm()) < 1e-12
