"""Transforms of up to 2048 points in small blocks (launches of many columns or
rows) against the large blocks of a single request.

Tolerance: FP32 grids a few roundings of 2^-24 of the grid's norm, FP64 ones of
2^-53 through two transforms of 2^11 points."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("lmax,nb", [(127, 16), (200, 8), (255, 8), (511, 4)])
@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("eps,prec,tol", [(1e-4, "mixed", 4 * 2.0 ** -24), (1e-7, "mixed", 4 * 2.0 ** -24),
                                          (1e-8, "fp64", 64 * 2.0 ** -53)])
def test_small_blocks_match_large_ones(built_lib, lmax, nb, spin, eps, prec, tol):
    import cunusht_gb300 as cu
    t = cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=eps, precision=prec, max_spin=spin)
    t.reserve_batch(nb)
    gen = torch.Generator(device="cuda").manual_seed(3)
    shape = (nb, 2 if spin else 1, t.nalm)
    g = torch.randn(shape, dtype=torch.complex128, device="cuda", generator=gen)
    d = torch.randn((nb, t.nalm), dtype=torch.complex128, device="cuda", generator=gen) * 1e-6 / t.nalm ** 0.5
    many = t.lensing_batch(g, d, spin)
    m = torch.randn(many.shape, dtype=torch.float64, device="cuda", generator=gen)
    back = t.delensing_batch(m, d, spin)
    for i in (0, nb - 1):
        one = t.lensing_batch(g[i:i + 1], d[i:i + 1], spin)
        assert torch.linalg.norm(many[i] - one[0]) <= tol * torch.linalg.norm(one)
        one = t.delensing_batch(m[i:i + 1], d[i:i + 1], spin)
        assert torch.linalg.norm(back[i] - one[0]) <= tol * torch.linalg.norm(one)
