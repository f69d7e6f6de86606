"""A lensing request alone gives bit for bit what it gives in a batch: its
transforms of up to 2048 points run in blocks of 512 threads alone and of 128 in
a launch with many columns, by the same operations, and no later stage mixes
requests or uses atomics."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("lmax,nb", [(127, 16), (255, 8), (300, 8), (511, 8)])
@pytest.mark.parametrize("spin", [0, 2])
@pytest.mark.parametrize("eps,precision", [(1e-4, "mixed"), (1e-7, "mixed"), (1e-8, "fp64")])
def test_alone_equals_batched(built_lib, lmax, nb, spin, eps, precision):
    import cunusht_gb300 as cu
    t = cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=eps, precision=precision, max_spin=spin)
    t.reserve_batch(nb)
    gen = torch.Generator(device="cuda").manual_seed(lmax)
    g = torch.randn((nb, 2 if spin else 1, t.nalm), dtype=torch.complex128, device="cuda", generator=gen)
    d = torch.randn((nb, t.nalm), dtype=torch.complex128, device="cuda", generator=gen) * 1e-6 / t.nalm ** 0.5
    many = t.lensing_batch(g, d, spin).clone()
    for i in range(0, nb, 3):
        assert torch.equal(t.lensing_batch(g[i:i + 1], d[i:i + 1], spin)[0], many[i])
