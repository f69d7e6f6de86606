"""FP64 plans' Legendre stages where the kernel or the block changes: spin 0
from lmax 96 on the tensor cores, and last blocks of one ring pair and of few."""
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _tol(lmax):
    """As between the tensor-core and the CUDA-core form: start values of
    either carry |log2 start| ln 2 2^-53, the recursion adds 2^-53 sqrt(lmax)."""
    return 8.0 * (lmax + 16) * 2.0 ** -53


def _plan(lmax):
    import cunusht_gb300 as cu
    return cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=1e-10, precision="fp64", max_spin=2)


def _inputs(t, lmax, spin):
    import cunusht_gb300 as cu
    gen = torch.Generator(device="cuda").manual_seed(lmax)
    shape = (2,) if spin else ()
    a = torch.randn(shape + (cu.Alm.getsize(lmax, lmax),), dtype=torch.complex128, device="cuda", generator=gen)
    a[..., :lmax + 1] = a[..., :lmax + 1].real + 0j
    return a, torch.randn(shape + (t.npix(),), dtype=torch.float64, device="cuda", generator=gen)


def _both(t, fn):
    from cunusht_gb300 import _lib
    out = []
    for on in (1, 0):
        _lib.check(t._lib.cunusht_plan_set_tensor_cores(t._plan, on))
        out.append(fn())
    return out


def _rel(a, b):
    return float((a - b).norm() / b.norm())


@pytest.mark.parametrize("lmax", [31, 95, 96, 97])
def test_spin0_threshold_against_the_oracle(built_lib, lmax):
    import oracle
    t = _plan(lmax)
    a, v = _inputs(t, lmax, 0)
    th, ph = t.get_grid_uniform().cpu().numpy()
    ref = torch.as_tensor(oracle.synth_points_c(lmax, 0, a.cpu().numpy(), th, ph)).cuda().reshape(-1)
    adj = torch.as_tensor(oracle.adjoint_synth_points_c(lmax, 0, v.cpu().numpy(), th, ph, ncomp=1)).cuda().reshape(-1)
    x, y = _both(t, lambda: t.synthesis(a, spin=0))
    assert torch.equal(x, y) == (lmax < 96)  # the CUDA cores whatever the switch says below 96
    assert _rel(x.reshape(-1), ref) < _tol(lmax) and _rel(y.reshape(-1), ref) < _tol(lmax)
    for z in _both(t, lambda: t.adjoint_synthesis(v, spin=0)):
        assert _rel(z.reshape(-1), adj) < _tol(lmax)


# ring pairs lmax / 2 + 1 in blocks of 256 (spin 0) and 128: 1, 2, 31, 32 in the last
@pytest.mark.parametrize("spin,lmax", [(0, 512), (0, 514), (0, 572), (0, 574), (0, 1024), (2, 256), (2, 258), (2, 316),
                                       (2, 318), (2, 512)])
def test_short_last_block(built_lib, spin, lmax):
    t = _plan(lmax)
    a, v = _inputs(t, lmax, spin)
    x, y = _both(t, lambda: t.synthesis(a, spin=spin))
    assert _rel(x, y) < _tol(lmax)
    x, y = _both(t, lambda: t.adjoint_synthesis(v, spin=spin))
    assert _rel(x, y) < _tol(lmax)


@pytest.mark.parametrize("spin", [0, 2])
def test_lmax_4095(built_lib, spin):
    """The largest size of the configurations: 32 windows of 128 l, 8 or 16 blocks of rings."""
    lmax = 4095
    t = _plan(lmax)
    a, v = _inputs(t, lmax, spin)
    x, y = _both(t, lambda: t.synthesis(a, spin=spin))
    assert _rel(x, y) < _tol(lmax)
    x, y = _both(t, lambda: t.adjoint_synthesis(v, spin=spin))
    assert _rel(x, y) < _tol(lmax)
