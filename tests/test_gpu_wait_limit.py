"""FP64 plans' tensor-core Legendre kernels when a bounded wait runs out
(cunusht_plan_set_wait_limit(plan, 0): every wait does, at once)."""
import ctypes

import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _plan(lmax):
    import cunusht_gb300 as cu
    return cu.get_transformer("GPU")(("gl", {"lmax": lmax}), nuFFTtype=2, epsilon=1e-10, precision="fp64", max_spin=2)


def _limit(t, polls):
    from cunusht_gb300 import _lib
    _lib.check(t._lib.cunusht_plan_set_wait_limit(t._plan, polls))


def _status(t):
    from cunusht_gb300 import _lib
    st = ctypes.c_int(-1)
    _lib.check(t._lib.cunusht_plan_device_status(t._plan, ctypes.byref(st)))
    return st.value


def _calls(t, lmax, spin):
    """(name, call) of both directions on both grids (rings; torus with its pole pair)."""
    import cunusht_gb300 as cu
    gen = torch.Generator(device="cuda").manual_seed(lmax + spin)
    shape = (2,) if spin else ()
    a = torch.randn(shape + (cu.Alm.getsize(lmax, lmax),), dtype=torch.complex128, device="cuda", generator=gen)
    a[..., :lmax + 1] = a[..., :lmax + 1].real + 0j
    v = torch.randn(shape + (t.npix(),), dtype=torch.float64, device="cuda", generator=gen)
    loc = t.get_grid_uniform().t().contiguous()
    return [("synthesis", lambda: t.synthesis(a, spin=spin)), ("nusht2d2", lambda: t.nusht2d2(lmax, lmax, a, loc, spin=spin)),
            ("adjoint_synthesis", lambda: t.adjoint_synthesis(v, spin=spin)),
            ("nusht2d1", lambda: t.nusht2d1(lmax, lmax, v, loc, spin=spin))]


# one window of 128 l and several; one block of rings and several
@pytest.mark.parametrize("lmax", [100, 300, 530])
@pytest.mark.parametrize("spin", [0, 2])
def test_block_that_gives_up_waits_for_its_own_copies(built_lib, lmax, spin):
    """The call returns with the status bit set, and the next one, whose blocks
    take the same shared and tensor memory, is right (order of the adjoint's
    atomic additions: 2^-46 of the norm, for sums of up to 2^6 terms per value)."""
    t = _plan(lmax)
    for name, call in _calls(t, lmax, spin):
        ref = call().clone()
        assert _status(t) == 0
        _limit(t, 0)
        call()
        assert _status(t) == 1, name
        _limit(t, 1 << 22)
        for _ in range(3):
            x = call()
            assert float((x - ref).norm() / ref.norm()) < 2.0 ** -50, name
        assert _status(t) == 0


# ring counts without a short tail, whose rings go to the CUDA cores
@pytest.mark.parametrize("lmax", [100, 400, 600])
@pytest.mark.parametrize("spin", [0, 2])
def test_results_of_a_block_that_gives_up_are_not_numbers(built_lib, lmax, spin):
    """Every pixel and every alm (l >= spin) is NaN, also after a call that left
    its numbers in the plan's buffers, and none in the call after it."""
    t = _plan(lmax)
    valid = torch.cat([torch.arange(m, lmax + 1) for m in range(lmax + 1)]).cuda() >= spin
    for name, call in _calls(t, lmax, spin):
        call()
        _limit(t, 0)
        x = call()
        assert _status(t) == 1
        assert bool(torch.isnan(x[..., valid] if x.is_complex() else x).all()), name
        _limit(t, 1 << 22)
        assert bool(torch.isfinite(call()).all()), name
