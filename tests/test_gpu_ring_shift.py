"""Ring synthesis by the chirp-z form with no ring, one ring or every ring
starting off zero (the phase table in shared memory belongs to the last two),
uniform rings of a prime length, against the FP64 direct sum at the pixels.

Tolerance: the transform's 2^-53 sqrt(log2 N) and the oracle's sums, 1e-11 of the
largest value (double-float rings of mixed plans: kernel rounding 2^-45 and
the Legendre stage's 1e-7)."""
import numpy as np
import pytest

import oracle
from oracle import oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("shifted", ["none", "first", "last", "all"])
@pytest.mark.parametrize("precision,tol", [("fp64", 1e-11), ("mixed", 2e-7)])
@pytest.mark.parametrize("lmax,nphi", [(30, 37), (30, 61), (120, 241)])
def test_first_longitudes(built_lib, monkeypatch, shifted, precision, tol, lmax, nphi):
    import cunusht_gb300 as cu
    from cunusht_gb300 import transformer
    geom = transformer.get_geom(("gl", {"lmax": lmax, "nphi": nphi}))
    n = geom.phi0.size
    geom.phi0[{"none": slice(0, 0), "first": slice(0, 1), "last": slice(n - 1, n), "all": slice(0, n)}[shifted]] = 0.37
    monkeypatch.setattr(transformer, "get_geom", lambda info: geom)
    t = cu.get_transformer("GPU")(("gl", {"lmax": lmax, "nphi": nphi}), nuFFTtype=2, epsilon=1e-7, precision=precision,
                                  max_spin=2)
    th, ph = geom.pixels()
    for spin in (0, 2):
        alm, _ = orc.make_inputs(lmax, spin, seed=2)
        a = alm if spin else alm[0]
        got = t.synthesis(torch.as_tensor(a, device="cuda"), spin=spin).cpu().numpy()
        assert t._lib.cunusht_plan_ring_transform(t._plan) == 1
        want = oracle.synth_points_c(lmax, spin, a, th, ph)
        assert np.max(np.abs(got.reshape(want.shape) - want)) < tol * np.max(np.abs(want))
