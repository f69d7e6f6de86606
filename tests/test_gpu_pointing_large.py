"""FP64 pointing of pixels next to a pole with deflections up to pi: the end
points lie anywhere on the sphere, the other pole included.

Tolerance: theta' = atan2(rho, nz) of components good to a few 2^-53, so 8 ulp
of pi next to the poles, where rho is a difference of terms of its own size."""
import numpy as np
import pytest

from oracle import oracle as orc

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


def _pointing(lib, th, dt, dp):
    """cunusht_pointing with one pixel per ring, phi = 0."""
    from cunusht_gb300 import _lib
    n = th.size
    dev = lambda a, t=torch.float64: torch.as_tensor(a, dtype=t, device="cuda")  # noqa: E731
    args = [dev(th), dev(np.zeros(n)), dev(np.ones(n), torch.int64), dev(np.arange(n), torch.int64), dev(dt), dev(dp)]
    out = torch.empty((3, n), dtype=torch.float64, device="cuda")
    p = [a.data_ptr() for a in args]
    _lib.check(lib.cunusht_pointing(n, p[0], p[1], p[2], p[3], n, p[4], p[5], *[o.data_ptr() for o in out],
                                    torch.cuda.current_stream().cuda_stream))
    return out.cpu().numpy()


@pytest.mark.parametrize("south", [False, True])
@pytest.mark.parametrize("length", [1e-4, 0.019, 0.5, 3.0, 3.1, 3.13, 3.14])
def test_rings_next_to_the_poles(built_lib, south, length):
    th, a = (x.ravel() for x in np.meshgrid([1e-3, 3e-3, 0.01, 0.0199, 0.05], 2 * np.pi * (np.arange(64) + 0.25) / 64))
    th = np.concatenate([th, [0.01, 3e-3]])  # straight over the pole
    a = np.concatenate([a, [0.0, np.pi]])
    if south:
        th = np.pi - th
    dt, dp = length * np.cos(a), length * np.sin(a)
    got = _pointing(built_lib, th, dt, dp)
    want, phi = orc.pointing(th, np.zeros_like(th), dt, dp)
    assert np.max(np.abs(got[0] - want)) < 8 * np.spacing(np.pi)
    d = np.remainder(got[1] - phi + np.pi, 2 * np.pi) - np.pi
    assert np.max(np.abs(d) * np.sin(want)) < 8 * np.spacing(np.pi)
