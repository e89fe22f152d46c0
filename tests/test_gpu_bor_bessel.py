"""Excitations and far-field weights at the edges of the Bessel evaluation: on and next to the
axis (the series below x = 1e-8), negative and large aspects (x < 0), both parities and signs of
the order, orders far above x, and both sides of the switch to the library at x = 2000."""
import numpy as np
import pytest

from oracle import bor as OB
from grim_20261007_b200 import synthetic as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


@pytest.mark.parametrize('k', [1e-3, 6.0, 2600.0])
@pytest.mark.parametrize('m', [0, 1, -1, 2, 5, -6, 40])
@pytest.mark.parametrize('far', [False, True])
def test_excitations_at_the_bessel_edges(k, m, far):
    from grim_20261007_b200.bor import solver as B
    pts = S.ogive_generatrix(2.0, 40.0, 9)
    dev = B.BorDevice(pts, k, 41, alpha=1.0)
    angles = np.array([0.0, 1e-9, -1e-9, 1e-7, 37.0, -37.0, 90.0, 180.0, 211.0, 50.1])
    th = torch.from_numpy(angles).cuda()
    got = dev.excitation(m, th, far).cpu().numpy().T
    body = OB.Body(pts)
    full = OB.excitation(body, k, angles, m, far=far)
    Q = OB.pole_transform(body, m)
    ref = (Q.T if far else Q.conj().T) @ full
    # the phase k z and the argument k rho carry their own rounding; weights 2 pi rho L
    pts = np.asarray(pts)
    scale = 4 * np.pi * np.max(pts[:, 0]) * np.max(np.hypot(*np.diff(pts, axis=0).T))
    reach = k * np.max(np.hypot(pts[:, 0], pts[:, 1]))
    assert np.max(np.abs(got - ref)) <= 16 * np.finfo(float).eps * (4 + reach) * scale * max(1, abs(m))
