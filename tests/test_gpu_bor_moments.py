"""Modal moments at the edges of the orders-per-lane split, against the FP64 oracle.

A lane keeps three orders up to 96 orders in all and four above, an even number of lane blocks
share a warp and leave between one and sixteen lanes per block.  The tolerance is the mode
matrices' 1e-11 of the largest entry, growing with the order: n times the phase rounding of
e^{j n xi} enters every moment."""
import numpy as np
import pytest

from oracle import bor as OB
from grim_20261007_b200 import synthetic as S

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


@pytest.mark.parametrize('mmax, alpha', [(0, 0.5), (5, 1.0), (5, 0.5), (94, 0.5), (95, 1.0), (126, 0.5)])
def test_mode_matrices_at_the_lane_splits(mmax, alpha):
    from grim_20261007_b200.bor import solver as B
    pts = S.ogive_generatrix(2.0, 40.0, 7)
    k = 6.0
    dev = B.BorDevice(pts, k, mmax, alpha=alpha)
    body = OB.Body(pts)
    asm = OB.Assembler(body, k, mmax, mfie=alpha < 1.0)
    for m in sorted({0, mmax // 2, mmax}):
        Q = OB.pole_transform(body, m)
        Zf = asm.matrix(m) if alpha == 1.0 else alpha * asm.matrix(m) + (1 - alpha) * OB.ETA0 * asm.mfie_matrix(m)
        Zr = Q.conj().T @ Zf @ Q
        Zg = dev.matrix(m).cpu().numpy().T
        assert np.max(np.abs(Zg - Zr)) <= 1e-11 * max(1.0, mmax / 10.0) * np.max(np.abs(Zr)), m
