"""FP64 tensor-core GEMM over its tile shapes (the launcher picks 64 x 64, 64 x 32 or 32 x 32 by
the load of the fullest SM): residuals R = B - A X against NumPy at ragged sizes and with padded
leading dimensions."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


@pytest.mark.parametrize('n, nrhs', [(1, 1), (31, 33), (64, 64), (65, 31), (200, 700), (777, 97), (1030, 721),
                                     (1601, 800)])
def test_residual_equals_numpy(n, nrhs):
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.device import context, ptr
    ctx = context()
    rng = np.random.default_rng(n)
    a, x, b = (rng.standard_normal((n, c)) + 1j * rng.standard_normal((n, c)) for c in (n, nrhs, nrhs))
    lda, ldx, ldb, ldr = n + 1, n + 2, n + 3, n + 5

    def dev(m, ld):
        out = torch.full((m.shape[1], ld), 5.0 + 1.0j, dtype=torch.complex128)
        out[:, :n] = torch.from_numpy(np.ascontiguousarray(m.T))
        return out.cuda()

    ad, xd, bd = dev(a, lda), dev(x, ldx), dev(b, ldb)
    rd = torch.full((nrhs, ldr), 5.0 + 1.0j, dtype=torch.complex128, device='cuda')
    _lib.check(ctx.lib.grim_residual(ctx.h, n, nrhs, ptr(ad), lda, 0, ptr(xd), ldx, ptr(bd), ldb, ptr(rd), ldr, 0))
    out = rd.cpu().numpy()
    assert np.all(out[:, n:] == 5.0 + 1.0j)
    # rounding of an n-term complex dot product
    bound = 8.0 * np.finfo(float).eps * n ** 0.5 * (np.max(np.abs(b)) + n ** 0.5 * np.max(np.abs(a)) * np.max(np.abs(x)))
    assert np.max(np.abs(out[:, :n].T - (b - a @ x))) <= bound


def test_millions_of_columns_keep_to_the_wide_tiles():
    """32 columns a tile would need more tiles than a grid's y extent."""
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.device import context, ptr
    ctx = context()
    n, nrhs = 16, 2_100_000
    gen = torch.Generator(device='cuda').manual_seed(1)
    a, x, b = (torch.randn((c, n), dtype=torch.complex128, device='cuda', generator=gen) for c in (n, nrhs, nrhs))
    r = torch.empty_like(b)
    _lib.check(ctx.lib.grim_residual(ctx.h, n, nrhs, ptr(a), n, 0, ptr(x), n, ptr(b), n, ptr(r), n, 0))
    ref = b - x @ a  # rows of the tensors are columns of the matrices
    assert float((r - ref).abs().max()) <= 8.0 * np.finfo(float).eps * 4.0 * n * float(x.abs().max() * a.abs().max())
