"""FP64 getrs in strips of eight columns against SciPy's lu_solve, at the edges of the 64-row
blocks and of the strips, with padded leading dimensions, and at a zero or infinite entry."""
import ctypes

import numpy as np
import pytest
import scipy.linalg as sla

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


def _getrs(lu, piv, b, lda, ldb):
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.device import context, ptr
    ctx = context()
    n, nrhs = b.shape
    a = torch.zeros((n, lda), dtype=torch.complex128)
    a[:, :n] = torch.from_numpy(np.ascontiguousarray(lu.T))
    x = torch.full((nrhs, ldb), 7.0 - 3.0j, dtype=torch.complex128)
    x[:, :n] = torch.from_numpy(np.ascontiguousarray(b.T))
    a, x = a.cuda(), x.cuda()
    ip = torch.from_numpy((piv + 1).astype(np.int32)).cuda()
    _lib.check(ctx.lib.grim_zgetrs(ctx.h, n, nrhs, ptr(a), lda, ptr(ip), ptr(x), ldb))
    out = x.cpu().numpy()
    assert np.all(out[:, n:] == 7.0 - 3.0j)  # the padding rows stay as they were
    return out[:, :n].T


@pytest.mark.parametrize('n', [1, 8, 63, 64, 65, 129, 200, 321])
@pytest.mark.parametrize('nrhs', [1, 7, 8, 9, 33])
def test_getrs_strips_equal_scipy(n, nrhs):
    rng = np.random.default_rng(1000 * n + nrhs)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    lu, piv = sla.lu_factor(a)
    x = _getrs(lu, piv, b, n + 3, n + 5)
    ref = sla.lu_solve((lu, piv), b)
    # normwise backward error of a substitution: a few n eps of |A| |x|
    res = np.max(np.abs(a @ x - b), axis=0)
    den = np.max(np.sum(np.abs(a), axis=1)) * np.max(np.abs(x), axis=0)
    assert np.max(res / den) < 1e-14
    assert np.max(np.abs(x - ref)) <= 1e-12 * np.linalg.cond(a) * np.max(np.abs(ref))


def test_getrs_strips_keep_columns_apart():
    """An infinite right-hand side entry stays in its own column."""
    n = 130
    rng = np.random.default_rng(5)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    b = rng.standard_normal((n, 11)) + 1j * rng.standard_normal((n, 11))
    lu, piv = sla.lu_factor(a)
    clean = _getrs(lu, piv, b, n, n)
    b2 = b.copy()
    b2[40, 3] = np.inf
    x = _getrs(lu, piv, b2, n, n)
    keep = [c for c in range(11) if c != 3]
    assert np.array_equal(x[:, keep], clean[:, keep])
    assert not np.all(np.isfinite(x[:, 3]))


def _solve(a, b, pivot, lda, ldb):
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.device import context, ptr
    ctx = context()
    n, nrhs = b.shape
    ad = torch.zeros((n, lda), dtype=torch.complex128)
    ad[:, :n] = torch.from_numpy(np.ascontiguousarray(a.T))
    x = torch.full((nrhs, ldb), 7.0 - 3.0j, dtype=torch.complex128)
    x[:, :n] = torch.from_numpy(np.ascontiguousarray(b.T))
    ad, x = ad.cuda(), x.cuda()
    info = ctypes.c_int(0)
    status = ctx.lib.grim_zgesv_mixed(ctx.h, n, nrhs, ptr(ad), lda, None, 0, ptr(x), ldb, _lib.PREC_FP64 | pivot,
                                      1e-10, 0, ctypes.byref(info), None)
    out = x.cpu().numpy()
    assert np.all(out[:, n:] == 7.0 - 3.0j)
    return status, info.value, out[:, :n].T


@pytest.mark.parametrize('n', [1, 63, 64, 65, 255, 256, 257, 321, 513])
@pytest.mark.parametrize('nrhs', [1, 8, 9, 33])
@pytest.mark.parametrize('mode', ['PREC_PARTIAL_PIVOT', 'PREC_TOURNAMENT_PIVOT'])
def test_elimination_beside_the_factorization(n, nrhs, mode):
    """Right-hand sides eliminated panel by panel (edges of panels and of the groups of four)."""
    from grim_20261007_b200 import _lib
    rng = np.random.default_rng(100 * n + nrhs)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    status, info, x = _solve(a, b, getattr(_lib, mode), n + 3, n + 5)
    assert status == 0 and info == 0
    res = np.max(np.abs(a @ x - b), axis=0)
    den = np.max(np.sum(np.abs(a), axis=1)) * np.max(np.abs(x), axis=0) + np.max(np.abs(b), axis=0)
    assert np.max(res / den) < 1e-14


# one, two and four panels a launch of the forward elimination (a launch is due by its rows from
# 1536 on, else by four panels); backward substitutions in strips and blocked on both sides of
# the rule (few columns above 1500 rows and third waves of strips take the blocked one)
@pytest.mark.parametrize('n, nrhs', [(64, 2369), (65, 1184), (65, 1185), (513, 3553), (1400, 9), (1601, 9), (1601, 361),
                                     (2048, 33), (2113, 9), (2113, 361), (3073, 8), (3073, 720)])
@pytest.mark.parametrize('pivot', ['partial', None])
def test_large_solves_on_both_sides_of_the_strip_rule(n, nrhs, pivot):
    """Whole solves (elimination beside a partial-pivoting factorization, or getrs after a
    certified one): normwise backward error of every column."""
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.device import context, ptr
    ctx = context()
    gen = torch.Generator(device='cuda').manual_seed(n + nrhs)
    at = torch.randn((n, n), dtype=torch.complex128, device='cuda', generator=gen)
    bt = torch.randn((nrhs, n), dtype=torch.complex128, device='cuda', generator=gen)
    x, info = bt.clone(), ctypes.c_int(-1)
    mode = _lib.PREC_FP64 | (_lib.PREC_PARTIAL_PIVOT if pivot else 0)
    _lib.check(ctx.lib.grim_zgesv_mixed(ctx.h, n, nrhs, ptr(at), n, None, 0, ptr(x), n, mode, 1e-10, 0,
                                        ctypes.byref(info), None))
    assert info.value == 0
    res = (x @ at - bt).abs().amax(1)  # rows of the tensors are columns of the matrices
    den = at.abs().sum(0).max() * x.abs().amax(1) + bt.abs().amax(1)
    assert float((res / den).max()) < 1e-14


def test_singular_matrix_leaves_the_right_hand_sides():
    from grim_20261007_b200 import _lib
    n = 300
    rng = np.random.default_rng(3)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n))
    a[:, 270] = 0.0
    b = rng.standard_normal((n, 10)) + 1j * rng.standard_normal((n, 10))
    status, info, x = _solve(a, b, _lib.PREC_PARTIAL_PIVOT, n, n)
    assert status != 0 and info == 271
    assert np.array_equal(x, b)
