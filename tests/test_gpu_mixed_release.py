"""What a mixed-precision solve returns when an iterate only just meets its backward-error target."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


def _solve(a, b, tol, max_iter, complex64=False):
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.device import context, ptr, to_device_colmajor, to_host_matrix
    ctx = context()
    n, nrhs = b.shape
    at, bt = to_device_colmajor(a, torch.complex64 if complex64 else torch.complex128), to_device_colmajor(b, torch.complex128)
    args = (None, n, ptr(at), n) if complex64 else (ptr(at), n, None, 0)
    info, st = ctypes.c_int(-1), _lib.GrimSolveInfo()
    _lib.check(ctx.lib.grim_zgesv_mixed(ctx.h, n, nrhs, *args, ptr(bt), n, _lib.PREC_MIXED_BERR, tol, max_iter,
                                        ctypes.byref(info), ctypes.byref(st)))
    x = to_host_matrix(bt)
    r = np.max(np.abs(a @ x - b), axis=0)
    den = np.max(np.sum(np.abs(a), axis=1)) * np.max(np.abs(x), axis=0) + np.max(np.abs(b), axis=0)
    return float(np.max(r / den)), st


@pytest.mark.parametrize('n, nrhs', [(96, 3), (300, 40)])
def test_iterates_in_the_last_decade_are_corrected_once_more(n, nrhs):
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * n ** 0.5 * np.eye(n)
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    first, st = _solve(a, b, 1.0, 4)  # the complex64 solution as it stands
    assert st.refinement_steps == 0 and 1e-9 < first < 1e-5
    # a target just above it: one correction, which a complex64 factor of a well-conditioned
    # system shortens the error by far more than ten times with
    got, st = _solve(a, b, 2.0 * first, 4)
    assert st.refinement_steps == 1 and got <= 0.1 * first
    # a target well above it, or no correction left: as it stands
    for tol, most in ((20.0 * first, 4), (2.0 * first, 0)):
        got, st = _solve(a, b, tol, most)
        assert st.refinement_steps == 0 and 0.5 * first <= got <= 2.0 * first


@pytest.mark.parametrize('n, nrhs', [(96, 3), (300, 40)])
def test_iterates_of_a_complex64_matrix_stay_as_they_are(n, nrhs):
    rng = np.random.default_rng(n)
    a = (rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 4.0 * n ** 0.5 * np.eye(n)).astype(np.complex64)
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    first, st = _solve(a.astype(complex), b, 1.0, 4)
    assert st.refinement_steps == 0 and 1e-9 < first < 1e-5
    for tol in (2.0 * first, 20.0 * first):
        got, st = _solve(a, b, tol, 4, complex64=True)
        assert st.refinement_steps == 0 and 0.5 * first <= got <= 2.0 * first


# exponent, half axes and phase of bodies whose fifth iterate has a backward error of
# 5e-11 to 9e-11 (tolerance 1e-10) and amplitudes 1.3e-9 to 2.9e-9 off
@pytest.mark.parametrize('p, a, b, phase', [(2.9188146577734972, 0.7364052813285286, 0.5030101002999807, 0.2014657372174874),
                                            (2.501660747442273, 0.8637627457638678, 0.37458943463838823, 0.9850504032756647),
                                            (2.4875701825175005, 0.7986149919634109, 0.3880252084505901, 0.6811946510427173)])
def test_large_mixed_amplitudes_are_those_of_the_fp64_solve(p, a, b, phase):
    """An accepted backward error of at most 1e-11, or 1e-10 and another correction, leaves at
    most 34 times 1e-11 in the amplitudes, the slices of the residual the rest."""
    from grim_20261007_b200.twod import operators as ops
    from grim_20261007_b200.twod.galerkin import GalerkinBody
    n = 4099
    t = -2.0 * np.pi * (np.arange(n) + phase) / n
    c, s = np.cos(t), np.sin(t)
    v = np.stack([a * np.sign(c) * np.abs(c) ** (2.0 / p), b * np.sign(s) * np.abs(s) ** (2.0 / p)], axis=1)
    k = 2.0 * np.pi * n / (10.0 * np.sum(np.hypot(*(np.roll(v, -1, axis=0) - v).T)))
    body, ang = GalerkinBody([v]), np.arange(181) * (360.0 / 181)
    amp = [ops.monostatic_solve(body, k, ang, 'TE', precision=m)['amplitude'].cpu().numpy() for m in ('mixed', 'double')]
    assert np.linalg.norm(amp[0] - amp[1]) <= 1e-9 * np.linalg.norm(amp[1])
