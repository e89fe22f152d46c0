"""Far pairs of the linear-Galerkin fill against plain quadrature with SciPy's Bessel functions.

Sizes sit at the edges of the 32-element tiles and on both sides of the switch between eight
threads and one thread per pair; the wavenumbers reach every interval of the Hankel
evaluation (x = 3, 4.5, 8, 25, 80) on one ring.  The tile orders hold a block within 1e-12 of
a converged rule, so the matrices agree to 1e-12 of their largest entry."""
import numpy as np
import pytest
from scipy import special

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


def _ring(count):
    rng = np.random.default_rng(count)
    theta = -2.0 * np.pi * (np.arange(count) + 0.2 * rng.uniform(-1, 1, count)) / count
    return np.stack([np.cos(theta), 0.8 * np.sin(theta)], axis=1)


def _far_entries(drawn, k, pol, rows, cols, order=12):
    """Node entries (rows, cols) whose four element pairs are all far, by a rule of `order` points."""
    n = len(drawn)
    a = drawn[(-np.arange(n)) % n]
    b = np.roll(a, -1, axis=0)
    length = np.hypot(*(b - a).T)
    nrm = np.stack([-(b - a)[:, 1], (b - a)[:, 0]], axis=1) / length[:, None]
    x, w = np.polynomial.legendre.leggauss(order)
    x, w = 0.5 * (x + 1.0), 0.5 * w
    hat = np.stack([1.0 - x, x])
    out = np.zeros(len(rows), complex)
    for eo, ao in ((rows, 0), ((rows - 1) % n, 1)):
        for es, bs in ((cols, 0), ((cols - 1) % n, 1)):
            po = a[eo][:, None, :] + x[None, :, None] * (b - a)[eo][:, None, :]
            ps = a[es][:, None, :] + x[None, :, None] * (b - a)[es][:, None, :]
            r = po[:, :, None, :] - ps[:, None, :, :]
            d = np.hypot(r[..., 0], r[..., 1])
            g = 0.25 * (special.y0(k * d) + 1j * special.j0(k * d))
            h = 0.25 * k * (special.y1(k * d) + 1j * special.j1(k * d))
            ll = length[eo] * length[es]
            wt = np.einsum('p,q->pq', w * hat[ao], w * hat[bs])
            s = ll * np.einsum('epq,pq->e', g, wt)
            if pol == 'TM':
                out += s + ll * np.einsum('epq,pq->e', h * np.einsum('epqx,ex->epq', r, nrm[es]) / d, wt) / (1j * k)
            else:
                kp = -ll * np.einsum('epq,pq->e', h * np.einsum('epqx,ex->epq', r, nrm[eo]) / d, wt)
                total = np.einsum('epq,pq->e', g, np.einsum('p,q->pq', w, w))
                sign = 1.0 if ao == bs else -1.0
                hyper = -k * k * np.einsum('ex,ex->e', nrm[eo], nrm[es]) * s + sign * total
                out += kp - hyper / (1j * k)
    return out


@pytest.mark.parametrize('n', [33, 64, 351, 352, 353, 385])
@pytest.mark.parametrize('kl', [0.1, 0.6, 1.4])
@pytest.mark.parametrize('pol', ['TM', 'TE'])
def test_far_entries_equal_plain_quadrature(n, kl, pol):
    from grim_20261007_b200.device import to_host_matrix
    from grim_20261007_b200.twod.galerkin import GalerkinBody
    drawn = _ring(n)
    k = kl * n / 5.6
    z = to_host_matrix(GalerkinBody([drawn]).fill_matrix(k, pol))
    rng = np.random.default_rng(1)
    rows = np.concatenate([rng.integers(0, n, 1500), np.repeat([0, 31, 32, n - 1], 40)])
    gap = np.concatenate([rng.integers(8, n - 7, 1500), np.tile(np.linspace(8, n - 8, 40).astype(int), 4)])
    cols = (rows + gap) % n
    ref = _far_entries(drawn, k, pol, rows, cols)
    assert np.max(np.abs(z[rows, cols] - ref)) <= 1e-12 * np.max(np.abs(z))


@pytest.mark.parametrize('kl', [0.02, 0.16, 0.46, 0.9, 1.4, 1.9, 2.6])
@pytest.mark.parametrize('floor', [8, 16])
@pytest.mark.parametrize('pol', ['TM', 'TE'])
def test_converged_orders_hold_every_floor(kl, floor, pol, monkeypatch):
    """A floor above the converged order changes nothing but rounding: entries against a 16-point
    rule over neighbouring tiles (ratios from 8) to far ones, elements of 1 : 3 lengths."""
    from grim_20261007_b200.device import to_host_matrix
    from grim_20261007_b200.twod.galerkin import GalerkinBody
    monkeypatch.setattr(GalerkinBody, 'far_min_order', lambda self, k, p: floor if p == 'TE' else 0)
    n = 400
    theta = -2.0 * np.pi * (np.arange(n) / n)
    theta = theta + 0.5 * np.sin(theta)
    drawn = np.stack([np.cos(theta), 0.8 * np.sin(theta)], axis=1)
    length = np.hypot(*(np.roll(drawn, -1, axis=0) - drawn).T)
    k = kl / length.max()
    z = to_host_matrix(GalerkinBody([drawn]).fill_matrix(k, pol))
    rows = np.arange(n).repeat(12)
    cols = (rows + np.tile([40, 47, 64, 90, 111, 150, 200, 260, 290, 333, 350, 360], n)) % n
    pts = drawn[(-np.arange(n)) % n]
    dist = np.hypot(*(pts[rows] - pts[cols]).T)
    sel = dist >= 12.0 * length.max()  # TM keeps the reference's lower orders nearer in
    rows, cols, dist = rows[sel], cols[sel], dist[sel]
    ref = _far_entries(drawn, k, pol, rows, cols, order=16)
    # the four element sums of an entry: kernel values carry a few ulp and the phase k r its own
    g = 0.25 * np.hypot(special.j0(k * dist), special.y0(k * dist))
    scale = g * (4.0 / k + 4.0 * length.max() + 4.0 * length.max() ** 2)
    eps = np.finfo(float).eps
    order_error = 2e-11 if pol == 'TM' else 0.0  # 5- to 8-point rules of the TM table
    assert np.all(np.abs(z[rows, cols] - ref) <= (8.0 * eps * (8.0 + k * dist) + order_error) * scale)


@pytest.mark.parametrize('stretch', [0.0, 0.5])
@pytest.mark.parametrize('kl', [0.02, 0.3, 0.8, 1.6, 2.6, 3.6])
@pytest.mark.parametrize('floor', [8, 16])
def test_converged_orders_hold_beside_the_near_pairs(kl, floor, stretch, monkeypatch):
    """TE entries of element pairs three to nine lengths apart (orders 10, 9, 8 and, past |k| L = 3,
    16), lengths of up to 1 : 2 and 1 : 5, against a 24-point rule."""
    from grim_20261007_b200.device import to_host_matrix
    from grim_20261007_b200.twod.galerkin import GalerkinBody
    monkeypatch.setattr(GalerkinBody, 'far_min_order', lambda self, k, p: floor)
    n = 400
    theta = -2.0 * np.pi * (np.arange(n) + np.random.default_rng(2).uniform(-0.15, 0.15, n)) / n
    theta = theta + stretch * np.sin(theta)
    drawn = np.stack([np.cos(theta), 0.8 * np.sin(theta)], axis=1)
    a = drawn[(-np.arange(n)) % n]
    b = np.roll(a, -1, axis=0)
    length, mid = np.hypot(*(b - a).T), 0.5 * (a + b)
    k = kl / length.max()
    z = to_host_matrix(GalerkinBody([drawn]).fill_matrix(k, 'TE'))
    rows = np.arange(n).repeat(6)
    cols = (rows + np.tile([4, 5, 6, 7, 8, 9], n)) % n
    ratio = np.min([np.hypot(*(mid[(rows - p) % n] - mid[(cols - q) % n]).T) /
                    np.maximum(length[(rows - p) % n], length[(cols - q) % n]) for p in (0, 1) for q in (0, 1)], axis=0)
    sel = ratio > 3.001  # all four element pairs far
    rows, cols = rows[sel], cols[sel]
    assert np.min(ratio[sel]) < 3.2 and np.max(ratio[sel]) > 7.0
    ref = _far_entries(drawn, k, 'TE', rows, cols, order=24)
    # every kernel value a few ulp, its phase and its distance of coordinates of order 1
    dist = np.hypot(*(a[rows] - a[cols]).T)
    near = np.maximum(dist - 1.5 * length.max(), 0.5 * dist)
    big = length.max()
    g = 0.25 * np.hypot(special.j0(k * near), special.y0(k * near))
    h = 0.25 * k * np.hypot(special.j1(k * near), special.y1(k * near))
    scale = 4.0 * (h * big ** 2 + k * g * big ** 2 + g / k)
    assert np.all(np.abs(z[rows, cols] - ref) <= 8.0 * np.finfo(float).eps * (8.0 + k * dist) * scale)
