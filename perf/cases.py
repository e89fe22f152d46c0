"""Performance cases of the RCS solve path, called through its public entry points.

A case is a dict of plain values: ``kind`` names the entry point, the rest its sizes.

* ``rcs2d``  ``twod.solver.solve_monostatic_rcs_2d``: geometry snapshot in, host samples of both
  polarisations out, one or more frequencies (the call of a user's program);
* ``solve``  ``twod.operators.monostatic_solve`` on a resident body: one (frequency, polarisation)
  system with all its angles, FP64 (the default) or mixed precision;
* ``fill``   ``GalerkinBody.fill_matrix``: the system matrix alone;
* ``hook``   ``twod.solver._solve_dense_gpu``: the reference's dense-solve hook on host arrays;
* ``far``    ``twod.farblock.far_block``: the reference's far-block quadrature on host arrays;
* ``bor``    ``bor.solver.solve_bor``: a body of revolution, every Fourier mode, VV and HH.

``exact`` restates the 2-D path (plain quadrature of the combined-field operators with the hat
bases, a dense solve, the far-field sum), the hook and the far block in 64-bit NumPy / torch.
"""
from __future__ import annotations

import contextlib
import math

import numpy as np
import torch

from grim_20261007_b200.bor.solver import solve_bor
from grim_20261007_b200.execution import linear_precision
from grim_20261007_b200.twod import farblock, galerkin, operators, solver
from grim_20261007_b200.synthetic import snapshot_from_polygons

C0 = 299_792_458.0
EXACT_MAX_ORDER = 1100     # above it, 2-D systems take the 64-bit restatement over 20 s
AIRFOIL, SUPER, CIRCLE = 'airfoil', 'superellipse', 'polygon'


def listed():
    return [
        # the smallest whole call: an interactive what-if on a coarse body, bound by launches and host work
        dict(name='rcs2d_96x37', kind='rcs2d', shape=SUPER, n=96, nang=37, nfreq=1, band=1.0, precision='double'),
        # an ordinary whole call: one frequency, half-degree cut, both polarisations
        dict(name='rcs2d_1024x361', kind='rcs2d', shape=AIRFOIL, n=1024, nang=361, nfreq=1, band=1.0,
             precision='double'),
        # a frequency sweep (ISAR, range profiles): every system its own mesh and size
        dict(name='sweep_12x700x181', kind='rcs2d', shape=CIRCLE, n=700, nang=181, nfreq=12, band=4.0,
             precision='double'),
        # a small odd system with few angles, geometry resident (serving, optimisation loops)
        dict(name='solve_fp64_333x19', kind='solve', shape=SUPER, n=333, nang=19, pol='TM', precision='double'),
        # the benchmark's body and angle count, default precision
        dict(name='solve_fp64_2048x720', kind='solve', shape=AIRFOIL, n=2048, nang=720, pol='TE', precision='double'),
        # the same in mixed precision
        dict(name='solve_mixed_2048x720', kind='solve', shape=AIRFOIL, n=2048, nang=720, pol='TM', precision='mixed'),
        # a large ragged system in mixed precision
        dict(name='solve_mixed_4099x181', kind='solve', shape=SUPER, n=4099, nang=181, pol='TE', precision='mixed'),
        # the system matrix alone at an odd order (callers that bring their own solver)
        dict(name='fill_te_1501', kind='fill', shape=SUPER, n=1501, pol='TE'),
        # the reference's dense hook with host matrices of an ordinary size
        dict(name='hook_900x181', kind='hook', n=900, nang=181),
        # one tile of the reference's far-field pass, host arrays, ragged
        dict(name='far_500x389', kind='far', rows=500, cols=389, order=6),
        # a small body of revolution: few modes, few aspects
        dict(name='bor_61x37', kind='bor', shape='sphere', segments=61, krho=4.0, nang=37, formulation='auto'),
        # the benchmark's ogive: 400 segments, |m| <= 40, half-degree aspects
        dict(name='bor_400x361', kind='bor', shape='ogive', segments=400, krho=25.0, nang=361, formulation='auto'),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['rcs2d', 'rcs2d', 'solve', 'solve', 'solve', 'fill', 'hook', 'far', 'bor', 'bor'])
    shape = rng.choice([AIRFOIL, SUPER, CIRCLE])
    even = 2 if shape == AIRFOIL else 1
    precision = rng.choice(['double', 'mixed'])
    pol = rng.choice(['TM', 'TE'])
    if kind == 'rcs2d':
        nfreq = rng.choice([1, 1, 2, 5, 8])
        n = _log(rng, 64, 1600 if nfreq == 1 else 600) // even * even
        return dict(kind=kind, shape=CIRCLE if nfreq > 1 else shape, n=n, nang=_log(rng, 1, 400), nfreq=nfreq,
                    band=round(rng.uniform(1.5, 5.0), 3) if nfreq > 1 else 1.0, precision=precision)
    if kind == 'solve':
        return dict(kind=kind, shape=shape, n=_log(rng, 64, 3500) // even * even, nang=_log(rng, 1, 720), pol=pol,
                    precision=precision)
    if kind == 'fill':
        return dict(kind=kind, shape=shape, n=_log(rng, 64, 4000) // even * even, pol=pol)
    if kind == 'hook':
        return dict(kind=kind, n=_log(rng, 48, 1500), nang=_log(rng, 1, 361))
    if kind == 'far':
        return dict(kind=kind, rows=_log(rng, 32, 700), cols=_log(rng, 32, 700), order=rng.choice([5, 6, 7, 8]))
    krho = rng.uniform(2.0, 20.0)
    return dict(kind=kind, shape=rng.choice(['sphere', 'ogive', 'spheroid']), krho=round(krho, 3),
                segments=max(24, int(krho * rng.uniform(6.0, 15.0))), nang=_log(rng, 1, 361),
                formulation=rng.choice(['auto', 'auto', 'efie']))


# ------------------------------------------------------------------ geometry
def _rng(case, seed):
    return np.random.default_rng([int(seed) & 0xffffffff, int(case.get('n', case.get('segments', case.get('rows', 0))))])


def _polygon(case, seed):
    """Closed clockwise polygon (n, 2) in metres, its proportions drawn from the seed."""
    rng, n = _rng(case, seed), case['n']
    if case['shape'] == AIRFOIL:
        # NACA 00tt, cosine node spacing, finite trailing edge closed by two base elements
        t, m = rng.uniform(0.08, 0.15), n // 2 - 1
        x = 0.5 * (1.0 + np.cos(np.pi * np.arange(m + 1) / m))
        y = 5.0 * t * (0.2969 * np.sqrt(x) - 0.1260 * x - 0.3516 * x ** 2 + 0.2843 * x ** 3 - 0.1015 * x ** 4)
        y[-1] = 0.0
        lower, upper = np.stack([x, -y], axis=1), np.stack([x[::-1], y[::-1]], axis=1)
        return np.concatenate([[[1.0, 0.0]], lower, upper[1:]], axis=0)
    a, b = rng.uniform(0.6, 1.0), rng.uniform(0.3, 0.6)
    if case['shape'] == SUPER:
        # superellipse, equal steps of the parameter
        p, th = rng.uniform(2.0, 3.0), -2.0 * np.pi * (np.arange(n) + rng.uniform(0.0, 1.0)) / n
        c, s = np.cos(th), np.sin(th)
        return np.stack([a * np.sign(c) * np.abs(c) ** (2.0 / p), b * np.sign(s) * np.abs(s) ** (2.0 / p)], axis=1)
    # an irregular 17-gon, each side cut into equal elements (n elements in all)
    th = -2.0 * np.pi * (np.arange(17) + rng.uniform(-0.2, 0.2, 17)) / 17
    corner = np.stack([a * np.cos(th), b * np.sin(th)], axis=1)
    cut = np.full(17, n // 17)
    cut[:n % 17] += 1
    nxt = np.roll(corner, -1, axis=0)
    return np.concatenate([corner[i] + (np.arange(cut[i]) / cut[i])[:, None] * (nxt[i] - corner[i]) for i in range(17)])


def _wavenumber(verts):
    """Ten elements to a wavelength on average."""
    d = np.roll(verts, -1, axis=0) - verts
    return 2.0 * math.pi * len(verts) / (10.0 * float(np.sum(np.hypot(d[:, 0], d[:, 1]))))


def _angles(case, seed):
    return _rng(case, seed).uniform(0.0, 0.5) + np.arange(case['nang']) * (360.0 / case['nang'])


def _generatrix(case, seed):
    rng, n = _rng(case, seed), case['segments']
    if case['shape'] == 'ogive':
        alpha, length = math.radians(rng.uniform(15.0, 30.0)), rng.uniform(2.0, 4.0)
        arc, ang = 0.5 * length / math.sin(alpha), np.linspace(alpha, -alpha, n + 1)
        pts = np.stack([np.maximum(arc * np.cos(ang) - arc * math.cos(alpha), 0.0), arc * np.sin(ang)], axis=1)
    else:
        t, a = np.linspace(0.0, np.pi, n + 1), 1.0 if case['shape'] == 'sphere' else rng.uniform(1.2, 2.0)
        r = rng.uniform(0.8, 1.2)
        pts = np.stack([r * np.sin(t), r * a * np.cos(t)], axis=1)
    pts[0, 0] = pts[-1, 0] = 0.0
    return pts, case['krho'] * (C0 / (2.0 * math.pi)) / float(np.max(pts[:, 0]))


def _hook_system(case, seed):
    """A well-conditioned dense system of the kind the hook receives: a decaying oscillatory
    kernel between points of a curve, a dominant diagonal, plane-wave right-hand sides."""
    rng, n = _rng(case, seed), case['n']
    th = 2.0 * np.pi * (np.arange(n) + rng.uniform(-0.2, 0.2, n)) / n
    p = np.stack([np.cos(th), rng.uniform(0.4, 0.9) * np.sin(th)], axis=1)
    k = n / 10.0
    r = np.hypot(p[:, None, 0] - p[None, :, 0], p[:, None, 1] - p[None, :, 1]) + 0.05 / n
    a = (2.0 * np.pi / n) * np.sqrt(k / r) * np.exp(-1j * k * r) / 4.0
    a[np.arange(n), np.arange(n)] += 0.5 + 0.2j
    ang = 2.0 * np.pi * np.arange(case['nang']) / case['nang']
    return a, -np.exp(1j * k * (p[:, :1] * np.cos(ang) + p[:, 1:] * np.sin(ang)))


def _far_tile(case, seed):
    """Observation and source elements of one far tile: two stretches of a curve, a few
    wavelengths apart, linear bases, every pair far."""
    rng, rows, cols, q = _rng(case, seed), case['rows'], case['cols'], case['order']
    x, w = np.polynomial.legendre.leggauss(q)
    h = 0.01

    def side(count, y0):
        s = np.arange(count + 1) * h
        ends = np.stack([s, y0 + 0.1 * np.sin(s + rng.uniform(0.0, 6.0))], axis=1)
        a, b = ends[:-1], ends[1:]
        t = (b - a) / np.linalg.norm(b - a, axis=1)[:, None]
        pts = a[:, None, :] * ((1.0 - x) / 2)[None, :, None] + b[:, None, :] * ((1.0 + x) / 2)[None, :, None]
        return np.ascontiguousarray(pts), np.ascontiguousarray(np.stack([t[:, 1], -t[:, 0]], axis=1))

    k = 2.0 * math.pi / (10.0 * h)
    obs, obs_n = side(rows, 0.0)
    src, src_n = side(cols, 0.5)
    phi = np.ascontiguousarray(np.stack([(1.0 - x) / 2, (1.0 + x) / 2], axis=-1))
    return dict(k=k, obs=obs, src=src, qw=np.ascontiguousarray(w * 0.5), phi=phi, obs_n=obs_n, src_n=src_n,
                far=np.ones((rows, cols), np.uint8))


def _sweep_snapshot(case, verts):
    """The 17-gon's sides as primitives meshed by wavelength (several frequencies) or the
    polygon's elements as they are (one frequency)."""
    if case['nfreq'] == 1:
        return snapshot_from_polygons([verts])
    cut = np.full(17, case['n'] // 17)
    cut[:case['n'] % 17] += 1
    snap = snapshot_from_polygons([verts[np.cumsum(cut) - cut]])
    snap['segments'][0]['properties'][1] = '-10'
    return snap


def _frequencies(case, verts):
    top = _wavenumber(verts) * C0 / (2.0 * math.pi) / 1e9
    return [float(f) for f in np.geomspace(top / case['band'], top, case['nfreq'])]


# ------------------------------------------------------------------ prepare / run
def prepare(case, seed):
    kind = case['kind']
    if kind == 'rcs2d':
        verts = _polygon(case, seed)
        return dict(case=case, snapshot=_sweep_snapshot(case, verts), freqs=_frequencies(case, verts),
                    angles=_angles(case, seed).tolist())
    if kind in ('solve', 'fill'):
        verts = _polygon(case, seed)
        state = dict(case=case, body=galerkin.GalerkinBody([verts]), k=_wavenumber(verts))
        if kind == 'solve':
            state['angles'] = _angles(case, seed)
            state['angles_dev'] = torch.as_tensor(state['angles'], device='cuda')
        return state
    if kind == 'hook':
        a, b = _hook_system(case, seed)
        return dict(case=case, a=a, b=b)
    if kind == 'far':
        t = _far_tile(case, seed)
        d = t['obs'].reshape(-1, 1, 2)[:, 0], t['src'].reshape(-1, 1, 2)[:, 0]
        reach = float(np.hypot(*(np.maximum(d[0].max(0), d[1].max(0)) - np.minimum(d[0].min(0), d[1].min(0)))))
        return dict(case=case, tile=t, table=farblock.KernelTable(t['k'], reach * 1.01))
    pts, freq = _generatrix(case, seed)
    return dict(case=case, points=pts, freq=freq, angles=np.arange(case['nang']) * (180.0 / max(1, case['nang'] - 1)))


def run(state):
    case = state['case']
    kind = case['kind']
    if kind == 'rcs2d':
        scope = linear_precision('mixed') if case['precision'] == 'mixed' else contextlib.nullcontext()
        with scope:
            res = solver.solve_monostatic_rcs_2d(state['snapshot'], state['freqs'], state['angles'],
                                                 geometry_units='meters')
        return {ch: np.array([complex(s['rcs_amp_real'], s['rcs_amp_imag']) for s in rows])
                for ch, rows in res['co_solved_samples'].items()}
    if kind == 'solve':
        return operators.monostatic_solve(state['body'], state['k'], state['angles'], case['pol'],
                                          precision=case['precision'], angles_dev=state['angles_dev'])['amplitude']
    if kind == 'fill':
        return state['body'].fill_matrix(state['k'], case['pol'])
    if kind == 'hook':
        return solver._solve_dense_gpu(state['a'], state['b'])[0]
    if kind == 'far':
        t = state['tile']
        return farblock.far_block(state['table'], t['k'], t['obs'], t['src'], t['qw'], t['phi'], t['obs_n'],
                                  t['src_n'], t['far'], 1, True, True, True)
    res = solve_bor(state['points'], state['freq'], state['angles'], formulation=case['formulation'])
    return {key: np.asarray(res[key]) for key in ('amp_vv', 'amp_hh')}


# ------------------------------------------------------------------ work
def _solve_work(n, nang):
    """(bytes, flops) of one 2-D system: the matrix written by the fill and read by the LU, the
    factor written; far pairs (both orientations from one set of kernel values, at least
    5 x 5 points, about 40 operations a point), LU and the two triangular solves."""
    return 3.0 * 16 * n * n + 2.0 * 16 * n * nang, 0.5 * n * n * 25 * 40 + 8.0 / 3 * n ** 3 + 8.0 * n * n * nang


def work(case):
    kind = case['kind']
    if kind == 'rcs2d':
        sizes = [case['n'] * f for f in np.geomspace(1.0 / case['band'], 1.0, case['nfreq'])]
        per = [_solve_work(n, case['nang']) for n in sizes]
        return dict(bytes=2.0 * sum(b for b, _f in per), flops=2.0 * sum(f for _b, f in per))
    if kind == 'solve':
        b, f = _solve_work(case['n'], case['nang'])
        return dict(bytes=b, flops=f)
    if kind == 'fill':
        return dict(bytes=16.0 * case['n'] ** 2, flops=0.5 * case['n'] ** 2 * 64 * 40)
    if kind == 'hook':
        n, r = case['n'], case['nang']
        return dict(bytes=16.0 * (n * n + 2 * n * r), flops=8.0 / 3 * n ** 3 + 8.0 * n * n * r)
    if kind == 'far':
        pairs = float(case['rows'] * case['cols'])
        return dict(bytes=pairs * 3 * 4 * 16, flops=pairs * case['order'] ** 2 * 120)
    # body of revolution: kernel samples of every point pair over half a turn (about 60
    # operations a sample), their moments at every order (10 real sums a sample and order for the
    # closed-body formulation, 2 for the EFIE), one dense system of order 2 n per order m >= 0
    n, modes = case['segments'], case['krho'] + max(12.0, 4.05 * case['krho'] ** (1.0 / 3.0) + 2.0)
    xi = 0.5 * (1.5 * (2.0 * case['krho'] + modes + 2) + 32.0)
    sums = 2.0 if case['formulation'] == 'efie' else 10.0
    samples = n * n * 9.0 * xi / 2
    order = 2.0 * n
    # a transform of a point pair's samples to its orders: about 2.5 log2(2 xi) operations a sample and sum
    return dict(bytes=modes * (3 * 16 * order ** 2 + 4 * 16 * order * case['nang']),
                flops=samples * (60 + 2.5 * math.log2(2 * xi) * sums) +
                modes * (8.0 / 3 * order ** 3 + 16.0 * order ** 2 * case['nang']))


# ------------------------------------------------------------------ exact (64 bits, no package code)
def _gauss(q):
    x, w = np.polynomial.legendre.leggauss(q)
    return torch.from_numpy(0.5 * (x + 1.0)), torch.from_numpy(0.5 * w)


def _hankel_low(x):
    """H0^(2), H1^(2) for x < 25: Miller's backward recurrence for J_n, Neumann's series for Y_0
    (DLMF 10.8, 10.23) and its derivative for Y_1 (torch.special's Bessel functions are single
    precision near x = 5)."""
    top = 72
    hi, cur = torch.zeros_like(x), torch.full_like(x, 1e-200)
    norm, y0, dy = torch.zeros_like(x), torch.zeros_like(x), torch.zeros_like(x)
    for n in range(top, 0, -1):
        hi, cur = cur, (2 * n / x) * cur - hi       # cur = J_{n-1}, hi = J_n (up to the scale)
        big = cur.abs() > 1e200
        if bool(big.any()):
            for v in (hi, cur, norm, y0, dy):
                v[big] *= 1e-200
        k, odd = divmod(n - 1, 2)
        if not odd and k > 0:                       # J_{2k} in hand, J_{2k+1} in hi
            norm += 2 * cur
            y0 += (-1) ** k / k * cur
            dy -= (-1) ** k / (2 * k) * hi
        if odd:                                     # J_{2k+1} = cur is J_{2(k+1)-1}
            dy += (-1) ** (k + 1) / (2 * (k + 1)) * cur
    norm += cur
    j0, j1, y0, dy = cur / norm, hi / norm, y0 / norm, dy / norm
    log = torch.log(x / 2) + 0.57721566490153286061
    y0 = (2 / math.pi) * (log * j0 - 2 * y0)
    y1 = -(2 / math.pi) * (j0 / x - log * j1 - 2 * dy)
    return torch.complex(j0, -y0), torch.complex(j1, -y1)


def _hankel_high(x, nu):
    """H_nu^(2) for x >= 25 by Hankel's expansion (DLMF 10.17.5-6)."""
    total, term = torch.zeros_like(x, dtype=torch.complex128), torch.ones_like(x, dtype=torch.complex128)
    for m in range(18):
        total += term
        term = term * ((4 * nu * nu - (2 * m + 1) ** 2) / ((m + 1) * 8)) * (-1j / x)
    phase = x - (0.5 * nu + 0.25) * math.pi
    return torch.sqrt(2 / (math.pi * x)) * torch.complex(torch.cos(phase), -torch.sin(phase)) * total


def _kernels(r, k):
    """(j/4) H0^(2)(k r) and (j/4) k H1^(2)(k r)."""
    x = k * r
    h0, h1 = torch.empty_like(x, dtype=torch.complex128), torch.empty_like(x, dtype=torch.complex128)
    low = x < 25.0
    h0[low], h1[low] = _hankel_low(x[low])
    high = ~low
    h0[high], h1[high] = _hankel_high(x[high], 0), _hankel_high(x[high], 1)
    return 0.25j * h0, 0.25j * k * h1


def _pair_blocks(a, b, nrm, length, eo, es, k, xo, xs, w):
    """S, D and K' blocks (pairs, 2, 2) of the element pairs (eo, es): points xo, xs in [0, 1] of
    either element with weight w (product rule or any other)."""
    po = a[eo][:, None, :] + xo[None, :, None] * (b - a)[eo][:, None, :]
    r = po - (a[es][:, None, :] + xs[None, :, None] * (b - a)[es][:, None, :])
    dist = torch.sqrt((r * r).sum(-1))
    g, h = _kernels(dist, k)
    fo, fs = torch.stack([1 - xo, xo]), torch.stack([1 - xs, xs])
    test = (w * fo[:, None] * fs[None, :]).reshape(4, -1).to(torch.complex128)
    scale = (length[eo] * length[es]).to(torch.complex128)[:, None]
    pn_s, pn_o = (r * nrm[es][:, None, :]).sum(-1) / dist, -(r * nrm[eo][:, None, :]).sum(-1) / dist
    return [(v @ test.T * scale).reshape(-1, 2, 2) for v in (g, h * pn_s, h * pn_o)]


def _graded(q, levels):
    """Gauss points on [0, 1] in parts halved ``levels`` times towards both ends."""
    x, w = _gauss(q)
    halves = 0.5 ** torch.arange(levels, 0, -1, dtype=torch.float64)
    cuts = torch.cat([halves.new_zeros(1), halves, 1 - halves.flip(0)[1:], halves.new_ones(1)])
    size = torch.diff(cuts)[:, None]
    return (cuts[:-1, None] + size * x[None, :]).reshape(-1), (size * w[None, :]).reshape(-1)


def _square(x, w):
    return x.repeat_interleave(len(x)), x.repeat(len(x)), (w[:, None] * w[None, :]).reshape(-1)


def _duffy(q, power):
    """Corner rule on the unit square: both triangles at (0, 0), graded as t^power from the corner
    and, for neighbours of very different lengths, towards both sides of each triangle."""
    (t, w), (s, ws) = _gauss(q), _graded(8, 9)
    u, du = t ** power, power * t ** (power - 1)
    big, small = (u[:, None] + 0 * s[None, :]).reshape(-1), (u[:, None] * s[None, :]).reshape(-1)
    wt = ((w * du * u)[:, None] * ws[None, :]).reshape(-1)
    return torch.cat([big, small]), torch.cat([small, big]), torch.cat([wt, wt])


def _exact_systems(verts, k, pols):
    """([matrix of each polarisation], elements) of the combined-field Galerkin systems of a drawn
    (clockwise) polygon: nodes reversed about the first one, element j from node j to node j + 1,
    normal (-t_y, t_x)."""
    n = len(verts)
    a = torch.from_numpy(np.ascontiguousarray(verts[(-np.arange(n)) % n]))
    b = torch.roll(a, -1, 0)
    length = torch.sqrt(((b - a) ** 2).sum(-1))
    t = (b - a) / length[:, None]
    nrm = torch.stack([-t[:, 1], t[:, 0]], -1)
    mid = 0.5 * (a + b)
    ratio = torch.cdist(mid, mid) / torch.maximum(length[:, None], length[None, :])
    idx = torch.arange(n)
    gap = (idx[:, None] - idx[None, :]) % n
    touch = (gap == 1) | (gap == n - 1)
    near = (ratio < 3.0) & ~touch & (gap != 0)
    S = torch.zeros(n, n, 2, 2, dtype=torch.complex128)
    D, K = torch.zeros_like(S), torch.zeros_like(S)

    def put(eo, es, blocks):
        for m, v in zip((S, D, K), blocks):
            m[eo, es] = v

    # near pairs of like lengths take 60 points of either element; next to a much longer element
    # (the base of a blunt trailing edge) a rule graded towards both ends
    uneven = torch.maximum(length[:, None], length[None, :]) > 2.0 * torch.minimum(length[:, None], length[None, :])
    for mask, rule, chunk in ((~near & ~touch & (gap != 0), _square(*_gauss(9)), 4000),
                              (near & ~uneven, _square(*_gauss(60)), 64),
                              (near & uneven, _square(*_graded(10, 14)), 8)):
        rows, cols = torch.nonzero(torch.triu(mask), as_tuple=True)
        for i in range(0, len(rows), chunk):
            eo, es = rows[i:i + chunk], cols[i:i + chunk]
            blocks = _pair_blocks(a, b, nrm, length, eo, es, k, *rule)
            put(eo, es, blocks)
            put(es, eo, [blocks[m].transpose(1, 2) for m in (0, 2, 1)])  # the pair seen from the other element
    x, y, w = _duffy(28, 4)
    for step, xo, xs in ((1, 1 - x, y), (-1, x, 1 - y)):  # the next element shares our end, the previous our start
        es = (idx + step) % n
        for i in range(0, n, 64):
            put(idx[i:i + 64], es[i:i + 64], _pair_blocks(a, b, nrm, length, idx[i:i + 64], es[i:i + 64], k, xo, xs,
                                                            w))
    # an element with itself: the distance alone enters, int_0^1 G(k L u) c(u) du, graded as t^5
    t1, w1 = _gauss(48)
    u, du = t1 ** 5, 5 * t1 ** 4
    g, _h = _kernels(length[:, None] * u[None, :], k)
    for (i, j), c in (((0, 0), 2 / 3 - u + u ** 3 / 3), ((0, 1), 1 / 3 - u ** 3 / 3)):
        v = (g * (w1 * du * c)[None, :]).sum(-1) * length ** 2
        S[idx, idx, i, j] = v
        S[idx, idx, 1 - i, 1 - j] = v
    gamma = 1.0 / (1j * k)
    mass = torch.diag(length.to(torch.complex128))[:, :, None, None] * torch.tensor([[1 / 3, 1 / 6], [1 / 6, 1 / 3]], dtype=torch.float64)
    out = []
    for pol in pols:
        if pol == 'TM':
            E = S + gamma * (D + 0.5 * mass)
        else:
            sign = torch.tensor([[1.0, -1.0], [-1.0, 1.0]], dtype=torch.float64)
            W = -k * k * (nrm @ nrm.T)[:, :, None, None] * S + \
                sign * (S.sum((2, 3)) / (length[:, None] * length[None, :]))[:, :, None, None]
            E = K - 0.5 * mass - gamma * W
        A = torch.zeros(n, n, dtype=torch.complex128)
        for i in range(2):
            for j in range(2):
                A += torch.roll(E[:, :, i, j], (i, j), (0, 1))
        out.append(A)
    return out, (a, b, nrm, length)


def _exact_amplitudes(verts, k, angles, pols):
    matrices, (a, b, nrm, length) = _exact_systems(verts, k, pols)
    phi = torch.from_numpy(np.radians(np.asarray(angles, dtype=np.float64)))
    d = torch.stack([torch.cos(phi), torch.sin(phi)], -1)
    x, w = _gauss(20)
    pts = a[:, None, :] + x[None, :, None] * (b - a)[:, None, :]
    wave = torch.exp(1j * k * torch.einsum('eqx,rx->eqr', pts, d))
    load = [torch.einsum('q,eqr->er', (w * f).to(torch.complex128), wave) * length[:, None] for f in (1 - x, x)]
    dn = (nrm @ d.T).to(torch.complex128)
    out = []
    for pol, A in zip(pols, matrices):
        fac = torch.ones_like(dn) if pol == 'TM' else 1j * k * dn
        X = torch.linalg.solve(A, -(load[0] * fac + torch.roll(load[1] * fac, 1, 0)))
        out.append(((load[0] * X + load[1] * torch.roll(X, -1, 0)) * (1.0 + dn)).sum(0).numpy())
    return out


def _mesh(case, verts, freq):
    """The elements of one frequency of an ``rcs2d`` case: a 17-gon's sides in ceil(10 L / lambda)
    equal pieces when there are several."""
    if case['nfreq'] == 1:
        return verts
    cut = np.full(17, case['n'] // 17)
    cut[:case['n'] % 17] += 1
    corner = verts[np.cumsum(cut) - cut]
    nxt = np.roll(corner, -1, axis=0)
    lam = C0 / (freq * 1e9)
    out = []
    for p, q in zip(corner, nxt):
        m = max(1, math.ceil(float(np.hypot(*(q - p))) * 10 / lam))
        out.append(p + (np.arange(m) / m)[:, None] * (q - p))
    return np.concatenate(out)


def exact(case, seed):
    kind = case['kind']
    if kind == 'bor':
        return None  # the modal operators of every order in 64-bit NumPy take minutes
    if kind == 'hook':
        a, b = _hook_system(case, seed)
        return np.linalg.solve(a, b)
    if kind == 'far':
        t = _far_tile(case, seed)
        out = [[] for _ in range(3)]
        obs, src, on, sn = (torch.from_numpy(t[key]) for key in ('obs', 'src', 'obs_n', 'src_n'))
        test = torch.from_numpy((t['qw'][:, None] * t['phi']).T).to(torch.complex128)
        for i in range(len(obs)):
            r = obs[i][None, :, None, :] - src[:, None, :, :]
            dist = torch.sqrt((r * r).sum(-1))
            g, h = _kernels(dist, t['k'])
            # the observation-normal kernel and its transpose with the source normal
            for o, v in zip(out, (g, -h * (r @ on[i]) / dist, h * torch.einsum('jpqx,jx->jpq', r, sn) / dist)):
                o.append(torch.einsum('ap,jpq,bq->abj', test, v, test))
            out[2][-1] = out[2][-1].transpose(0, 1)  # the mirrored block: the source's basis first
        return tuple(torch.stack([v.reshape(4, -1) for v in o], 1).numpy() for o in out)
    if kind == 'rcs2d':
        verts, cost = _polygon(case, seed), sum((case['n'] * f) ** 2 for f in
                                                np.geomspace(1.0 / case['band'], 1.0, case['nfreq'])) * 2
        if cost > 2 * EXACT_MAX_ORDER ** 2:
            return None
        ang = _angles(case, seed)
        out = {ch: [] for ch in ('VV', 'HH')}
        for f in _frequencies(case, verts):
            mesh, k = _mesh(case, verts, f), 2.0 * math.pi * f * 1e9 / C0
            for ch, amp in zip(out, _exact_amplitudes(mesh, k, ang, ('TE', 'TM'))):
                out[ch].append(amp)
        return {ch: np.concatenate(v) for ch, v in out.items()}
    if case['n'] > EXACT_MAX_ORDER:
        return None
    verts = _polygon(case, seed)
    if kind == 'fill':
        return _exact_systems(verts, _wavenumber(verts), [case['pol']])[0][0].T.contiguous()
    return _exact_amplitudes(verts, _wavenumber(verts), _angles(case, seed), [case['pol']])[0]
