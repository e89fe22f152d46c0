"""Host-buffer entry points around the sizes where their copies change: below 4 MiB up and 2 MiB
down one plain copy, above it 1 MiB chunks through the handle's pinned slots on several threads; row-major
systems are transposed on the device."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip('torch')


@pytest.mark.parametrize('n, nrhs', [(1, 1), (33, 5), (361, 1), (363, 40), (600, 129)])
@pytest.mark.parametrize('layout', ['C', 'F', 'strided'])
def test_dense_hook_takes_every_layout(n, nrhs, layout):
    from grim_20261007_b200.twod.solver import _solve_dense_gpu
    rng = np.random.default_rng(n)

    def lay(v):
        if layout == 'strided':
            out = np.zeros((2 * v.shape[0], 2 * v.shape[1]), complex)[::2, ::2]
            out[...] = v
            return out
        return np.array(v, order=layout)

    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3.0 * n ** 0.5 * np.eye(n)
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    al, bl = lay(a), lay(b)
    x, _name = _solve_dense_gpu(al, bl)
    res = np.max(np.abs(a @ x - b)) / (np.max(np.sum(np.abs(a), axis=1)) * np.max(np.abs(x)))
    assert res < 1e-14
    assert np.array_equal(al, a) and np.array_equal(bl, b)  # the inputs are borrowed
    assert x.flags.c_contiguous if bl.flags.c_contiguous else x.flags.f_contiguous
    v, _name = _solve_dense_gpu(al, np.ascontiguousarray(b[:, 0]))
    assert v.shape == (n,) and np.max(np.abs(v - x[:, 0])) <= 1e-13 * np.max(np.abs(x))


@pytest.mark.parametrize('n, nrhs', [(511, 1), (512, 1), (500, 262), (500, 263)])
@pytest.mark.parametrize('order', ['C', 'F'])
def test_dense_hook_on_both_sides_of_the_staged_copies(n, nrhs, order):
    """4 MiB of matrix and right-hand sides up, 2 MiB of solution down."""
    from grim_20261007_b200.twod.solver import _solve_dense_gpu
    rng = np.random.default_rng(n + nrhs)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3.0 * n ** 0.5 * np.eye(n)
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    x, _name = _solve_dense_gpu(np.array(a, order=order), np.array(b, order=order))
    assert np.max(np.abs(a @ x - b)) < 1e-14 * (np.max(np.sum(np.abs(a), axis=1)) * np.max(np.abs(x)))


@pytest.mark.parametrize('n, nrhs', [(2, 2600), (16, 300), (16, 310), (60, 70), (60, 2500), (121, 1), (122, 1)])
def test_dense_hook_on_both_sides_of_the_row_major_rule(n, nrhs):
    """n (n + 3 nrhs) from 15000 on goes up row-major; few rows and many columns among them."""
    from grim_20261007_b200.twod.solver import _solve_dense_gpu
    rng = np.random.default_rng(n + nrhs)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3.0 * n ** 0.5 * np.eye(n)
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    x, _name = _solve_dense_gpu(a, b)
    assert np.max(np.abs(a @ x - b)) < 1e-14 * (np.max(np.sum(np.abs(a), axis=1)) * np.max(np.abs(x)))


@pytest.mark.parametrize('mode, nrhs', [('PREC_FP64', 64), ('PREC_FP64', 3500), ('PREC_MIXED', 64), ('PREC_MIXED', 3)])
def test_row_major_systems_keep_no_more_memory_than_column_major_ones(mode, nrhs):
    """The device memory that a call leaves held, and the answer with its rows in a buffer of the
    solve (a matrix of 140 MB: one host array after the other goes through it)."""
    import ctypes
    from grim_20261007_b200 import _lib
    lib = _lib.load()
    n = 3000
    rng = np.random.default_rng(nrhs)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3.0 * n ** 0.5 * np.eye(n)
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    held, xs = [], []
    for rows in (False, True):
        h, info, free, total = ctypes.c_void_p(), ctypes.c_int(-1), ctypes.c_size_t(), ctypes.c_size_t()
        _lib.check(lib.grim_create(0, ctypes.byref(h)))
        try:
            _lib.check(lib.grim_mem_info(h, ctypes.byref(free), ctypes.byref(total)))
            before = free.value
            if rows:
                x = np.empty_like(b)
                _lib.check(lib.grim_zgesv_rowmajor(h, n, nrhs, a.ctypes.data, b.ctypes.data, x.ctypes.data,
                                                   getattr(_lib, mode), ctypes.byref(info)))
            else:
                af, x = np.asfortranarray(a), np.asfortranarray(b)
                _lib.check(lib.grim_zgesv_batched(h, n, nrhs, af.ctypes.data, n, x.ctypes.data, n, getattr(_lib, mode),
                                                  ctypes.byref(info)))
            _lib.check(lib.grim_synchronize(h))
            _lib.check(lib.grim_mem_info(h, ctypes.byref(free), ctypes.byref(total)))
            held.append(before - free.value)
            xs.append(x)
        finally:
            lib.grim_destroy(h)
    assert np.max(np.abs(xs[1] - xs[0])) <= 1e-11 * np.max(np.abs(xs[0]))
    extra = max(0, nrhs - n) * n * 16  # right-hand sides wider than the matrix
    assert held[1] <= held[0] + extra + (64 << 20), held


def test_row_major_systems_take_millions_of_columns():
    """More 32-column tiles of the solution than a grid's y extent."""
    import ctypes
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.device import context
    ctx = context()
    a = np.array([[2.0 + 1.0j, 0.5], [1.0j, 3.0]])
    b = np.stack([np.arange(2_100_000) + 0j, np.arange(2_100_000)[::-1] * 1j])
    x, info = np.empty_like(b), ctypes.c_int(-1)
    _lib.check(ctx.lib.grim_zgesv_rowmajor(ctx.h, 2, b.shape[1], a.ctypes.data, b.ctypes.data, x.ctypes.data,
                                           _lib.PREC_FP64, ctypes.byref(info)))
    assert np.max(np.abs(a @ x - b)) <= 1e-14 * np.max(np.abs(b))


@pytest.mark.parametrize('rows', [False, True])
def test_dense_systems_on_the_per_thread_stream(rows):
    """cudaStreamPerThread (handle value 2) is another stream on every thread: copies from a team of
    threads would not be ordered with the solve."""
    import ctypes
    from grim_20261007_b200 import _lib
    lib = _lib.load()
    n, nrhs = 700, 90
    rng = np.random.default_rng(n)
    a = rng.standard_normal((n, n)) + 1j * rng.standard_normal((n, n)) + 3.0 * n ** 0.5 * np.eye(n)
    b = rng.standard_normal((n, nrhs)) + 1j * rng.standard_normal((n, nrhs))
    h, info = ctypes.c_void_p(), ctypes.c_int(-1)
    _lib.check(lib.grim_create(0, ctypes.byref(h)))
    try:
        _lib.check(lib.grim_set_stream(h, ctypes.c_void_p(2)))
        if rows:
            x = np.empty_like(b)
            _lib.check(lib.grim_zgesv_rowmajor(h, n, nrhs, a.ctypes.data, b.ctypes.data, x.ctypes.data, _lib.PREC_FP64,
                                               ctypes.byref(info)))
        else:
            af, x = np.asfortranarray(a), np.asfortranarray(b)
            _lib.check(lib.grim_zgesv_batched(h, n, nrhs, af.ctypes.data, n, x.ctypes.data, n, _lib.PREC_FP64,
                                              ctypes.byref(info)))
    finally:
        lib.grim_destroy(h)
    assert np.max(np.abs(a @ x - b)) < 1e-14 * (np.max(np.sum(np.abs(a), axis=1)) * np.max(np.abs(x)))


@pytest.mark.parametrize('rows, cols', [(3, 2), (130, 131), (181, 182), (300, 257)])
def test_far_block_from_zero_equals_accumulating(rows, cols):
    """Fresh accumulators equal sums into zeros; sums into other values keep them."""
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.twod import farblock
    rng = np.random.default_rng(rows)
    q, k = 5, 20.0
    x, w = np.polynomial.legendre.leggauss(q)
    s = np.linspace(0.0, 0.05, q)
    obs = np.ascontiguousarray(np.stack([np.arange(rows)[:, None] * 0.06 + s, 0.01 * np.ones((rows, q))], -1))
    src = np.ascontiguousarray(np.stack([np.arange(cols)[:, None] * 0.06 + s, np.full((cols, q), 1.0)], -1))
    phi = np.ascontiguousarray(np.stack([(1 - x) / 2, (1 + x) / 2], -1))
    qw = np.ascontiguousarray(w / 2)
    on, sn = np.tile([0.0, 1.0], (rows, 1)), np.tile([0.6, 0.8], (cols, 1))
    far = (rng.uniform(size=(rows, cols)) < 0.8).astype(np.uint8)
    table = farblock.KernelTable(k, 25.0)
    got = farblock.far_block(table, k, obs, src, qw, phi, on, sn, far, 1, True, True, True)
    start = [rng.standard_normal((4, rows, cols)) + 1j * rng.standard_normal((4, rows, cols)) for _ in range(3)]
    acc = [v.copy() for v in start]
    coeff = np.ascontiguousarray(table.normalized_power)
    lib = _lib.load()
    assert lib.ghost_far_block(rows, cols, q, 2, obs.ctypes.data, src.ctypes.data, qw.ctypes.data, phi.ctypes.data,
                               on.ctypes.data, sn.ctypes.data, far.ctypes.data, 1, 1, 1, 1, k, 0.0,
                               len(table.bounds) - 1, table.bounds.ctypes.data, coeff.shape[1] - 1, coeff.ctypes.data,
                               *(v.ctypes.data for v in acc)) == 0
    for g, a, s0 in zip(got, acc, start):
        assert np.all(g[:, far == 0] == 0)
        assert np.array_equal(a[:, far == 0], s0[:, far == 0])
        assert np.max(np.abs(a - s0 - g)) <= 1e-15 * np.max(np.abs(s0)) * 4


def test_far_block_threads_give_their_memory_back():
    """Each host thread has a handle of its own (70 MB of accumulators on the device, 16 MiB of pinned
    slots): nothing of it stays when the thread has ended."""
    import ctypes
    import threading
    from grim_20261007_b200 import _lib
    from grim_20261007_b200.device import context
    from grim_20261007_b200.twod import farblock
    ctx = context()
    count, q, k = 600, 5, 20.0
    x, w = np.polynomial.legendre.leggauss(q)
    s = np.linspace(0.0, 0.05, q)
    pts = [np.ascontiguousarray(np.stack([np.arange(count)[:, None] * 0.06 + s, np.full((count, q), y)], -1))
           for y in (0.01, 1.0)]
    phi = np.ascontiguousarray(np.stack([(1 - x) / 2, (1 + x) / 2], -1))
    norms = np.tile([0.0, 1.0], (count, 1))
    far = np.ones((count, count), np.uint8)
    table = farblock.KernelTable(k, 45.0)
    sums = []

    def run():
        sums.append(farblock.far_block(table, k, *pts, np.ascontiguousarray(w / 2), phi, norms, norms, far, 1, True, True,
                                       True)[0].sum())

    def free():
        got, total = ctypes.c_size_t(), ctypes.c_size_t()
        _lib.check(ctx.lib.grim_mem_info(ctx.h, ctypes.byref(got), ctypes.byref(total)))
        return got.value

    def turn():
        t = threading.Thread(target=run)
        t.start()
        t.join()
    turn()
    torch.cuda.synchronize()
    before = free()
    for _ in range(5):
        turn()
    torch.cuda.synchronize()
    assert len(set(sums)) == 1
    assert before - free() <= 64 << 20
