"""Positive QR and LQ against Householder factors in extended conditions.

Q' Q = 1 and Q R = A hold to a few n eps whatever the condition number (both the Gram route and
the Householder routine it falls back to); the factors themselves differ from another algorithm's
by n eps cond(A)."""
import numpy as np
import pytest

import mpsgb

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def ctx():
    return mpsgb.Context(0)


def _ref(a):
    q, r = np.linalg.qr(a)
    ph = np.diagonal(r).copy()
    ph[ph == 0] = 1
    ph = ph / np.abs(ph)
    return q * ph, np.conj(ph)[:, None] * r


def _check(a, q, r, cond):
    m, n = a.shape
    k = min(m, n)
    assert np.linalg.norm(q.conj().T @ q - np.eye(k)) <= 8 * n * EPS
    assert np.linalg.norm(a - q @ r) <= 8 * n * EPS * np.linalg.norm(a)
    assert np.all(np.tril(r, -1) == 0)
    d = np.diagonal(r)[:k]
    assert np.all(d.real >= 0) and np.all(d.imag == 0)
    if cond is not None:
        q0, r0 = _ref(a)
        assert np.linalg.norm(q - q0) <= 8 * n * EPS * cond
        assert np.linalg.norm(r - r0) <= 8 * n * EPS * cond * np.linalg.norm(r0)


def _matrix(rng, m, n, cx, cond):
    a = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cx else 0)
    if cond:
        u, _, v = np.linalg.svd(a, full_matrices=False)
        a = u * np.logspace(0, -np.log10(cond), min(m, n)) @ v
        return a, cond
    s = np.linalg.svd(a, compute_uv=False)
    return a, s[0] / s[-1]


# one column, block rows and their edges, one block row of the update more, wide matrices, block
# rows longer than a pass of the chip
SHAPES = [(2, 1), (6, 3), (32, 16), (40, 17), (64, 33), (96, 48), (130, 65), (512, 256),
          (700, 300), (20, 34), (64, 100), (256, 256), (1100, 1024), (1100, 1025)]


@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("m,n", SHAPES)
def test_left_and_right(ctx, m, n, cx):
    rng = np.random.default_rng(m * n)
    if m % 2:
        m += 1
    a, cond = _matrix(rng, m, n, cx, None)
    al, c = mpsgb.left_orth(mpsgb.DeviceTensor.from_numpy(
        ctx, "mps", a.reshape(m // 2, 2, n, order="F")))
    _check(a, al.numpy().reshape(m, -1, order="F"), c.numpy(), cond if m >= n else None)
    # LQ of the adjoint: the same factors
    b = a.conj().T
    c2, ar = mpsgb.right_orth(mpsgb.DeviceTensor.from_numpy(
        ctx, "mps", b.reshape(n, 2, m // 2, order="F")))
    _check(a, ar.numpy().reshape(-1, m, order="F").conj().T, c2.numpy().conj().T,
           cond if m >= n else None)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("cond", [1e3, 1e5, 1e7, 1e10, 1e15])
@pytest.mark.parametrize("cx", [False, True])
def test_ill_conditioned(ctx, cx, cond):
    """From one correction to several and to the Householder fallback."""
    rng = np.random.default_rng(int(np.log10(cond)))
    a, c = _matrix(rng, 200, 90, cx, cond)
    al, r = mpsgb.left_orth(mpsgb.DeviceTensor.from_numpy(
        ctx, "mps", a.reshape(100, 2, 90, order="F")))
    _check(a, al.numpy().reshape(200, 90, order="F"), r.numpy(), c if cond <= 1e10 else None)


def test_rank_deficient_scaled_and_non_finite(ctx):
    rng = np.random.default_rng(9)
    a = rng.standard_normal((80, 30))
    a[:, 20:] = 0  # an enlarged bond: zero columns appended
    q, r = (t.numpy() for t in mpsgb.left_orth(mpsgb.DeviceTensor.from_numpy(
        ctx, "mps", a.reshape(40, 2, 30, order="F"))))
    _check(a, q.reshape(80, 30, order="F"), r, None)
    for scale in (1e-150, 1e150):  # squares leave the range of FP64 only beyond this
        b = scale * rng.standard_normal((80, 30))
        b[:, ::2] *= 1e-4
        q, r = (t.numpy() for t in mpsgb.left_orth(mpsgb.DeviceTensor.from_numpy(
            ctx, "mps", b.reshape(40, 2, 30, order="F"))))
        _check(b, q.reshape(80, 30, order="F"), r, None)
    for scale in (1e-200, 1e200):  # the Gram matrix under- or overflows: Householder
        b = scale * rng.standard_normal((80, 30))
        q, r = (t.numpy() for t in mpsgb.left_orth(mpsgb.DeviceTensor.from_numpy(
            ctx, "mps", b.reshape(40, 2, 30, order="F"))))
        assert np.linalg.norm(q.reshape(80, 30, order="F").T @ q.reshape(80, 30, order="F")
                              - np.eye(30)) <= 8 * 30 * EPS
        assert np.all(np.abs(b - q.reshape(80, 30, order="F") @ r) <= 240 * EPS * np.abs(b).max())
    assert ctx.device_status() == 0


def _factors(ctx, a):
    """Positive QR of `a` (rows a multiple of two) and, from the LQ of its adjoint, again."""
    m, n = a.shape
    q, r = mpsgb.left_orth(mpsgb.DeviceTensor.from_numpy(
        ctx, "mps", a.reshape(m // 2, 2, n, order="F")))
    yield q.numpy().reshape(m, -1, order="F"), r.numpy()
    c, q = mpsgb.right_orth(mpsgb.DeviceTensor.from_numpy(
        ctx, "mps", a.conj().T.reshape(n, 2, m // 2, order="F")))
    yield q.numpy().reshape(-1, m, order="F").conj().T, c.numpy().conj().T


@pytest.mark.parametrize("triangular", [False, True])
@pytest.mark.parametrize("shape", [(200, 90), (512, 256)])  # FMA products, digit products
@pytest.mark.parametrize("cx", [False, True])
def test_condition_numbers_of_several_passes(ctx, cx, shape, triangular):
    """Condition numbers of 1e6 to 1e9, where the factor of the Gram matrix needs from one to
    several corrections or is given up: Q R = A throughout.  Also as a gauge step meets them, an
    isometry times a triangular bond matrix."""
    m, n = shape
    rng = np.random.default_rng(m)
    for cond in 1e6 * 2.0 ** np.arange(11):
        a, _ = _matrix(rng, m, n, cx, cond)
        if triangular:
            a = _matrix(rng, m, n, cx, None)[0]
            v = np.linalg.qr(_matrix(rng, n, n, cx, None)[0])[0]
            a = np.linalg.qr(a)[0] @ np.linalg.qr(np.logspace(0, -np.log10(cond), n)[:, None] * v)[1]
        for q, r in _factors(ctx, a):
            _check(a, q, r, None)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("decades", [4, 8, 12])
@pytest.mark.parametrize("shape", [(200, 90), (512, 256), (128, 300)])
@pytest.mark.parametrize("cx", [False, True])
def test_graded_columns(ctx, cx, shape, decades):
    """Columns of very different norm, as a site tensor times its Schmidt values has them.  Each is
    held to its own norm (a backward error of Householder's size per column), and Q is that of the
    matrix without the grading.  Alone (rows), the grading of the rows changes nothing either."""
    m, n = shape
    rng = np.random.default_rng(m + decades)
    a, cond = _matrix(rng, m, n, cx, None)
    k = min(m, n)
    if m < n:
        s = np.linalg.svd(a[:, :m], compute_uv=False)
        cond = s[0] / s[-1]
    q0, _ = _ref(a)
    d = np.logspace(0, -decades, n)[rng.permutation(n)]
    b = a * d
    q, r = next(_factors(ctx, b))
    assert np.linalg.norm(q.conj().T @ q - np.eye(k)) <= 8 * n * EPS
    assert np.all(np.linalg.norm(b - q @ r, axis=0) <= 8 * n * EPS * np.linalg.norm(b, axis=0))
    assert np.linalg.norm(q - q0[:, :k]) <= 8 * n * EPS * cond
    if m >= n:
        c = np.logspace(0, -decades, m)[rng.permutation(m)][:, None] * a
        for q, r in _factors(ctx, c):
            assert np.linalg.norm(q.conj().T @ q - np.eye(k)) <= 8 * n * EPS
            assert np.all(np.linalg.norm(c - q @ r, axis=0) <= 8 * n * EPS * np.linalg.norm(c, axis=0))
    assert ctx.device_status() == 0


@pytest.mark.parametrize("cx", [False, True])
def test_where_the_products_would_be_slow(ctx, cx):
    """More rows than the digits' contraction takes and too many for the small tiles: the library's
    panels, as their four launches tell; the Gram route on either side of it."""
    rng = np.random.default_rng(4)
    for m, n, gram in ((200000, 4, not cx), (270000, 8, False), (131072 if cx else 262144, 8, True)):
        a = rng.standard_normal((m, n)) + (1j * rng.standard_normal((m, n)) if cx else 0)
        t = mpsgb.DeviceTensor.from_numpy(ctx, "mps", a.reshape(m // 2, 2, n, order="F"))
        before = ctx.kernel_launches()
        q, r = mpsgb.left_orth(t)
        assert (ctx.kernel_launches() - before > 6) == gram, (m, n)
        _check(a, q.numpy().reshape(m, n, order="F"), r.numpy(), None)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("shape", [(64, 33), (512, 256)])
@pytest.mark.parametrize("cx", [False, True])
def test_factorisations_that_stop_early(ctx, cx, shape):
    """Low rank (a pivot runs out on the way), zero and non-finite columns anywhere: the panels'
    factors, and the counters ready for the next factorisation."""
    m, n = shape
    rng = np.random.default_rng(6)
    good, cond = _matrix(rng, m, n, cx, None)
    low = _matrix(rng, m, n // 3, cx, None)[0] @ _matrix(rng, n // 3, n, cx, None)[0]
    first, last = good.copy(), good.copy()
    first[:, 0] = 0
    last[:, -1] = 0
    nan = good.copy()
    nan[5, 7] = np.nan
    for a in (low, first, last, nan):
        q, r = next(_factors(ctx, a))
        if a is nan:
            assert not np.isfinite(r).all()
        else:
            _check(a, q, r, None)
        q, r = next(_factors(ctx, good))
        _check(good, q, r, cond)
    assert ctx.device_status() == 0
