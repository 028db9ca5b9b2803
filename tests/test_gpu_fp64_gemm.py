"""Plain-precision products of the device against extended precision.

Entry bound: the digits keep every entry of a row (column) to half a unit of 2^-54 of its
largest part, and the product digits left out are smaller still, so over K terms
|C - C*| <= 2 K 2^-54 a b + 2^-53 |C*| with a, b the largest parts of the row and the column
(four real products per complex one).  The plain-FMA kernel used for small products is within
K 2^-53 sum |a_k| |b_k| <= K^2 2^-53 a b."""
import numpy as np
import pytest

import mpsgb
from mpsgb import _lib as L

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return mpsgb.Context(0)


def _rand(rng, shape, cx, spread):
    x = rng.standard_normal(shape)
    if cx:
        x = x + 1j * rng.standard_normal(shape)
    if spread:  # magnitudes over many decades inside every row and column
        x = x * 10.0 ** rng.uniform(-spread, 0, shape)
    return x


def _wide(a):
    return a.astype(np.clongdouble if np.iscomplexobj(a) else np.longdouble)


def _part(a, axis):
    return np.maximum(np.abs(a.real), np.abs(a.imag) if np.iscomplexobj(a) else 0).max(axis=axis)


def _check(C, A, B, small):
    """C = A B for 2-d arrays."""
    K = A.shape[1]
    ref = _wide(A) @ _wide(B)
    err = np.abs(_wide(C) - ref).astype(np.float64)
    n = 4.0 if np.iscomplexobj(C) else 1.0
    scale = np.outer(_part(A, 1), _part(B, 0))
    bound = n * (K * K * 2.0 ** -53 if small else 2 * K * 2.0 ** -54) * scale
    bound = bound + 2.0 ** -52 * np.abs(ref).astype(np.float64)
    assert np.all(err <= bound), float((err / np.maximum(bound, 1e-300)).max())
    return float(np.linalg.norm(err) / np.linalg.norm(ref.astype(C.dtype)))


# (rows / 2, K, columns): tile edges of 128 x 64 and 128 x 32, k-blocks of 64, one and many
# splits, single rows and columns
SHAPES = [(64, 384, 256, 0), (64, 385, 255, 3), (65, 191, 513, 0), (150, 290, 149, 8),
          (301, 550, 37, 0), (1, 4097, 1500, 0), (1500, 4097, 1, 0), (33, 3000, 65, 0),
          (510, 70, 600, 2), (160, 128, 129, 0), (11, 23, 69, 0), (8, 700, 9, 0), (2, 1, 3, 0)]


@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("shape", SHAPES)
def test_mul_tail(ctx, shape, cx):
    h, K, N, spread = shape
    rng = np.random.default_rng(hash(shape) % 1000)
    A = _rand(rng, (h, 2, K), cx, spread)
    C = _rand(rng, (K, N), cx, spread)
    out = mpsgb.states.mul_tail(mpsgb.DeviceTensor.from_numpy(ctx, "mps", A),
                                mpsgb.DeviceTensor.from_numpy(ctx, "bond", C)).numpy()
    mac = 2 * h * K * N * (4 if cx else 1)
    _check(out.reshape(2 * h, N, order="F"), A.reshape(2 * h, K, order="F"), C, mac < 1.2e7)
    assert ctx.device_status() == 0


@pytest.mark.parametrize("cx", [False, True])
def test_conjugated_and_accumulating_products(ctx, cx):
    """Y - X (X' Y): a product with a conjugate transpose on the left, one that accumulates
    with alpha = -1."""
    rng = np.random.default_rng(5)
    X = _rand(rng, (150, 2, 141), cx, 0) / 17.0
    Y = _rand(rng, (150, 2, 333), cx, 0)  # 1.4e7 products
    yd = mpsgb.DeviceTensor.from_numpy(ctx, "mps", Y)
    mpsgb.states.project_complement_(yd, mpsgb.DeviceTensor.from_numpy(ctx, "mps", X))
    x, y = _wide(X.reshape(300, 141, order="F")), _wide(Y.reshape(300, 333, order="F"))
    ref = y - x @ (x.conj().T @ y)
    got = yd.numpy().reshape(300, 333, order="F")
    assert np.linalg.norm((got - ref).astype(got.dtype)) <= 4e-15 * np.linalg.norm(
        ref.astype(got.dtype))


@pytest.mark.parametrize("cx", [False, True])
def test_batched_products(ctx, cx):
    """Both environment steps: a batch over MPO channels, right operand conjugated."""
    rng = np.random.default_rng(6)
    dt = np.complex128 if cx else np.float64
    W = np.asarray(mpsgb.heisenberg_XXX(6, dtype=dt).W[2])
    Dl, Dr = 93, 110
    GL = _rand(rng, (Dl, W.shape[0], Dl), cx, 0)
    GR = _rand(rng, (Dr, W.shape[3], Dr), cx, 0)
    A = _rand(rng, (Dl, 2, Dr), cx, 0)
    dev = lambda k, a: mpsgb.DeviceTensor.from_numpy(ctx, k, a)
    left = mpsgb.transfer_left(dev("gl", GL), W, dev("mps", A)).numpy()
    right = mpsgb.transfer_right(dev("gr", GR), W, dev("mps", A)).numpy()
    rl = np.einsum("bwk,kta->bwta", GL, A, optimize=True)
    rl = np.einsum("bwta,wstv->bsva", rl, W, optimize=True)
    rl = np.einsum("bsva,bsc->cva", rl, A.conj(), optimize=True)
    rr = np.einsum("atq,qvr->atvr", A, GR, optimize=True)
    rr = np.einsum("atvr,wstv->awsr", rr, W, optimize=True)
    rr = np.einsum("awsr,bsr->awb", rr, A.conj(), optimize=True)
    assert np.linalg.norm(left - rl) <= 3e-15 * np.linalg.norm(rl)
    assert np.linalg.norm(right - rr) <= 3e-15 * np.linalg.norm(rr)


@pytest.mark.parametrize("cx", [False, True])
def test_zero_blocks_and_extremes(ctx, cx):
    """Exact zeros stay exact zeros; huge, tiny and subnormal rows keep their scale."""
    rng = np.random.default_rng(7)
    h, K, N = 160, 320, 200  # 2e7 products
    A = _rand(rng, (2 * h, K), cx, 0)
    B = _rand(rng, (K, N), cx, 0)
    A[:130, 64:] = 0
    A[200:] = 0
    B[:64, 70:] = 0
    B[192:256] = 0
    A[5] *= 1e300
    A[6] *= 1e-300
    B[:, 3] *= 1e-20
    A[7, :] = 0
    A[8] *= 0
    A[8, 3] = 5e-324
    out = mpsgb.states.mul_tail(
        mpsgb.DeviceTensor.from_numpy(ctx, "mps", A.reshape(h, 2, K, order="F")),
        mpsgb.DeviceTensor.from_numpy(ctx, "bond", B)).numpy().reshape(2 * h, N, order="F")
    ref = A @ B
    assert np.array_equal(out == 0, (np.abs(A) != 0).astype(float) @ (np.abs(B) != 0) == 0) or \
        np.all(out[(np.abs(A) != 0).astype(float) @ (np.abs(B) != 0) == 0] == 0)
    for r in (5, 6, 0, 131):
        assert np.linalg.norm(out[r] - ref[r]) <= 1e-14 * np.linalg.norm(ref[r]), r
    assert np.all(np.abs(out[8] - ref[8]) <= 1e-323)


@pytest.mark.parametrize("cx", [False, True])
def test_non_finite_entries(ctx, cx):
    """A row or column with Inf or NaN gives what FMAs give; the others are unaffected."""
    rng = np.random.default_rng(8)
    h, K, N = 160, 320, 160
    A, B = _rand(rng, (2 * h, K), cx, 0), _rand(rng, (K, N), cx, 0)
    clean = A @ B
    A[17, 20] = np.inf
    A[140, 30] = np.nan
    B[50, 77] = np.nan
    out = mpsgb.states.mul_tail(
        mpsgb.DeviceTensor.from_numpy(ctx, "mps", A.reshape(h, 2, K, order="F")),
        mpsgb.DeviceTensor.from_numpy(ctx, "bond", B)).numpy().reshape(2 * h, N, order="F")
    bad = np.zeros(out.shape, bool)
    bad[[17, 140]] = True
    bad[:, 77] = True
    assert not np.isfinite(out[bad]).any()
    assert np.isnan(out[140]).all() and np.isnan(out[:, 77]).all()
    assert np.linalg.norm((out - clean)[~bad]) <= 1e-14 * np.linalg.norm(clean[~bad])


@pytest.mark.parametrize("h,K", [(12, 24), (75, 150), (128, 256)])
def test_chained_launches(ctx, h, K):
    """Products that feed one another, queued without a wait: the same bits as one at a time."""
    rng = np.random.default_rng(11)
    C = [mpsgb.DeviceTensor.from_numpy(
        ctx, "bond", np.linalg.qr(_rand(rng, (K, K), True, 0))[0]) for _ in range(3)]
    a0 = mpsgb.DeviceTensor.from_numpy(ctx, "mps", _rand(rng, (h, 2, K), True, 0))

    def run(wait):
        a = a0
        for i in range(40):
            a = mpsgb.states.mul_tail(a, C[i % 3])
            if wait:
                ctx.synchronize()
        return a.numpy()

    assert np.array_equal(run(True), run(False))


@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("Dl,Dr", [(1, 1), (3, 5), (7, 64), (65, 33), (90, 91), (160, 170)])
def test_left_and_right_products_together(ctx, Dl, Dr, cx):
    """A one-site operator whose products with the two environments share a launch (all but the
    largest), every tile of the small products and its remainders among them.  Each product errs
    by at most 4e-16 sqrt(K) of its terms' norm."""
    rng = np.random.default_rng(Dl + Dr)
    dt = np.complex128 if cx else np.float64
    H = mpsgb.heisenberg_XXX(6, dtype=dt)
    W = np.asarray(H.W[2])
    GL, GR = _rand(rng, (Dl, W.shape[0], Dl), cx, 0), _rand(rng, (Dr, W.shape[3], Dr), cx, 0)
    GL[:, 0, :] = np.eye(Dl)  # the channels "not started" and "finished"
    GR[:, -1, :] = np.eye(Dr)
    x = _rand(rng, (Dl, 2, Dr), cx, 0)
    dev = lambda k, a: mpsgb.DeviceTensor.from_numpy(ctx, k, a)
    op = mpsgb.DerivativeOperator(ctx, mpsgb._lib.GB_HEFF_AC, dev("gl", GL),
                                  H.device(ctx, dt)[2], None, dev("gr", GR),
                                  mpsgb.GB300Backend("fp64"))
    ref = np.einsum("bwk,kta->bwta", GL, x, optimize=True)
    ref = np.einsum("bwta,wstv->bsva", ref, W, optimize=True)
    scale = np.linalg.norm(np.einsum("bsva,avc->bsc", np.abs(ref), np.abs(GR), optimize=True))
    ref = np.einsum("bsva,avc->bsc", ref, GR, optimize=True)
    assert np.linalg.norm(op(dev("mps", x)).numpy() - ref) <= 4e-15 * scale


def _entry_bounds(A, B):
    """The bounds of an entry: by its row and column (digits), by its terms (FMAs)."""
    K = A.shape[1]
    four = 4.0 if np.iscomplexobj(A) else 1.0
    row = four * 2 * K * 2.0 ** -54 * np.outer(_part(A, 1), _part(B, 0))
    terms = four * K * 2.0 ** -53 * (np.abs(A) @ np.abs(B))
    return row, terms


# real multiply-adds just below and above 3.5 million, where digits take over, and far above
@pytest.mark.parametrize("shape,digits", [((64, 170, 160), False), ((64, 172, 160), True),
                                          ((160, 128, 129), True), ((256, 512, 256), True)])
@pytest.mark.parametrize("cx", [False, True])
def test_entry_bounds_at_the_threshold(ctx, shape, digits, cx):
    """Both sides of the rule meet the bound of their own kernel, on operands graded within rows and
    columns."""
    h, K, N = shape
    if cx:
        K //= 4
    rng = np.random.default_rng(K)
    A, B = _rand(rng, (2 * h, K), cx, 8), _rand(rng, (K, N), cx, 8)
    out = mpsgb.states.mul_tail(
        mpsgb.DeviceTensor.from_numpy(ctx, "mps", A.reshape(h, 2, K, order="F")),
        mpsgb.DeviceTensor.from_numpy(ctx, "bond", B)).numpy().reshape(2 * h, N, order="F")
    ref = _wide(A) @ _wide(B)
    err = np.abs(_wide(out) - ref).astype(np.float64)
    row, terms = _entry_bounds(A, B)
    assert np.all(err <= (row if digits else terms) + 2.0 ** -52 * np.abs(ref).astype(np.float64))


@pytest.mark.parametrize("cx", [False, True])
def test_entries_of_graded_operands_by_fmas(cx):
    """With 'fp64_fma' every entry keeps the bound of its own terms: columns of A graded down and rows
    of B graded up, so that results are made of entries far below the largest ones; also an operator
    built before the switch, whose constants are in digits.  Back at 0: the same bits as before."""
    ctx = mpsgb.Context(0)
    rng = np.random.default_rng(3)
    h, K, N = 160, 320, 200
    s = 10.0 ** -np.linspace(0, 20, K)
    A = _rand(rng, (2 * h, K), cx, 0) * s
    B = _rand(rng, (K, N), cx, 0) / s[:, None]
    B[: K // 2] = 0
    A[:, 0] = 1.0
    a = mpsgb.DeviceTensor.from_numpy(ctx, "mps", A.reshape(h, 2, K, order="F"))
    b = mpsgb.DeviceTensor.from_numpy(ctx, "bond", B)
    D = 160
    H = mpsgb.heisenberg_XXX(6, dtype=A.dtype)
    n = np.asarray(H.W[2]).shape[0]
    G = _rand(rng, (D, n, D), cx, 0)
    G[:, 0, :] = G[:, -1, :] = np.eye(D)
    dev = lambda k, v: mpsgb.DeviceTensor.from_numpy(ctx, k, v)
    op = mpsgb.DerivativeOperator(ctx, L.GB_HEFF_AC, dev("gl", G), H.device(ctx, A.dtype)[2], None,
                                  dev("gr", G), mpsgb.GB300Backend("fp64"))
    x = dev("mps", _rand(rng, (D, 2, D), cx, 0))
    y0, c0 = op(x).numpy(), mpsgb.states.mul_tail(a, b).numpy()
    ctx.set_option("fp64_fma", 1)
    out = mpsgb.states.mul_tail(a, b).numpy().reshape(2 * h, N, order="F")
    y1 = op(x).numpy()
    ctx.set_option("fp64_fma", 0)
    ref = _wide(A) @ _wide(B)
    err = np.abs(_wide(out) - ref).astype(np.float64)
    assert np.all(err <= _entry_bounds(A, B)[1])
    assert np.linalg.norm(y1 - y0) <= 1e-14 * np.linalg.norm(y0) and not np.array_equal(y1, y0)
    assert np.array_equal(op(x).numpy(), y0)
    assert np.array_equal(mpsgb.states.mul_tail(a, b).numpy(), c0)
