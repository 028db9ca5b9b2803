"""The leg mixes at sizes on both sides of the split between a block per 128 entries and blocks
that walk columns, over copied rows (one unit coefficient) and summed ones.

Bound: the products before and after the mix err by at most 4e-16 sqrt(K) of their terms' norm,
the mix by an eps per entry: 3e-15 of the result."""
import numpy as np
import pytest

import mpsgb

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def ctx():
    return mpsgb.Context(0)


@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("Dl,Dr", [(3, 5), (129, 127), (385, 421)])
def test_environment_step(ctx, Dl, Dr, cx):
    rng = np.random.default_rng(Dl)
    dt = np.complex128 if cx else np.float64

    def rand(*s):
        a = rng.standard_normal(s)
        return a + 1j * rng.standard_normal(s) if cx else a

    W = np.asarray(mpsgb.heisenberg_XXX(6, dtype=dt).W[2]).copy()
    W[1, 0, 0, 1] = 0.5  # a row of two entries
    GL, A = rand(Dl, W.shape[0], Dl), rand(Dl, 2, Dr)
    GL[Dl // 2] = 0
    GL[0, :, 0] = -0.0
    got = mpsgb.transfer_left(mpsgb.DeviceTensor.from_numpy(ctx, "gl", GL), W,
                              mpsgb.DeviceTensor.from_numpy(ctx, "mps", A)).numpy()
    ref = np.einsum("bwk,kta->bwta", GL, A, optimize=True)
    ref = np.einsum("bwta,wstv->bsva", ref, W, optimize=True)
    ref = np.einsum("bsva,bsc->cva", ref, A.conj(), optimize=True)
    assert np.linalg.norm(got - ref) <= 3e-15 * np.linalg.norm(ref)


@pytest.mark.parametrize("prec", ["bf16x3", "tf32x3"])
@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("Dl,Dr", [(5, 3), (37, 41), (131, 128), (300, 257)])
def test_chain_mix_in_planes(ctx, Dl, Dr, cx, prec):
    """The mix that writes split planes: rows of one input with a coefficient that FP32 does not
    hold, rows of several, columns around the numbers in flight.  A plane pair keeps 16 (bf16) or
    22 bits (tf32: at least the 16) of each of four roundings, and the product of the low planes
    is dropped: 4 2^-17 + 2 2^-16 = 2^-14 of the result at most."""
    rng = np.random.default_rng(Dl * Dr)
    dt = np.complex128 if cx else np.float64
    n = 4
    W = np.zeros((n, 2, 2, n), dtype=dt)
    sz, sp = np.diag([0.5, -0.5]), np.array([[0.0, 1.0], [0.0, 0.0]])
    W[0, :, :, 0] = W[-1, :, :, -1] = np.eye(2)
    for c, o in ((1, sz), (2, sp + sp.T)):  # exponentially decaying couplings
        W[0, :, :, c] = rng.uniform(0.5, 1.0) * o
        W[c, :, :, c] = rng.uniform(0.1, 0.9) * np.eye(2)
        W[c, :, :, -1] = o
    W[1, :, :, 2] = 0.3 * sz  # an output of two inputs
    W[0, :, :, -1] = 0.7 * sp + 0.7 * sp.T

    def env(D):
        g = rng.standard_normal((D, n, D)) / np.sqrt(D)
        return (g + 1j * rng.standard_normal((D, n, D)) / np.sqrt(D)).astype(dt) if cx else g

    GL, GR = env(Dl), env(Dr)
    GL[:, 0, :] = np.eye(Dl)
    GR[:, -1, :] = np.eye(Dr)
    x = rng.standard_normal((Dl, 2, Dr, 2)).astype(dt)
    dev = lambda k, a: mpsgb.DeviceTensor.from_numpy(ctx, k, a)
    w = dev("mpo", W)

    def apply(p, times):
        op = mpsgb.DerivativeOperator(ctx, mpsgb._lib.GB_HEFF_AC2, dev("gl", GL), w, w,
                                      dev("gr", GR), mpsgb.GB300Backend(p))
        xd = dev("ac2", x)
        for _ in range(times):
            y = op(xd)
        return y.numpy()

    ref = apply("fp64", 1)
    got = apply(prec, 1)
    assert np.linalg.norm(got - ref) <= 2.0 ** -14 * np.linalg.norm(ref)
    assert np.array_equal(apply(prec, 3), got)  # over planes and maps of an earlier apply


@pytest.mark.parametrize("prec", ["bf16x3", "tf32x3"])
@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("Dl,Dr", [(3, 2), (40, 41), (128, 130), (200, 256)])
def test_both_products_in_one_launch(ctx, Dl, Dr, cx, prec):
    """A one-site operator in split precision whose products with the two environments share a
    launch: within the planes' 2^-14 of FP64, and the same bits from apply to apply (sums of two
    values do not depend on their order)."""
    rng = np.random.default_rng(Dl + 7 * Dr)
    dt = np.complex128 if cx else np.float64
    H = mpsgb.heisenberg_XXX(6, dtype=dt)
    n = np.asarray(H.W[2]).shape[0]

    def env(D, unit):
        g = rng.standard_normal((D, n, D)) + (1j * rng.standard_normal((D, n, D)) if cx else 0)
        g[:, unit, :] = np.eye(D)
        return g.astype(dt)

    GL, GR = env(Dl, 0), env(Dr, -1)
    dev = lambda k, a: mpsgb.DeviceTensor.from_numpy(ctx, k, a)
    x = dev("mps", rng.standard_normal((Dl, 2, Dr)).astype(dt))

    def op(p):
        return mpsgb.DerivativeOperator(ctx, mpsgb._lib.GB_HEFF_AC, dev("gl", GL),
                                        H.device(ctx, dt)[2], None, dev("gr", GR),
                                        mpsgb.GB300Backend(p))

    ref = op("fp64")(x).numpy()
    o = op(prec)
    got = [o(x).numpy() for _ in range(3)]
    assert np.linalg.norm(got[0] - ref) <= 2.0 ** -14 * np.linalg.norm(ref)
    assert np.array_equal(got[0], got[1]) and np.array_equal(got[0], got[2])


@pytest.mark.parametrize("kind", ["AC", "AC2"])
@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("prec", ["fp64", "bf16x3", "tf32x3"])
def test_long_range_operator_repeats_bit_for_bit(ctx, kind, cx, prec):
    """Decaying couplings: a chain over the continuing channels writes y beside the two products
    that may share a launch.  The same bits from apply to apply, at sizes on both sides of the rule
    that puts the two together, and the operator itself against einsum."""
    dt = np.complex128 if cx else np.float64
    sp, sz, eye = np.array([[0, 1], [0, 0]]), np.diag([0.5, -0.5]), np.eye(2)
    W = np.zeros((5, 2, 2, 5))
    W[0, :, :, 0] = W[4, :, :, 4] = eye
    for c, (a, b) in enumerate(((sp, sp.T), (sp.T, sp), (sz, sz))):
        W[0, :, :, 1 + c], W[1 + c, :, :, 1 + c], W[1 + c, :, :, 4] = a, 0.6 * eye, b
    W = W.astype(dt)
    dev = lambda k, a: mpsgb.DeviceTensor.from_numpy(ctx, k, a)
    for D in ((130, 200, 256) if kind == "AC" else (72, 100, 150)):
        rng = np.random.default_rng(D)
        rand = lambda *s: (rng.standard_normal(s) + (1j * rng.standard_normal(s) if cx else 0))
        GL, GR = rand(D, 5, D).astype(dt), rand(D, 5, D).astype(dt)
        GL[:, 0, :] = GR[:, -1, :] = np.eye(D)
        Wd = dev("mpo", W)
        if kind == "AC":
            x = rand(D, 2, D)
            op = mpsgb.DerivativeOperator(ctx, mpsgb._lib.GB_HEFF_AC, dev("gl", GL), Wd, None,
                                          dev("gr", GR), mpsgb.GB300Backend(prec))
            ref = np.einsum("bwk,kta->bwta", GL, x, optimize=True)
            ref = np.einsum("bwta,wstv->bsva", ref, W, optimize=True)
            ref = np.einsum("bsva,avc->bsc", ref, GR, optimize=True)
            xd = dev("mps", x)
        else:
            x = rand(D, 2, D, 2)
            op = mpsgb.DerivativeOperator(ctx, mpsgb._lib.GB_HEFF_AC2, dev("gl", GL), Wd, Wd,
                                          dev("gr", GR), mpsgb.GB300Backend(prec))
            ref = np.einsum("bwk,ktau->bwtau", GL, x, optimize=True)
            ref = np.einsum("bwtau,wstv->bsvau", ref, W, optimize=True)
            ref = np.einsum("bsvau,vzuq->bsqza", ref, W, optimize=True)
            ref = np.einsum("bsqza,aqc->bscz", ref, GR, optimize=True)
            xd = dev("ac2", x)
        got = [op(xd).numpy() for _ in range(25)]
        if prec == "fp64":
            assert np.linalg.norm(got[0] - ref) <= 1e-14 * np.linalg.norm(ref)
        else:  # the products one by one (a fixed tile width): the same addends, summed in FP64
            ctx.set_gemm_schedule("grouped", 128)
            try:
                apart = op(xd).numpy()
            finally:
                ctx.set_gemm_schedule("grouped", 0)
            assert np.linalg.norm(got[0] - apart) <= 1e-15 * np.linalg.norm(ref)
        for g in got[1:]:
            assert np.array_equal(got[0], g)
