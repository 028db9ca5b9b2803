"""The one-launch Krylov step: orthogonality and decomposition of what it returns.

With k orthonormal vectors V, w_in = V h + w_out with V' w_out = 0: each projection is a dot
product and an update of rounding at most a few eps of |w|, so both relations hold to 16 k eps
(of |w_out| and |w_in|; a pass that loses more than half of |w|^2 is repeated)."""
import ctypes

import numpy as np
import pytest

import mpsgb
from mpsgb import _lib as L

pytestmark = pytest.mark.gpu
EPS = np.finfo(np.float64).eps


@pytest.fixture(scope="module")
def ctx():
    return mpsgb.Context(0)


def _orthogonalize(ctx, V, w):
    n, k = V.shape
    basis = mpsgb.DeviceTensor.from_numpy(ctx, "generic", V)
    x = mpsgb.DeviceTensor.from_numpy(ctx, "generic", w)
    h = np.zeros(2 * k)
    L.check(L.lib().gb_basis_orthogonalize(ctx.handle, basis.handle, k, x.handle,
                                           h.ctypes.data_as(ctypes.POINTER(ctypes.c_double))))
    h = h[0::2] + 1j * h[1::2] if np.iscomplexobj(w) else h[0::2]
    return x.numpy(), h


# pieces of 64 entries on 152 multiprocessors: one, two and all blocks, one entry more; pieces
# in shared memory and too long for it; one to five vectors (one barrier or two), the longest
# list and one past it; the longest vectors of a single cluster and one entry more
@pytest.mark.parametrize("cx", [False, True])
@pytest.mark.parametrize("n,k", [(3, 2), (64, 5), (65, 9), (130, 4), (9728, 3), (9729, 30),
                                 (40000, 8), (400001, 13), (900000, 7), (700, 128), (700, 129),
                                 (2048, 15), (2049, 15), (4096, 20), (4097, 3)])
def test_decomposition(ctx, n, k, cx):
    rng = np.random.default_rng(n + k)
    V = rng.standard_normal((n, k)) + (1j * rng.standard_normal((n, k)) if cx else 0)
    V = np.linalg.qr(V)[0]
    for near in (1.0, 1e-9):  # a generic vector, one almost in the span
        w = V @ (rng.standard_normal(k) + (1j * rng.standard_normal(k) if cx else 0))
        u = rng.standard_normal(n) + (1j * rng.standard_normal(n) if cx else 0)
        u = u - V @ (V.conj().T @ u)
        u = u - V @ (V.conj().T @ u)
        w = w + near * u / np.linalg.norm(u)
        out, h = _orthogonalize(ctx, V, w)
        assert np.linalg.norm(w - V @ h - out) <= 16 * k * EPS * np.linalg.norm(w)
        if n > k:
            assert np.linalg.norm(V.conj().T @ out) <= 16 * k * EPS * np.linalg.norm(out)
            # the input's own rounding is eps of |w| in every direction
            assert np.linalg.norm(out - near * u / np.linalg.norm(u)) <= 16 * k * EPS * (
                np.linalg.norm(w) + near)
    assert ctx.device_status() == 0


def test_non_finite_input_is_reported(ctx):
    H = mpsgb.heisenberg_XXX(8, dtype=np.float64)
    As = mpsgb.states.random_tensors(8, 2, 16, seed=3, dtype=np.float64)
    psi = mpsgb.FiniteMPS.from_tensors(As, ctx, center=4)
    envs = mpsgb.FiniteEnvironments(psi, H)
    op = mpsgb.AC_hamiltonian(4, psi, H, envs)
    x = psi.ac(4).numpy()
    x[0, 0, 0] = np.nan
    with pytest.raises(mpsgb._lib.GBError) as e:
        mpsgb.fixedpoint(op, mpsgb.DeviceTensor.from_numpy(ctx, "mps", x))
    assert e.value.code == L.GB_ERR_NAN
    with pytest.raises(mpsgb._lib.GBError) as e:
        mpsgb.fixedpoint(op, mpsgb.DeviceTensor.from_numpy(ctx, "mps", 0 * np.nan_to_num(x)))
    assert e.value.code == L.GB_ERR_ARG


@pytest.mark.parametrize("D", [2, 4, 16])
def test_solve_that_exhausts_its_space(ctx, D):
    """More Krylov vectors asked for than the space holds: the step that finds nothing left ends
    the solve with the exact eigenpair."""
    H = mpsgb.heisenberg_XXX(6, dtype=np.float64)
    As = mpsgb.states.random_tensors(6, 2, D, seed=4, dtype=np.float64)
    psi = mpsgb.FiniteMPS.from_tensors(As, ctx, center=3)
    envs = mpsgb.FiniteEnvironments(psi, H)
    op = mpsgb.C_hamiltonian(2, psi, H, envs)
    x0 = psi.C[3]
    n = x0.size
    M = np.zeros((n, n))
    for i in range(n):
        e = np.zeros(n)
        e[i] = 1
        y = op(mpsgb.DeviceTensor.from_numpy(ctx, "bond", e.reshape(x0.dims, order="F")))
        M[:, i] = y.numpy().reshape(-1, order="F")
    val, vec, info = mpsgb.fixedpoint(op, x0, "SR", mpsgb.Lanczos(40, 4, 1e-12))
    assert abs(val - np.linalg.eigvalsh(M)[0]) <= 1e-11 * np.abs(M).max()
    v = vec.numpy().reshape(-1, order="F")
    assert np.linalg.norm(M @ v - val * v) <= 1e-10 * np.abs(M).max()


@pytest.mark.parametrize("dtype", [np.float64, np.complex128])
@pytest.mark.parametrize("Dl,Dr", [(190, 190), (275, 280), (500, 340)])
def test_solve_over_pieces_short_and_long(ctx, Dl, Dr, dtype):
    """Pieces of 480, 1024 and 2240 entries per multiprocessor (short and long lists of sums in the
    steps and in the final combination): the returned vector has norm one and the returned value
    is its expectation value, each to the rounding of 2 Dl Dr squares added pairwise in parts."""
    H = mpsgb.transverse_field_ising(8, dtype=dtype)
    W = H.device(ctx, dtype)[3]
    rng = np.random.default_rng(Dl)

    def env(D, wide):
        g = rng.standard_normal((D, wide, D)) / np.sqrt(D)
        return (g + g.transpose(2, 1, 0)).astype(dtype)

    op = mpsgb.DerivativeOperator(
        ctx, L.GB_HEFF_AC, mpsgb.DeviceTensor.from_numpy(ctx, "gl", env(Dl, 3)),
        W, None, mpsgb.DeviceTensor.from_numpy(ctx, "gr", env(Dr, 3)),
        mpsgb.GB300Backend("fp64"))
    x = rng.standard_normal((Dl, 2, Dr)).astype(dtype)
    x0 = mpsgb.DeviceTensor.from_numpy(ctx, "mps", x / np.linalg.norm(x))
    val, vec, _ = mpsgb.fixedpoint(op, x0, "SR", mpsgb.Lanczos(12, 1, 1e-12, True))
    v = vec.numpy()
    assert abs(np.linalg.norm(v) - 1) <= 64 * EPS
    y = op(vec).numpy()
    assert abs(np.vdot(v, y) - val) <= 1e-12 * np.linalg.norm(y)
    assert ctx.device_status() == 0


def test_long_lists_after_a_solve_that_ended_early(ctx):
    """A solve that stops with a step still queued, then more dot products than the pinned results
    have room for: the room grows once the queued step has written its numbers."""
    own = mpsgb.Context(0)
    H = mpsgb.heisenberg_XXX(10, dtype=np.float64)
    As = mpsgb.states.random_tensors(10, 2, 32, seed=4, dtype=np.float64)
    psi = mpsgb.FiniteMPS.from_tensors(As, own, center=5)
    envs = mpsgb.FiniteEnvironments(psi, H)
    op = mpsgb.AC_hamiltonian(5, psi, H, envs)
    rng = np.random.default_rng(5)
    n, k = 2000, 700  # 1400 doubles; the steps' own slots are 1040
    V = np.linalg.qr(rng.standard_normal((n, k)))[0]
    w = rng.standard_normal(n)
    for _ in range(3):
        lam, _, info = mpsgb.fixedpoint(op, psi.ac(5), "SR", mpsgb.Lanczos(30, 1, 1e-3, True))
        assert info.numops < 30 and np.isfinite(lam)
        out, h = _orthogonalize(own, V, w)
        assert np.linalg.norm(w - V @ h - out) <= 16 * k * EPS * np.linalg.norm(w)
        assert np.linalg.norm(V.T @ out) <= 16 * k * EPS * np.linalg.norm(out)
    assert own.device_status() == 0
