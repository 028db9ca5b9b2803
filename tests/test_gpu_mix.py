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
