"""W = orth(A) of the refined complex64 cycles: two passes of Cholesky QR, checked in 64 bits.

The second pass leaves the rounding of its Gram sums (13 additions in FP32 at most, 13 2^-24 = 8e-7) and of
its products with R^-1 (3xTF32, a few 2^-22 an element: 1e-6 in an inner product at most): 2e-6."""
import numpy as np
import pytest

import gdmr

pytestmark = pytest.mark.gpu


def _vectors(k, n, condition, seed=6):
    """k vectors of very different lengths, whose angles give the normalised ones about that condition."""
    rng = np.random.default_rng(seed)
    A = rng.standard_normal((k, n), np.float32) + 1j * rng.standard_normal((k, n), np.float32)
    A /= np.linalg.norm(A, axis=1)[:, None]
    A[1:] += (1 - 1 / condition) * A[0]
    return (A * 10.0 ** np.linspace(-3, 3, k)[:, None]).astype(np.complex64)


@pytest.mark.parametrize("n,k,condition", [
    (884736, 24, 1.0),
    (262144, 24, 3.0),
    (100345, 16, 1.0),     # odd n
    (4096, 8, 3.0),        # the fewest vectors
    (2000, 32, 1.0),       # the most
    (33, 8, 1.0),          # one chunk of rows
])
def test_orthonormal_to_fp32(n, k, condition):
    A = _vectors(k, n, condition)
    W, R, failed = gdmr.orthonormalise_check(A)
    assert not failed
    Wd, Ad = W.astype(np.complex128), A.astype(np.complex128)
    G = Wd.conj() @ Wd.T
    print(f"n {n} k {k}: {np.abs(G - np.eye(k)).max():.2e}")
    assert np.abs(G - np.eye(k)).max() <= 2e-6
    assert np.abs(np.tril(R, -1)).max() == 0.0
    assert (np.linalg.norm(Ad - R.T @ Wd, axis=1) <= 4e-6 * np.linalg.norm(Ad, axis=1)).all()


def test_dependent_vectors_are_reported():
    A = _vectors(12, 5000, 1.0)
    A[7] = 2 * A[2]
    W, R, failed = gdmr.orthonormalise_check(A)
    assert failed and not W.any() and not R.any()
