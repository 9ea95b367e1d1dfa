"""Refined complex64 batches whose blocked cycles break down: nothing but the failing cycle is lost.

The blocked Krylov loop runs when n x systems reaches 3 * 2^17."""
import numpy as np
import pytest

import gdmr
import problems

pytestmark = pytest.mark.gpu

TOL = 1e-10
N = 3 * 2 ** 17


def _diagonal(d):
    n = d.size
    return problems.CSR(n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d.astype(np.complex128))


def _unit_vectors(n, k):
    Z = np.zeros((k, n), complex)
    Z[np.arange(k), np.arange(k)] = 1.0
    return Z


def _rhs(n, nrhs, seed=50):
    return np.stack([problems.unit_gaussian_rhs(n, seed + i) for i in range(nrhs)])


def _check(A, B, X, stats):
    for b, x, st in zip(B, X, stats):
        assert st["status"] == 0, st
        assert np.linalg.norm(b - A.data * x) <= (TOL + 1e-12) * np.linalg.norm(b)


@pytest.mark.parametrize("nrhs", [1, 2, 8])
def test_space_exhausted_at_the_last_single_step(nrhs):
    # m - k = 22: four single steps.  The deflated operator has four eigenvalues that the right-hand sides
    # see, and one 1e5 times as large on 64 rows where they are 1e-27.  The fourth step leaves rounding of
    # the first four, far above the absolute breakdown threshold of 1e-6, and by then the 64 rows are part of
    # it: the block's products grow by about 1e6 each, and the squared norm of the third leaves FP32.
    # Only that cycle may be lost.
    d = 2.0 ** 13 * np.array([1, -1, 0.5, -0.5])[np.arange(N) % 4]
    d[-64:] = 2.0 ** 13 * 1e5
    A = _diagonal(d)
    B = _rhs(N, nrhs)
    B[:, -64:] = 1e-27
    s = gdmr.System(A, 30, 8, capacity=nrhs, precision="mixed")
    s.import_deflation(_unit_vectors(N, 8))
    X, stats = s.solve_batch(B, tol=TOL, max_cycles=200)
    _check(A, B, X, stats)
    s.close()
