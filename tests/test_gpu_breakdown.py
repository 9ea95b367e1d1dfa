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


@pytest.mark.parametrize("after", ["solve", "multi"])
def test_factor_that_failed_in_an_unused_loop_is_forgotten(after):
    # with the overlapped residual, the deflation loop of a next cycle is enqueued before the host knows
    # that every system is done (zero right-hand sides are, at once); its factor fails on a singular space
    A = problems.helmholtz((20, 19, 18), 5.0, 0.1)
    B = _rhs(A.n, 2)
    Z = _rhs(A.n, 16, 900)
    Z[9] = Z[3]

    def system():
        s = gdmr.System(A, 40, 16, capacity=2, precision="mixed")
        s.set_graphs(False)
        return s

    s = system()
    ref = [t["cycles"] for t in s.solve_batch(B, tol=TOL, max_cycles=200)[1]]
    s.close()
    s = system()
    s.solve_batch(B, tol=TOL, max_cycles=200)
    s.import_deflation(Z)
    prev = gdmr.overlap_residual(1)
    try:
        assert [t["cycles"] for t in s.solve_batch(np.zeros_like(B), tol=TOL, max_cycles=200)[1]] == [0, 0]
    finally:
        gdmr.overlap_residual(prev)
    s.drop_deflation()
    if after == "solve":
        stats = s.solve_batch(B, tol=TOL, max_cycles=200)[1]
        assert [t["cycles"] for t in stats] == ref
    else:
        prev = gdmr.multi_tail(0)      # lockstep to the end
        try:
            (X, stats), = gdmr.multi_solve([s], [B], tol=TOL, max_cycles=200)
        finally:
            gdmr.multi_tail(prev)
    assert [t["status"] for t in stats] == [0, 0], stats
    s.close()
