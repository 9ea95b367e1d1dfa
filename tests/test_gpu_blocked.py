"""Blocked Krylov steps of the refined complex64 batches (gdmr_block.cu) and the constant-plane operator.

The blocked loop runs when n x systems reaches 3 * 2^17; every shape here is just above that."""
import numpy as np
import pytest

import gdmr
import problems

pytestmark = pytest.mark.gpu

TOL = 1e-10


def _rhs(n, nrhs):
    return np.stack([problems.unit_gaussian_rhs(n, 50 + i) for i in range(nrhs)])


def _scaled(A, factor):
    return problems.CSR(A.n, A.indptr, A.indices, A.data * factor)


def _check(A, B, X, stats):
    S = A.to_scipy()
    for b, x, st in zip(B, X, stats):
        assert st["status"] == 0, st
        # the library's own FP64 residual met TOL; the host's differs by rounding of order
        # eps ||A|| ||x|| / ||b||, below 1e-12 for these operators
        assert np.linalg.norm(b - S @ x) <= (TOL + 1e-12) * np.linalg.norm(b)


@pytest.mark.parametrize("shape,nrhs,m,k", [
    ((41, 39, 33), 8, 40, 16),     # odd n: 8-byte loads; tensor-core deflator at its smallest batch
    ((64, 40, 32), 5, 48, 24),     # even n, deflator on the CUDA cores
    ((70, 70, 81), 1, 30, 8),      # one system
    ((24, 24, 12), 64, 40, 10),    # the largest tensor-core batch, short vectors
    ((22, 21, 14), 65, 30, 8),     # above it
    ((40, 36, 30), 10, 20, 0),     # no deflation space
    ((40, 36, 30), 10, 12, 4),     # the smallest loop that is blocked: two single steps, two blocks
])
def test_blocked_batches_converge_as_complex128_cycles(shape, nrhs, m, k):
    A = problems.helmholtz(shape, 5.0, 0.1)
    B = _rhs(A.n, nrhs)
    cycles = {}
    for precision in ("mixed", "fp64"):
        s = gdmr.System(A, m, k, capacity=nrhs, precision=precision)
        X, stats = s.solve_batch(B, tol=TOL, max_cycles=400)
        s.close()
        _check(A, B, X, stats)
        cycles[precision] = np.mean([st["cycles"] for st in stats])
    # the same Krylov spaces up to complex64 rounding: as the recycled-sequence parity tests
    assert abs(cycles["mixed"] - cycles["fp64"]) <= 2 + 0.1 * cycles["fp64"], cycles


@pytest.mark.parametrize("factor", [1e-9, 1e12, 0.6 + 0.8j])
def test_blocked_steps_follow_the_operator_scale(factor):
    A = problems.helmholtz((41, 39, 33), 5.0, 0.1)
    B = _rhs(A.n, 8)
    got = {}
    for f in (1.0, factor):
        s = gdmr.System(_scaled(A, f), 40, 16, capacity=8, precision="mixed")
        X, stats = s.solve_batch(B, tol=TOL, max_cycles=400)
        s.close()
        _check(_scaled(A, f), B, X, stats)
        got[f] = np.mean([st["cycles"] for st in stats])
    assert abs(got[factor] - got[1.0]) <= 2, got


@pytest.mark.parametrize("eigenvalues", [5, 12])
def test_exhausted_krylov_space_falls_back(eigenvalues):
    # few distinct eigenvalues: the Krylov space is exhausted inside a block, whose basis is then noise
    n = 3 * 2 ** 17
    d = (1.0 + np.arange(n) % eigenvalues) * (1 + 0.1j)
    A = problems.CSR(n, np.arange(n + 1, dtype=np.int32), np.arange(n, dtype=np.int32), d.astype(np.complex128))
    B = _rhs(n, 2)
    s = gdmr.System(A, 30, 8, capacity=2, precision="mixed")
    for _ in range(2):      # the second solve starts from the first one's deflation space
        X, stats = s.solve_batch(B, tol=TOL, max_cycles=60)
        _check(A, B, X, stats)
    s.close()


@pytest.mark.parametrize("case", ["random", "repeated"])
def test_imported_deflation_spaces_through_the_cholesky_factor(case):
    # W = orth(A Z) by Cholesky QR: any independent Z works; a singular one costs
    # the cycle and goes on step by step
    A = problems.helmholtz((41, 39, 33), 5.0, 0.1)
    B = _rhs(A.n, 4)
    Z = np.stack([problems.unit_gaussian_rhs(A.n, 900 + i) for i in range(16)])
    if case == "repeated":
        Z[9] = Z[3]
    s = gdmr.System(A, 40, 16, capacity=4, precision="mixed")
    s.import_deflation(Z)
    for _ in range(2):                   # then from the space that the first solve left
        X, stats = s.solve_batch(B, tol=TOL, max_cycles=400)
        _check(A, B, X, stats)
    s.close()


@pytest.mark.parametrize("shape,nrhs,factor,precision", [
    ((41, 39, 33), 8, 1.0, "mixed"),            # real off-diagonal planes, partial tiles, shifted products
    ((41, 39, 33), 8, 0.6 + 0.8j, "mixed"),     # complex planes
    ((67, 45), 3, 1.0, "mixed"),                # 2D, step by step
    ((20, 12, 19), 1, 1.0, "fp64"),
    ((20, 12, 19), 2, 0.6 + 0.8j, "fp64e"),
])
def test_constant_plane_operator_matches_sell(shape, nrhs, factor, precision):
    # the terms and their order are the SELL kernel's, so whole solves agree bit for bit
    A = _scaled(problems.helmholtz(shape, 5.0, 0.1), factor)
    B = _rhs(A.n, nrhs)
    out = []
    for grid in (True, False):
        gdmr.grid_operator(grid)
        try:
            s = gdmr.System(A, 30, 8, capacity=nrhs, precision=precision)
            s.set_fused(False)
            s.solve_batch(B, tol=TOL, max_cycles=400)      # every launch's kernel variant settled
            s.drop_deflation()
            X, stats = s.solve_batch(B, tol=TOL, max_cycles=400)
            s.close()
        finally:
            gdmr.grid_operator(True)
        _check(A, B, X, stats)
        out.append(X)
    assert np.array_equal(out[0], out[1])
