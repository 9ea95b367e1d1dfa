"""The blocked Krylov loop on every operator kernel that has the shifted product y = sigma (A x - t x).

Each shape is just above the 3 * 2^17 unknowns from which the loop runs in blocks."""
import numpy as np
import pytest

import gdmr
import problems

pytestmark = pytest.mark.gpu

TOL = 1e-10
SHAPE, DAMPING = (41, 39, 33), 0.1


def _solve(A, nrhs, precision="mixed", stencil=None):
    B = np.stack([problems.unit_gaussian_rhs(A.n, 50 + i) for i in range(nrhs)])
    s = gdmr.System(A, 40, 16, capacity=nrhs, precision=precision)
    if stencil:
        s.set_stencil(*stencil)
    before = gdmr.cycle_counts()["blocked"]
    X, stats = s.solve_batch(B, tol=TOL, max_cycles=400)
    blocked = gdmr.cycle_counts()["blocked"] - before
    s.close()
    S = A.to_scipy()
    for b, x, st in zip(B, X, stats):
        assert st["status"] == 0, st
        assert np.linalg.norm(b - S @ x) <= (TOL + 1e-12) * np.linalg.norm(b)
    cycles = [st["cycles"] for st in stats]
    # a batch that has shrunk below the line goes on step by step
    assert blocked == sum(cycles) if precision == "mixed" and nrhs == 1 else (blocked > 0) == (precision == "mixed")
    return X, np.mean(cycles)


def _agree(mixed, fp64):
    assert abs(mixed - fp64) <= 2 + 0.1 * fp64, (mixed, fp64)


def test_stencil():
    A = problems.helmholtz(SHAPE, 5.0, DAMPING)
    st = (SHAPE,) + tuple(problems.helmholtz_stencil(SHAPE, 5.0, DAMPING))
    X, cycles = _solve(A, 8, stencil=st)
    Y, csr = _solve(A, 8)
    assert abs(cycles - csr) <= 1 and np.linalg.norm(X - Y) <= 1e-6 * np.linalg.norm(Y)


def test_one_system_of_variable_coefficients():       # k_spmv2 with the grid form off, k_grid_spmm with it on
    A = problems.variable_helmholtz((75, 74, 71), 4.0, DAMPING, 3)
    out = []
    for grid in (False, True):
        gdmr.grid_operator(grid)
        try:
            out.append(_solve(A, 1))
        finally:
            gdmr.grid_operator(True)
    assert out[0][1] == out[1][1]
    _agree(out[0][1], _solve(A, 1, "fp64")[1])


@pytest.mark.parametrize("systems", [0, 1, 2, 4])     # 0: k_spmm; else systems a thread of k_grid_spmm
def test_batch_of_variable_coefficients(systems):
    A = problems.variable_helmholtz(SHAPE, 4.0, DAMPING, 3)
    gdmr.grid_batch(systems)
    try:
        X, cycles = _solve(A, 9)                      # a group of systems that is not full
    finally:
        gdmr.grid_batch(0)
    _agree(cycles, _solve(A, 9, "fp64")[1])
