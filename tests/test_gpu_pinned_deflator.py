"""gdmrTuneForce pins the blocked cycles' deflator: nothing is left to the tuner, and every form solves."""
import numpy as np
import pytest

import gdmr
import problems

pytestmark = pytest.mark.gpu

A = problems.helmholtz((41, 39, 31), 5.0, 0.1)       # a size of its own: the tuner's choices are per n
B = np.stack([problems.unit_gaussian_rhs(A.n, 50 + i) for i in range(8)])


@pytest.mark.parametrize("pair", [(0, 0), (1, 1), (9, 6), (9, 7), (10, 8), (10, 9), (10, 10), (9, 11)])
def test_pinned_cycles_ask_no_tuner(pair):
    blocked = gdmr.cycle_counts()["blocked"]
    gdmr.tune_force(*pair)
    try:
        s = gdmr.System(A, 30, 8, capacity=8, precision="mixed")
        X, stats = s.solve_batch(B, tol=1e-10, max_cycles=400)
        s.close()
    finally:
        gdmr.tune_force(-1, -1)
    for b, x, st in zip(B, X, stats):
        assert st["status"] == 0 and np.linalg.norm(b - A.to_scipy() @ x) <= 1.01e-10
    assert gdmr.cycle_counts()["blocked"] > blocked
    assert f"n={A.n} " not in gdmr.tune_report()
