"""Every cycle graph holds tuned variants: a shrinking batch's classes are timed, not captured unsettled."""
import numpy as np
import pytest

import gdmr
import problems

pytestmark = pytest.mark.gpu


def test_a_shrinking_batch_settles_each_width_class():
    A = problems.helmholtz((17, 13, 11), 5.0, 0.1)        # a size of its own: classes are per n
    tol = np.repeat([1e-5, 1e-7, 1e-9, 1e-11], [16, 12, 8, 4])
    B = np.stack([problems.unit_gaussian_rhs(A.n, 50 + i) for i in range(tol.size)])
    s = gdmr.System(A, 20, 8, capacity=tol.size, precision="mixed")
    X, stats = s.solve_batch(B, tol=tol, max_cycles=400)
    s.close()
    for b, x, t, st in zip(B, X, tol, stats):
        assert st["status"] == 0 and np.linalg.norm(b - A.to_scipy() @ x) <= 1.01 * t
    # 40, 24, 12 and 4 systems in flight, one class each, met in graphs after the first two cycles
    assert len({st["cycles"] for st in stats}) >= 4
    rep = [q for q in gdmr.tune_report().splitlines() if f"n={A.n} " in q and "projection" in q and "shared-only" in q]
    assert len(rep) == 4, rep
