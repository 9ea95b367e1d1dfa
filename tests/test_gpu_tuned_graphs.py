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


@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64e"])
def test_repeat_solves_take_the_same_kernels_whatever_came_before(precision):
    # the batch's graphs are captured before the single-system classes are settled, which the deflation loop's
    # short launches share: the first system's repeat solve must match a system's that found all settled
    A = problems.helmholtz((19, 14, 13) if precision == "mixed" else (18, 14, 13), 5.0, 0.1)
    B = np.stack([problems.unit_gaussian_rhs(A.n, 50 + i) for i in range(2)])
    out = []
    for _ in range(2):
        s = gdmr.System(A, 30, 8, capacity=2, precision=precision)
        s.set_fused(False)
        for _ in range(2):
            s.drop_deflation()
            X = s.solve_batch(B, tol=[1e-6, 1e-10], max_cycles=400)[0]
        s.close()
        out.append(X)
    assert np.array_equal(out[0], out[1])
