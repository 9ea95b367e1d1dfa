"""A right-hand side holding NaN is refused alone: the slot it used answers the next one."""
import numpy as np
import pytest

import gdmr
import problems

pytestmark = pytest.mark.gpu

A = problems.helmholtz((24, 24), 5.0, 0.1)
TOL = 1e-8


def _pair():
    b = problems.unit_gaussian_rhs(A.n, 5)
    bad = b.copy()
    bad[7] = np.nan
    return b, bad


def _check(b, x, st):
    assert st["status"] == 0, st
    assert np.linalg.norm(b - A.to_scipy() @ x) <= 1.01 * TOL


@pytest.mark.parametrize("precision", ["mixed", "fp64", "fp64e"])
def test_batched_solve_after_a_nan(precision):
    b, bad = _pair()
    s = gdmr.System(A, 30, 8, capacity=1, precision=precision)
    with pytest.raises(gdmr.GDMRError) as e:
        s.solve_batch(bad[None], tol=TOL, max_cycles=500)
    assert e.value.status == 9
    X, stats = s.solve_batch(b[None], tol=TOL, max_cycles=500)
    _check(b, X[0], stats[0])
    s.close()


def test_served_request_after_a_nan():
    b, bad = _pair()
    srv = gdmr.Server(budget_bytes=1 << 30)
    op = srv.add_operator(A, 30, 8, capacity=1, precision="mixed")
    srv.start()
    assert srv.wait(srv.submit(op, bad, tol=TOL), timeout=60)[1]["status"] == 9
    _check(b, *srv.wait(srv.submit(op, b, tol=TOL), timeout=60))
    srv.close()
