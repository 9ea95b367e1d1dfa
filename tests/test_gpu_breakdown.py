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


def _spread(n):
    """A diagonal operator of 997 eigenvalues over a factor of 200, far enough from zero that no step of an
    exhausted space falls below the absolute breakdown threshold, and a unit vector that sees two of them."""
    i = np.arange(n) % 997
    b = np.where((i == 0) | (i == 500), problems.unit_gaussian_rhs(n, 7), 0.0)
    return _diagonal(2.0 ** 13 * (1 + 0.05j) * 200.0 ** (i / 996.0)), b / np.linalg.norm(b)


def _counts(before=None):
    c = gdmr.cycle_counts()
    return c if before is None else {k: c[k] - before[k] for k in c}


def _check(A, B, X, stats):
    for b, x, st in zip(B, X, stats):
        assert st["status"] == 0, st
        assert np.linalg.norm(b - A.to_scipy() @ x) <= (TOL + 1e-12) * np.linalg.norm(b)


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


def test_one_systems_breakdown_leaves_the_others_blocked():
    # the first right-hand side lies in an invariant space of dimension 2: its first block is dropped, and
    # the batch runs step by step until it has left
    A, two = _spread(N // 3 + 41)      # three systems reach the blocked loop
    B = np.concatenate([two[None], _rhs(A.n, 9)])
    s = gdmr.System(A, 30, 8, capacity=4, precision="mixed")
    alone = s.solve_batch(B[1:], tol=TOL, max_cycles=200)[1]
    s.drop_deflation()
    c0 = _counts()
    X, stats = s.solve_batch(B, tol=TOL, max_cycles=200)
    c = _counts(c0)
    _check(A, B, X, stats)
    assert c["dropped"] == 1, c
    # all cycles but those beside the first system after its breakdown (three others) and those of the
    # last one or two systems
    beside = 4 * (stats[0]["cycles"] - 1)
    tail = 2 * max(t["cycles"] for t in stats)
    assert c["blocked"] >= sum(t["cycles"] for t in stats) - beside - tail > 0, (c, stats)
    assert c["blocked"] > 4, c
    assert c["factored"] > c["factor_failed"], c
    ref, got = (np.mean([t["cycles"] for t in q]) for q in (alone, stats[1:]))
    assert abs(got - ref) <= 1.5, (got, ref)
    s.close()


def test_served_requests_after_a_breakdown_run_blocked():
    A, two = _spread(N + 1)
    srv = gdmr.Server(budget_bytes=8 << 30)
    op = srv.add_operator(A, 30, 8, capacity=1, precision="mixed")
    srv.start()
    for b, dropped in ((two, 1), (_rhs(A.n, 1)[0], 0)):
        c0 = _counts()
        x, st = srv.wait(srv.submit(op, b, tol=TOL), timeout=120)
        _check(A, [b], [x], [st])
        c = _counts(c0)
        assert c["dropped"] == dropped, c
    assert c["blocked"] == st["cycles"] > 0, (c, st)
    srv.close()


def test_cholesky_factor_returns_after_a_failure():
    A = problems.helmholtz((20, 19, 18), 12.0, 0.02)
    Z = _rhs(A.n, 8, 900)
    Z[5] = Z[2]
    s = gdmr.System(A, 20, 8, capacity=1, precision="mixed")
    s.import_deflation(Z)
    c0 = _counts()
    X, stats = s.solve_batch(_rhs(A.n, 1), tol=TOL, max_cycles=2000)
    c = _counts(c0)
    _check(A, _rhs(A.n, 1), X, stats)
    # the failed cycle, 16 without, then every one
    assert stats[0]["cycles"] > 20 and c["factor_failed"] == 1, (c, stats)
    assert c["factored"] == stats[0]["cycles"] - 16, (c, stats)
    s.close()


def test_a_lead_that_breaks_down_leaves_the_deflation_space():
    # one system, whose cycles from the third on are graphs: the cycle's update of the space comes from an
    # incomplete Hessenberg and is undone, in both buffers' parities
    A, two = _spread(N + 2)
    s = gdmr.System(A, 30, 8, capacity=1, precision="mixed")
    Z = _unit_vectors(A.n, 8)
    dropped = []
    for warm in range(4):
        for _ in range(1 + warm % 2):
            _check(A, _rhs(A.n, 1), *s.solve_batch(_rhs(A.n, 1), tol=TOL, max_cycles=200))
        s.import_deflation(Z)
        c0 = _counts()
        stats = s.solve_batch(two[None], tol=TOL, max_cycles=1)[1]
        dropped.append(_counts(c0)["dropped"])
        assert stats[0]["status"] == 3 and np.array_equal(s.export_deflation(), Z)
        _check(A, [two], *s.solve_batch(two[None], tol=TOL, max_cycles=200))
    assert dropped == [1, 1, 1, 1]
    s.close()
