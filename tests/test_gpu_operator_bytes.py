"""The operator class books what its kernels move: x and y alone on constant planes, the CSR formula elsewhere."""
import numpy as np
import pytest

import gdmr
import problems

pytestmark = pytest.mark.gpu


def _operator_class(A, precision):
    s = gdmr.System(A, 30, 8, capacity=1, precision=precision)
    s.set_fused(False)
    gdmr.profile_reset()
    gdmr.profile(True)
    try:
        s.solve_batch(problems.unit_gaussian_rhs(A.n, 5)[None], tol=1e-8, max_cycles=2)
    finally:
        gdmr.profile(False)
    s.close()
    return gdmr.profile_read()["operator"]


@pytest.mark.parametrize("precision,size", [("mixed", 8), ("fp64", 16), ("fp64e", 16)])
def test_constant_planes_book_two_or_three_vectors_a_product(precision, size):
    A = problems.helmholtz((20, 18, 16), 5.0, 0.1)
    c = _operator_class(A, precision)
    # one launch each: x and y, v too in a folded step; the deflation loop's batched product has 8 systems
    assert 2 * size * A.n * c["launches"] <= c["bytes"] <= size * A.n * (3 * c["launches"] + 2 * 8), c
    V = problems.variable_helmholtz((20, 18, 16), 5.0, 0.1, 3)
    c = _operator_class(V, precision)
    assert c["bytes"] >= c["launches"] * (V.indices.size * (size + 4) + 2 * size * V.n), c
