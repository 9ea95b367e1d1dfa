"""The shared-basis projection W^H Y of a batch (k_wdots, projection variant 9) against variant 0.

One restart cycle from an imported deflation space with four own steps.  The right-hand sides live on the
first and last rows, so that a coefficient that misses a row of the edge is off in its first digits.  A
coefficient's rounding is at most 128 products of an FP32 chain, 128 * 2^-24 = 8e-6; the least squares of
four steps on operators whose spectrum spans about two decades multiplies it by 100 at most: 1e-3."""
import numpy as np
import pytest

import gdmr
import problems

pytestmark = pytest.mark.gpu


def _case(shape, nrhs, k):
    A = problems.helmholtz(shape, 5.0, 0.1)
    rng = np.random.default_rng(11)
    B = np.zeros((nrhs, A.n), complex)
    for rows in (slice(0, 2), slice(A.n - 3, A.n)):
        B[:, rows] = rng.standard_normal(B[:, rows].shape) + 1j * rng.standard_normal(B[:, rows].shape)
    Z = rng.standard_normal((k, A.n)) + 1j * rng.standard_normal((k, A.n))
    return A, B, Z


@pytest.mark.parametrize("shape,nrhs,k", [
    ((10, 10), 3, 4),           # shorter than one chunk of rows
    ((16, 16), 2, 1),           # two whole chunks, one vector
    ((13, 11, 7), 3, 5),        # odd n: 8-byte copies
    ((13, 11, 7), 33, 24),      # the systems in three groups, the last of one
    ((16, 12, 10), 65, 32),     # the most vectors; groups of twelve
    ((16, 12, 10), 64, 7),
    ((41, 39, 33), 2, 32),      # several chunks a CTA
])
def test_one_cycle_matches_the_general_projection(shape, nrhs, k):
    A, B, Z = _case(shape, nrhs, k)
    out = {}
    for variant in (0, 9):
        gdmr.tune_force(variant, 0)
        try:
            s = gdmr.System(A, k + 4, k, capacity=nrhs, precision="mixed")
            s.import_deflation(Z)
            out[variant] = s.solve_batch(B, tol=1e-10, max_cycles=1)[0]
            s.close()
        finally:
            gdmr.tune_force(-1, -1)
    err = np.linalg.norm(out[9] - out[0], axis=1) / np.linalg.norm(out[0], axis=1)
    assert np.all(np.linalg.norm(out[0], axis=1) > 0) and err.max() < 1e-3, err
